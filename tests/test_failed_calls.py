"""A call that ends in an error between the fork and the join of its chains waits for them (settle) before it returns.
On the host, read as source: the functions that fork are reached through settle only.  On the device: the projection
after such an error, in the plain form, which runs on the caller's stream and shares the workspace."""

import math
import os
import re

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), os.pardir, "taurus_vap_gb300", "csrc")


def functions(src):
    """name -> body of the functions at the start of a line"""
    out = {}
    for m in re.finditer(r"^int (\w+)\([^;{]*\) \{\n(.*?)^\}", src, re.M | re.S):
        out[m.group(1)] = m.group(2)
    return out


def test_chains_are_forked_under_settle():
    src = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "projection.cu")).read())
    fns = functions(src)
    forks = {k for k, b in fns.items() if "cudaEventRecord(c->ev_fork" in b}
    assert forks == {"project_angles", "project_chains", "project_observables_device"}
    # project_chains (and project_angles through it) only from project_device, whose result is settled
    assert [k for k, b in fns.items() if "project_chains(" in b] == ["project_device"]
    assert [k for k, b in fns.items() if "project_angles(" in b] == ["project_chains"]
    assert "settle(c, project_chains(" in fns["project_device"]
    # the observables fork in a local function; no return between it and the end but the settled one
    body = fns["project_observables_device"]
    head, tail = body[:body.index("auto run =")], body[body.index("\n  };\n", body.index("auto run =")):]
    assert "ev_fork" not in head and "settle(c, run())" in tail
    assert tail.index("settle(c, run())") < tail.index("return")


def test_every_stream_is_waited_for():
    src = open(os.path.join(CSRC, "tvap_context.cu")).read()
    body = re.search(r"^void sync_streams\(.*?^\}", src, re.M | re.S).group(0)
    ctx = open(os.path.join(CSRC, "tvap_internal.cuh")).read()
    ctx = ctx[ctx.index("struct tvap_ctx {"):]
    streams = set(re.findall(r"cudaStream_t (\w+)(?:\[\d\])? = ", ctx[:ctx.index("\n};")]))
    assert streams == {"stream", "stream2", "stream3", "streamM", "streamM2", "streamB"}
    assert all(f"c->{k}" in body for k in streams)
    # the caller may have set the default stream, whose handle is null
    assert re.search(r"^  cudaStreamSynchronize\(c->stream\);", body, re.M)


@pytest.mark.parametrize("source,pointer,size", [("ozaki.cu", "sc->buf", "sc->bytes"),
                                                 ("ozaki.cu", "sc->ex", "sc->ex_count"),
                                                 ("tvap_context.cu", "c->scratch", "c->scratch_count"),
                                                 ("tvap_context.cu", "c->fields_buf", "c->fields_bytes")])
def test_a_failed_growth_leaves_no_size_behind(source, pointer, size):
    # grown buffers are freed first: were the old size kept when the allocation fails, the next call would find the
    # null pointer large enough
    src = open(os.path.join(CSRC, source)).read()
    at = src.index(f"cudaMalloc(&{pointer},")
    before = src[src.rindex(f"cudaFree({pointer})", 0, at):at]
    assert re.search(re.escape(pointer) + r" = nullptr;", before) and re.search(re.escape(size) + r" = 0;", before)


@pytest.mark.gpu
@pytest.mark.parametrize("call", ["observables", "projection"])
def test_projection_after_an_error(call):
    from taurus_vap_gb300 import model as M
    from taurus_vap_gb300.native import Context, TvapError

    mdl = M.noncore_model(3, seed=1)
    n = mdl.n
    U, V = M.random_bogoliubov(mdl.basis, 8, 8, seed=2)
    args = (3, 3, 2 * math.pi, 8, 8)
    ref, Href = Context(mdl.basis, mdl.ham).project(U, V, *args, mode=1)
    # one state alone partly occupied: an odd number of paired states, found when the chains run
    v = np.zeros(n)
    v[:n // 2] = 1.0
    v[0] = 0.6
    badU, badV = np.diag(np.sqrt(1.0 - v * v)), np.diag(v)
    ctx = Context(mdl.basis, mdl.ham)
    ops = mdl.observable_operators()
    for _ in range(3):
        with pytest.raises(TvapError) as e:
            if call == "observables":
                ctx.project_observables(badU, badV, 9, 9, 2 * math.pi, 8, 8, ops)
            else:
                ctx.project(badU, badV, 9, 9, 2 * math.pi, 8, 8)
        assert e.value.code == 16
        p, H = ctx.project(U, V, *args, mode=1)
        assert abs(p.c("ener") - ref.c("ener")) <= 1e-10 * abs(ref.c("ener"))
        assert np.abs(H - Href).max() <= 1e-9 * np.abs(Href).max()
