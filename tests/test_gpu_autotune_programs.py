"""tvap_autotune chooses between programs: candidates that launch the same one (the same tile columns, groups, cap and
look-ahead once the size and the angles are known) are timed once and share its time."""

import math

import pytest

from taurus_vap_gb300 import model as M
from taurus_vap_gb300.native import Context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shells,mphi,gemm_mode", [(0, 5, 2), (0, 19, 2), (6, 5, 2), (6, 5, 0), (6, 5, 1)])
def test_same_program_same_time(shells, mphi, gemm_mode):
    if shells:
        sh = M.shells_up_to(6)[:shells]
        mdl = M.synthetic(sh, [10.0 * (k + 1) for k in range(shells)], hw=20.0, valence_Z=4, valence_N=4, seed=1)
    else:
        mdl = M.sd_model(seed=2)
    U, V = M.random_bogoliubov(mdl.basis, 4, 4, seed=3)
    ctx = Context(mdl.basis, mdl.ham)
    ctx.set_gemm_mode(gemm_mode)
    table = ctx.autotune(U, V, mphi, mphi, 2 * math.pi, 4, 4, reps=2)
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    two_groups = (mphi * mphi + 1) // 2 > sms
    programs = {}
    for (bn, groups, cap, la, pf), ms in table.items():
        key = (pf,)
        if gemm_mode:
            # beside the panels of more than half the SMs, cap 0 comes to cap 1 (half the SMs)
            key += ("half" if cap < 2 else "none",) if two_groups and groups == 2 else ()
            key += (la,) if mdl.n > 32 else ()  # one panel up to 32: nothing to look ahead to
        if gemm_mode == 2:
            key += (bn == 2,)
        programs.setdefault(key, set()).add(ms)
    assert len(table) == 48
    assert all(len(times) == 1 for times in programs.values()), programs
    assert ctx.tuning() == min(table, key=table.get)
