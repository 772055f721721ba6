"""The calls whose time counts: what a user of this framework has it do, through its public entry points.

The work is that of a TAURUS_vap user: gradient iterations on the model spaces of the repository's benchmark (sd; the
no-core spaces emax = 2 to 6, n = 40 to 336 single-particle states) with 3 to 15 gauge angles per species, and the
calls around them: the fields of given densities, overlaps (Pfaffians), the Thouless evolution, the constraint
adjustment, the adjoint of the projected energy, the printed observables, many seeds at once.  The interaction is the
repository's synthetic one; a case's seed draws the state (a random Bogoliubov state) or the matrices.

``exact`` restates the formulas in plain torch (float64 and complex128): the gauge angles unfolded, the overlap as the
Pfaffian of the two Thouless matrices, the fields as a sparse matrix of the element list.
"""

import ctypes
import functools
import math

import numpy as np
import torch

from taurus_vap_gb300 import model as M
from taurus_vap_gb300 import native as N
from taurus_vap_gb300.autograd import projected_energy

ETA, MU = 0.002, 0.3  # step size and momentum of the no-core spaces (sd: 0.02)
SHELLS = M.shells_up_to(6)  # emax = 2, 3, 4, 5, 6: the first 6, 10, 15, 21, 28 shells


def listed():
    return [
        # the smallest use: a valence-space minimisation, called from host arrays; launches and host work count
        {"name": "iterate_sd_m9", "kind": "iterate", "shells": 0, "Mp": 9, "Mn": 9, "Z": 4, "N": 4, "host": True},
        # a middle space, odd proton number (one blocked quasiparticle), different numbers of angles per species
        {"name": "iterate_e3_odd_m11x7", "kind": "iterate", "shells": 10, "Mp": 11, "Mn": 7, "Z": 9, "N": 8,
         "host": False},
        # the headline: emax = 4, 15 x 15 angles, the state kept on the device
        {"name": "iterate_e4_m15", "kind": "iterate", "shells": 15, "Mp": 15, "Mn": 15, "Z": 8, "N": 8, "host": False},
        # the largest space (12.9 million elements)
        {"name": "iterate_e6_m15", "kind": "iterate", "shells": 28, "Mp": 15, "Mn": 15, "Z": 10, "N": 10,
         "host": False},
        # calculate_fields at its Fortran call site: one density, host arrays
        {"name": "fields_one_e4", "kind": "fields", "shells": 15, "cols": 1, "host": True},
        # the fields of a whole angle grid at once, densities and fields on the device
        {"name": "fields_batch_e4", "kind": "fields", "shells": 15, "cols": 113, "host": False},
        # the overlaps of an angle grid for a caller with its own overlap code (ZSKPFA)
        {"name": "pfaffian_113x140", "kind": "pfaffian", "batch": 113, "m": 140},
        # one Thouless evolution (a line search or a mean-field step), host arrays
        {"name": "evolve_e4", "kind": "evolve", "shells": 15},
        # the constraint Newton loop of a constrained step: Z, N and Q20
        {"name": "constraints_e4", "kind": "constraints", "shells": 15, "q20": 4.0},
        # energy and dE/dZ through autograd, as an optimiser calls it
        {"name": "adjoint_e4_m15", "kind": "adjoint", "shells": 15, "Mp": 15, "Mn": 15, "Z": 8, "N": 8},
        # the printed observables of a converged state: energies, J^2, multipoles, occupations, parity, density
        {"name": "observables_e3_m9", "kind": "observables", "shells": 10, "Mp": 9, "Mn": 9, "Z": 8, "N": 8},
        # a minima search: even and odd seeds on two spaces, worker contexts sharing the device
        {"name": "many_16sd_4e4_m15", "kind": "many", "small": 16, "large": 4, "shells": 15, "Mp": 15, "Mn": 15},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["iterate", "iterate", "iterate", "fields", "pfaffian", "evolve", "constraints", "adjoint",
                       "observables", "many"])
    if kind == "iterate":
        k = rng.choice([0] + list(range(5, 25)))
        z = rng.choice([4, 5] if k == 0 else [4, 5, 6] if k < 8 else [6, 7, 8, 10])
        return {"kind": kind, "shells": k, "Mp": rng.randint(3, 15), "Mn": rng.randint(3, 15), "Z": z,
                "N": 4 if k == 0 or k < 8 else rng.choice([6, 8, 10]), "host": rng.random() < 0.5}
    if kind == "fields":
        return {"kind": kind, "shells": rng.randint(5, 21), "cols": _log_int(rng, 1, 120),
                "host": rng.random() < 0.3}
    if kind == "pfaffian":
        m = 2 * _log_int(rng, 5, 140)
        return {"kind": kind, "batch": _log_int(rng, 2, 225), "m": m}
    if kind == "evolve":
        return {"kind": kind, "shells": rng.choice([0] + list(range(4, 29)))}
    if kind == "constraints":
        return {"kind": kind, "shells": rng.randint(6, 21), "q20": round(rng.uniform(-4.0, 4.0), 3)}
    if kind == "adjoint":
        return {"kind": kind, "shells": rng.randint(6, 17), "Mp": rng.randint(3, 15), "Mn": rng.randint(3, 15),
                "Z": rng.choice([4, 6]), "N": rng.choice([4, 6])}
    if kind == "observables":
        return {"kind": kind, "shells": rng.randint(6, 15), "Mp": rng.randint(3, 11), "Mn": rng.randint(3, 11),
                "Z": rng.choice([4, 6]), "N": rng.choice([4, 6])}
    return {"kind": "many", "small": rng.randint(4, 24), "large": rng.randint(1, 4), "shells": rng.randint(8, 15),
            "Mp": rng.randint(5, 15), "Mn": rng.randint(5, 15)}


# ---------------------------------------------------------------------------
# what a program keeps: the model space with its interaction, and a context that has it on the device
# ---------------------------------------------------------------------------


@functools.lru_cache(maxsize=None)
def _model(shells):
    """0: the sd valence space; k: the first k no-core shells."""
    if shells == 0:
        return M.sd_model(seed=1)
    sh = SHELLS[:shells]
    spe = [20.0 * ((2 * (s // 1000) + (s % 1000) // 100) + 1.5) / 2.0 for s in sh]
    return M.synthetic(sh, spe, hw=20.0, valence_Z=8, valence_N=8, seed=1, scale=1.0, damp=8.0)


@functools.lru_cache(maxsize=None)
def _context(shells, worker=0):
    m = _model(shells)
    return N.Context(m.basis, m.ham)


def _dim(shells):
    return 24 if shells == 0 else 2 * sum(s % 100 + 1 for s in SHELLS[:shells])


def _state(shells, Z, Nn, seed):
    """A random Bogoliubov state; an odd proton number blocks one quasiparticle."""
    return M.random_bogoliubov(_model(shells).basis, Z, Nn, seed=seed, block=3 if Z % 2 else 0)


def _thouless(n, seed, scale):
    B = np.random.default_rng(seed).normal(0.0, scale, (n, n))
    return np.asfortranarray((B - B.T) / math.sqrt(2.0))


def _densities(shells, cols, seed):
    """Transition densities of a state with its gauge-rotated copies are full complex matrices of rapidly varying
    size: a Hermitian-like part of order 1 on the low states and a small general part; the pairing tensors skew."""
    n = _dim(shells)
    g = torch.Generator(device="cuda").manual_seed(seed)

    def rnd():
        return torch.randn(cols, n, n, generator=g, device="cuda", dtype=torch.complex128)

    d = torch.exp(-3.0 * torch.arange(n, device="cuda", dtype=torch.float64) / n)
    rho = rnd() * (d[:, None] * d[None, :])
    kl, kr = rnd(), rnd()
    return rho, kl - kl.transpose(1, 2), kr - kr.transpose(1, 2)


def _cm(a):
    """A host matrix as a device vector in column-major order."""
    return torch.tensor(np.asarray(a).reshape(-1, order="F"), device="cuda")


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def _eta(case):
    return 0.02 if case["shells"] == 0 else ETA


def _constraint_ops(shells):
    n = _dim(shells)
    m = _model(shells)
    q = m.multipoles()
    nz, nn = np.zeros((n, n)), np.zeros((n, n))
    nz[np.arange(n // 2), np.arange(n // 2)] = 1.0
    nn[np.arange(n // 2, n), np.arange(n // 2, n)] = 1.0
    return np.stack([nz.reshape(-1), nn.reshape(-1), q[1, 0, 0] + q[1, 1, 0]])


def _constraint_target(case, U, V):
    """Particle numbers as the state has them after rounding to the aimed ones, Q20 moved by case["q20"] fm^2."""
    ops = _constraint_ops(case["shells"])
    n = U.shape[0]
    rho = V @ V.T
    q = float(np.sum(ops[2].reshape(n, n, order="F") * rho.T))
    return ops, [6.0, 6.0, q + case["q20"]]


def _many(case, seed):
    """(shells, worker, Z, U, V) of every state: the small space's first."""
    out = []
    for k in range(case["small"]):
        Z = 5 if k % 2 else 4
        out.append((0, k % 4, Z, 4) + _state(0, Z, 4, seed * 100 + k))
    for k in range(case["large"]):
        Z = 9 if k % 2 else 8
        out.append((case["shells"], k % 2, Z, 8) + _state(case["shells"], Z, 8, seed * 100 + 50 + k))
    return out


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "case": case}
    if kind == "pfaffian":
        g = torch.Generator(device="cuda").manual_seed(seed)
        A = torch.randn(case["batch"], case["m"], case["m"], generator=g, device="cuda", dtype=torch.complex128)
        s["A"] = (A - A.transpose(1, 2)).contiguous()
        s["ctx"] = _context(0)
        s["pf"] = torch.zeros(case["batch"], dtype=torch.complex128, device="cuda")
        return s
    if kind == "many":
        st = _many(case, seed)
        s["ctxs"] = [_context(q[0], q[1]) for q in st]
        s["U"], s["V"] = [q[4] for q in st], [q[5] for q in st]
        s["Zm"] = [np.zeros(u.size) for u in s["U"]]
        s["opts"] = [dict(Mphip=case["Mp"], Mphin=case["Mn"], facpi=2 * math.pi, valence_Z=q[2], valence_N=q[3])
                     for q in st]
        s["eta"] = [0.02 if q[0] == 0 else ETA for q in st]
        return s
    n = _dim(case["shells"])
    ctx = s["ctx"] = _context(case["shells"])
    if kind == "fields":
        rho, kl, kr = _densities(case["shells"], case["cols"], seed)
        if case["host"]:
            s["in"] = tuple(x.cpu().numpy() for x in (rho, kl, kr))
        else:
            s["in"] = tuple(x.transpose(1, 2).contiguous() for x in (rho, kl, kr))  # column-major matrices
            s["out"] = tuple(torch.empty_like(s["in"][0]) for _ in range(4))
        return s
    Z, Nn = case.get("Z", 6), case.get("N", 6)
    U, V = s["U"], s["V"] = _state(case["shells"], Z, Nn, seed)
    if kind == "iterate":
        s["Zm"] = np.zeros(n * n)
        if not case["host"]:
            s["dU"], s["dV"], s["dZm"] = _cm(U), _cm(V), _cm(s["Zm"])
            s["out"] = {k: torch.empty(n * n, dtype=torch.float64, device="cuda") for k in ("Zi", "U1", "V1", "H20v")}
            s["o"] = N.TvapProjOpts(case["Mp"], case["Mn"], 2 * math.pi, Z, Nn, 1.0, 0.0, 0, 0)
            s["pnp"], s["norm"] = N.TvapPnp(), ctypes.c_double()
    elif kind == "evolve":
        s["Z"] = _thouless(n, seed + 1, 0.05)
    elif kind == "constraints":
        s["ops"], s["targets"] = _constraint_target(case, U, V)
        s["Z"] = _thouless(n, seed + 1, 1e-3).reshape(-1, order="F")
    elif kind == "adjoint":
        s["Z"] = torch.tensor(np.ascontiguousarray(_thouless(n, seed + 1, 0.02)), device="cuda")
    elif kind == "observables":
        s["ops"] = _model(case["shells"]).observable_operators()
    assert ctx.n == n
    return s


PNP = ("over", "ener", "prot", "neut", "prot2", "neut2")


def _sums(pnp):
    return np.array([pnp.c(k) for k in PNP])


def run(s):
    kind, case = s["kind"], s["case"]
    if kind == "iterate" and case["host"]:
        pnp, Zi, norm, U1, V1, H = s["ctx"].iterate(s["U"], s["V"], s["Zm"], case["Mp"], case["Mn"], 2 * math.pi,
                                                    case["Z"], case["N"], _eta(case), MU, want_H20v=True)
        return {"sums": _sums(pnp), "Zi": Zi, "norm": norm, "U1": U1, "V1": V1, "H20v": H}
    if kind == "iterate":
        o = s["out"]
        N._check(N.lib().tvap_iterate(s["ctx"].h, _ptr(s["dU"]), _ptr(s["dV"]), ctypes.byref(s["o"]), _eta(case), MU,
                                      _ptr(s["dZm"]), _ptr(o["Zi"]), _ptr(o["U1"]), _ptr(o["V1"]),
                                      ctypes.byref(s["pnp"]), _ptr(o["H20v"]), ctypes.byref(s["norm"])),
                 "tvap_iterate")
        return {"sums": _sums(s["pnp"]), "norm": s["norm"].value, **o}
    if kind == "fields" and case["host"]:
        if case["cols"] == 1:
            return list(s["ctx"].calculate_fields(*(x[0] for x in s["in"])))
        return list(s["ctx"].calculate_fields_batched(*s["in"]))
    if kind == "fields":
        N._check(N.lib().tvap_calculate_fields_batched(s["ctx"].h, case["cols"], *[_ptr(x) for x in s["in"]],
                                                       *[_ptr(x) for x in s["out"]]), "tvap_calculate_fields_batched")
        return list(s["out"])
    if kind == "pfaffian":
        # (the library reads the matrices column-major: the transposed of what the tensor holds)
        N._check(N.lib().tvap_zskpfa_batched(s["ctx"].h, case["batch"], case["m"], _ptr(s["A"]), _ptr(s["pf"])),
                 "tvap_zskpfa_batched")
        return s["pf"]
    if kind == "evolve":
        return list(s["ctx"].evolve(s["U"], s["V"], s["Z"]))
    if kind == "constraints":
        U1, V1, Zi, C20, steps = s["ctx"].adjust_constraints(s["U"], s["V"], s["Z"], s["ops"], s["targets"])
        return {"U1": U1, "V1": V1, "Zi": Zi, "C20": C20, "steps": steps}
    if kind == "adjoint":
        z = s["Z"].clone().requires_grad_(True)
        e = projected_energy(z, s["ctx"], s["U"], s["V"], case["Mp"], case["Mn"], case["Z"], case["N"])
        e.backward()
        return {"E": e.detach(), "dEdZ": z.grad}
    if kind == "observables":
        r = s["ctx"].project_observables(s["U"], s["V"], case["Mp"], case["Mn"], 2 * math.pi, case["Z"], case["N"],
                                         s["ops"])
        return {k: r[k] for k in ("scal", "obo", "sq", "occnum", "rho")}
    res = N.iterate_many(s["ctxs"], s["U"], s["V"], s["Zm"], s["opts"], s["eta"], [MU] * len(s["U"]))
    out = {}
    for part, at in (("even_small", slice(0, case["small"], 2)), ("odd_small", slice(1, case["small"], 2)),
                     ("even_large", slice(case["small"], None, 2)), ("odd_large", slice(case["small"] + 1, None, 2))):
        r = res[at]
        if r:
            out[part] = {"sums": np.stack([_sums(q[0]) for q in r]), "Zi": np.stack([q[1] for q in r]),
                         "norm": np.array([q[2] for q in r]), "U1": np.stack([q[3] for q in r]),
                         "V1": np.stack([q[4] for q in r])}
    return out


def work(case):
    """One pass: the inputs read and the outputs written once (the element list, 13 bytes an element, among them), and
    the multiply-adds of the path in double precision, two operations each.  Per computed gauge angle (conjugate pairs
    once) of a space of n states: the Thouless solve 10.7 n^3, the wave functions 8, the densities 12, the gradient
    40, the overlap 5.4; the fields 8 complex terms for each of about 1.65 uses of an element."""
    kind = case["kind"]
    if kind == "pfaffian":
        m, b = case["m"], case["batch"]
        return {"bytes": 16 * b * (m * (m - 1) // 2 + 1), "flops": b * 8 * m ** 3 / 6}
    if kind == "many":
        a = work({"kind": "iterate", "shells": 0, "Mp": case["Mp"], "Mn": case["Mn"]})
        c = work({"kind": "iterate", "shells": case["shells"], "Mp": case["Mp"], "Mn": case["Mn"]})
        return {k: case["small"] * a[k] + case["large"] * c[k] for k in a}
    n = _dim(case["shells"])
    if kind == "evolve":
        return {"bytes": 8 * 5 * n * n, "flops": 2 * n ** 3 * (1 + 2 + 1 / 6 + 1)}
    if kind == "constraints":  # a handful of Newton steps: one evolution, two densities, three operators each
        return {"bytes": 8 * 12 * n * n, "flops": 5 * 2 * n ** 3 * (4.2 + 2 + 12)}
    S = _model(case["shells"]).ham.S
    if kind == "fields":
        c = case["cols"]
        return {"bytes": 13 * S + 16 * n * n * 7 * c, "flops": 4 * 8 * 1.65 * S * c}
    G = case["Mp"] * case["Mn"]
    if kind != "observables":
        G = (G + 1) // 2
    flops = G * (76 * n ** 3 + 4 * 8 * 1.65 * S)
    if kind == "observables":
        flops = G * (36 * n ** 3 + 4 * 8 * 1.65 * S + 3 * 3 * 8 * n ** 3)
    return {"bytes": 13 * S + 16 * n * n + 8 * n * n * 7, "flops": flops}


# ---------------------------------------------------------------------------
# the same in plain torch, 64 bits
# ---------------------------------------------------------------------------
_TR = torch.tensor([[0, 1, 2, 3], [1, 0, 2, 3], [0, 1, 3, 2], [1, 0, 3, 2],
                    [2, 3, 0, 1], [2, 3, 1, 0], [3, 2, 0, 1], [3, 2, 1, 0]])


def _sparse(rows, cols, vals, n2):
    t = torch.sparse_coo_tensor(torch.stack([rows, cols]), vals, (n2, n2)).coalesce()
    return t.to_sparse_csr()


@functools.lru_cache(maxsize=2)
def _field_matrices(shells):
    """(Gamma, Delta) as sparse matrices over the row-major entries of rho and kappa."""
    m = _model(shells)
    n, dev = m.basis.n, "cuda"
    ind = torch.tensor(m.ham.abcd.reshape(-1, 4).astype(np.int64) - 1, device=dev)
    h = torch.tensor(m.ham.h2.astype(np.float64), device=dev)
    code = torch.tensor(m.ham.trperm.astype(np.int64), device=dev)
    tr = torch.tensor(m.basis.sp_tr.astype(np.int64) - 1, device=dev)
    mj = torch.tensor(m.basis.sp_2mj.astype(np.int64), device=dev)
    # the time-reversed partner of every element whose M is not zero
    has = mj[ind[:, 0]] + mj[ind[:, 1]] != 0
    p = code[has]
    part = torch.gather(tr[ind[has]], 1, _TR.to(dev)[torch.where(p < 0, p + 8, p)])
    ind = torch.cat([ind, part])
    h = torch.cat([h, torch.where(p < 0, -h[has], h[has])])
    a, b, c, d = ind.unbind(1)
    f = torch.where((a == c) & (b == d), torch.zeros_like(h), h)
    at = lambda i, j: i * n + j  # noqa: E731
    gamma = _sparse(torch.cat([at(a, c), at(a, d), at(b, c), at(b, d), at(c, a), at(c, b), at(d, a), at(d, b)]),
                    torch.cat([at(d, b), at(c, b), at(d, a), at(c, a), at(b, d), at(a, d), at(b, c), at(a, c)]),
                    torch.cat([h, -h, -h, h, f, -f, -f, f]), n * n)
    delta = _sparse(torch.cat([at(b, a), at(d, c)]), torch.cat([at(d, c), at(b, a)]), torch.cat([h, f]), n * n)
    return gamma, delta


def _apply(op, X):
    """op on a batch (g, n, n) of complex matrices."""
    g, n, _ = X.shape
    y = op @ torch.view_as_real(X).permute(1, 2, 0, 3).reshape(n * n, 2 * g).contiguous()
    return torch.view_as_complex(y.reshape(n, n, g, 2).permute(2, 0, 1, 3).contiguous())


def _fields(shells, rho, kl, kr):
    gamma, delta = _field_matrices(shells)
    H1 = torch.tensor(_model(shells).ham.H1, device=rho.device)
    gam = _apply(gamma, rho)

    def skew(X):
        low = torch.tril(_apply(delta, X))
        return low - torch.tril(low, -1).transpose(1, 2)

    return gam, gam + H1, skew(kl), skew(kr)


def _pfaffian(A):
    """Pfaffians of a batch of skew matrices: Parlett-Reid elimination with partial pivoting (A is overwritten)."""
    b, m, _ = A.shape
    pf = torch.ones(b, dtype=A.dtype, device=A.device)
    every = torch.arange(b, device=A.device)
    for k in range(0, m - 1, 2):
        kp = k + 1 + A[:, k + 1:, k].abs().argmax(1)
        pf = torch.where(kp == k + 1, pf, -pf)
        r0, r1 = A[:, k + 1, :].clone(), A[every, kp, :].clone()
        A[:, k + 1, :] = r1
        A[every, kp, :] = r0
        c0, c1 = A[:, :, k + 1].clone(), A[every, :, kp].clone()
        A[:, :, k + 1] = c1
        A[every, :, kp] = c0
        piv = A[:, k, k + 1]
        pf = pf * piv
        if k + 2 < m:
            tau, col = A[:, k, k + 2:] / piv[:, None], A[:, k + 2:, k + 1].clone()
            A[:, k + 2:, k + 2:] += tau[:, :, None] * col[:, None, :] - col[:, :, None] * tau[:, None, :]
    return pf


def _overlaps(U, V, R):
    """<Phi| R |Phi> for diagonal rotations R (g, n) of the basis: the Pfaffian of the Thouless matrices of the two
    states, divided by that of the state with itself."""
    g, n = R.shape
    T = torch.linalg.solve(U.T, V.T).T.to(R.dtype)  # V U^-1 (real)
    T = 0.5 * (T - T.T)
    one = torch.eye(n, dtype=R.dtype, device=R.device).expand(g + 1, n, n)
    R = torch.cat([torch.ones(1, n, dtype=R.dtype, device=R.device), R])
    T1 = R[:, :, None] * T * R[:, None, :]
    A = torch.cat([torch.cat([T1, -one], 2), torch.cat([one, -T.expand(g + 1, n, n)], 2)], 1)
    pf = _pfaffian(A)
    return pf[1:] / pf[0]


def _grid(case, Z, Nn, n):
    """Rotations (g, n) and weights of the gauge angles."""
    def angles(count):
        j = torch.arange(count, dtype=torch.float64, device="cuda")
        return 2 * math.pi * (j if count % 2 else j + 0.5) / count

    p, q = angles(case["Mp"]), angles(case["Mn"])
    p, q = p.repeat_interleave(len(q)), q.repeat(len(p))
    w = torch.exp(-1j * (p * Z + q * Nn)) / len(p)
    R = torch.cat([torch.exp(1j * p)[:, None].expand(-1, n // 2), torch.exp(1j * q)[:, None].expand(-1, n // 2)], 1)
    return R, w


def _rotated(U, V, R):
    """A_phi, U~, V~ and the transition densities."""
    Uc, Vc = U.to(R.dtype), V.to(R.dtype)
    Ub, Vb = R[:, :, None] * Uc, R.conj()[:, :, None] * Vc
    Up, Vp = Vc.T @ Vb + Uc.T @ Ub, Vc.T @ Ub + Uc.T @ Vb
    A = torch.linalg.solve(Up.transpose(1, 2), Vp.transpose(1, 2)).transpose(1, 2).conj()
    Ut, Vt = Uc + Vc @ A, Vc + Uc @ A
    return A, Ut, Vt, Vt @ Vc.T, Vt @ Uc.T, Vc @ Ut.transpose(1, 2)


def _trace(X):
    return X.diagonal(dim1=1, dim2=2).sum(1)


def _numbers(rho, kl, kr):
    h = rho.shape[1] // 2
    out = []
    for at in (slice(0, h), slice(h, None)):
        r = rho[:, at, at]
        t = _trace(r)
        out += [t, t + t * t - (r * r.transpose(1, 2)).sum((1, 2)) + (kr[:, at, at] * kl[:, at, at]).sum((1, 2))]
    return out[0], out[2], out[1], out[3]  # protons, neutrons, and their squares


def _projected(case, shells, U, V, Z, Nn):
    """The projected sums and field_H20v (n x n) of the state."""
    n = U.shape[0]
    ham = _model(shells).ham
    R, w = _grid(case, Z, Nn, n)
    f = w * _overlaps(U, V, R)
    A, Ut, Vt, rho, kl, kr = _rotated(U, V, R)
    gam, h, dl, dr = _fields(shells, rho, kl, kr)
    H1 = torch.tensor(ham.H1, device="cuda")
    e = ham.H0 + (H1.T * rho).sum((1, 2)) + 0.5 * ((gam.transpose(1, 2) * rho).sum((1, 2)) + (dl * kr).sum((1, 2)))
    t = lambda X: X.transpose(1, 2)  # noqa: E731
    H20 = t(Ut) @ h @ Vt
    H20 = H20 - t(H20) + t(Ut) @ dl @ Ut - t(Vt) @ dr @ Vt
    sums = torch.stack([(f * x).sum() for x in (torch.ones_like(f), e, *_numbers(rho, kl, kr))])
    pA, pH, pAH = ((f * x)[:, None, None] * y for x, y in ((1, A), (1, H20), (e, A)))
    pA, pH, pAH = (0.5 * (x.sum(0) - x.sum(0).T) / sums[0] for x in (pA, pH, pAH))
    return sums, (pAH - sums[1] / sums[0] * pA + pH).real


def _evolved(U, V, Z):
    L = torch.linalg.cholesky(torch.eye(len(Z), dtype=Z.dtype, device=Z.device) + Z.T @ Z)
    back = lambda X: torch.linalg.solve_triangular(L, X.T, upper=False).T  # noqa: E731
    return back(U + V @ Z), back(V + U @ Z), L


def _iterated(case, shells, U, V, Z, Nn, eta):
    """One gradient step from Z_{i-1} = 0: sums, H20v, Z_i, |Z_i| / eta, U1, V1."""
    sums, H = _projected(case, shells, U, V, Z, Nn)
    Zi = -eta * H
    U1, V1, _ = _evolved(U, V, Zi)
    return sums, H, Zi, float(torch.linalg.norm(Zi)) / eta, U1, V1


def _dev(a):
    return torch.tensor(np.ascontiguousarray(a), device="cuda")


def _vec(X):
    return X.T.reshape(-1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "pfaffian":
        # the path reads the matrices column-major: the transposed, that is minus, of what the tensor holds
        return _pfaffian(prepare(case, seed)["A"].transpose(1, 2).clone())
    if kind == "fields":
        rho, kl, kr = _densities(case["shells"], case["cols"], seed)
        out = _fields(case["shells"], rho, kl, kr)
        if case["host"]:
            return [(x[0] if case["cols"] == 1 else x) for x in out]
        return [x.transpose(1, 2) for x in out]
    if kind == "many":
        out = {}
        st = _many(case, seed)
        for part, at, shells in (("even_small", slice(0, case["small"], 2), 0),
                                 ("even_large", slice(case["small"], None, 2), case["shells"])):
            r = [_iterated(case, shells, _dev(q[4]), _dev(q[5]), q[2], q[3], 0.02 if shells == 0 else ETA)
                 for q in st[at]]
            if r:
                out[part] = {"sums": torch.stack([q[0] for q in r]), "Zi": torch.stack([_vec(q[2]) for q in r]),
                             "norm": np.array([q[3] for q in r]), "U1": torch.stack([q[4] for q in r]),
                             "V1": torch.stack([q[5] for q in r])}
        return out  # (odd states: their U is singular, the Thouless matrices of _overlaps do not exist)
    Z, Nn = case.get("Z", 6), case.get("N", 6)
    n = _dim(case["shells"])
    Uh, Vh = _state(case["shells"], Z, Nn, seed)
    U, V = _dev(Uh), _dev(Vh)
    if kind == "evolve":
        return list(_evolved(U, V, _dev(_thouless(n, seed + 1, 0.05)))[:2])
    if kind == "constraints":
        ops, target = _constraint_target(case, Uh, Vh)
        C = [_dev(x.reshape(n, n, order="F")) for x in ops]
        T = torch.tensor(target, dtype=torch.float64, device="cuda")
        Zi = _dev(_thouless(n, seed + 1, 1e-3))
        for step in range(1, 101):
            U1, V1, _ = _evolved(U, V, Zi)
            rho = V1 @ V1.T
            off = T - torch.stack([(c * rho.T).sum() for c in C])
            C20 = []
            for c in C:
                x = U1.T @ c @ V1 - V1.T @ c.T @ U1
                C20.append(0.5 * (x - x.T))
            if float(off.abs().max()) <= 1e-6:
                break
            gram = torch.stack([torch.stack([(x * y).sum() for y in C20]) for x in C20])
            for x, c20 in zip(torch.linalg.solve(gram, off).tolist(), C20):
                Zi = Zi + x * c20
        return {"U1": U1, "V1": V1, "Zi": _vec(Zi), "C20": torch.stack([_vec(x) for x in C20]), "steps": step}
    if Z % 2:
        return None  # odd states: as above
    if kind == "iterate":
        sums, H, Zi, norm, U1, V1 = _iterated(case, case["shells"], U, V, Z, Nn, _eta(case))
        if case["host"]:
            return {"sums": sums, "Zi": _vec(Zi), "norm": norm, "U1": U1, "V1": V1, "H20v": _vec(H)}
        return {"sums": sums, "norm": norm, "Zi": _vec(Zi), "U1": _vec(U1), "V1": _vec(V1), "H20v": _vec(H)}
    if kind == "adjoint":
        U1, V1, L = _evolved(U, V, _dev(_thouless(n, seed + 1, 0.02)))
        sums, H = _projected(case, case["shells"], U1, V1, Z, Nn)
        G = torch.linalg.solve_triangular(L.T, torch.linalg.solve_triangular(L, H, upper=False, left=False),
                                          upper=True)
        return {"E": (sums[1] / sums[0]).real, "dEdZ": G}
    # observables
    m = _model(case["shells"])
    ops = m.observable_operators()
    R, w = _grid(case, Z, Nn, n)
    f = w * _overlaps(U, V, R)
    _, _, _, rho, kl, kr = _rotated(U, V, R)
    gam, _, dl, _ = _fields(case["shells"], rho, kl, kr)
    H1 = torch.tensor(m.ham.H1, device="cuda")
    h = n // 2
    halves = (slice(0, h), slice(h, None))
    rows = lambda X, Y, at: (X[..., at, :] * Y.transpose(1, 2)[:, at, :]).sum((1, 2))  # noqa: E731
    one = [rows(H1, rho, at) for at in halves]
    ph = [0.5 * (gam[:, i, j] * rho[:, j, i].transpose(1, 2)).sum((1, 2)) for i in halves for j in halves]
    pp = [0.5 * (dl[:, i, j] * kr[:, i, j]).sum((1, 2)) for i in halves for j in halves]
    both = [one[t] + ph[2 * t] + ph[2 * t + 1] + pp[2 * t] + pp[2 * t + 1] for t in (0, 1)]
    par = torch.tensor(ops["parity"].astype(np.float64), device="cuda")
    scal = [(f * x).sum() for x in (torch.ones_like(f), m.ham.H0 + both[0] + both[1], *_numbers(rho, kl, kr))]
    scal += [(w * _overlaps(U, V, R * par)).sum()] + [(f * x).sum() for x in one + ph + pp + both]
    obo = torch.stack([torch.stack([(f * rows(_dev(B), rho, at)).sum() for at in halves]) for B in ops["obo"]])
    sq = []
    for O, O2 in ops["sq"]:
        O, O2 = _dev(O), _dev(O2)
        r = O @ rho
        t1 = _trace(r)
        sq.append((f * (t1 * t1 + (O2.T * rho).sum((1, 2)) - (r * r.transpose(1, 2)).sum((1, 2))
                        + ((O.T @ kr.transpose(1, 2)) * (O @ kl).transpose(1, 2)).sum((1, 2)))).sum())
    occ = (f[:, None] * rho.diagonal(dim1=1, dim2=2)).sum(0).reshape(2, h)
    ends = np.concatenate([[0], np.cumsum(ops["shell_size"])])
    occ = torch.stack([torch.stack([occ[t, a:b].sum() for t in (0, 1)]) for a, b in zip(ends[:-1], ends[1:])])
    return {"scal": torch.stack(scal), "obo": obo, "sq": torch.stack(sq), "occnum": occ,
            "rho": (f[:, None, None] * rho).sum(0)}
