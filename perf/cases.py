"""Performance cases of the G-MCTDH core: the calls a propagation program makes.

A driver calls the C-ABI of ``include/macaw_gb300.h`` on its own (page-locked)
host arrays: one equation of motion (``mctdh_calc_derivs``), one Runge-Kutta
attempt (``mctdh_rk_attempt``), one CMF2 step of a given length
(``mctdh_cmf2_attempt``); it reads observables of the resident state at every
output time; and it advances ensembles of small wavepackets together.  The
states have the structure of a wavepacket some way into its propagation: complex
SPFs that differ between the electronic states and natural populations that fall
from one to about 1e-6 over the SPFs of a mode.

The step-error numbers of the attempts are left out of the outputs:
sqrt|2 (1 - Re<1|2> / sqrt(<1|1><2|2>))| is at the rounding floor of
1 - Re<1|2> for steps of the lengths that a propagation accepts.
"""
import ctypes as C
import random

import numpy as np
import torch

from macaw_gb300.capi import DP, Ensemble, GpuCore
from macaw_gb300.generate import ensemble_member, gmctdh16, lvc5, qvc, qvc12
from macaw_gb300.model import AU2FS, OP_DQ2, initial_wavefunction

MODEL_SEED = 20261203


def listed():
    return [
        # the smallest models of teaching inputs and tests: 2 states, 3 modes; latency only
        _case("eom_small", "eom", "qvc", nstates=2, modes=3, dofs=1, grid=16, nspf=4, ncoup=1, precision=0),
        # 2-state / 5-mode linear vibronic coupling, 6 SPFs: one Calc_Derivs in FP64 ...
        _case("eom_lvc5", "eom", "lvc5", nspf=6, precision=0),
        # ... and what its RK45 propagation spends its time on: a Cash-Karp attempt
        _case("rk_lvc5", "rk", "lvc5", nspf=6, precision=0, dt_fs=0.02),
        # uneven SPF counts (5..9) and odd grids, compensated arithmetic
        _case("eom_uneven_split", "eom", "qvc", nstates=3, modes=5, dofs=1, grid=27, nspf=7, ncoup=3, precision=2,
              uneven=True),
        # 3-state / 12-DOF / 6-mode QVC model, 8 SPFs (786,432 coefficients): FP64 EOM
        _case("eom_qvc12", "eom", "qvc12", nspf=8, precision=0),
        # the same model with 12 SPFs (143 MB of coefficients, beyond L2), the mixed-precision path
        _case("eom_qvc12_12spf_mixed", "eom", "qvc12", nspf=12, precision=5),
        # one CMF2 step: a small model with odd sizes, then the benchmark model in FP64
        # and in the mixed precision of its headline
        _case("cmf2_small", "cmf2", "qvc", nstates=3, modes=4, dofs=2, grid=7, nspf=5, ncoup=3, precision=0,
              dt_fs=0.03),
        _case("cmf2_qvc12", "cmf2", "qvc12", nspf=8, precision=0, dt_fs=0.03),
        _case("cmf2_qvc12_mixed", "cmf2", "qvc12", nspf=8, precision=5, dt_fs=0.03),
        # scans over initial conditions and couplings: 24 uneven wavepackets, FP32 products
        _case("ensemble_eom", "ens", "ens", members=24, max_conf=1 << 14, precision=1),
        # variational Gaussians: 4 grid modes and one 12-DOF mode of 32 Gaussians per state
        _case("eom_gaussian", "eom", "gmctdh16", precision=0),
        # an output time: energy, populations, norm, C(t) and natural populations
        _case("output_qvc12", "out", "qvc12", nspf=8, precision=0),
    ]


def _case(name, kind, model, **kw):
    c = {"kind": kind, "model": model, **kw}
    if name:
        c["name"] = name
    return c


def draw(rng):
    """Calls of the same kinds on vibronic models of 2-4 states and 3-7 modes, equal
    or uneven SPF counts of 3-12, grids of 6-40 points per DOF, one or two DOFs
    per mode, 1-4 coupling terms; ensembles of 4-24 members."""
    kind = rng.choice(["eom", "eom", "eom", "rk", "cmf2", "out", "ens"])
    if kind == "ens":
        return _case("", "ens", "ens", members=rng.randint(4, 24), max_conf=int(2 ** rng.uniform(8, 14)),
                     precision=rng.choice([0, 1, 2]), shape=rng.randint(1, 10 ** 6))
    precision = rng.choice([0, 0, 2, 5, 1] if kind == "eom" else [0, 0, 5] if kind == "cmf2" else [0])
    most = 2 ** (16 if kind == "cmf2" else 19 if precision == 0 else 20)
    total = 2 ** rng.uniform(8, np.log2(most))   # coefficients of all states
    while True:
        nstates, modes, nspf = rng.randint(2, 4), rng.randint(3, 7), rng.randint(3, 12)
        if 0.5 * total <= nstates * nspf ** modes <= 1.4 * total:
            break
    dofs = rng.choice([1, 1, 2])
    grid = rng.randint(14, 40) if dofs == 1 else rng.randint(6, 20)
    c = _case("", kind, "qvc", nstates=nstates, modes=modes, dofs=dofs, grid=grid, nspf=nspf,
              ncoup=rng.randint(1, min(4, modes)), precision=precision, uneven=rng.random() < 0.5,
              shape=rng.randint(1, 10 ** 6))
    if kind in ("rk", "cmf2"):
        c["dt_fs"] = round(rng.uniform(0.01, 0.03), 4)
    return c


# --------------------------------------------------------------------------
# models and states
# --------------------------------------------------------------------------
def _model(case):
    if case["model"] == "lvc5":
        return lvc5(nspf=case["nspf"])
    if case["model"] == "qvc12":
        return qvc12(nspf=case["nspf"])
    if case["model"] == "gmctdh16":
        return gmctdh16()
    shape = case.get("shape", 1)
    nst, ndof = case["nstates"], case["modes"] * case["dofs"]
    m = qvc(nst, ndof, case["grid"], case["nspf"], case["ncoup"], MODEL_SEED + shape, (200.0, 3500.0),
            (0.05, 0.2), [0.35 * s for s in range(nst)], "qvc", dofs_per_mode=case["dofs"])
    if case.get("uneven"):
        rng = np.random.default_rng(shape)
        low = max(2, case["nspf"] - 2)
        m.nspf = rng.integers(low, case["nspf"] + 3, (m.nmodes, nst))
        m.ngp = [int(g) for g in rng.integers(max(5, case["grid"] - 3), case["grid"] + 4, ndof)]
        m = m.finalize()
    return m


def _members(case):
    rng = np.random.default_rng(MODEL_SEED + case.get("shape", 1))
    return [ensemble_member(rng, i, case["max_conf"]) for i in range(case["members"])]


def _state(model, rng):
    """(A, psi) of a correlated wavepacket: SPFs of every state displaced in momentum
    and mixed, coefficients of random phase that fall off with the SPF index."""
    psi = initial_wavefunction(model)[1]
    for m in range(model.nmodes):
        for s in range(model.nstates):
            n, o = int(model.nspf[m, s]), int(model.ipsispf[m, s])
            if model.is_gwp_mode[m]:
                k = n * len(model.mode_dofs[m])
                psi[o:o + k] += 0.1 * (rng.standard_normal(k) + 1j * rng.standard_normal(k))
                continue
            G = model.ngpm[m]
            phase = np.zeros(1)
            for d in reversed(model.mode_dofs[m]):   # first DOF fastest
                phase = (phase[:, None] + rng.uniform(-0.8, 0.8) * model.grid[d][None, :]).reshape(-1)
            phi = psi[o:o + G * n].reshape(G, n, order="F") * np.exp(1j * phase)[:, None]
            mix = np.eye(n) + 0.3 * (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)))
            psi[o:o + G * n] = np.linalg.qr(phi @ mix)[0].reshape(-1, order="F")
    parts = []
    for s in range(model.nstates):
        ns = [int(x) for x in model.nspf[:, s]]
        w = np.ones(1)
        for n in ns:   # mode 1 fastest
            w = (10.0 ** (-2.0 * np.arange(n) / max(n - 1, 1))[:, None] * w[None, :]).reshape(-1)
        a = (rng.standard_normal(w.size) + 1j * rng.standard_normal(w.size)) * w
        parts.append(a * (np.sqrt(1.0 + s) / np.linalg.norm(a)))
    A = np.concatenate(parts)
    return A / np.linalg.norm(A), psi


def _pinned(x):
    return torch.from_numpy(np.ascontiguousarray(x, dtype=np.complex128)).pin_memory()


def _p(t):
    return C.cast(t.data_ptr(), DP)


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    if case["kind"] == "ens":
        models = _members(case)
        ens = Ensemble(models, precision=case["precision"], autotune=False)
        for i, m in enumerate(models):
            ens.set_state(i, *_state(m, rng))
        return {"kind": "ens", "ens": ens}
    model = _model(case)
    A, psi = _state(model, rng)   # also fixes the widths of Gaussian SPFs, part of the set-up
    core = GpuCore(model, precision=case["precision"])
    st = {"kind": case["kind"], "core": core, "A": _pinned(A), "psi": _pinned(psi)}
    if case["kind"] == "out":
        core.set_state(*_state(model, rng), as_start=True)
        core.set_state(A, psi, as_start=False)
    elif case["kind"] in ("eom", "rk"):
        st["dA"], st["dpsi"] = torch.empty_like(st["A"]).pin_memory(), torch.empty_like(st["psi"]).pin_memory()
    if case["kind"] == "rk":   # the derivative at the start of the step, as the time loop has it
        core._check(core.lib.mctdh_calc_derivs(core.h, _p(st["A"]), _p(st["psi"]), _p(st["dA"]), _p(st["dpsi"]), 0.0))
        st["A0"], st["psi0"] = st["A"].clone(), st["psi"].clone()
    if "dt_fs" in case:
        st["dt"] = case["dt_fs"] / AU2FS
    return st


def run(st):
    if st["kind"] == "ens":
        return st["ens"].calc_derivs()
    core = st["core"]
    lib = core.lib
    if st["kind"] == "eom":
        core._check(lib.mctdh_calc_derivs(core.h, _p(st["A"]), _p(st["psi"]), _p(st["dA"]), _p(st["dpsi"]), 0.0))
        return {"dA": st["dA"], "dpsi": st["dpsi"]}
    err = C.c_double()
    if st["kind"] == "rk":     # every attempt from the same state, like a step that is retried
        st["A"].copy_(st["A0"])
        st["psi"].copy_(st["psi0"])
        core._check(lib.mctdh_rk_attempt(core.h, _p(st["A"]), _p(st["psi"]), _p(st["dA"]), _p(st["dpsi"]), 0.0,
                                         st["dt"], 1, C.byref(err)))
        return {"A": st["A"], "psi": st["psi"]}
    if st["kind"] == "cmf2":   # in place: the next pass is the next step of the propagation
        core._check(lib.mctdh_cmf2_attempt(core.h, _p(st["A"]), _p(st["psi"]), 0.0, st["dt"], C.byref(err)))
        return {"A": st["A"], "psi": st["psi"]}
    o = core.observables(0.0)
    return {"energy": np.float64(o["energy"]), "pop": o["pop"], "norm": np.float64(o["norm"]),
            "auto": np.array([o["auto"].real, o["auto"].imag]), "natpop": core.natpop()[0]}


# --------------------------------------------------------------------------
# the work of one pass
# --------------------------------------------------------------------------
def _eom_flops(model):
    """Complex multiply-adds (8 FLOP each) of one EOM: per state and mode the pre-summed
    one-mode operators and the density contraction; per coupling term the product
    over all modes, and per conjugate pair of them one mean field for each mode
    with the partial products it needs; the operators on the SPFs."""
    size = [float(np.prod(model.nspf[:, s])) for s in range(model.nstates)]
    fl = 0.0
    for s in range(model.nstates):
        fl += 2 * 8 * size[s] * float(model.nspf[:, s].sum())
    for t in model.terms:
        if t.lhs != t.rhs:
            fl += 8 * size[t.rhs] * float(model.nspf[:, t.lhs].sum()) * (1 + 0.5 + 0.5)
    for m in model.modes_dvr:
        for s in range(model.nstates):
            n = float(model.nspf[m, s])
            fl += 8 * model.ngpm[m] * n * n * (len(model.mode_dofs[m]) * 2 + 3)
    return fl


def work(case):
    models = _members(case) if case["kind"] == "ens" else [_model(case)]
    fl = sum(_eom_flops(m) for m in models)
    n = sum(16.0 * (m.naconftot + m.dimpsi) for m in models)
    if case["kind"] == "rk":       # five evaluations; state and derivative in, state out
        return {"bytes": 3 * n, "flops": 5 * fl}
    if case["kind"] == "cmf2":     # two mean-field evaluations, about 20 products H_B B
        return {"bytes": 2 * n, "flops": 12 * fl}
    if case["kind"] == "out":
        return {"bytes": 2 * n, "flops": 1.5 * fl}
    return {"bytes": 2 * n, "flops": fl}


# --------------------------------------------------------------------------
# the same quantities in plain 64-bit numpy
# --------------------------------------------------------------------------
def exact(case, seed):
    """None for the Gaussian mode (its integrals and regularised parameter solve have no
    short plain form), the CMF2 step (adaptive inner integrations) and models whose
    products would take minutes on the host."""
    rng = np.random.default_rng(seed)
    if case["kind"] == "ens":
        return [_eom(m, *_state(m, rng))[:2] for m in _members(case)]
    model = _model(case)
    if case["kind"] == "cmf2" or model.modes_gwp or model.naconftot > 2_000_000:
        return None
    A, psi = _state(model, rng)
    if case["kind"] == "eom":
        dA, dpsi = _eom(model, A, psi)[:2]
        return {"dA": dA, "dpsi": dpsi}
    if case["kind"] == "rk":
        return _cash_karp(model, A, psi, case["dt_fs"] / AU2FS)
    start = _state(model, rng)
    dA, _, rho = _eom(model, A, psi)
    pop = np.array([np.trace(rho[0, s]).real for s in range(model.nstates)])
    nat = np.zeros((int(model.nspf.max()), model.nmodes, model.nstates), order="F")
    for (m, s), r in rho.items():
        nat[:len(r), m, s] = np.linalg.eigvalsh(r)[::-1]
    auto = 0.0
    for s in range(model.nstates):
        B = _tensor(model, A, s)
        for m in range(model.nmodes):
            B = _apply(_spf(model, start[1], m, s).conj().T @ _spf(model, psi, m, s), B, m)
        auto += np.vdot(_tensor(model, start[0], s), B)
    return {"energy": np.vdot(A, 1j * dA).real / pop.sum(), "pop": pop, "norm": pop.sum(),
            "auto": np.array([auto.real, auto.imag]), "natpop": nat}


def _cash_karp(model, A, psi, dt):
    b = [[0.2], [3 / 40, 9 / 40], [0.3, -0.9, 1.2], [-11 / 54, 2.5, -70 / 27, 35 / 27],
         [1631 / 55296, 175 / 512, 575 / 13824, 44275 / 110592, 253 / 4096],
         [37 / 378, 0.0, 250 / 621, 125 / 594, 0.0, 512 / 1771]]
    k = []
    y = (A, psi)
    for row in b:
        k.append(_eom(model, *y)[:2])
        y = tuple(v + dt * sum(c * q[i] for c, q in zip(row, k)) for i, v in enumerate((A, psi)))
    return {"A": y[0], "psi": y[1]}


def _tensor(model, A, s):
    size = [int(np.prod(model.nspf[:, q])) for q in range(model.nstates)]
    o = sum(size[:s])
    return A[o:o + size[s]].reshape([int(x) for x in model.nspf[:, s]], order="F")


def _spf(model, psi, m, s):
    n, o, G = int(model.nspf[m, s]), int(model.ipsispf[m, s]), model.ngpm[m]
    return psi[o:o + G * n].reshape(G, n, order="F")


def _apply(M, T, m):
    return np.moveaxis(np.tensordot(M, T, axes=(1, m)), 0, m)


def _hole(X, Y, m):
    n1, n2 = X.shape[m], Y.shape[m]
    return np.moveaxis(X, m, 0).reshape(n1, -1).conj() @ np.moveaxis(Y, m, 0).reshape(n2, -1).T


def _grid_op(model, m, ops, phi):
    """The product of the DOF operators `ops` ({dof: code}) of mode m on the SPFs."""
    dofs = model.mode_dofs[m]
    x = phi.reshape([model.ngp[d] for d in dofs] + [-1], order="F")
    for k, d in enumerate(dofs):
        if d not in ops:
            continue
        if ops[d] == OP_DQ2:
            x = _apply(np.asarray(model.d2[d]).T, x, k)
        else:
            q = np.asarray(model.grid[d]) ** ops[d]
            x = x * q.reshape([-1 if i == k else 1 for i in range(x.ndim)])
    return x.reshape(phi.shape, order="F")


def _eom(model, A, psi):
    """dA, dpsi and the density matrices of a grid model with one SPF set per state."""
    f, ns = model.nmodes, model.nstates
    T = [_tensor(model, A, s) for s in range(ns)]
    phi = {(m, s): _spf(model, psi, m, s) for m in range(f) for s in range(ns)}
    rho = {(m, s): _hole(T[s], T[s], m) for m in range(f) for s in range(ns)}
    HA = [np.zeros_like(t) for t in T]
    one = {}                       # (m, s) -> sum of the one-mode operators of the state
    drive = {k: 0.0 for k in phi}  # (m, s) -> sum of O phi (rho^-1 MF)^T before rho^-1
    inv = {}
    for k, r in rho.items():
        w, U = np.linalg.eigh(0.5 * (r + r.conj().T))
        e = model.eps_rho
        inv[k] = (U / np.where(w < e, 0.5 * (e + w * w / e), w)) @ U.conj().T
    for t in model.terms:
        mode_of = {m: {d: c for d, c in t.dof_ops.items() if d in model.mode_dofs[m]} for m in range(f)}
        a, b = t.lhs, t.rhs
        act = [m for m in range(f) if mode_of[m]]
        if a == b and len(act) <= 1:
            if not act:
                HA[a] = HA[a] + t.coeff * T[a]
                continue
            m = act[0]
            o = _grid_op(model, m, mode_of[m], phi[m, a])
            h = phi[m, a].conj().T @ o
            one[m, a] = one.get((m, a), 0.0) + t.coeff * 0.5 * (h + h.conj().T)
            drive[m, a] = drive[m, a] + o @ (inv[m, a] @ (t.coeff * rho[m, a])).T
            continue
        o = {m: _grid_op(model, m, mode_of[m], phi[m, b]) for m in range(f)}
        h = {m: phi[m, a].conj().T @ o[m] for m in range(f)}
        left, right = [T[a]], [T[b]]
        for m in range(f - 1):
            left.append(_apply(h[m].conj().T, left[-1], m))
        for m in range(f - 1, -1, -1):
            right.append(_apply(h[m], right[-1], m))
        HA[a] = HA[a] + t.coeff * right[f]
        for m in range(f):
            mf = t.coeff * _hole(left[m], right[f - 1 - m], m)
            drive[m, a] = drive[m, a] + o[m] @ (inv[m, a] @ mf).T
    for (m, s), h in one.items():
        HA[s] = HA[s] + _apply(h, T[s], m)
    dA = np.concatenate([-1j * x.reshape(-1, order="F") for x in HA])
    dpsi = np.zeros_like(psi)
    for (m, s), d in drive.items():
        p = phi[m, s]
        d = -1j * d
        d = d - p @ np.linalg.solve(p.conj().T @ p, p.conj().T @ d)
        o = int(model.ipsispf[m, s])
        dpsi[o:o + d.size] = d.reshape(-1, order="F")
    return dA, dpsi, rho


if __name__ == "__main__":
    r = random.Random(1)
    for c in listed() + [draw(r) for _ in range(6)]:
        print(c, work(c))
