"""Operands of very different size in one vector: the digit products share an exponent per
fibre, row or column, and have to hold the bound of an FP64 chain all the same,
|error| <= 2 N 2^-53 sum |x||y| for N complex terms (two products each), for every element.

The references are sums in long double (or, for diagonal matrices, products); SPFs are
unit vectors of the grid, so that the matrices are known exactly.
"""
import numpy as np
import pytest

from macaw_gb300.generate import gmctdh16
from macaw_gb300.model import Model, Term
from oracle.mctdh import Oracle
from tests.helpers import random_state

pytestmark = pytest.mark.gpu

U = 2.0 ** -53
LD = np.clongdouble


def _model(sizes, nstates, terms, grid=34):
    f = len(sizes)
    return Model(nstates=nstates, mode_dofs=[[k] for k in range(f)], multiset=[True] * f,
                 nspf=np.array([[n] * nstates for n in sizes]), dvr_type=["HO"] * f, ngp=[grid] * f,
                 dvrpar=[(0.0, 1.0)] * f, terms=terms, init_state=0, label="graded").finalize()


def _unit_spfs(model):
    psi = np.zeros(model.dimpsi, dtype=complex)
    for m in range(model.nmodes):
        for s in range(model.nstates):
            o, G, n = int(model.ipsispf[m, s]), model.ngpm[m], int(model.nspf[m, s])
            psi[o:o + G * n] = np.eye(G, n).reshape(-1, order="F")
    return psi


def _phases(rng, shape):
    return np.exp(2j * np.pi * rng.random(shape))


# densities: one operand block of columns and more, short and full last blocks
@pytest.mark.parametrize("sizes", [(2, 8, 8, 8), (5, 17, 16), (8, 9, 31), (9, 8, 8, 8), (13, 31, 9), (16, 8, 8, 8), (31, 20)])
@pytest.mark.parametrize("grade", ["opposite", "along", "elements"])
def test_contractions(sizes, grade):
    from macaw_gb300.capi import GpuCore
    model = _model(sizes, 1, [Term(0.01 + 0j, 0, 0, {0: 1})])
    rng = np.random.default_rng(sum(sizes))
    n, P = sizes[0], int(np.prod(sizes[1:]))
    at = np.linspace(0.0, 12.0, P)
    if grade == "opposite":     # neighbouring columns fall and rise
        power = np.where(np.arange(n)[:, None] % 2, at[::-1], at)
    elif grade == "along":      # all fall, the weaker columns by more
        power = at * (1.0 + np.arange(n)[:, None] / n) / 2
    else:
        power = rng.uniform(0.0, 14.0, (n, P))
    X = 10.0 ** -power * _phases(rng, (n, P))
    core = GpuCore(model)
    core.set_state(X.reshape(-1, order="F"), _unit_spfs(model))
    rho = core.densmat(0, 0)
    ref = np.array([[(X[i].astype(LD).conj() * X[j].astype(LD)).sum() for j in range(n)] for i in range(n)])
    bound = 2 * P * U * (np.abs(X) @ np.abs(X).T)
    assert (np.abs((rho - ref).astype(complex)) <= bound).all()


# mode products: output groups of four, the odd last one, more than 16; from (8, 8, 8, 8, 8, 5)
# on enough fibres for the tcgen05 form, with short last tiles
@pytest.mark.parametrize("sizes", [(3, 2, 2), (8, 7, 9), (9, 4, 12), (13, 8, 6), (24, 6, 25), (32, 5, 9), (8, 8, 8, 8, 8, 5),
                                   (6, 7, 8, 8, 6, 6), (9, 12, 10, 11, 9), (13, 14, 5, 16, 8)])
@pytest.mark.parametrize("grade", ["index", "elements", "late"])
def test_mode_products(sizes, grade):
    from macaw_gb300.capi import GpuCore
    lam = 0.01
    model = _model(sizes, 2, [Term(lam + 0j, 0, 1, {0: 1}), Term(lam + 0j, 1, 0, {0: 1})])
    rng = np.random.default_rng(sum(sizes))
    x = _phases(rng, sizes)
    if grade == "index":        # weakly occupied SPFs
        for m, n in enumerate(sizes):
            x *= (10.0 ** (-9.0 * np.arange(n) / n)).reshape([n if k == m else 1 for k in range(len(sizes))])
    elif grade == "elements":
        x *= 10.0 ** -rng.uniform(0.0, 14.0, sizes)
    else:                       # columns that are zero in the first fibres, and strong later
        late = np.arange(int(np.prod(sizes[1:]))).reshape(sizes[1:], order="F") > np.prod(sizes[1:]) // 2
        x[1::2] *= np.where(late, 1e6, 0.0)
    n1 = int(np.prod(sizes))
    A = np.concatenate([np.zeros(n1), x.reshape(-1, order="F")])
    dA = GpuCore(model).calc_derivs(A, _unit_spfs(model), 0.0)[0]
    q = np.asarray(model.grid[0])[:sizes[0]]
    ref = (-1j * lam * q.reshape([-1] + [1] * (len(sizes) - 1)) * x).reshape(-1, order="F")
    # a product per mode, the coefficient's and the factor's
    bound = (2 * sum(sizes) + 8) * U * np.abs(ref)
    assert (np.abs(dA[:n1] - ref) <= bound).all()


# operator sums of the SPF derivatives: q with weight 1, q^12 with one that makes them alike
# at the grid's end; the coefficients are the unit matrix, so that rho^-1 MF is diagonal
@pytest.mark.parametrize("n", [1, 4, 8, 9, 12, 17])
def test_operator_sums(n):
    from macaw_gb300.capi import GpuCore
    grid = 70                    # two tiles of rows
    q = np.asarray(_model((n, n), 1, [Term(1.0 + 0j, 0, 0, {0: 1})], grid).grid[0])
    weight = {1: 1.0, 3: 0.25, 12: float(1.0 / np.abs(q).max() ** 11)}
    model = _model((n, n), 1, [Term(w + 0j, 0, 0, {0: p}) for p, w in weight.items()], grid)
    rng = np.random.default_rng(n)
    phi = np.linalg.qr(rng.standard_normal((grid, n)) + 1j * rng.standard_normal((grid, n)))[0]
    psi = _unit_spfs(model)
    o = int(model.ipsispf[0, 0])
    psi[o:o + grid * n] = phi.reshape(-1, order="F")
    dpsi = GpuCore(model).calc_derivs(np.eye(n).reshape(-1) + 0j, psi, 0.0)[1][o:o + grid * n].reshape(grid, n, order="F")
    p = phi.astype(LD)
    op = sum(w * (q ** k).astype(LD) for k, w in weight.items())
    size = sum(w * np.abs(q) ** k for k, w in weight.items())
    S = p.conj().T @ p
    X = p.conj().T @ (op[:, None] * p)
    for _ in range(3):           # S = 1 up to rounding: S^-1 X by iteration
        X = X - (S @ X - p.conj().T @ (op[:, None] * p))
    ref = -1j * (op[:, None] * p - p @ X)
    a = np.abs(phi)
    # 2 x 3 n terms, the operators' own roundings (powers), the projection: phi^H O phi over the
    # grid and n terms of phi X
    bound = U * ((6 * n + 40) * size[:, None] * a + a @ ((2 * grid + 4 * n + 40) * (a.T @ (size[:, None] * a))))
    assert (np.abs((dpsi - ref).astype(complex)) <= bound).all()


# Gaussian parameters of weakly occupied SPFs: panels of graded rows and columns; tolerance as
# in test_gpu_gwp_solve
@pytest.mark.parametrize("ngwp, dofs", [(3, 3), (6, 5), (11, 3)])
def test_graded_parameter_equations(ngwp, dofs):
    from macaw_gb300.capi import GpuCore
    model = gmctdh16(ngwp=ngwp, gwp_dofs=dofs, dvr_grid=6, dvr_nspf=3)
    A, psi = random_state(model, seed=11, gwp_shift=0.5)
    m = model.modes_gwp[0]
    o = 0
    for s in range(model.nstates):
        shape = [int(n) for n in model.nspf[:, s]]
        a = A[o:o + int(np.prod(shape))].reshape(shape, order="F")
        a *= (10.0 ** (-5.0 * np.arange(ngwp) / ngwp)).reshape([ngwp if k == m else 1 for k in range(len(shape))])
        A[o:o + a.size] = a.reshape(-1, order="F")
        o += a.size
    A /= np.sqrt(Oracle(model).norm_wf(A, psi))
    rng = np.random.default_rng(0)
    ulp = np.finfo(float).eps
    ref = Oracle(model).calc_derivs(A, psi, 0.0)
    moved = Oracle(model).calc_derivs(A * (1 + ulp * rng.standard_normal(A.size)),
                                      psi * (1 + ulp * rng.standard_normal(psi.size)), 0.0)
    out = GpuCore(model).calc_derivs(A, psi, 0.0)
    rel = lambda a, b: np.linalg.norm(a - b) / np.linalg.norm(b)
    assert rel(out[0], ref[0]) < max(1e-12, 1e3 * rel(moved[0], ref[0]))
    for s in range(model.nstates):
        b = int(model.ipsispf[m, s])
        b = slice(b, b + ngwp * dofs)
        assert rel(out[1][b], ref[1][b]) < max(1e-12, 1e3 * rel(moved[1][b], ref[1][b]))
