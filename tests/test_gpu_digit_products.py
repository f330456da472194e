"""The mode products and contractions of FP64 accuracy (exact 8-bit digit products on
the tensor cores) through one EOM evaluation against the oracle, at the SPF counts
where their tiles end (4 outputs and 16 fibres per MMA, 8 x 8 pair blocks), and for
operands outside the exponent range the digits cover.

Tolerance: the EOM parity of the FP64 path, 1e-11 relative, on random states whose
density matrices are well conditioned (the digit products round below FP64's own
rounding); scaling A by a power of two scales dA exactly up to FP64 rounding.
"""
import numpy as np
import pytest

from macaw_gb300.generate import qvc
from oracle.mctdh import Oracle
from tests.helpers import random_state
from tests.test_gpu_parity import _rel

pytestmark = pytest.mark.gpu

RTOL = 1e-11
SIZES = [(2, 3, 2), (4, 5, 3), (8, 7, 9), (9, 12, 4), (13, 8, 6), (16, 17, 5), (24, 6, 25), (32, 5, 9)]


@pytest.fixture(scope="module")
def capi():
    from macaw_gb300 import capi
    return capi


def _model(sizes):
    m = qvc(2, 3, 34, 4, 2, 11, (200.0, 3500.0), (0.05, 0.2), (0.0, 0.4), "digits", dofs_per_mode=1)
    m.nspf = np.array([[n, sizes[(i + 1) % 3]] if i else [n, n] for i, n in enumerate(sizes)])
    return m.finalize()


@pytest.mark.parametrize("precision", [0, 2])
@pytest.mark.parametrize("sizes", SIZES)
def test_eom_at_tile_edges(capi, sizes, precision):
    model = _model(sizes)
    A, psi = random_state(model, seed=sum(sizes))
    ref = Oracle(model).calc_derivs(A, psi, 0.0)
    out = capi.GpuCore(model, precision=precision).calc_derivs(A, psi, 0.0)
    tol = RTOL if precision == 0 else 1e-10
    assert _rel(out[0], ref[0]) < tol
    assert _rel(out[1], ref[1]) < tol


@pytest.mark.parametrize("power", [-430, -380, 0, 380, 430])
def test_scaled_coefficients(capi, power):
    model = _model((5, 6, 8))
    A, psi = random_state(model, seed=3)
    core = capi.GpuCore(model)
    dA = core.calc_derivs(A, psi, 0.0)[0]
    scaled = core.calc_derivs(np.ldexp(1.0, power) * A, psi, 0.0)[0]
    assert _rel(scaled * np.ldexp(1.0, -power), dA) < 1e-13


def test_zero_and_non_finite_coefficients(capi):
    model = _model((5, 6, 8))
    A, psi = random_state(model, seed=4)
    core = capi.GpuCore(model)
    n0 = int(np.prod(model.nspf[:, 0]))
    A[:n0] = 0.0
    ref = Oracle(model).calc_derivs(A, psi, 0.0)[0]
    assert _rel(core.calc_derivs(A, psi, 0.0)[0], ref) < RTOL
    A[n0 + 3] = np.inf
    try:
        dA = core.calc_derivs(A, psi, 0.0)[0]
    except capi.MctdhError:
        return
    assert not np.isfinite(dA).all()
