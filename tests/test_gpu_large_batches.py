"""Batches large enough for the tcgen05 form of the FP64 mode products (128 fibres a
tile, eight, twelve or sixteen outputs) through one EOM evaluation against the oracle:
SPF counts and fibre numbers that leave remainders in every direction, and operands
outside the exponent range of the digits, which its threads multiply in FP64.

Tolerance: the EOM parity of the FP64 path, 1e-11 relative (the digit products round
below FP64's own rounding); scaling A by a power of two scales dA exactly up to FP64
rounding; the SPF derivatives 1e-10, their solve with phi^H phi takes a digit.
"""
import numpy as np
import pytest

from macaw_gb300.generate import qvc
from oracle.mctdh import Oracle
from tests.helpers import random_state
from tests.test_gpu_parity import _rel

pytestmark = pytest.mark.gpu

SIZES = [(6, 7, 8, 8, 6, 6), (8, 8, 8, 8, 8, 5), (9, 12, 10, 11, 9), (13, 14, 5, 16, 8)]


def _model(sizes):
    n = len(sizes)
    m = qvc(2, n, 18, 4, 2, 11, (200.0, 3500.0), (0.05, 0.2), (0.0, 0.4), "large", dofs_per_mode=1)
    m.nspf = np.array([[k, k if i else k - 1] for i, k in enumerate(sizes)])
    return m.finalize()


@pytest.mark.parametrize("precision", [0, 2])
@pytest.mark.parametrize("sizes", SIZES)
def test_eom(sizes, precision):
    from macaw_gb300.capi import GpuCore
    model = _model(sizes)
    A, psi = random_state(model, seed=sum(sizes))
    ref = Oracle(model).calc_derivs(A, psi, 0.0)
    dA, dpsi = GpuCore(model, precision=precision).calc_derivs(A, psi, 0.0)
    assert _rel(dA, ref[0]) < 1e-11
    assert _rel(dpsi, ref[1]) < 1e-10


@pytest.mark.parametrize("power", [-430, 430])
def test_scaled_coefficients(power):
    from macaw_gb300.capi import GpuCore
    model = _model(SIZES[0])
    A, psi = random_state(model, seed=3)
    core = GpuCore(model)
    dA = core.calc_derivs(A, psi, 0.0)[0]
    scaled = core.calc_derivs(np.ldexp(1.0, power) * A, psi, 0.0)[0]
    assert _rel(scaled * np.ldexp(1.0, -power), dA) < 1e-13
