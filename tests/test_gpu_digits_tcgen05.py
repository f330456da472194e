"""The tcgen05 form of the FP64-accurate mode products (batches of two tiles per CTA and
more) at all its instantiations: fibres and matrices outside the exponent range of the
digits, which it multiplies in FP64, and no wait for an MMA that ran out.  That these
sizes reach it is checked on the CPU (test_tensor_core_settings).

Scaling all coefficients of the state, or of the Hamiltonian, by a power of two scales
dA exactly, up to FP64 rounding (1e-13, as in test_gpu_large_batches).
"""
import numpy as np
import pytest

from tests.helpers import random_state
from tests.test_gpu_large_batches import SIZES, _model
from tests.test_gpu_parity import _rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", SIZES)
def test_outside_the_exponent_range(sizes):
    from macaw_gb300.capi import GpuCore, tensor_core_status
    model = _model(sizes)
    A, psi = random_state(model, seed=3)
    core = GpuCore(model)
    dA = core.calc_derivs(A, psi, 0.0)[0]
    for power in (-430, 430):
        scaled = core.calc_derivs(np.ldexp(1.0, power) * A, psi, 0.0)[0]
        assert _rel(scaled * np.ldexp(1.0, -power), dA) < 1e-13
    core.close()
    for power in (-430, 430):    # the pre-summed one-mode operators leave the range
        strong = _model(sizes)
        for t in strong.terms:
            t.coeff = t.coeff * np.ldexp(1.0, power)
        strong.finalize()
        core = GpuCore(strong)
        scaled = core.calc_derivs(A, psi, 0.0)[0]
        assert _rel(scaled * np.ldexp(1.0, -power), dA) < 1e-13
        core.close()
    assert tensor_core_status()["timeouts"] == 0
