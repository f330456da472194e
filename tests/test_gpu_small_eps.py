"""The 'poly' regularisation of rho with eps_rho far below FP32's range of squares: an
eigenvalue below eps is replaced by (eps + w^2 / eps) / 2, whatever eps is.

The state occupies two SPFs per mode with disjoint coefficients, so that the density
matrices are exactly diagonal, 1 and `weak`; the derivative of the weak SPF is
proportional to 1 / w_reg.  Tolerance: parity of the SPF derivatives, 1e-9 relative,
where the plain inverse is off by eps / (2 weak).
"""
import numpy as np
import pytest

from macaw_gb300.model import Model, OP_DQ2, Term
from oracle.mctdh import Oracle
from tests.helpers import random_state

pytestmark = pytest.mark.gpu


def _model():
    """Two anharmonic oscillators with a bilinear coupling, two SPFs each."""
    terms = [Term(0.01 + 0j, 0, 0, {0: 1, 1: 1})]
    for k in range(2):
        terms += [Term(-0.005 + 0j, 0, 0, {k: OP_DQ2}), Term(0.005 + 0j, 0, 0, {k: 2}), Term(0.001 + 0j, 0, 0, {k: 3})]
    return Model(nstates=1, mode_dofs=[[0], [1]], multiset=[True] * 2, nspf=np.full((2, 1), 2), dvr_type=["HO"] * 2,
                 ngp=[14] * 2, dvrpar=[(0.0, 1.0)] * 2, terms=terms, init_state=0, label="weak").finalize()


@pytest.mark.parametrize("eps, weak", [(1e-21, 1e-24), (1e-21, 1e-18), (1e-30, 1e-32), (1e-160, 1e-162)])
def test_small_eps(eps, weak):
    from macaw_gb300.capi import GpuCore
    model = _model()
    model.eps_rho = eps
    A, psi = random_state(model, seed=2)
    A = np.diag([1.0, np.sqrt(weak)]).astype(complex).reshape(-1, order="F")
    ref = Oracle(model).calc_derivs(A, psi, 0.0)[1]
    out = GpuCore(model).calc_derivs(A, psi, 0.0)[1]
    for m in range(2):
        o, G = int(model.ipsispf[m, 0]), model.ngpm[m]
        for j in range(2):
            b = slice(o + G * j, o + G * (j + 1))
            assert np.linalg.norm(out[b] - ref[b]) < 1e-9 * np.linalg.norm(ref[b])
