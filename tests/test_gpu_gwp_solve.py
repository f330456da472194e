"""The Gaussian parameter equations at the sizes where the solve's panels, tiles and
back-substitution blocks end: C x = Y of n_gaussians * n_dofs unknowns per state.

The tolerance follows from the state's condition: the oracle's own change when its
inputs move by one unit in the last place, times 1000 (the number of roundings of the
eliminations at these sizes adds up to a few hundred such moves), at least 1e-12.
"""
import numpy as np
import pytest

from macaw_gb300.generate import gmctdh16
from oracle.mctdh import Oracle
from tests.helpers import random_state

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


# unknowns: 1 (one pivot), 7 | 8 | 9 (panel), 15 | 16 (MMA rows), 30 | 32 | 33 (tile, warp), 65, 128
@pytest.mark.parametrize("ngwp, dofs", [(1, 1), (1, 7), (2, 4), (3, 3), (3, 5), (4, 4), (6, 5), (4, 8), (11, 3), (13, 5),
                                        (32, 4)])
def test_parameter_solve_sizes(ngwp, dofs):
    from macaw_gb300.capi import GpuCore
    model = gmctdh16(ngwp=ngwp, gwp_dofs=dofs, dvr_grid=6, dvr_nspf=3)
    A, psi = random_state(model, seed=11, gwp_shift=0.5)
    rng = np.random.default_rng(0)
    ulp = np.finfo(float).eps
    ref = Oracle(model).calc_derivs(A, psi, 0.0)
    moved = Oracle(model).calc_derivs(A * (1 + ulp * rng.standard_normal(A.size)),
                                      psi * (1 + ulp * rng.standard_normal(psi.size)), 0.0)
    dA, dpsi = GpuCore(model).calc_derivs(A, psi, 0.0)
    assert _rel(dA, ref[0]) < max(1e-12, 1e3 * _rel(moved[0], ref[0]))
    m = model.modes_gwp[0]
    for s in range(model.nstates):
        o = int(model.ipsispf[m, s])
        b = slice(o, o + ngwp * dofs)
        assert _rel(dpsi[b], ref[1][b]) < max(1e-12, 1e3 * _rel(moved[1][b], ref[1][b]))
