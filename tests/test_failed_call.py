"""A failed EOM evaluation leaves the caller's arrays as they were, for coefficient
vectors of any length (from 32768 on they are copied beside the evaluation).  On the
stand-in runtime, which puts the failure into the status word."""
import numpy as np
import pytest

from macaw_gb300 import capi
from macaw_gb300.generate import qvc
from tests import fake
from tests.helpers import random_state


@pytest.fixture(scope="module")
def library(tmp_path_factory):
    return fake.fake_runtime(tmp_path_factory.mktemp("fake"))


@pytest.mark.parametrize("status, code", [(1, -2), (2, -2), (4, -5), (8, -6)])
@pytest.mark.parametrize("modes", [3, 5])
def test_outputs_stay(library, monkeypatch, modes, status, code):
    rt = fake.use(monkeypatch, library)
    model = qvc(2, modes, 18, 8, 2, 5, (200.0, 3500.0), (0.05, 0.2), (0.0, 0.4), "failing", dofs_per_mode=1)
    A, psi = random_state(model)
    core = capi.GpuCore(model)
    dA, dpsi = np.full_like(A, 7.0), np.full_like(psi, 7.0)
    for _ in range(3):   # issued, captured, replayed
        rt.lib.fake_status(status)
        rc = core.lib.mctdh_calc_derivs(core.h, capi._ptr(A), capi._ptr(psi), capi._ptr(dA), capi._ptr(dpsi), 0.0)
        rt.lib.fake_status(0)
        assert rc == code
        assert (dA == 7.0).all() and (dpsi == 7.0).all()
    core.calc_derivs(A, psi)
