"""A kernel launch that the runtime refuses makes the call that issued it fail with the
CUDA status, whether the launch is issued directly, captured or replayed; the context
works again afterwards.  On the stand-in runtime, which refuses launches by name."""
import numpy as np
import pytest

from macaw_gb300 import capi
from macaw_gb300.generate import ensemble_member
from macaw_gb300.model import INT_CMF2
from tests import fake
from tests.helpers import random_state, small_lvc, small_qvc

ECUDA = -6


@pytest.fixture(scope="module")
def library(tmp_path_factory):
    return fake.fake_runtime(tmp_path_factory.mktemp("fake"))


def _refused(rt, name, call):
    rt.lib.fake_fail(name.encode())
    try:
        with pytest.raises(capi.MctdhError) as e:
            call()
    finally:
        rt.lib.fake_fail(b"")
    return e.value.code


# calls before the failing one: it is issued directly, captured, replayed
@pytest.mark.parametrize("before", [0, 1])
@pytest.mark.parametrize("kernel", ["h1_kernel", "prod_fx", "hole_fx", "termsum", "reginv", "spf_drive8"])
def test_eom(library, monkeypatch, kernel, before):
    rt = fake.use(monkeypatch, library)
    model = small_lvc()
    core = capi.GpuCore(model)
    A, psi = random_state(model)
    for _ in range(before):
        core.calc_derivs(A, psi)
    assert _refused(rt, kernel, lambda: core.calc_derivs(A, psi)) == ECUDA
    rt.kernels()
    for _ in range(3):   # complete again, also what is captured from now on
        core.calc_derivs(A, psi)
        assert any(kernel in k for k in rt.kernels())


def test_other_entry_points(library, monkeypatch):
    rt = fake.use(monkeypatch, library)
    model = small_qvc(integrator=INT_CMF2)
    core = capi.GpuCore(model)
    A, psi = random_state(model)
    core.set_state(A, psi)
    assert _refused(rt, "natpop", core.natpop) == ECUDA
    assert _refused(rt, "prod_fx", lambda: core.observables(0.0)) == ECUDA
    assert _refused(rt, "lan_normalize", lambda: core.cmf2_attempt(A, psi, 0.0, 1.0)) == ECUDA
    ens = capi.Ensemble([ensemble_member(np.random.default_rng(1), i, 1 << 8) for i in range(2)], autotune=False)
    assert _refused(rt, "termsum", ens.calc_derivs) == ECUDA


def test_an_error_of_the_caller_stays_its_own(library, monkeypatch):
    rt = fake.use(monkeypatch, library)
    model = small_lvc()
    core = capi.GpuCore(model)
    A, psi = random_state(model)
    rt.lib.fake_pending(700)
    for _ in range(3):
        core.calc_derivs(A, psi)
    assert rt.lib.cudaPeekAtLastError() == 700
    assert _refused(rt, "termsum", lambda: core.observables(0.0)) == ECUDA
