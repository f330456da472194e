"""Context creation on a second device of one process: kernels that need more dynamic
shared memory than 48 KB are allowed it on every device, so that each launch of an EOM
evaluation is accepted there too.  On the stand-in runtime, which has two devices."""
import pytest

from macaw_gb300 import capi
from macaw_gb300.generate import ensemble_member, qvc
from tests import fake
from tests.helpers import random_state


@pytest.fixture(scope="module")
def library(tmp_path_factory):
    return fake.fake_runtime(tmp_path_factory.mktemp("fake"))


def _model(nspf, modes=3):
    return qvc(2, modes, 40, nspf, 2, 5, (200.0, 3500.0), (0.05, 0.2), (0.0, 0.4), "second device", dofs_per_mode=1)


# SPF derivatives of n <= 8 in one and (two DOFs) two launches, the wide contractions, products of
# more than 24 and the tcgen05 ones
@pytest.mark.parametrize("precision", [0, 1, 5])
@pytest.mark.parametrize("nspf, modes", [(4, 3), (12, 3), (30, 3), (8, 6), (11, 5), (14, 5)])
def test_same_launches_on_either_device(library, monkeypatch, nspf, modes, precision):
    rt = fake.use(monkeypatch, library)
    model = _model(nspf, modes)
    A, psi = random_state(model)
    seen = []
    for device in (0, 1):
        rt.lib.fake_device(device)
        core = capi.GpuCore(model, precision=precision)
        core.calc_derivs(A, psi)
        seen.append(rt.kernels())
        core.close()
    assert any("spf_" in k for k in seen[0])
    assert seen[1] == seen[0]


def test_ensemble_on_second_device(library, monkeypatch):
    import numpy as np
    rt = fake.use(monkeypatch, library)
    models = [ensemble_member(np.random.default_rng(1), i, 1 << 8) for i in range(3)]
    seen = []
    for device in (0, 1):
        rt.lib.fake_device(device)
        ens = capi.Ensemble(models, autotune=False)
        ens.calc_derivs()
        seen.append(rt.kernels())
        ens.close()
    assert seen[0] and seen[1] == seen[0]


def test_grids_follow_the_device(tmp_path, monkeypatch):
    """Two blocks a matrix where the device has two SMs for each, four where it has more."""
    rt = fake.use(monkeypatch, fake.fake_runtime(tmp_path))   # its own copy: SM counts are kept
    model = _model(4)                                         # 2 states x 3 modes
    rt.lib.fake_sms(1, 13)
    A, psi = random_state(model)
    for device, blocks in ((0, 4), (1, 2)):
        rt.lib.fake_device(device)
        core = capi.GpuCore(model)
        rt.launches()
        core.calc_derivs(A, psi)
        assert [x[1:] for x in rt.launches() if "reginv" in x[0]] == [(6, blocks)]
        core.close()
