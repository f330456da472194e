"""The tensor-core settings choose the kernels of the calls made after them, also where
an EOM evaluation is replayed from a graph; MACAW_GB300_TC=0 keeps every tcgen05 kernel
out; FP64-accurate mode products of two tiles per CTA and more take its digit kernel.  On the stand-in runtime, by the names of the launched kernels."""
import pytest

from macaw_gb300 import capi
from macaw_gb300.generate import gmctdh16, qvc
from tests import fake
from tests.helpers import random_state
from tests.test_gpu_large_batches import SIZES, _model as large


def _model(modes):
    return qvc(2, modes, 18, 8, 2, 5, (200.0, 3500.0), (0.05, 0.2), (0.0, 0.4), "settings", dofs_per_mode=1)


@pytest.mark.parametrize("modes", [3, 5])   # one graph; copies beside the operators
def test_settings_reach_replayed_calls(tmp_path, monkeypatch, modes):
    rt = fake.use(monkeypatch, fake.fake_runtime(tmp_path))
    model = _model(modes)
    core = capi.GpuCore(model, precision=1)
    A, psi = random_state(model)
    for min_n, name in ((17, "prod_kernel"), (4, "prod_tc_kernel"), (17, "prod_kernel")):
        capi.tensor_core_config(min_n=min_n)
        for _ in range(3):
            core.calc_derivs(A, psi)
            launched = [k for k in rt.kernels() if "prod" in k]
            assert launched and all(name in k for k in launched)


# 262,144 coefficients and fewer than 152 x 8 tiles
@pytest.mark.parametrize("value, modes, digits", [("1", 6, True), ("0", 6, False), ("1", 3, False)])
def test_switch_covers_the_digit_products(tmp_path, monkeypatch, value, modes, digits):
    monkeypatch.setenv("MACAW_GB300_TC", value)
    rt = fake.use(monkeypatch, fake.fake_runtime(tmp_path))
    model = _model(modes)
    core = capi.GpuCore(model)
    A, psi = random_state(model)
    core.calc_derivs(A, psi)
    assert any("prod_digits_kernel" in k for k in rt.kernels()) == digits
    assert capi.tensor_core_status()["enabled"] == int(value)


# the sizes of test_gpu_large_batches, whose first products fill two tiles per CTA
@pytest.mark.parametrize("sizes, form", list(zip(SIZES, "2234")))
def test_large_batches_take_the_digit_kernel(tmp_path, monkeypatch, sizes, form):
    rt = fake.use(monkeypatch, fake.fake_runtime(tmp_path))
    model = large(sizes)
    core = capi.GpuCore(model)
    core.calc_derivs(*random_state(model))
    products = [k for k in rt.kernels() if "prod_" in k]
    assert f"prod_digits_kernelILi{form}E" in products[0]


# 65,536 fibres of a Gaussian mode for each of two states: S^-1 A, then dA -= tau A
def test_accumulating_batches_do_not(tmp_path, monkeypatch):
    rt = fake.use(monkeypatch, fake.fake_runtime(tmp_path))
    model = gmctdh16(ngwp=16, gwp_dofs=2, dvr_grid=18, dvr_nspf=16)
    core = capi.GpuCore(model)
    core.calc_derivs(*random_state(model))
    products = [k for k in rt.kernels() if "prod_" in k]
    assert all("prod_digits_kernelILi4E" in k for k in products[:-1])
    assert "prod_fx_kernelILi4E" in products[-1]
