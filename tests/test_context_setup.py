"""What a context's creation asks of the CUDA runtime (no GPU: tests/fake_cudart.c)."""
import pytest

import fake_runtime
from cases import build_case


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return fake_runtime.load(str(tmp_path_factory.mktemp("fake")))


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("name", ["2d_ep", "3d_evp", "3d_heat_jitter_multimat"])
def test_no_kernel_runs_before_the_uploads_have_arrived(lib, name, prec):
    from dynearthsol_gb300 import capi
    from dynearthsol_gb300.solver import DeviceModel
    wl, _ = build_case(name)
    with fake_runtime.installed(lib):
        m = DeviceModel(wl, precision=capi.PREC_FP64 if prec == "fp64" else capi.PREC_MIXED)
        assert lib.fake_launches() >= 2
        assert lib.fake_violations() == 0, lib.fake_first_violation().decode()
        m.close()
