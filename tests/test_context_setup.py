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


# bytes of device memory per element, facets and nodes of these meshes
# included: the state, the topology and one block of step scratch
@pytest.mark.parametrize("name,cells,prec,most", [("c0_2d_ep", (120, 60), "fp64", 341),
                                                  ("c1_3d_evp", (24, 20, 18), "fp64", 484),
                                                  ("c1_3d_evp", (24, 20, 18), "mixed", 744)])
def test_device_memory_of_a_context(lib, name, cells, prec, most):
    from dynearthsol_gb300 import capi
    from dynearthsol_gb300.config import make_workload
    from dynearthsol_gb300.solver import DeviceModel
    wl = make_workload(name, cells=cells)
    with fake_runtime.installed(lib):
        m = DeviceModel(wl, precision=capi.PREC_FP64 if prec == "fp64" else capi.PREC_MIXED)
        assert lib.fake_allocated() / wl.mesh.nelem <= most
        m.close()


@pytest.mark.parametrize("room", [False, True])
def test_host_step_without_room_for_the_pipeline(lib, room):
    """The pipelined host step's own buffers do not fit: the general path."""
    from dynearthsol_gb300.config import initial_state, make_workload
    from dynearthsol_gb300.solver import DeviceModel
    wl = make_workload("c1_3d_evp", cells=(16, 6, 4))
    with fake_runtime.installed(lib):
        st, cp = initial_state(wl)
        m = DeviceModel(wl, comp_pressure=cp)
        lib.fake_pinned(1)
        m.upload(st, (0.0, 1.0, 0))
        if not room:
            lib.fake_malloc_limit(0)
        before = lib.fake_allocated()
        for _ in range(2):
            m.step_host(st, 1, (0.0, 1.0, 0))
        assert (lib.fake_allocated() > before) == room
        m.close()
