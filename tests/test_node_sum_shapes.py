"""The shape that a launch's node sums and force terms take by its size (no GPU:
tests/fake_cudart.c).  A staged node sum has blocks of 192 threads, a walk 64
or 128.  The sizes lie on either side of the lines at which the two shapes take
the same time."""
import pytest

import fake_runtime


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return fake_runtime.load(str(tmp_path_factory.mktemp("fake")))


@pytest.mark.parametrize("name,cells,prec,staged,split", [
    ("c0_2d_ep", (200, 20), "fp64", True, True),        # 8,000 triangles, 4,221 nodes
    ("c0_2d_ep", (200, 40), "fp64", True, False),       # 16,000, 8,241
    ("c0_2d_ep", (240, 50), "fp64", False, False),      # 24,000, 12,291: staged 18 % slower
    ("c0_2d_ep", (400, 90), "fp64", False, False),      # 72,000, 36,491: staged 36 % slower than unstaged
    ("c1_3d_evp", (20, 20, 6), "fp64", True, True),     # 14,400 tets, 3,087 nodes
    ("c1_3d_evp", (28, 28, 9), "fp64", True, False),    # 42,336, 8,410
    ("c1_3d_evp", (32, 32, 12), "fp64", False, False),  # 73,728, 14,157
    ("c1_3d_evp", (32, 32, 12), "mixed", True, None),
    ("c1_3d_evp", (48, 48, 12), "mixed", False, None)])  # 165,888, 31,213
def test_shape_by_size(lib, name, cells, prec, staged, split):
    from dynearthsol_gb300 import capi
    from dynearthsol_gb300.config import initial_state, make_workload
    from dynearthsol_gb300.solver import DeviceModel
    wl = make_workload(name, cells=cells)
    nd = wl.mesh.ndims
    with fake_runtime.installed(lib):
        st, cp = initial_state(wl)
        m = DeviceModel(wl, comp_pressure=cp, precision=capi.PREC_FP64 if prec == "fp64" else capi.PREC_MIXED)
        m.upload(st, (0.0, 1.0, 0))
        lib.fake_reset()
        m.step(2)
        for kernel in (b"k_node_pass", b"k_nmd_gather", b"k_force", b"k_mass_sum"):
            assert (lib.fake_block_of(kernel) == 192) == staged, kernel
        if split is not None:   # k_elem_force<nd, true, true, false, SPLIT>
            on, off = (lib.fake_block_of(b"k_elem_forceILi%dELb1ELb1ELb0ELb%dE" % (nd, k)) for k in (1, 0))
            assert (on > 0, off > 0) == (split, not split)
        if prec == "mixed":   # its heat terms are costlier: staged up to 38,912 nodes
            m.call("update_temperature")
            assert lib.fake_block_of(b"k_heat_gather_mixed3") == 192
        m.close()


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_entry_points_launch_their_own_kernels(lib, prec):
    """A copy and compute_dt's terms are not the geometry pass; the light updates have blocks of 256."""
    from dynearthsol_gb300 import capi
    from dynearthsol_gb300.config import initial_state, make_workload
    from dynearthsol_gb300.solver import DeviceModel
    wl = make_workload("c1_3d_evp", cells=(32, 32, 12))
    with fake_runtime.installed(lib):
        st, cp = initial_state(wl)
        m = DeviceModel(wl, comp_pressure=cp, precision=capi.PREC_FP64 if prec == "fp64" else capi.PREC_MIXED)
        m.upload(st, (0.0, 1.0, 0))
        lib.fake_reset()
        m.call("swap_volume")
        m.call("compute_dt")
        assert lib.fake_block_of(b"k_geometry") == 0
        for name, kernel in (("update_velocity", b"k_velocity"), ("apply_vbcs", b"k_vbcs"),
                             ("update_coordinate", b"k_coordinate")):
            m.call(name)
            assert lib.fake_block_of(kernel) == 256, kernel
        m.close()


def test_layout_conversions_have_blocks_of_256(lib):
    from dynearthsol_gb300.config import initial_state, make_workload
    from dynearthsol_gb300.solver import DeviceModel
    wl = make_workload("c0_2d_ep", cells=(60, 10))
    with fake_runtime.installed(lib):
        st, cp = initial_state(wl)
        m = DeviceModel(wl, comp_pressure=cp)
        m.upload(st, (0.0, 1.0, 0))
        m.download()
        assert lib.fake_block_of(b"k_aos_to_soa") == lib.fake_block_of(b"k_soa_to_aos") == 256
        m.close()
