"""The shapes that a kernel takes by mesh size give the same bits.

A mesh of more than one wave of the GPU sums its nodes by a walk over the
support lists and collects the mixed step's FP64 branches per block; a small
mesh stages the entries in shared memory and runs the FP64 branches in place.
The slab-pipelined host step launches the same kernels on slabs of the same
mesh, small enough for the other shape: three chained steps on the whole mesh
against three pipelined calls, every field and the clock, on meshes just above
the lines (elements and nodes of odd counts per block) whose band is at the
Mohr-Coulomb surface, with softening and per-element cohesions.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _workload(name):
    from dataclasses import replace
    from dynearthsol_gb300 import capi
    from dynearthsol_gb300.config import make_workload, weak_band
    if name == "2d":
        return make_workload("c0_2d_ep", cells=(240, 163))
    wl = make_workload("c1_3d_evp", cells=(64, 31, 29))
    if name == "band":
        return weak_band(wl)
    # one weak material, the cohesion per element
    wl.mat = replace(wl.mat, cohesion0=(1e6,), cohesion1=(1e5,), friction_angle0=(10.0,), friction_angle1=(5.0,))
    noise = 1 + 0.05 * np.random.default_rng(3).standard_normal(wl.mesh.nelem)
    wl.elem_fields = {capi.EF_COHESION0: 1e6 * noise, capi.EF_COHESION1: 1e5 * noise}
    return wl


@pytest.mark.parametrize("name,prec", [("2d", "fp64"), ("band", "fp64"), ("band", "mixed"), ("noise", "mixed")])
def test_whole_mesh_and_slabs_give_the_same_bits(name, prec):
    from dynearthsol_gb300 import capi
    from dynearthsol_gb300.config import initial_state
    from dynearthsol_gb300.solver import DeviceModel
    from test_gpu_pipelined_step import _pinned
    precision = capi.PREC_FP64 if prec == "fp64" else capi.PREC_MIXED
    wl = _workload(name)
    st0, cp = initial_state(wl)
    rng = np.random.default_rng(1)
    if name != "2d":
        p = -st0["stress"][:, 2]
        st0["stress"][:, 0] += (0.295 + 0.01 * rng.uniform(-1, 1, p.size)) * p + 8.5e5
        st0["plstrain"] += np.where(rng.uniform(size=p.size) < 0.5, 0.02 * rng.uniform(size=p.size), 0.0)
    ref = DeviceModel(wl, comp_pressure=cp, precision=precision)
    init = ref.init_fields(st0)
    clk = (0.0, ref.clock()[1], 8)   # dt is recomputed after the second step
    ref.upload({k: v.copy() for k, v in init.items()}, clk)
    ref.step(3)
    want = ref.download()
    if name != "2d":
        assert np.count_nonzero(want["plstrain"] != init["plstrain"]) > 100
    m = DeviceModel(wl, comp_pressure=cp, precision=precision)
    st, keep = _pinned(init)
    c, n0 = clk, m.launches()
    for _ in range(3):
        c = m.step_host(st, 1, c)
    assert m.launches() - n0 > 3 * 33   # the pipelined path
    assert c == ref.clock()
    for k in want:
        np.testing.assert_array_equal(st[k], want[k], err_msg=k)
