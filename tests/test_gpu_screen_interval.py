"""Softening intervals that are empty or inverted, on a large mixed mesh.

pls1 <= pls0 drops the strength to the saturated values at once.  A mesh of
more than one wave screens its elements with FP32 material terms; the slabs of
the pipelined host step are small enough for the form that reads the FP64
properties.  With stresses between the start and the saturated yield surface,
three chained steps on the whole mesh and three pipelined calls give the same
bits, and the elements yield.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("l0,l1", [(0.0, 0.0), (0.02, 0.02), (0.02, 0.01)])
@pytest.mark.parametrize("markers", [False, True])
def test_empty_softening_interval(l0, l1, markers):
    from dataclasses import replace
    from dynearthsol_gb300 import capi
    from dynearthsol_gb300.config import initial_state, make_workload, weak_band
    from dynearthsol_gb300.solver import DeviceModel
    from test_gpu_pipelined_step import _pinned
    wl = make_workload("c1_3d_evp", cells=(64, 31, 29))
    if markers:
        wl = weak_band(wl)
        wl.mat = replace(wl.mat, pls0=(0.0, l0), pls1=(0.1, l1))
        weak = wl.mat.elemmarkers[:, 1] > 0
    else:
        wl.mat = replace(wl.mat, cohesion0=(1e6,), cohesion1=(1e5,), friction_angle0=(10.0,),
                         friction_angle1=(5.0,), pls0=(l0,), pls1=(l1,))
        weak = np.ones(wl.mesh.nelem, bool)
    st0, cp = initial_state(wl)
    ref = DeviceModel(wl, comp_pressure=cp, precision=capi.PREC_MIXED)
    p = -st0["stress"][:, 2]
    st0["stress"][:, 0] += np.where(weak, 0.22 * p + 3e5, 0.0)
    st0["plstrain"][:] = l0
    init = ref.init_fields(st0)
    clk = (0.0, ref.clock()[1], 8)
    ref.upload({k: v.copy() for k, v in init.items()}, clk)
    ref.step(3)
    want = ref.download()
    assert np.count_nonzero(want["plstrain"] != init["plstrain"]) > 100
    m = DeviceModel(wl, comp_pressure=cp, precision=capi.PREC_MIXED)
    st, keep = _pinned(init)
    c, n0 = clk, m.launches()
    for _ in range(3):
        c = m.step_host(st, 1, c)
    assert m.launches() - n0 > 3 * 33   # the pipelined path
    assert c == ref.clock()
    for k in want:
        np.testing.assert_array_equal(st[k], want[k], err_msg=k)
