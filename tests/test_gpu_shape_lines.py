"""Both shapes of the node sums and of the FP64 force terms at their lines.

Meshes just beyond the line at which an FP64 launch walks its support lists,
against their slabs, which stage them: three chained steps and three pipelined
calls, every field and the clock bit for bit.  The force terms with a thread
per (element, slot) and a thread per element, on either side of 14,592
elements, against NumPy.
"""
import numpy as np
import pytest

from test_gpu_force_terms import test_force_terms as _force_terms

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,cells", [("c0_2d_ep", (300, 41)), ("c1_3d_evp", (32, 17, 19))])
def test_walk_and_staged_give_the_same_bits(name, cells):
    from dynearthsol_gb300.config import initial_state, make_workload
    from dynearthsol_gb300.solver import DeviceModel
    from test_gpu_pipelined_step import _pinned
    wl = make_workload(name, cells=cells)
    st0, cp = initial_state(wl)
    st0["stress"] += 1e6 * np.random.default_rng(2).standard_normal(st0["stress"].shape)
    ref = DeviceModel(wl, comp_pressure=cp)
    init = ref.init_fields(st0)
    clk = (0.0, ref.clock()[1], 8)   # dt is recomputed after the second step
    ref.upload({k: v.copy() for k, v in init.items()}, clk)
    ref.step(3)
    want = ref.download()
    m = DeviceModel(wl, comp_pressure=cp)
    st, keep = _pinned(init)
    c, n0 = clk, m.launches()
    for _ in range(3):
        c = m.step_host(st, 1, c)
    assert m.launches() - n0 > 3 * 33   # the pipelined path
    assert c == ref.clock()
    for k in want:
        np.testing.assert_array_equal(st[k], want[k], err_msg=k)


@pytest.mark.parametrize("name,cells", [("c0_2d_ep", (152, 48)), ("c0_2d_ep", (152, 49)),
                                        ("c1_3d_evp", (16, 8, 19)), ("c1_3d_evp", (17, 11, 13))])
def test_force_terms_at_the_split(name, cells):
    _force_terms(name, cells)
