"""The reverse mode's forward window leaves the context as its steps do.

A taped step works on its tape records and the window's end brings the
context's arrays back from the last one.  A window of five steps between two
updates of dt is five steps: every field and the clock, bit for bit, whatever
the segments (one step each, with a rest, the whole window), and again after
the backward, which recomputes the untaped segments on the same arrays.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells,thermal", [((1, 1, 1), 1), ((3, 4, 3), 1), ((3, 4, 3), 0)])
@pytest.mark.parametrize("every", [1, 2, 5, 9])
def test_window_is_its_steps(cells, thermal, every):
    from dataclasses import replace
    from dynearthsol_gb300.config import initial_state, make_workload
    from dynearthsol_gb300.solver import DeviceModel
    wl = make_workload("c1_3d_evp", cells=cells)
    wl.params = replace(wl.params, damping_option=2, has_thermal_diffusion=thermal)
    st, cp = initial_state(wl)
    m = DeviceModel(wl, comp_pressure=cp)
    m.init_fields(st)
    m.step(4)
    start, clk = m.download(), m.clock()
    m.step(5)
    want, want_clk = m.download(), m.clock()
    m.upload({k: v.copy() for k, v in start.items()}, clk)
    m.adjoint_forward(5, every)
    got = m.download()
    assert m.clock() == want_clk
    for k in want:
        np.testing.assert_array_equal(got[k], want[k], err_msg=k)
    m.adjoint_backward({"vel": np.ones_like(want["vel"])})
    after = m.download()
    assert m.clock() == want_clk
    for k in want:
        np.testing.assert_array_equal(after[k], want[k], err_msg=k)
