"""The force of des_update_force against NumPy's FP64 sums of the element terms.

The FP64 terms are formed a thread per (element, node slot) on a mesh of at
most a quarter of a wave's elements and a thread per element beyond: the
smallest meshes, odd sizes, and one on either side of that line (77,824
elements), in 2D and 3D.  The force with a random stress less the force with
none is the sum of -(sigma . dN/dx) vol: everything else that the entry point
adds does not depend on the stress.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,cells", [("c0_2d_ep", (1, 1)), ("c0_2d_ep", (7, 5)), ("c0_2d_ep", (256, 152)),
                                        ("c0_2d_ep", (256, 153)), ("c1_3d_evp", (1, 1, 1)), ("c1_3d_evp", (5, 3, 3)),
                                        ("c1_3d_evp", (32, 16, 25)), ("c1_3d_evp", (32, 16, 26))])
def test_force_terms(name, cells):
    from dynearthsol_gb300 import capi
    from dynearthsol_gb300.config import initial_state, make_workload
    from dynearthsol_gb300.solver import DeviceModel
    wl = make_workload(name, cells=cells)
    st, cp = initial_state(wl)
    m = DeviceModel(wl, comp_pressure=cp, precision=capi.PREC_FP64)
    m.set_params(damping_option=0)
    st = m.init_fields(st)
    clk = m.clock()

    def force(stress):
        m.upload(dict(st, stress=stress), clk)
        m.call("update_force")
        return m.download_fields(["force"])["force"]

    f0 = force(np.zeros_like(st["stress"]))
    s = 1e8 * np.random.default_rng(5).standard_normal(st["stress"].shape)
    got = force(s) - f0
    nd = wl.mesh.ndims
    voigt = [[0, 2], [2, 1]] if nd == 2 else [[0, 3, 4], [3, 1, 5], [4, 5, 2]]
    shp = [st["shpdx"], st["shpdz"]] if nd == 2 else [st["shpdx"], st["shpdy"], st["shpdz"]]
    conn = np.asarray(wl.mesh.connectivity).reshape(-1, nd + 1)
    want, mag = np.zeros_like(got), np.abs(f0)
    for d in range(nd):
        for k in range(nd):
            t = -s[:, voigt[d][k], None] * shp[k] * st["volume"][:, None]
            np.add.at(want[:, d], conn, t)
            np.add.at(mag[:, d], conn, np.abs(t))
    # up to ~100 roundings of partial sums that mag bounds
    assert np.all(np.abs(got - want) <= 100 * np.finfo(float).eps * mag + np.finfo(float).tiny)
