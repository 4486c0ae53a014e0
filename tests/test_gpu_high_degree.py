"""Nodes whose support is longer than one chunk of the staged node sums.

A small mesh sums 8 nodes to a block, whose support entries and boundary
facets are staged in shared memory 224 (3D) or 64 (2D) at a time.  A box mesh
never has more in a block; here a spindle of 300 tetrahedra around one edge
(both its ends hold all of them, and 300 facets each) and a fan of 300
triangles, with shuffled elements and corners, take several chunks, with nodes
that begin or end within one.  The rheology is elastic and the damping
continuous, so that the results are smooth in the inputs.
"""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu

N = 300


def _mesh(nd):
    from dynearthsol_gb300.mesh import BOUNDZ0, BOUNDZ1, Mesh, _boundary_products, boundary_normals
    rng = np.random.default_rng(nd)
    a = 2 * np.pi * np.arange(N) / N
    first = nd - 1                # the ring's nodes follow the axis or the centre
    ring, nxt = first + np.arange(N), first + (np.arange(N) + 1) % N
    if nd == 3:
        axis = [[0, 0, -1e4], [0, 0, 0]]
        xy = 1e4 * np.stack([np.cos(a), np.sin(a)], axis=1)
        coord = np.concatenate([axis, np.concatenate([xy, np.full((N, 1), -5e3)], axis=1)])
        conn = np.stack([np.zeros(N, int), np.ones(N, int), ring, nxt], axis=1)
        even = [(0, 1, 2, 3), (1, 2, 0, 3), (2, 0, 1, 3), (1, 0, 3, 2), (3, 2, 1, 0), (0, 3, 1, 2)]
        flag = np.full(N + 2, BOUNDZ0 | BOUNDZ1)
        flag[:2] = BOUNDZ0, BOUNDZ1
    else:
        coord = np.concatenate([[[0, -5e3]], np.stack([1e4 * np.cos(a), -5e3 + 5e3 * np.sin(a)], axis=1)])
        conn = np.stack([np.zeros(N, int), ring, nxt], axis=1)
        even = [(0, 1, 2), (1, 2, 0), (2, 0, 1)]
        flag = np.concatenate([[0], np.where(np.sin(a) < 0, BOUNDZ0, BOUNDZ1)])
    coord[:, 0] += 5e4
    pick = rng.integers(len(even), size=N)
    conn = np.stack([c[list(even[k])] for c, k in zip(conn, pick)])[rng.permutation(N)]
    conn, flag = np.ascontiguousarray(conn, np.int32), flag.astype(np.uint32)
    m = Mesh(nd, np.ascontiguousarray(coord, np.float64), conn, flag, *_boundary_products(nd, flag, conn),
             lengths=(1e5, 1e5 if nd == 3 else 0.0, 1e4), cells=(1, 1, 1))
    boundary_normals(m)
    return m


def _workload(nd):
    from dataclasses import replace
    from dynearthsol_gb300 import capi
    from dynearthsol_gb300.config import WeakZone, make_workload
    wl = make_workload("c1_3d_evp" if nd == 3 else "c0_2d_ep", cells=(2,) * nd)
    wl.mesh, wl.weakzone = _mesh(nd), WeakZone(option=0)
    wl.mat = replace(wl.mat, rheol_type=capi.RH_ELASTIC)
    wl.params = replace(wl.params, damping_option=2)
    return wl


def _model(wl, prec, noise=True):
    """A model and a state with velocities and deviatoric stresses."""
    from dynearthsol_gb300.config import initial_state
    from dynearthsol_gb300.solver import DeviceModel
    st, cp = initial_state(wl)
    m = DeviceModel(wl, comp_pressure=cp, precision=prec)
    st = m.init_fields(st)
    clk = m.clock()
    rng = np.random.default_rng(9)
    st["vel"] += 1e-9 * rng.standard_normal(st["vel"].shape)
    st["stress"] += 1e7 * rng.standard_normal(st["stress"].shape)
    st["dpressure"] += 1e6 * rng.standard_normal(st["dpressure"].shape)
    st["strain_rate"] += 1e-14 * rng.standard_normal(st["strain_rate"].shape)
    m.upload(st, clk)
    return m, st, clk, cp


def _nodal(wl, terms):
    """The elements' terms added to their nodes one after the other in element order."""
    out = np.zeros(wl.mesh.nnode)
    np.add.at(out, wl.mesh.connectivity.ravel(), np.repeat(terms, wl.mesh.ndims + 1))
    return out


@pytest.mark.parametrize("nd", [2, 3])
def test_fp64_sums_have_the_bits_of_the_serial_order(nd):
    from dynearthsol_gb300 import capi
    wl = _workload(nd)
    m, st, clk, _ = _model(wl, capi.PREC_FP64)
    np.testing.assert_array_equal(st["volume_n"], _nodal(wl, st["volume"]))
    tr = st["strain_rate"][:, 0] + st["strain_rate"][:, 1]
    if nd == 3:
        tr = tr + st["strain_rate"][:, 2]
    m.call("compute_dvoldt")
    np.testing.assert_array_equal(m.download_fields(["ntmp"])["ntmp"],
                                  _nodal(wl, tr * st["volume"]) / st["volume_n"])
    m.call("NMD_stress")
    np.testing.assert_array_equal(m.download_fields(["ntmp"])["ntmp"],
                                  _nodal(wl, st["dpressure"] * st["volume"]) / st["volume_n"])


@pytest.mark.parametrize("nd", [2, 3])
def test_fp64_steps_agree_with_the_oracle(nd):
    """Three chained steps; 1e-9 is the FP64 path's stated bound after a thousand."""
    from dynearthsol_gb300 import capi
    from oracle.oracle import Oracle, state_copy
    wl = _workload(nd)
    m, st, clk, cp = _model(wl, capi.PREC_FP64)
    o = Oracle(wl, state_copy(st), cp, clock=clk)
    m.step(3)
    assert o.run(3) == 0
    out = m.download()
    for k in ("coord", "vel", "force", "temperature", "mass", "tmass", "volume_n", "stress", "strain", "ntmp"):
        assert rel_err(out[k], o.st[k]) <= 1e-9, k


def test_mixed_sums_agree_with_fp64():
    """The double-word sums: a term's split (2^-48) and a compensated sum (2^-44) of each magnitude."""
    from dynearthsol_gb300 import capi
    wl = _workload(3)
    out = {}
    for prec in (capi.PREC_FP64, capi.PREC_MIXED):
        m, st, _, _ = _model(wl, prec)
        m.call("update_force")
        m.call("NMD_stress")
        out[prec] = m.download()
        m.step(2)
        out[prec]["T2"] = m.download()["temperature"] - st["temperature"]
    a, b = out[capi.PREC_FP64], out[capi.PREC_MIXED]
    vol, conn = a["volume"], wl.mesh.connectivity
    shp = np.stack([np.abs(a[k]) for k in ("shpdx", "shpdy", "shpdz")], axis=2).max(axis=2)
    mag = np.zeros(wl.mesh.nnode)   # bounds the sum of the terms' magnitudes
    s = 3 * np.abs(st["stress"]).max(axis=1) * vol
    np.add.at(mag, conn, s[:, None] * shp + (1e4 * vol)[:, None])
    assert np.all(np.abs(b["force"] - a["force"]) <= 1e-11 * mag[:, None])
    dp = _nodal(wl, np.abs(st["dpressure"]) * vol) / a["volume_n"]
    assert np.all(np.abs(b["ntmp"] - a["ntmp"]) <= 1e-11 * dp)
    for k in ("volume_n", "mass"):
        assert rel_err(b[k], a[k]) <= 1e-11, k
    # the heat terms are FP32 values
    assert np.abs(a["T2"]).max() > 0
    assert rel_err(b["T2"], a["T2"]) <= 1e-4


def test_reverse_step_agrees_with_differences():
    from dynearthsol_gb300 import capi
    from dynearthsol_gb300.adjoint import Window, adjoint_dot, central_fd
    wl = _workload(3)
    m, _, clk, _ = _model(wl, capi.PREC_FP64)
    win = Window(m, m.download(), clk, 2, 1)
    rng = np.random.default_rng(4)
    fields = ("coord", "vel", "temperature", "stress")
    seed = {k: rng.standard_normal(v.shape) / np.abs(v).max() for k, v in win.run().items() if k in fields}
    start, grad = win.gradients(seed)
    for k in fields:
        d = {k: 1e-6 * rng.standard_normal(win.start[k].shape) * (1e4 if k == "coord" else np.abs(win.start[k]).max())}
        ad, fd = adjoint_dot(start, grad, d, None), central_fd(win, seed, d, None)
        assert abs(ad - fd) <= 1e-5 * max(abs(ad), abs(fd)), (k, ad, fd)
