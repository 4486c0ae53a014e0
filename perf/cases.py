"""Timed cases of the explicit step: what a program that uses this library has it do.

Four kinds of pass, each through the public entry points:

* ``advance``    a run segment of a device-resident model: the state of a
                 restart is uploaded, ``steps`` explicit steps run, and the
                 fields of an output frame come back to page-locked arrays
                 (DeviceModel.upload / step / download);
* ``host``       one des_step_host call on page-locked arrays that stay the
                 caller's (the drop-in form; the arrays are advanced in place);
* ``functions``  the reference's time loop through the per-function entry
                 points, device resident (DeviceModel.call);
* ``adjoint``    one iteration of an inversion: a taped window of ``steps``
                 steps, the misfit of the top-surface velocities, and the
                 reverse sweep to every parameter gradient (adjoint.Window).

Meshes, physics and sizes are the named workloads of
``dynearthsol_gb300.config.make_workload`` at their full or smaller cell
counts.  The start states are those of a run under way: the boundary
speeds' extension spread over the box, a linear geotherm, a lithostatic
stress with a horizontal extension that grows with depth, and smooth seeded
perturbations of a few per cent on all of them.  The mixed runs of several
steps take the continuous damping option 2: with the default option's
copysign any rounding difference grows by orders of magnitude within a few
dozen steps, in the reference's own FP64 step too, so that the results of
two correct runs could not be compared.
"""
from __future__ import annotations

import functools
import math
from dataclasses import replace

import numpy as np
import torch

from dynearthsol_gb300 import adjoint, capi
from dynearthsol_gb300.config import make_workload, weak_band
from dynearthsol_gb300.solver import DeviceModel

RHEOLOGY = {"elastic": capi.RH_ELASTIC, "maxwell": capi.RH_MAXWELL, "ep": capi.RH_EP, "evp": capi.RH_EVP}
PRECISION = {"fp64": capi.PREC_FP64, "mixed": capi.PREC_MIXED}
INPUTS = ("coord", "vel", "temperature", "volume_old", "stress", "strain", "plstrain")
FRAME = ("coord", "vel", "force", "temperature", "mass", "tmass", "volume", "stress", "strain", "strain_rate",
         "plstrain", "delta_plstrain", "dpressure", "edvoldt")
START = ("coord", "vel", "temperature", "stress", "plstrain", "volume_old")
LOOP = ("update_temperature", "update_strain_rate", "compute_dvoldt", "compute_edvoldt", "update_stress",
        "NMD_stress", "update_force", "update_velocity", "apply_vbcs", "update_mesh", "rotate_stress")
DEV = "cuda" if torch.cuda.is_available() else "cpu"


def _case(name, kind, mesh, cells, precision, steps, rheology="evp", damping=1, band=False, checkpoint=0):
    nx, ny, nz = cells
    return {"name": name, "kind": kind, "mesh": mesh, "nx": nx, "ny": ny, "nz": nz, "precision": precision,
            "steps": steps, "rheology": rheology, "damping": damping, "band": band, "checkpoint": checkpoint}


def listed():
    return [
        # the 2D workload at its full size: 8,000 triangles, where launches and latency count
        _case("ep2d_8k_fp64", "advance", "c0_2d_ep", (200, 0, 20), "fp64", 200, rheology="ep"),
        # the smallest meshes: a set-up check, a parameter study of tiny boxes
        _case("evp3d_648_fp64", "advance", "c1_3d_evp", (6, 6, 3), "fp64", 100),
        # a small yielding model: two materials, the band at the Mohr-Coulomb surface
        _case("band3d_14k_mixed", "advance", "c1_3d_evp", (20, 20, 6), "mixed", 100, damping=2, band=True),
        # the headline workload, mixed and FP64
        _case("evp3d_998k_mixed", "advance", "c1_3d_evp", (80, 80, 26), "mixed", 50, damping=2),
        _case("evp3d_998k_fp64", "advance", "c1_3d_evp", (80, 80, 26), "fp64", 20),
        # the same mesh with a yielding band of a second material
        _case("band3d_998k_mixed", "advance", "c1_3d_evp", (80, 80, 26), "mixed", 30, damping=2, band=True),
        # the largest workload: 7,987,200 tets, per-element cohesion
        _case("noise3d_8m_mixed", "advance", "c2_3d_evp_noise", (160, 160, 52), "mixed", 30, damping=2),
        # jittered nodes, permuted elements, odd cell counts: the gathers lose their locality
        _case("heat3d_1m_permuted_mixed", "advance", "c4_3d_heat_jitter", (127, 63, 21), "mixed", 30, damping=2),
        # a caller whose host arrays stay authoritative
        _case("host3d_998k_mixed", "host", "c1_3d_evp", (80, 80, 26), "mixed", 1),
        # the reference's own loop over the C ABI
        _case("functions3d_118k_fp64", "functions", "c1_3d_evp", (37, 41, 13), "fp64", 10),
        # an inversion's iteration: small with checkpoints, and at the headline size with the whole window taped
        _case("adjoint3d_14k", "adjoint", "c1_3d_evp", (20, 20, 6), "fp64", 50, damping=2, checkpoint=10),
        _case("adjoint3d_998k", "adjoint", "c1_3d_evp", (80, 80, 26), "fp64", 40, damping=2, checkpoint=40),
    ]


def draw(rng):
    """One more case of the same ranges: sizes from 500 to 4 million elements."""
    kind = rng.choices(("advance", "host", "functions", "adjoint"), (6, 1, 1, 2))[0]
    top = {"advance": 4.0e6, "host": 1.0e6, "functions": 3.0e5, "adjoint": 5.0e5}[kind]
    ne = math.exp(rng.uniform(math.log(500), math.log(top)))
    mesh, precision = "c1_3d_evp", rng.choice(("fp64", "mixed", "mixed"))
    rheology, band = rng.choice(("evp", "evp", "ep", "maxwell", "elastic")), False
    if kind == "adjoint":
        precision, rheology = "fp64", "evp"
    elif kind == "advance":
        mesh = rng.choice(("c0_2d_ep", "c1_3d_evp", "c1_3d_evp", "c2_3d_evp_noise", "c4_3d_heat_jitter"))
        band = mesh == "c1_3d_evp" and rheology in ("ep", "evp") and rng.random() < 0.4
    if mesh == "c0_2d_ep":
        ne, precision = min(ne, 4.0e5), "fp64"
        nz = max(2, round(math.sqrt(ne / 2 / rng.uniform(4, 12))))
        cells = (max(3, round(ne / 2 / nz)), 0, nz)
        rheology = "ep"
    else:
        nz = max(2, round((ne / 6 / rng.uniform(4, 12)) ** (1 / 3)))
        ny = max(2, round(math.sqrt(ne / 6 / nz / rng.uniform(0.7, 1.4))))
        cells = (max(3, round(ne / 6 / nz / ny)), ny, nz)
    steps = 1 if kind == "host" else int(min({"advance": 100, "functions": 20, "adjoint": 40}[kind],
                                             max(10, 4.0e7 / ne * rng.uniform(0.5, 1.0))))
    damping = 2 if kind == "adjoint" or (precision == "mixed" and steps > 1) else rng.choice((1, 1, 2))
    checkpoint = max(1, steps // rng.choice((1, 1, 4))) if kind == "adjoint" else 0
    case = _case("", kind, mesh, cells, precision, steps, rheology, damping, band, checkpoint)
    return {k: v for k, v in case.items() if k != "name"}


def _sizes(case):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if case["mesh"] == "c0_2d_ep":
        return 2, (nx + 1) * (nz + 1), 2 * nx * nz
    return 3, (nx + 1) * (ny + 1) * (nz + 1), 6 * nx * ny * nz


def work(case):
    """Bytes and operations of one pass.  A step reads and writes its state
    once: connectivity, stress, strain, plstrain and volume per element, the
    support lists, and coordinates, velocity, temperature and the boundary
    flag per node; around it the inputs come in and the frame goes out once.
    A reverse step reads its tape record and reads and writes the adjoint
    state.  Operations: the strain rate, heat stencil, rheology, force and
    geometry of an element, about a thousand in 3D."""
    nd, nn, ne = _sizes(case)
    nstr, npe = nd * (nd + 1) // 2, nd + 1
    step = ne * (8 * npe + 32 * nstr + 32) + nn * (32 * nd + 24)
    flops = ne * (1000 if nd == 3 else 400)
    moved = 8 * (ne * (2 * nstr + 2) + nn * (2 * nd + 1)) + 8 * (ne * (3 * nstr + 5) + nn * (3 * nd + 3))
    n = case["steps"]
    if case["kind"] == "host":
        moved = 8 * (ne * (2 * nstr + 3) + nn * (2 * nd + 2)) + 8 * (ne * (3 * nstr + 6 + nd * npe) + nn * (3 * nd + 5))
    if case["kind"] == "functions":
        moved += n * 8 * (ne * (2 * nstr + 3 * nd * npe) + nn * 3 * nd)   # what one call hands to the next
    if case["kind"] == "adjoint":
        tape = 8 * (ne * (18 + 12 + 7) + nn * 16)
        return {"bytes": n * (step + 2 * tape + 2 * 8 * (ne * 20 + nn * 10)) + moved, "flops": 4 * n * flops}
    return {"bytes": n * step + moved, "flops": n * flops}


# --------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------
@functools.lru_cache(maxsize=2)
def _mesh_workload(mesh, cells, permutation):
    wl = make_workload(mesh, cells=[c for c in cells if c], seed=permutation)
    conn = torch.from_numpy(wl.mesh.connectivity).to(DEV).long()
    return wl, conn


def _workload(case, seed):
    cells = (case["nx"], case["ny"], case["nz"])
    base, conn = _mesh_workload(case["mesh"], cells, seed % 5 if case["mesh"] == "c4_3d_heat_jitter" else 12345)
    wl = replace(base, params=replace(base.params, damping_option=case["damping"]),
                 mat=replace(base.mat, rheol_type=RHEOLOGY[case["rheology"]]), elem_fields=dict(base.elem_fields))
    ne = wl.mesh.nelem
    if case["mesh"] == "c2_3d_evp_noise":
        noise = 1 + 0.05 * np.random.default_rng(seed).standard_normal(ne)
        wl.elem_fields = {capi.EF_COHESION0: wl.mat.cohesion0[0] * noise, capi.EF_COHESION1: wl.mat.cohesion1[0] * noise}
    if case["band"]:
        wl = weak_band(wl)
    if case["kind"] == "adjoint":
        m = wl.mat
        wl.elem_fields = {capi.EF_LOG10_VISC: _log10_visc(wl, conn, seed),
                          capi.EF_SHEAR_MODULUS: np.full(ne, m.shear_modulus[0]),
                          capi.EF_COHESION0: np.full(ne, m.cohesion0[0]), capi.EF_COHESION1: np.full(ne, m.cohesion1[0]),
                          capi.EF_FRICTION0: np.full(ne, m.friction_angle0[0]),
                          capi.EF_FRICTION1: np.full(ne, m.friction_angle1[0])}
    return wl, conn


def _box(wl):
    """The box's side lengths in the order of the coordinates."""
    lx, ly, lz = wl.lengths
    return torch.tensor([lx, ly, lz] if wl.mesh.ndims == 3 else [lx, lz], dtype=torch.float64, device=DEV)


def _smooth(xi, rng, modes=4):
    """A sum of a few seeded plane waves over the unit box, of size about 1."""
    f = torch.zeros(xi.shape[0], dtype=torch.float64, device=xi.device)
    for _ in range(modes):
        k = torch.tensor(rng.uniform(0.5, 3.0, xi.shape[1]), device=xi.device)
        f += float(rng.uniform(0.3, 0.7)) * torch.cos(2 * math.pi * ((xi @ k) + float(rng.uniform())))
    return f


def _log10_visc(wl, conn, seed):
    x = torch.from_numpy(wl.mesh.coord).to(DEV)
    ctr = x[conn].mean(1) / _box(wl)
    return (21 + 0.4 * _smooth(ctr, np.random.default_rng(seed + 77))).cpu().numpy()


def _inputs(case, seed):
    """(workload, connectivity, start state in the reference's layout)."""
    wl, conn = _workload(case, seed)
    m, p, mt = wl.mesh, wl.params, wl.mat
    nd = m.ndims
    rng = np.random.default_rng(seed)
    x = torch.from_numpy(m.coord).to(DEV)
    box = _box(wl)
    xi, ctr = x / box, x[conn].mean(1)
    ci = ctr / box
    v0, v1 = p.vbc_values[0], p.vbc_values[1]
    vel = torch.zeros_like(x)
    vel[:, 0] = v0 + (v1 - v0) * xi[:, 0] + 0.05 * v1 * _smooth(xi, rng) * torch.sin(math.pi * xi[:, 0])
    vel[:, -1] = -(v1 - v0) * x[:, -1] / box[0] * 0.5 + 0.02 * v1 * _smooth(xi, rng)
    if nd == 3:
        vel[:, 1] = 0.02 * v1 * _smooth(xi, rng)
    bc = torch.from_numpy(m.bcflag.astype(np.int64)).to(DEV)
    vel[(bc & 1) != 0, 0] = v0
    vel[(bc & 2) != 0, 0] = v1
    T = wl.t_top + (wl.t_bottom - wl.t_top) * (-xi[:, -1]) + 5.0 * _smooth(xi, rng) * torch.sin(math.pi * -xi[:, -1])
    pr = mt.rho0[0] * p.gravity * -ctr[:, -1]
    # horizontal extension: a share of the lithostatic pressure that, in a weak band, reaches its yield surface
    d = ((0.295 + 0.01 * _smooth(ci, rng)) * pr + 8.5e5) if case["band"] else (0.10 + 0.01 * _smooth(ci, rng)) * pr
    nstr = nd * (nd + 1) // 2
    s = torch.zeros(m.nelem, nstr, dtype=torch.float64, device=DEV)
    s[:, :nd] = -pr[:, None]
    s[:, 0] += d
    if nd == 3:
        s[:, 1] += 0.02 * d   # the sides carry the reference pressure
    for c in range(nd, nstr):
        s[:, c] = 2e5 * _smooth(ci, rng)
    es = s / (3 * mt.bulk_modulus[0])
    pls = wl.weakzone.plstrain * ((ctr[:, 0] - 0.5 * box[0]).abs() < 1.5 * wl.resolution).double()
    if case["band"]:
        pls = pls + 0.02 * (1 + _smooth(ci, rng).clamp(-1, 1))
    back = 0.1 * wl.resolution / (p.max_vbc_val() * p.inertial_scaling)   # about the last step's dt
    st = {"coord": x, "vel": vel, "temperature": T, "volume_old": _volume(x - back * vel, conn), "stress": s, "strain": es,
          "plstrain": pls}
    return wl, conn, st


def _pinned(shape):
    a = torch.empty(shape, dtype=torch.float64, pin_memory=torch.cuda.is_available()).numpy()
    return a


def _to_pinned(t):
    a = _pinned(tuple(t.shape))
    torch.from_numpy(a).copy_(t)
    return a


def prepare(case, seed):
    wl, conn, st = _inputs(case, seed)
    m = wl.mesh
    nd, nn, ne = m.ndims, m.nnode, m.nelem
    comp = wl.mat.rho0[0] * wl.params.gravity * wl.lengths[2]
    model = DeviceModel(wl, comp_pressure=comp, precision=PRECISION[case["precision"]])
    start = {k: _to_pinned(v) for k, v in st.items()}
    model.upload(start)
    dt = model.call("compute_dt")
    state = {"case": case, "model": model, "start": start, "clock": (0.0, dt, 0)}
    if case["kind"] == "adjoint":
        state["window"] = adjoint.Window(model, start, (0.0, dt, 0), case["steps"], case["checkpoint"])
        state["top"] = adjoint.top_nodes(m)
        state["target"] = st["vel"].cpu().numpy() * 1.1
        return state
    if case["kind"] == "host":
        nstr, npe = nd * (nd + 1) // 2, nd + 1
        per_node = {"coord": nd, "coord0": nd, "vel": nd, "force": nd, "temperature": 0, "mass": 0, "tmass": 0,
                    "volume_n": 0, "ntmp": 0}
        per_elem = {"stress": nstr, "strain": nstr, "strain_rate": nstr, "shpdx": npe, "shpdy": npe, "shpdz": npe}
        full = {}
        for k in capi.STATE_ARRAYS:
            n, w = (nn, per_node[k]) if k in per_node else (ne, per_elem.get(k, 0))
            full[k] = _pinned((n, w) if w else (n,))
        full["shpdy"][:] = 0
        state["host"] = model.download(full)
        return state
    width = {"coord": nd, "vel": nd, "force": nd, **dict.fromkeys(("stress", "strain", "strain_rate"), nd * (nd + 1) // 2)}
    state["frame"] = {}
    for i, k in enumerate(FRAME):
        n = nn if i < 6 else ne
        state["frame"][k] = _pinned((n, width[k]) if k in width else (n,))
    return state


def run(state):
    case, model = state["case"], state["model"]
    if case["kind"] == "host":
        state["clock"] = model.step_host(state["host"], 1, state["clock"])
        return {k: state["host"][k] for k in FRAME}
    if case["kind"] == "adjoint":
        win = state["window"]
        vel = win.run_vel()
        loss, seed = adjoint.surface_velocity_misfit(vel, state["target"], state["top"])
        start, grad = win.gradients({"vel": seed})
        return {"loss": loss, "vel": vel, "start": start, "grad": {str(k): v for k, v in grad.items()}}
    model.upload(state["start"], state["clock"])
    if case["kind"] == "advance":
        model.step(case["steps"])
    else:
        for k in range(case["steps"]):
            for name in LOOP:
                model.call(name)
            if (k + 1) % 10 == 0:
                model.call("compute_dt")
    return model.download(state["frame"])


# --------------------------------------------------------------------------
# the same in plain torch, 64 bits
# --------------------------------------------------------------------------
def _volume(x, conn):
    a = x[conn]
    e = a[:, 1:] - a[:, :1]
    if x.shape[1] == 2:
        return (e[:, 0, 0] * e[:, 1, 1] - e[:, 0, 1] * e[:, 1, 0]).abs() / 2
    return (e[:, 0] * torch.linalg.cross(e[:, 1], e[:, 2])).sum(-1) / 6


def _gradients(x, conn):
    """dN_i/dx of linear simplices [ne][npe][nd]."""
    a = x[conn]
    e = a[:, 1:] - a[:, :1]
    if x.shape[1] == 2:
        det = e[:, 0, 0] * e[:, 1, 1] - e[:, 0, 1] * e[:, 1, 0]
        g1 = torch.stack([e[:, 1, 1], -e[:, 1, 0]], -1) / det[:, None]
        g2 = torch.stack([-e[:, 0, 1], e[:, 0, 0]], -1) / det[:, None]
        g = torch.stack([g1, g2], 1)
    else:
        c = [torch.linalg.cross(e[:, i], e[:, j]) for i, j in ((1, 2), (2, 0), (0, 1))]
        det = (e[:, 0] * c[0]).sum(-1)
        g = torch.stack(c, 1) / det[:, None, None]
    return torch.cat([-g.sum(1, keepdim=True), g], 1)


class _Plain:
    """The step's equations on torch tensors: one material law per element."""

    def __init__(self, case, seed):
        self.wl, self.conn, st = _inputs(case, seed)
        wl, conn = self.wl, self.conn
        m, self.p, mt = wl.mesh, wl.params, wl.mat
        self.nd, self.nn, self.ne = m.ndims, m.nnode, m.nelem
        self.mt = mt
        full = lambda v: torch.full((self.ne,), float(v), dtype=torch.float64, device=DEV)  # noqa: E731
        which = None if mt.elemmarkers is None else torch.from_numpy(mt.elemmarkers.argmax(1)).to(DEV)
        per = {}
        for key, name in ((capi.EF_COHESION0, "cohesion0"), (capi.EF_COHESION1, "cohesion1"),
                          (capi.EF_FRICTION0, "friction_angle0"), (capi.EF_FRICTION1, "friction_angle1"),
                          (capi.EF_SHEAR_MODULUS, "shear_modulus"), (capi.EF_THERM_COND, "therm_cond")):
            if key in wl.elem_fields:
                per[key] = torch.from_numpy(wl.elem_fields[key]).to(DEV)
            elif which is not None:
                per[key] = torch.tensor(getattr(mt, name), dtype=torch.float64, device=DEV)[which]
            else:
                per[key] = full(getattr(mt, name)[0])
        if capi.EF_LOG10_VISC in wl.elem_fields:
            per[capi.EF_LOG10_VISC] = torch.from_numpy(wl.elem_fields[capi.EF_LOG10_VISC]).to(DEV)
        self.per = per
        self.vbc = torch.tensor(self.p.vbc_values, dtype=torch.float64, device=DEV)
        self.vmax = self.p.max_vbc_val()
        self.bc = torch.from_numpy(m.bcflag.astype(np.int64)).to(DEV)
        self.facets = []
        nof = [[1, 2, 3], [0, 3, 2], [0, 1, 3], [0, 2, 1]] if self.nd == 3 else [[1, 2], [2, 0], [0, 1]]
        nof = torch.tensor(nof, device=DEV)
        for b in range(6):
            lo, hi = int(m.bfacet_offsets[b]), int(m.bfacet_offsets[b + 1])
            if hi > lo and self.p.vbc_types[b] == 0:
                f = torch.from_numpy(m.bfacets[lo:hi].astype(np.int64)).to(DEV)
                self.facets.append((b, f[:, 0], conn[f[:, 0][:, None], nof[f[:, 1]]]))
        self.S = {"x": st["coord"], "v": st["vel"], "T": st["temperature"], "s": st["stress"], "es": st["strain"],
                  "pls": st["plstrain"], "volo": st["volume_old"]}

    def scatter(self, a):
        """Sum of per-(element, slot) values over the nodes."""
        out = torch.zeros((self.nn, *a.shape[2:]), dtype=torch.float64, device=a.device)
        return out.index_add(0, self.conn.reshape(-1), a.reshape(-1, *a.shape[2:]))

    def rho(self, T):
        return self.mt.rho0[0] * (1 - self.mt.alpha[0] * (T[self.conn].mean(1) - 273))

    def masses(self, vol, rho):
        npe, ps = self.nd + 1, self.vmax * self.p.inertial_scaling
        spread = lambda a: self.scatter(a[:, None].expand(-1, npe))  # noqa: E731
        mass = spread(self.mt.bulk_modulus[0] / (ps * ps) * vol / npe)
        return mass, spread(rho * self.mt.heat_capacity[0] * vol / npe), spread(vol)

    def derive(self):
        S = self.S
        S["vol"], S["g"] = _volume(S["x"], self.conn), _gradients(S["x"], self.conn)
        S["mass"], S["tmass"], S["voln"] = self.masses(S["vol"], self.rho(S["T"]))

    def compute_dt(self):
        S, p = self.S, self.p
        a = S["x"][self.conn]
        if self.nd == 3:
            area = [torch.linalg.cross(a[:, j] - a[:, i], a[:, k] - a[:, i]).norm(dim=-1) / 2
                    for i, j, k in ((0, 1, 2), (0, 1, 3), (2, 3, 0), (2, 3, 1))]
            minl = float((3 * S["vol"] / torch.stack(area).max(0).values).min())
        else:
            side = [(a[:, j] - a[:, i]).norm(dim=-1) for i, j in ((0, 1), (1, 2), (0, 2))]
            minl = float((2 * S["vol"] / torch.stack(side).max(0).values).min())
        G = float(self.per[capi.EF_SHEAR_MODULUS].max())
        return p.dt_fraction * min(0.5 * minl / (self.vmax * p.inertial_scaling), 0.5 * self.mt.visc_min / (1e-40 + G),
                                   0.5 * minl / self.vmax, 0.5 * minl * minl / self.mt.therm_diff_max)

    def plastic(self, pls):
        mt, P = self.mt, self.per
        l0, l1 = mt.pls0[0], mt.pls1[0]
        q = ((pls - l0) / (l1 - l0)).clamp(0, 1)
        c = P[capi.EF_COHESION0] + q * (P[capi.EF_COHESION1] - P[capi.EF_COHESION0])
        phi = P[capi.EF_FRICTION0] + q * (P[capi.EF_FRICTION1] - P[capi.EF_FRICTION0])
        hard = torch.where((pls >= l0) & (pls < l1), (P[capi.EF_COHESION1] - P[capi.EF_COHESION0]) / (l1 - l0), 0.0)
        sphi = torch.sin(phi * (math.pi / 180))
        anphi = (1 + sphi) / (1 - sphi)
        ten = torch.clamp(c / torch.tan(phi * (math.pi / 180)), max=mt.tension_max)
        return 2 * c * torch.sqrt(anphi), anphi, hard, ten

    def matrix(self, s):
        rows = ((0, 3, 4), (3, 1, 5), (4, 5, 2)) if self.nd == 3 else ((0, 2), (2, 1))
        return torch.stack([torch.stack([s[:, c] for c in r], -1) for r in rows], -2)

    def return_map(self, K, G, s, pls):
        """Mohr-Coulomb return of the trial stress (no dilation)."""
        nd = self.nd
        amc, anphi, hard, ten = self.plastic(pls)
        depls = torch.zeros_like(pls)
        with torch.no_grad():   # closed-form principal stresses: which elements yield
            A = self.matrix(s)
            mean = s[:, :nd].mean(-1)
            if nd == 3:
                B = A - mean[:, None, None] * torch.eye(3, dtype=torch.float64, device=s.device)
                r = torch.sqrt((B * B).sum((-1, -2)) / 6).clamp(min=1e-300)
                ang = torch.acos((torch.linalg.det(B / r[:, None, None]) / 2).clamp(-1, 1)) / 3
                p0, p2 = mean + 2 * r * torch.cos(ang + 2 * math.pi / 3), mean + 2 * r * torch.cos(ang)
            else:
                r = torch.sqrt(((s[:, 0] - s[:, 1]) / 2) ** 2 + s[:, 2] ** 2)
                p0, p2 = mean - r, mean + r
            hit = ~((p0 - p2 * anphi + amc > 0) & (p2 - ten < 0))
            at = hit.nonzero()[:, 0]
        if at.numel() == 0:
            return s, depls
        amc, anphi, hard, ten, K, G = (a[at] for a in (amc, anphi, hard, ten, K, G))
        w, V = (torch.cat(a) for a in zip(*(torch.linalg.eigh(part) for part in self.matrix(s[at]).split(8192))))
        lo, hi = w[:, 0], w[:, -1]
        fs, ft = lo - hi * anphi + amc, hi - ten
        pa = torch.sqrt(1 + anphi * anphi) + anphi
        shear = hi - ten + pa * (lo - (ten * anphi - amc)) < 0
        a1, a2 = K + 4 / 3 * G, K - 2 / 3 * G
        al = torch.where(shear, fs / (a1 - a2 + a1 * anphi - a2 * anphi + 2 * torch.sqrt(anphi) * hard), ft / a1)
        first = torch.where(shear, a1 - a2, a2)
        last = torch.where(shear, a2 - a1, a1)
        mid = torch.where(shear, torch.zeros_like(a2), a2)
        corr = torch.stack([first, mid, last] if nd == 3 else [first, last], -1) * al[:, None]
        tension = torch.full_like(al, math.sqrt(7 / 18 if nd == 3 else 3 / 8))
        depls = depls.index_copy(0, at, al.abs() * torch.where(shear, torch.ones_like(al), tension))
        R = (V * (w - corr)[:, None, :]) @ V.transpose(-1, -2)
        pick = ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2)) if nd == 3 else ((0, 0), (1, 1), (0, 1))
        return s.index_copy(0, at, torch.stack([R[:, i, j] for i, j in pick], -1)), depls

    def j2(self, t):
        if self.nd == 3:
            d = t[:, :3] - t[:, :3].mean(-1, keepdim=True)
            return 0.5 * (d * d).sum(-1) + (t[:, 3:] ** 2).sum(-1)
        return 0.25 * (t[:, 0] - t[:, 1]) ** 2 + t[:, 2] ** 2

    def viscosity(self, edot, T):
        mt = self.mt
        if capi.EF_LOG10_VISC in self.per:
            v = 10.0 ** self.per[capi.EF_LOG10_VISC]
        else:
            n, A, Q = mt.visc_exponent[0], mt.visc_coefficient[0], mt.visc_activation_energy[0]
            ed = torch.sqrt(self.j2(edot)).clamp(min=1e-30)
            v = 0.25 * ed ** (1 / n - 1) * (0.75 * A) ** (-1 / n) * torch.exp(Q / (n * 8.3144 * T[self.conn].mean(1))) * 1e6
        return v.clamp(mt.visc_min, mt.visc_max)

    def step(self, dt):
        S, p, mt, conn, nd = self.S, self.p, self.mt, self.conn, self.nd
        g, vol = S["g"], S["vol"]
        k = self.per[capi.EF_THERM_COND]
        # heat
        heat = torch.einsum("eij,ej->ei", g @ g.transpose(-1, -2), S["T"][conn]) * (k * vol)[:, None]
        heat = heat - (mt.radiogenic_heating[0] / mt.heat_capacity[0] * vol)[:, None]
        T = S["T"] - self.scatter(heat) * dt / S["tmass"]
        T = torch.where((self.bc & 32) != 0, torch.as_tensor(p.surface_temperature, dtype=torch.float64, device=T.device), T)
        # strain rate, nodal volume rate
        L = torch.einsum("eid,eik->edk", S["v"][conn], g)
        pairs = ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2)) if nd == 3 else ((0, 0), (1, 1), (0, 1))
        edot = torch.stack([0.5 * (L[:, i, j] + L[:, j, i]) for i, j in pairs], -1)
        tr = edot[:, :nd].sum(-1)
        dvol = self.scatter((tr * vol)[:, None].expand(-1, nd + 1)) / S["voln"]
        edv = dvol[conn].mean(1)
        edot = torch.cat([edot[:, :nd] + ((edv - tr) / nd)[:, None], edot[:, nd:]], -1)
        # rheology
        de = edot * dt
        es = S["es"] + de
        K = torch.full_like(vol, mt.bulk_modulus[0])
        G = self.per[capi.EF_SHEAR_MODULUS]
        trd, s = de[:, :nd].sum(-1), S["s"]
        rt = mt.rheol_type
        depls = None
        if rt != capi.RH_MAXWELL:
            sp = s + 2 * G[:, None] * de
            sp = torch.cat([sp[:, :nd] + ((K - 2 / 3 * G) * trd)[:, None], sp[:, nd:]], -1)
            if rt != capi.RH_ELASTIC:
                sp, depls = self.return_map(K, G, sp, S["pls"])
        if rt in (capi.RH_MAXWELL, capi.RH_EVP):
            tmp = 0.5 * dt * G / self.viscosity(edot, T)
            f1, f2 = 1 - tmp, 1 / (1 + tmp)
            s0 = s[:, :nd].mean(-1)
            dv = vol / S["volo"] - 1
            n = ((s[:, :nd] - s0[:, None]) * f1[:, None] + 2 * G[:, None] * (de[:, :nd] - trd[:, None] / nd)) * f2[:, None]
            off = (s[:, nd:] * f1[:, None] + 2 * G[:, None] * de[:, nd:]) * f2[:, None]
            sv = torch.cat([n + (s0 + K * dv)[:, None], off], -1)
        if rt == capi.RH_MAXWELL:
            new = sv
        elif rt == capi.RH_EVP:
            relax = self.j2(sv) < self.j2(sp)
            new = torch.where(relax[:, None], sv, sp)
            depls = torch.where(relax, torch.zeros_like(depls), depls)
        else:
            new = sp
        pls = S["pls"] if depls is None else S["pls"] + depls
        dp = new[:, :nd].sum(-1) - s[:, :nd].sum(-1)
        # nodal mixed pressure
        dpn = self.scatter((dp * vol)[:, None].expand(-1, nd + 1)) / S["voln"]
        new = torch.cat([new[:, :nd] + ((dpn[conn].mean(1) - dp) / nd)[:, None], new[:, nd:]], -1)
        # force
        rho = self.rho(T)
        t = torch.einsum("eij,enj->eni", self.matrix(new), g)
        lift = torch.zeros(nd, dtype=torch.float64, device=t.device)
        lift[-1] = 1.0
        t = t + (rho * p.gravity / (nd + 1))[:, None, None] * lift
        f = -self.scatter(t * vol[:, None, None])
        for b, e, nodes in self.facets:
            c = S["x"][nodes]
            if nd == 3:
                nrm = torch.linalg.cross(c[:, 1] - c[:, 0], c[:, 2] - c[:, 0]) / 2
            else:
                d = c[:, 1] - c[:, 0]
                nrm = torch.stack([d[:, 1], -d[:, 0]], -1)
            z = c[:, :, -1].mean(1)
            if b == 4:
                comp = mt.rho0[0] * p.gravity * self.wl.lengths[2]
                pr = comp - (rho[e] + p.winkler_delta_rho) * p.gravity * (z + self.wl.lengths[2])
            elif b == 5:
                pr = torch.where(z < 0, -1030 * p.gravity * z, torch.zeros_like(z))
            else:
                pr = -mt.rho0[0] * p.gravity * z
            f = f.index_add(0, nodes.reshape(-1), -((pr[:, None] * nrm) / nd).repeat_interleave(nd, 0))
        if p.damping_option == 1:
            f = torch.where(S["v"].abs() > 1e-13, f - p.damping_factor * torch.copysign(f, S["v"]), f)
        else:
            f = f - p.damping_factor * f
        # motion
        v = S["v"] + dt * f / S["mass"][:, None]
        vx = torch.where((self.bc & 1) != 0, self.vbc[0], v[:, 0])
        vx = torch.where((self.bc & 2) != 0, self.vbc[1], vx)
        v = torch.cat([vx[:, None], v[:, 1:]], -1)
        x = S["x"] + v * dt
        gn, voln = _gradients(x, conn), _volume(x, conn)
        # Jaumann rotation
        W = torch.einsum("eid,eik->edk", v[conn], gn)
        W = 0.5 * (W - W.transpose(-1, -2))
        turned = []
        for a in (new, es):
            M = self.matrix(a)
            R = (M @ W - W @ M) if nd == 3 else (W @ M - M @ W)   # the reference's sign of the 3D spin
            turned.append(a + dt * torch.stack([R[:, i, j] for i, j in pairs], -1))
        mass, tmass, vn = self.masses(voln, rho)
        self.S = {"x": x, "v": v, "T": T, "s": turned[0], "es": turned[1], "pls": pls, "volo": vol, "vol": voln, "g": gn,
                  "mass": mass, "tmass": tmass, "voln": vn}
        self.out = {"force": f, "strain_rate": edot, "delta_plstrain": depls if depls is not None else torch.zeros_like(pls),
                    "dpressure": dp, "edvoldt": edv}

    def frame(self):
        S = self.S
        named = {"coord": "x", "vel": "v", "temperature": "T", "mass": "mass", "tmass": "tmass", "volume": "vol",
                 "stress": "s", "strain": "es", "plstrain": "pls"}
        return {k: (S[named[k]] if k in named else self.out[k]) for k in FRAME}


def exact(case, seed):
    m = _Plain(case, seed)
    if case["kind"] == "adjoint":
        return _exact_adjoint(case, m)
    m.derive()
    dt = m.compute_dt()
    for k in range(case["steps"]):
        m.step(dt)
        if (k + 1) % 10 == 0:
            dt = m.compute_dt()
    out = m.frame()
    # an element keeps its last plastic increment while it does not yield: after several steps no one step's value
    if case["rheology"] != "elastic" and case["steps"] > 1:
        out["delta_plstrain"] = None
    return out


def _exact_adjoint(case, m):
    """The gradients by automatic differentiation, one step's graph at a time."""
    if m.ne * case["steps"] > 6.0e7:
        return None
    target = m.S["v"] * 1.1
    top = torch.from_numpy(np.nonzero(m.wl.mesh.bcflag & 32)[0]).to(DEV)
    with torch.no_grad():
        m.derive()
        dt = m.compute_dt()
        states = []
        for _ in range(case["steps"]):
            states.append(m.S)
            m.step(dt)
    seed = torch.zeros_like(target)
    seed[top] = m.S["v"][top] - target[top]
    loss = 0.5 * float((seed * seed).sum())
    vel = m.S["v"]
    grads = {k: torch.zeros(m.ne, dtype=torch.float64, device=DEV) for k in range(capi.EF_COUNT)}
    gvbc = torch.zeros(capi.NBDRY, dtype=torch.float64, device=DEV)
    adj = {k: torch.zeros_like(a) for k, a in m.S.items()}
    adj["v"] = seed

    def pull(S, call, adj, params):
        """Adjoints of S (and of the parameters) from those of what call() leaves in m.S."""
        leaf = {k: a.detach().requires_grad_() for k, a in S.items()}
        m.S = dict(leaf)
        call()
        outs = [(m.S[k], adj[k]) for k in adj if k in m.S and m.S[k].requires_grad]
        names = list(leaf)
        got = torch.autograd.grad([o for o, _ in outs], [leaf[k] for k in names] + params, [a for _, a in outs],
                                  allow_unused=True)
        new = {k: (torch.zeros_like(leaf[k]) if x is None else x) for k, x in zip(names, got)}
        return new, got[len(names):]

    keys = list(m.per)
    for S in reversed(states):
        for k in keys:
            m.per[k] = m.per[k].detach().requires_grad_()
        m.vbc = m.vbc.detach().requires_grad_()
        adj, got = pull(S, lambda: m.step(dt), adj, [m.per[k] for k in keys] + [m.vbc])
        for k, x in zip(keys, got):
            if x is not None:
                grads[k] += x
        if got[-1] is not None:
            gvbc += got[-1]
    first = {k: states[0][k] for k in ("x", "v", "T", "s", "es", "pls", "volo")}
    adj, _ = pull(first, m.derive, adj, [])
    start = {"coord": adj["x"], "vel": adj["v"], "temperature": adj["T"], "stress": adj["s"], "plstrain": adj["pls"],
             "volume_old": adj["volo"]}
    return {"loss": loss, "vel": vel, "start": start, "grad": {**{str(k): v for k, v in grads.items()}, "vbc_values": gvbc}}
