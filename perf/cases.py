"""Performance cases: the work that a program using this framework has it do.

Each case goes through the public Python API over the C ABI (mpaso.gpu):
resident RK4 steps of the sw and ocean apps, the adjoint, an ensemble, the
host-buffer exchange and the task-by-task drop-in entries, on generated
spheres (icosahedral levels 3-7) and periodic hex planes, with seeded smooth
fields.  `exact` restates the same step in plain torch float64.
"""
import math
import os
import random
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "mpas-o-flecsi-2.0_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import mpaso  # noqa: E402
import mpaso.gpu as G  # noqa: E402
from mpaso._lib import check, lib  # noqa: E402
from mpaso.setup import fct_statics  # noqa: E402

DEV = "cuda" if torch.cuda.is_available() else "cpu"
F64 = torch.float64
GRAVITY = 9.80616
KAPPA, NU = 1e4, 1e4


# --------------------------------------------------------------------- cases
def listed():
    return [
        # the reference's own CPU configuration (64 x 64 planar hex, FCT tracer):
        # a small research run, where launches and latency count
        dict(name="sw_hex64_fct", kind="sw", mesh="hex", nx=64, ny=64, L=1, T=1, fct=True, steps=10),
        # the smallest call: one plain step of a coarse sphere without tracers, as a
        # coupler that advances step by step makes it
        dict(name="sw_sphere3_one", kind="sw", mesh="icosa", level=3, L=1, T=0, fct=False, steps=1),
        # the benchmark's workload: level-7 sphere, FCT + del2 tracer, resident time loop
        dict(name="sw_sphere7_fct", kind="sw", mesh="icosa", level=7, L=1, T=1, fct=True, steps=5),
        # an uneven plane with a few layers and the sw app's own centred tracer flux
        dict(name="sw_hex151x98_centred", kind="sw", mesh="hex", nx=151, ny=98, L=5, T=2, fct=False, steps=4),
        # the ocean app's production column: 60 levels x 3 tracers on a level-6 sphere
        dict(name="ocean_sphere6_60x3", kind="ocean", mesh="icosa", level=6, L=60, T=3, fct=True, steps=1),
        # a regional ocean run: odd plane, few levels, one tracer
        dict(name="ocean_hex77x54_7x1", kind="ocean", mesh="hex", nx=77, ny=54, L=7, T=1, fct=True, steps=4),
        # data assimilation window, (h, u) only: forward with checkpoints, then the gradient
        dict(name="adjoint_sphere5_hu", kind="adj_hu", mesh="icosa", level=5, L=1, T=0, fct=False, steps=40,
             every=10),
        # the same with an FCT tracer, whole window stored
        dict(name="adjoint_sphere5_tracer", kind="adj_tr", mesh="icosa", level=5, L=1, T=1, fct=True, steps=6,
             every=0),
        # tracer inversion of the ocean app, checkpoint every 2 steps
        dict(name="adjoint_ocean5_20x3", kind="adj_oc", mesh="icosa", level=5, L=20, T=3, fct=True, steps=4,
             every=2),
        # an ensemble of uneven members in one context
        dict(name="ensemble_48", kind="ens", members=48, pick=11, L=1, T=1, fct=True, steps=4),
        # a host model that keeps its fields in page-locked memory: copy in, one step, copy out
        dict(name="host_sphere7_fct", kind="host", mesh="icosa", level=7, L=1, T=1, fct=True, steps=1),
        # the drop-in boundary: one tracer stage task by task, as the reference's run.cc executes them
        dict(name="tasks_ocean5_20x3", kind="tasks_oc", mesh="icosa", level=5, L=20, T=3, fct=True, steps=1),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _cells(case):
    if case["kind"] == "ens":
        return sum(s[1] * s[2] if s[0] == "hex" else 10 * 4 ** s[1] + 2 for s in _members(case))
    return case["nx"] * case["ny"] if case["mesh"] == "hex" else 10 * 4 ** case["level"] + 2


def draw(rng):
    kind = rng.choice(["sw", "sw", "sw", "ocean", "ocean", "adj_hu", "adj_tr", "adj_oc", "ens", "host",
                       "tasks_oc", "tasks_sw"])
    c = dict(kind=kind)
    if kind == "ens":
        c.update(members=_log_int(rng, 3, 64), pick=rng.randrange(1000), L=1, T=rng.choice([0, 1, 1, 2]),
                 steps=rng.randint(1, 6))
        c["fct"] = c["T"] > 0 and rng.random() < 0.8
        return c
    if rng.random() < 0.5:
        c.update(mesh="icosa", level=rng.choice([3, 4, 5, 6, 7]))
    else:
        c.update(mesh="hex", nx=_log_int(rng, 16, 400), ny=2 * _log_int(rng, 8, 200))
    oc = kind in ("ocean", "adj_oc", "tasks_oc")
    c["L"] = _log_int(rng, 1, 60) if oc else rng.choice([1, 1, 1, 2, 3, 5, _log_int(rng, 4, 20)])
    c["T"] = 0 if kind == "adj_hu" else rng.randint(1, 3) if kind != "sw" else rng.choice([0, 1, 1, 2, 3])
    c["fct"] = c["T"] > 0 and (oc or kind == "adj_tr" or rng.random() < 0.7)
    adj = kind.startswith("adj")
    c["steps"] = _log_int(rng, 2, 24 if kind == "adj_hu" else 4) if adj else _log_int(rng, 1, 10)
    if kind.startswith("tasks"):
        c["steps"] = 1
    if adj:
        c["every"] = rng.choice([0, 1, 2, 5])
    # no dearer than the largest listed case, with an adjoint step counted as four
    # and kept to what its restatement's tape may hold
    most = 40962 * 180 // (12 if adj else 1)

    def cost():
        return _cells(c) * c["L"] * max(1, c["T"]) * c["steps"]

    while cost() > most:
        if c["steps"] > (2 if adj else 1):
            c["steps"] -= 1
        elif c["L"] > 8:
            c["L"] = c["L"] * 2 // 3
        elif c["mesh"] == "icosa":
            c["level"] -= 1
        else:
            c["nx"] = max(16, c["nx"] * 2 // 3)
    return c


# -------------------------------------------------------------------- inputs
_MESH = {}


def _mesh(spec, L, fct):
    """(host mesh, FCT statics, per-level-count): generated once per size and kept, as the
    mesh file that a program reads."""
    if spec not in _MESH:
        _MESH[spec] = (mpaso.Mesh.hex(spec[1], spec[2], 10e3, 1e-4) if spec[0] == "hex"
                       else mpaso.Mesh.icosa(spec[1])), {}
    mesh, st = _MESH[spec]
    if fct and L not in st:
        st[L] = fct_statics(mesh, L)
    return mesh, (st[L] if fct else None)


def _members(case):
    r = random.Random(case["pick"])
    out = []
    for _ in range(case["members"]):
        if r.random() < 0.25:
            out.append(("icosa", r.choice([3, 4, 5])))
        else:
            out.append(("hex", r.randint(12, 128), 2 * r.randint(8, 64)))
    return out


def _specs(case):
    if case["kind"] == "ens":
        return _members(case)
    return [("hex", case["nx"], case["ny"]) if case["mesh"] == "hex" else ("icosa", case["level"])]


def _waves(mesh, where, rng, count):
    """`count` smooth fields with values in about [-1, 1] at the mesh's cells or vertices:
    sums of plane waves (periodic ones on the plane)."""
    f = mesh.fields
    if mesh.on_sphere:
        x = np.stack([f[a + where] for a in "xyz"], 1)
        x = torch.tensor(x / np.linalg.norm(x, axis=1, keepdims=True), dtype=F64, device=DEV)
        k = rng.uniform(-5.0, 5.0, (6, 3, count))
    else:
        x = torch.tensor(np.stack([f["x" + where] / mesh.Lx, f["y" + where] / mesh.Ly], 1), dtype=F64, device=DEV)
        k = 2 * np.pi * rng.integers(-3, 4, (6, 2, count))
    amp, ph = rng.uniform(0.3, 1.0, (6, count)), rng.uniform(0, 2 * np.pi, (6, count))
    k, amp, ph = (torch.tensor(np.asarray(a, float), device=DEV) for a in (k, amp, ph))
    out = torch.zeros(x.shape[0], count, dtype=F64, device=DEV)
    for m in range(6):
        a = ph[m].expand_as(out).clone()
        for d in range(x.shape[1]):
            a += x[:, d:d + 1] * k[m, d]
        out += amp[m] * torch.sin(a)
    return out / amp.sum(0)


def _flow(mesh, rng, L, peak):
    """Rotational velocity of a streamfunction at the vertices."""
    psi = _waves(mesh, "Vertex", rng, L)
    v = torch.tensor(mesh.fields["verticesOnEdge"] - 1, dtype=torch.long, device=DEV)
    dv = torch.tensor(mesh.fields["dvEdge"], dtype=F64, device=DEV)[:, None]
    u = -(psi[v[:, 1]] - psi[v[:, 0]]) / dv
    return peak * u / u.abs().amax(0)


def _fields(case, seed):
    """h, u, tracers (concatenated over the members), and the ocean's edge thickness."""
    rng = np.random.default_rng([seed, 77])
    L, T = case["L"], case["T"]
    oc = case["kind"] in ("ocean", "adj_oc", "tasks_oc")
    hs, us, ts, es = [], [], [], []
    for spec in _specs(case):
        mesh, _ = _mesh(spec, L, False)
        if oc:
            depth = torch.arange(0.5, L, device=DEV, dtype=F64) / L
            hs.append(torch.full((mesh.nCells, L), 100.0, dtype=F64, device=DEV))
            es.append(torch.full((mesh.nEdges, L), 100.0, dtype=F64, device=DEV))
            us.append(_flow(mesh, rng, L, 0.3) * (1.0 - 0.8 * depth))
            w = _waves(mesh, "Cell", rng, L * T).reshape(-1, L, T)
            # temperature, salinity, a passive tracer
            if case["kind"] == "adj_oc":
                w[:, :, 0] = 15.0 + 10.0 * w[:, :, 0]
            else:
                w[:, :, 0] = (30.0 * (1.0 - depth) + 2.0 * w[:, :, 0]).clamp(0.0, 30.0)
            if T > 1:
                w[:, :, 1] = 35.0 + 0.9 * w[:, :, 1]
            if T > 2:
                w[:, :, 2:] = 0.5 + 0.5 * w[:, :, 2:]
            ts.append(w)
        else:
            h0, ha, up = (8000.0, 100.0, 30.0) if mesh.on_sphere else (1000.0, 10.0, 1.0)
            hs.append(h0 + ha * _waves(mesh, "Cell", rng, L))
            us.append(_flow(mesh, rng, L, up))
            ts.append((0.5 + 0.5 * _waves(mesh, "Cell", rng, L * T)).reshape(-1, L, T) if T else
                      torch.zeros(mesh.nCells, L, 0, dtype=F64, device=DEV))
    out = dict(h=torch.cat(hs).contiguous(), u=torch.cat(us).contiguous(), tr=torch.cat(ts).contiguous())
    if oc:
        out["hE"] = torch.cat(es)
    return out


def _dt(case):
    if case["kind"] == "ens":
        return 30.0
    if case["mesh"] == "hex":
        return 300.0 if case["kind"] in ("ocean", "adj_oc", "tasks_oc") else 30.0
    return (300.0 if case["kind"] in ("ocean", "adj_oc", "tasks_oc") else 60.0) * 1.5 ** (7 - case["level"])


def _cotangents(case, seed, f):
    g = torch.Generator(device="cpu").manual_seed(seed * 31 + 5)
    return {k: torch.randn(f[k].shape, generator=g, dtype=F64).to(DEV) for k in ("h", "u", "tr")}


def prepare(case, seed):
    L, T, kind = case["L"], case["T"], case["kind"]
    pairs = [_mesh(s, L, case["fct"]) for s in _specs(case)]
    fcts = [p[1] for p in pairs]
    if kind == "ens":
        dm = G.DeviceMesh.ensemble([p[0] for p in pairs], fcts=fcts if case["fct"] else None)
    else:
        dm = G.DeviceMesh(pairs[0][0], fct=fcts[0])
    f = _fields(case, seed)
    s = dict(case=case, kind=kind, dm=dm, dt=_dt(case), n=case["steps"], **f)
    if kind.startswith("tasks"):
        nC, nE, nV = dm.nC, dm.nE, dm.nV

        def new(n, t=0):
            return torch.zeros((n, L, t) if t else (n, L), dtype=F64, device=DEV)

        s["stream"] = torch.cuda.Stream()
        if kind == "tasks_oc":
            s["b"] = dict(ntf=new(nE), hProv=new(nC), hInv=new(nC), hNew=new(nC), lo=new(nE, T), ho=new(nE, T),
                          fin=new(nC, T), fout=new(nC, T), tend=new(nC, T), mx=new(nC, T), mn=new(nC, T),
                          prov=new(nC, T), trNew=new(nC, T), trPrev=new(nC, T))
        else:
            s["b"] = dict(h_edge=new(nE), h_vertex=new(nV), circulation=new(nV), vorticity=new(nV), ke=new(nC),
                          pv_edge=new(nE), pv_vertex=new(nV), th=new(nC), tu=new(nE), tt=new(nC, T),
                          u1=new(nE), h1=new(nC), t1=new(nC, T), u2=new(nE), h2=new(nC), t2=new(nC, T))
        return s
    oc = kind in ("ocean", "adj_oc")
    st = G.State(dm, app=G.APP_OCEAN if oc else G.APP_SW, nlev=L, ntr=T, fct=case["fct"],
                 hmix=T > 0, kappa=KAPPA, nu=0.0 if oc else NU)
    s["st"] = st
    if oc:
        st.set(G.FIELD_LAYER_THICKNESS_EDGE, f["hE"])
    if kind == "host":
        for k in ("h", "u", "tr"):
            s[k] = f[k].cpu().pin_memory() if f[k].numel() else f[k].cpu()
    else:
        s["out"] = {k: torch.empty_like(f[k]) for k in ("h", "u", "tr")}
    if kind.startswith("adj"):
        s["g"] = _cotangents(case, seed, f)
        s["g0"] = {k: torch.empty_like(f[k]) for k in ("h", "u", "tr")}
    return s


# ---------------------------------------------------------------------- runs
def _set(s):
    st = s["st"]
    st.set(G.FIELD_H, s["h"])
    st.set(G.FIELD_U, s["u"])
    if s["case"]["T"]:
        st.set(G.FIELD_TRACERS, s["tr"])


def _get(s, only_tracers=False):
    st, o = s["st"], s["out"]
    out = {}
    if not only_tracers:
        out["h"] = st.get(G.FIELD_H, o["h"])
        out["u"] = st.get(G.FIELD_U, o["u"])
    if s["case"]["T"]:
        out["tr"] = st.get(G.FIELD_TRACERS, o["tr"])
    return out


def _run_steps(s):
    _set(s)
    if s["n"] == 1:
        s["st"].step(s["dt"], 1)
    else:
        s["st"].step_graph(s["dt"], s["n"])
    return _get(s, s["kind"] == "ocean")


def _run_adjoint(s):
    st, g, o = s["st"], s["g"], s["g0"]
    _set(s)
    st.forward(s["dt"], s["n"], s["case"]["every"])
    out = _get(s, s["kind"] == "adj_oc")
    if s["kind"] == "adj_hu":
        st.vjp(g["h"], g["u"], out=(o["h"], o["u"]))
        out.update(gh=o["h"], gu=o["u"])
    else:
        st.vjp_tracers(g["h"], g["u"], g["tr"], out=(o["h"], o["u"], o["tr"]))
        out.update(gt=o["tr"])
        if s["kind"] == "adj_tr":
            out.update(gh=o["h"], gu=o["u"])
    return out


def _run_host(s):
    s["st"].step_host(s["dt"], s["n"], s["h"], s["u"], s["tr"] if s["case"]["T"] else None)
    return {k: s[k] for k in (("h", "u", "tr") if s["case"]["T"] else ("h", "u"))}


def _task(s, name, *args):
    """One C-ABI task entry on the program's stream."""
    conv = [s["dm"].handle]
    for a in args:
        conv.append(G.ctypes.c_double(a) if isinstance(a, float) else
                    G.ctypes.c_int32(a) if isinstance(a, int) else G.ctypes.c_void_p(a.data_ptr()))
    conv.append(G.ctypes.c_void_p(s["stream"].cuda_stream))
    check(getattr(lib(), "mpaso_" + name)(*conv))


def _run_tasks_ocean(s):
    L, T, dt, b = s["case"]["L"], s["case"]["T"], s["dt"], s["b"]
    with torch.cuda.stream(s["stream"]):
        b["tend"].zero_()
        b["trNew"].copy_(s["tr"])
    _task(s, "oc_calc_normal_thickness_flux", L, s["hE"], s["u"], b["ntf"])
    _task(s, "oc_calc_provisional_layer_thicknesses", L, s["h"], b["ntf"], b["hProv"], b["hInv"], b["hNew"], dt)
    _task(s, "oc_calc_horiz_tracer_advection_flux_mono_low_order", L, T, b["ntf"], s["tr"], b["lo"])
    _task(s, "oc_calc_horiz_tracer_advection_flux_mono_high_order", L, T, b["ntf"], s["tr"], b["ho"])
    _task(s, "oc_correct_and_rescale_high_order_mono_horiz_flux", L, T, b["hInv"], s["h"], b["ntf"], b["lo"],
          s["tr"], b["ho"], b["fin"], b["fout"], b["tend"], b["mx"], b["mn"], dt)
    _task(s, "oc_accumulate_horiz_tracer_advection_tend_mono_FCT", L, T, b["hInv"], s["h"], b["ho"], s["tr"],
          b["prov"], b["tend"], dt)
    _task(s, "oc_tracer_hmix_del2_tend", L, T, s["hE"], s["tr"], b["tend"], KAPPA)
    _task(s, "oc_step_tracers_forward", L, T, b["tend"], s["tr"], b["trNew"], b["trPrev"], dt / 6, dt / 2)
    return {k: b[k] for k in ("tend", "prov", "trNew", "trPrev", "ho", "lo", "hProv")}


def _run_tasks_sw(s):
    L, T, dt, b = s["case"]["L"], s["case"]["T"], s["dt"], s["b"]
    with torch.cuda.stream(s["stream"]):
        b["u2"].copy_(s["u"])
        b["h2"].copy_(s["h"])
        b["t2"].copy_(s["tr"] * s["h"][:, :, None])
    _task(s, "sw_compute_solve_diagnostics", L, s["h"], s["u"], b["h_edge"], b["h_vertex"], b["circulation"],
          b["vorticity"], b["ke"], b["pv_edge"], b["pv_vertex"])
    _task(s, "sw_compute_tend", L, b["h_edge"], s["h"], s["u"], b["ke"], b["pv_edge"], b["th"], b["tu"])
    _task(s, "sw_compute_scalar_tend", L, T, b["h_edge"], s["u"], s["tr"], b["tt"])
    _task(s, "sw_compute_substep", L, T, b["u1"], s["u"], b["tu"], b["h1"], s["h"], b["th"], b["t1"], s["tr"],
          b["tt"], dt / 2, 0)
    _task(s, "sw_accumulate_update", L, T, b["u2"], b["tu"], b["h2"], b["th"], b["t2"], b["tt"], dt / 6)
    return {k: b[k] for k in ("vorticity", "ke", "pv_edge", "th", "tu", "tt", "u1", "h1", "t1", "u2", "h2", "t2")}


_RUN = dict(sw=_run_steps, ocean=_run_steps, ens=_run_steps, host=_run_host, adj_hu=_run_adjoint,
            adj_tr=_run_adjoint, adj_oc=_run_adjoint, tasks_oc=_run_tasks_ocean, tasks_sw=_run_tasks_sw)


def run(state):
    return _RUN[state["kind"]](state)


# ---------------------------------------------------------------------- work
def work(case):
    """Least traffic and arithmetic of a pass.  Per entity of a stage and level (a cell, its
    3 edges and 2 vertices): the prognostic fields read and written once, the static mesh and
    stencil arrays read once; multiplies and adds of the reference's task formulas."""
    kind, L, T = case["kind"], case["L"], case["T"]
    nc = _cells(case)
    cl = nc * L
    oc = kind in ("ocean", "adj_oc", "tasks_oc")
    # statics per cell (all levels share them): TRiSK 10 x (4 + 8), FCT 10 x (4 + 8 + 8) per edge,
    # connectivity and geometry about 150 bytes
    stat = nc * ((0 if oc else 3 * 10 * 12) + (3 * 10 * 20 if case["fct"] else 0) + 150)
    state = 8 * cl * ((3 if oc else 4) + T)  # u (3 edges) and h, tracers
    tracer = T * ((3 * (2 * 10 + 5) + 6 * 4 + 20 + 6 * 3) if case["fct"] else 3 * 5 + 6 * 2)
    flow = 0 if oc else 3 * (4 * 10 + 20) + 6 * 6 + 2 * 14
    stage_flops = cl * (tracer + (3 * 12 if case["fct"] else 0) + flow + 3 * (2 + 2 * T) + T * 9)
    stage_bytes = stat + 3 * state
    if kind.startswith("tasks"):
        if oc:
            return dict(bytes=8 * cl * (3 + 1 + 3 + T + (3 + 3 + 6 * T + 6 * T + 6 * T)), flops=stage_flops)
        return dict(bytes=8 * cl * (4 + T + 3 * 5 + 12 + 5 * T), flops=stage_flops)
    n = case["steps"]
    stages = 4 * n
    by, fl = stage_bytes * stages, stage_flops * stages
    if kind.startswith("adj"):  # the forward, and a reverse of about twice its arithmetic
        by, fl = 3 * by, 3 * fl
    return dict(bytes=by + 2 * state, flops=fl)


# --------------------------------------------------------------------- exact
def _pad(off, idx):
    """CRS rows padded to the widest: (index [n][w], valid [n][w])."""
    cnt = np.diff(off)
    w = int(cnt.max())
    valid = np.arange(w)[None, :] < cnt[:, None]
    out = np.zeros(valid.shape, np.int64)
    out[valid] = idx
    return torch.tensor(out, device=DEV), torch.tensor(valid, device=DEV)


def _max(a, b):
    return torch.where(a < b, b, a)


def _min(a, b):
    return torch.where(b < a, b, a)


class _Ref:
    """One mesh's RK4 stages in plain torch float64 (task formulas of the reference's
    apps/sw/tasks/solve.cc and apps/ocean/tasks/solve.cc)."""

    def __init__(self, mesh, fct, case):
        def t(a, dtype=F64):
            return torch.tensor(np.ascontiguousarray(a), dtype=dtype, device=DEV)

        f, crs = mesh.fields, mesh.crs()
        self.oc = case["kind"] in ("ocean", "adj_oc", "tasks_oc")
        self.fct, self.T, self.L = case["fct"], case["T"], case["L"]
        c12 = t(crs["e2c"][1], torch.long).reshape(-1, 2)
        self.c1, self.c2 = c12[:, 0], c12[:, 1]
        v12 = t(crs["e2v"][1], torch.long).reshape(-1, 2)
        self.v1, self.v2 = v12[:, 0], v12[:, 1]
        self.ce, ok = _pad(*crs["c2e"])
        me = torch.arange(mesh.nCells, device=DEV)[:, None]
        self.cs = torch.where(self.c1[self.ce] == me, -1.0, 1.0).to(F64) * ok  # inward positive
        self.cok = ok
        cc, ok2 = _pad(*crs["c2c"])
        self.cc = torch.where(ok2, cc, me)
        self.vc = t(crs["v2c"][1], torch.long).reshape(-1, 3)
        self.ve = t(crs["v2e"][1], torch.long).reshape(-1, 3)
        mv = torch.arange(mesh.nVertices, device=DEV)[:, None]
        self.vs = torch.where(self.v2[self.ve] == mv, 1.0, -1.0).to(F64)
        self.ee, eok = _pad(*crs["e2e"])
        self.ew = t(f["weightsOnEdge"])[:, :self.ee.shape[1]] * eok
        self.dc, self.dv, self.area, self.atri, self.fv = (
            t(f[k])[:, None] for k in ("dcEdge", "dvEdge", "areaCell", "areaTriangle", "fVertex"))
        self.kite = t(f["kiteAreasOnVertex"])
        if fct is not None:
            na = t(fct["nAdvCellsForEdge"], torch.long)
            w = int(na.max())
            aok = torch.arange(w, device=DEV)[None, :] < na[:, None]
            self.ac = t(fct["advCellsForEdge"][:, :w], torch.long) * aok
            self.a1 = t(fct["advCoef"])[:, :w] * aok
            self.a3 = t(fct["advCoef_3rd"])[:, :w] * aok * 0.25
            self.mask = t(fct["highOrderAdvMask"])[:, :self.L, None]
            self.msd = t(fct["meshScalingDel2"])[:, None, None]
        else:
            self.msd = torch.ones(mesh.nEdges, 1, 1, dtype=F64, device=DEV)

    def cell_sum(self, x):
        """sum over the cell's edges of edgeSign x / area."""
        out = 0.0
        for j in range(self.ce.shape[1]):
            s = self.cs[:, j].reshape((-1,) + (1,) * (x.dim() - 1))
            out = out + s * x[self.ce[:, j]]
        return out / (self.area if x.dim() == 2 else self.area[:, :, None])

    def diagnostics(self, h, u):
        circ = hv = 0.0
        for j in range(3):
            e = self.ve[:, j]
            circ = circ + self.vs[:, j:j + 1] * (self.dc * u)[e]
            hv = hv + self.kite[:, j:j + 1] * h[self.vc[:, j]]
        vort, hv = circ / self.atri, hv / self.atri
        ke = 0.0
        for j in range(self.ce.shape[1]):
            e = self.ce[:, j]
            ke = ke + self.cok[:, j:j + 1] * (0.25 * self.dc * self.dv * u * u)[e]
        pvv = (self.fv + vort) / hv
        return 0.5 * (h[self.c1] + h[self.c2]), ke / self.area, 0.5 * (pvv[self.v1] + pvv[self.v2]), vort

    def flow_tend(self, h, u, nu):
        he, ke, pve, vort = self.diagnostics(h, u)
        q, F = 0.0, u * he
        for j in range(self.ee.shape[1]):
            o = self.ee[:, j]
            q = q + self.ew[:, j:j + 1] * F[o] * (0.5 * (pve + pve[o]))
        c1, c2 = self.c1, self.c2
        tu = q - (ke[c2] - ke[c1] + GRAVITY * (h[c2] - h[c1])) / self.dc
        if nu:
            div = -self.cell_sum(self.dv * u)
            tu = tu + nu * ((div[c2] - div[c1]) / self.dc - (vort[self.v2] - vort[self.v1]) / self.dv)
        return self.cell_sum(self.dv * F), tu

    def fluxes(self, ntf, tr):
        f = ntf[:, :, None]
        dv, c1, c2 = self.dv[:, :, None], self.c1, self.c2
        lo = dv * (torch.where(f > 0, f, 0.0 * f) * tr[c1] + torch.where(f < 0, f, 0.0 * f) * tr[c2])
        ho = 0.0
        sg = torch.sign(f).detach()
        for j in range(self.ac.shape[1]):
            co = self.a1[:, j, None, None] + self.a3[:, j, None, None] * sg
            ho = ho + tr[self.ac[:, j]] * (f * self.mask * co)
        return lo, ho

    def tracer_tend(self, h, u, tr, dt, he=None):
        c1, c2 = self.c1, self.c2
        he = 0.5 * (h[c1] + h[c2]) if he is None else he
        ntf, dv = u * he, self.dv[:, :, None]
        if self.fct:
            hpi = (1.0 / (h + dt * self.cell_sum(self.dv * ntf)))[:, :, None]
            lo, ho = self.fluxes(ntf, tr)
            ho = ho + (1.0 - self.mask) * (0.5 * dv) * ntf[:, :, None] * (tr[c1] + tr[c2]) - lo
            tend, ho = self.limit(h, hpi, lo, ho, tr, dt)
        elif not self.oc:
            tend = self.cell_sum(dv * ntf[:, :, None] * (0.5 * (tr[c1] + tr[c2])))
        else:
            tend = 0.0 * tr
        return tend - self.mix(he, tr)

    def mix(self, he, tr):
        dv = self.dv[:, :, None]
        return self.cell_sum(he[:, :, None] * (tr[self.c2] - tr[self.c1]) * (self.msd * KAPPA * dv / self.dc[:, :, None]))

    def limit(self, h, hpi, lo, ho, tr, dt):
        mx, mn = tr, tr
        for j in range(self.cc.shape[1]):
            x = tr[self.cc[:, j]]
            mx, mn = _max(mx, x), _min(mn, x)
        td = self.cell_sum(lo)
        fin = fout = 0.0
        for j in range(self.ce.shape[1]):
            x = self.cs[:, j, None, None] * ho[self.ce[:, j]]
            fin, fout = fin + torch.where(x > 0, x, 0.0 * x), fout + torch.where(x < 0, x, 0.0 * x)
        fin, fout = fin / self.area[:, :, None], fout / self.area[:, :, None]
        up = (tr * h[:, :, None] + dt * td) * hpi
        eps, one = 1e-10, torch.ones((), dtype=F64, device=DEV)
        zero = 0.0 * one

        def factor(num, den):
            return _min(one, _max(zero, num / (den + eps)))

        rp = factor(mx - up, dt * fin * hpi)
        rm = factor(up - mn, -dt * fout * hpi)
        c1, c2 = self.c1, self.c2
        r = torch.where(ho > 0, _min(rm[c1], rp[c2]), _min(rp[c1], rm[c2]))
        ho = ho * r
        return td + self.cell_sum(ho), ho

    def sw(self, h, u, tr, dt, n, nu=NU):
        w, sub = (dt / 6, dt / 3, dt / 3, dt / 6), (dt / 2, dt / 2, dt)
        for _ in range(n):
            hp, up, tp = h, u, tr
            hn, un, qn = h, u, tr * h[:, :, None]
            for k in range(4):
                th, tu = self.flow_tend(hp, up, nu)
                tq = self.tracer_tend(hp, up, tp, dt) if self.T else None
                if k < 3:
                    hp, up = h + sub[k] * th, u + sub[k] * tu
                    if self.T:
                        tp = (h[:, :, None] * tr + sub[k] * tq) / hp[:, :, None]
                hn, un = hn + w[k] * th, un + w[k] * tu
                if self.T:
                    qn = qn + w[k] * tq
            h, u = hn, un
            if self.T:
                tr = qn / hn[:, :, None]
        return h, u, tr

    def ocean(self, h, hE, u, tr, dt, n):
        w, sub = (dt / 6, dt / 3, dt / 3, dt / 6), (dt / 2, dt / 2, dt)
        for _ in range(n):
            tp, tn = tr, tr
            for k in range(4):
                tq = self.tracer_tend(h, u, tp, dt, hE)
                tn = tn + w[k] * tq
                if k < 3:
                    tp = tr + sub[k] * tq
            tr = tn
        return tr


def exact(case, seed):
    kind, L, T, n, dt = case["kind"], case["L"], case["T"], case["steps"], _dt(case)
    pairs = [_mesh(s, L, case["fct"]) for s in _specs(case)]
    f = _fields(case, seed)
    if kind == "ens":
        out, c, e = [], 0, 0
        for mesh, fct in pairs:
            cs, es = slice(c, c + mesh.nCells), slice(e, e + mesh.nEdges)
            c, e = cs.stop, es.stop
            out.append(_Ref(mesh, fct, case).sw(f["h"][cs], f["u"][es], f["tr"][cs], dt, n))
        r = [torch.cat(x) for x in zip(*out)]
        return dict(h=r[0], u=r[1], **({"tr": r[2]} if T else {}))
    R = _Ref(pairs[0][0], pairs[0][1], case)
    if kind in ("sw", "host"):
        h, u, tr = R.sw(f["h"], f["u"], f["tr"], dt, n)
        out = dict(h=h, u=u, **({"tr": tr} if T else {}))
        return {k: v.cpu() for k, v in out.items()} if kind == "host" else out
    if kind == "ocean":
        return dict(tr=R.ocean(f["h"], f["hE"], f["u"], f["tr"], dt, n))
    if kind.startswith("adj"):
        g = _cotangents(case, seed, f)
        x = {k: f[k].clone().requires_grad_(True) for k in ("h", "u", "tr")}
        if kind == "adj_oc":
            tr = R.ocean(f["h"], f["hE"], f["u"], x["tr"], dt, n)
            (gt,) = torch.autograd.grad((tr * g["tr"]).sum(), x["tr"])
            return dict(tr=tr.detach(), gt=gt)
        h, u, tr = R.sw(x["h"], x["u"], x["tr"], dt, n)
        J = (h * g["h"]).sum() + (u * g["u"]).sum()
        out = dict(h=h.detach(), u=u.detach())
        if kind == "adj_hu":
            out["gh"], out["gu"] = torch.autograd.grad(J, (x["h"], x["u"]))
            return out
        out["tr"] = tr.detach()
        out["gh"], out["gu"], out["gt"] = torch.autograd.grad(J + (tr * g["tr"]).sum(), (x["h"], x["u"], x["tr"]))
        return out
    if kind == "tasks_oc":
        h, hE, u, tr = f["h"], f["hE"], f["u"], f["tr"]
        ntf = u * hE
        hp = h + dt * R.cell_sum(R.dv * ntf)
        hpi = (1.0 / hp)[:, :, None]
        lo, ho = R.fluxes(ntf, tr)
        ho = ho + (1.0 - R.mask) * (0.5 * R.dv[:, :, None]) * ntf[:, :, None] * (tr[R.c1] + tr[R.c2]) - lo
        td, ho = R.limit(h, hpi, lo, ho, tr, dt)
        prov = (tr * h[:, :, None] + dt * td) * hpi
        td = td - R.mix(hE, tr)
        return dict(tend=td, prov=prov, trNew=tr + dt / 6 * td, trPrev=tr + dt / 2 * td, ho=ho, lo=lo, hProv=hp)
    h, u, tr = f["h"], f["u"], f["tr"]
    he, ke, pve, vort = R.diagnostics(h, u)
    th, tu = R.flow_tend(h, u, 0.0)
    tt = R.cell_sum(R.dv[:, :, None] * (u * he)[:, :, None] * (0.5 * (tr[R.c1] + tr[R.c2])))
    h1 = h + dt / 2 * th
    return dict(vorticity=vort, ke=ke, pv_edge=pve, th=th, tu=tu, tt=tt, u1=u + dt / 2 * tu, h1=h1,
                t1=(h[:, :, None] * tr + dt / 2 * tt) / h1[:, :, None], u2=u + dt / 6 * tu, h2=h + dt / 6 * th,
                t2=tr * h[:, :, None] + dt / 6 * tt)
