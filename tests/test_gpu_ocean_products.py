"""The ocean kernels' integer-pipe products at and outside their exponent windows
(factors 2^-128 .. 2^128, products 2^-895 .. 2^129), against the oracle value
for value: zeros, subnormals and values on both sides of each end, one to
three tracers, on stencils of exactly ten cells and of run-time width."""
import numpy as np
import pytest

import mpaso
from mpaso.initial import ocean_state
from mpaso.setup import fct_statics
from oracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ntr", [1, 2, 3])
@pytest.mark.parametrize("spec", [("icosa", 2), ("hex", 9, 6)])
@pytest.mark.parametrize("exp2", [-1060, -960, -920, -880, -300, -130, 0, 100, 125, 300])
def test_ocean_step_at_the_window_of_the_integer_products(exp2, spec, ntr):
    import mpaso.gpu as G
    mesh = mpaso.Mesh.icosa(spec[1]) if spec[0] == "icosa" else mpaso.Mesh.hex(spec[1], spec[2], 20e3, 1e-4)
    L, dt = 3, 100.0
    f = fct_statics(mesh, L)
    h, hE, u, _ = ocean_state(mesh, 4, L, ntr)
    rng = np.random.default_rng(7)
    tr = np.ldexp(rng.uniform(-1.0, 1.0, (mesh.nCells, L, ntr)), exp2)
    tr[rng.uniform(size=tr.shape) < 0.2] = 0.0
    u[rng.uniform(size=u.shape) < 0.1] = 0.0
    opts = dict(fct=True, hmix=True, kappa=1e4)
    S = Oracle("restatement")
    want = S.ocean_run(mesh, S.static(mesh, f), S.config(L, ntr, **opts), dt, 2, h, hE, u, tr)
    dm = G.DeviceMesh(mesh, fct=f)
    st = G.State(dm, app=G.APP_OCEAN, nlev=L, ntr=ntr, **opts)
    for field, a in ((G.FIELD_H, h), (G.FIELD_LAYER_THICKNESS_EDGE, hE), (G.FIELD_U, u), (G.FIELD_TRACERS, tr)):
        st.set(field, a)
    st.step(dt, 2)
    got = st.get(G.FIELD_TRACERS)
    assert np.isfinite(want).all()
    assert np.array_equal(got, np.asarray(want).reshape(got.shape))


@pytest.mark.parametrize("ntr", [1, 3, 4])
@pytest.mark.parametrize("exp2", [-1060, -900, -130, 0, 125, 300])
def test_ocean_tasks_at_the_window_of_the_integer_products(exp2, ntr):
    """The same through the per-task entries, on columns of uneven depth."""
    import mpaso.gpu as G
    mesh = mpaso.Mesh.icosa(2)
    L, T, dt = 4, ntr, 100.0
    maxlev = np.random.default_rng(1).integers(1, L + 1, mesh.nCells).astype(np.int32)
    f = fct_statics(mesh, L, maxLevelCell=maxlev)
    h, hE, u, _ = ocean_state(mesh, 4, L, ntr)
    rng = np.random.default_rng(8)
    nC, nE = mesh.nCells, mesh.nEdges
    tr = np.ldexp(rng.uniform(-1.0, 1.0, (nC, L, T)), exp2)
    tr[rng.uniform(size=tr.shape) < 0.2] = 0.0
    u[rng.uniform(size=u.shape) < 0.1] = 0.0
    z = lambda *s: np.zeros(s)  # noqa: E731
    a = dict(ntf=u * hE, hp=z(nC, L), hpi=z(nC, L), hni=z(nC, L), lo=z(nE, L, T), ho=z(nE, L, T), fi=z(nC, L, T),
             fo=z(nC, L, T), tend=z(nC, L, T), mx=z(nC, L, T), mn=z(nC, L, T), tp=z(nC, L, T))
    b = {k: v.copy() for k, v in a.items()}
    dm = G.DeviceMesh(mesh, fct=f)
    S = Oracle("restatement")
    om, st, cfg = S.mesh(mesh), S.static(mesh, f), S.config(L, T)
    dm.call("oc_calc_provisional_layer_thicknesses", L, h, a["ntf"], a["hp"], a["hpi"], a["hni"], dt)
    dm.call("oc_calc_horiz_tracer_advection_flux_mono_low_order", L, T, a["ntf"], tr, a["lo"])
    dm.call("oc_calc_horiz_tracer_advection_flux_mono_high_order", L, T, a["ntf"], tr, a["ho"])
    dm.call("oc_correct_and_rescale_high_order_mono_horiz_flux", L, T, a["hpi"], h, a["ntf"], a["lo"], tr, a["ho"],
            a["fi"], a["fo"], a["tend"], a["mx"], a["mn"], dt)
    dm.call("oc_accumulate_horiz_tracer_advection_tend_mono_FCT", L, T, a["hpi"], h, a["ho"], tr, a["tp"], a["tend"],
            dt)
    dm.call("oc_tracer_hmix_del2_tend", L, T, hE, tr, a["tend"], 1e4)
    S.call("oc_provisional_layer_thicknesses", om, st, cfg, h, b["ntf"], b["hp"], b["hp"], b["hpi"], b["hni"], dt)
    S.call("oc_low_order", om, st, cfg, b["ntf"], tr, b["lo"])
    S.call("oc_high_order", om, st, cfg, b["ntf"], tr, b["ho"])
    S.call("oc_correct_and_rescale", om, st, cfg, b["hpi"], h, b["ntf"], b["lo"], tr, b["ho"], b["fi"], b["fo"],
           b["tend"], b["mx"], b["mn"], dt)
    S.call("oc_accumulate_fct", om, st, cfg, b["hpi"], h, b["ho"], tr, b["tp"], b["tend"], dt)
    S.call("oc_hmix_del2", om, st, cfg, hE, tr, b["tend"], 1e4)
    for k in a:
        assert np.array_equal(a[k], b[k]), k


def test_prepared_thickness_on_a_mesh_that_fills_the_gpu():
    """The thickness flux and 1/hProv in two launches (158,000 cell-levels and more)
    against the oracle: a level-5 sphere of 16 levels, one step, value for value."""
    import mpaso.gpu as G
    mesh = mpaso.Mesh.icosa(5)
    L, T, dt = 16, 1, 600.0
    f = fct_statics(mesh, L)
    h, hE, u, tr = ocean_state(mesh, 6, L, T)
    rng = np.random.default_rng(9)
    h, hE = h * rng.uniform(0.9, 1.1, h.shape), hE * rng.uniform(0.9, 1.1, hE.shape)
    u[rng.uniform(size=u.shape) < 0.1] = 0.0
    opts = dict(fct=True, hmix=True, kappa=1e4)
    S = Oracle("restatement")
    want = S.ocean_run(mesh, S.static(mesh, f), S.config(L, T, **opts), dt, 1, h, hE, u, tr)
    dm = G.DeviceMesh(mesh, fct=f)
    st = G.State(dm, app=G.APP_OCEAN, nlev=L, ntr=T, **opts)
    for field, a in ((G.FIELD_H, h), (G.FIELD_LAYER_THICKNESS_EDGE, hE), (G.FIELD_U, u), (G.FIELD_TRACERS, tr)):
        st.set(field, a)
    st.step(dt, 1)
    got = st.get(G.FIELD_TRACERS)
    assert np.array_equal(got, np.asarray(want).reshape(got.shape))
