"""The level-0 sphere: twelve pentagons, the one mesh whose cells all have fewer
than the six slots that the kernels unroll.  Steps against the oracle at the
bars of the other meshes (1e-12 after one step, the ocean's value for value),
gradients by the dot-product identity against the complex-step tangent (1e-10
of the sum of |terms|)."""
import numpy as np
import pytest

import mpaso
from helpers import rel_max
from mpaso.initial import ocean_state, sw_state
from mpaso.setup import fct_statics
from oracle import Oracle

pytestmark = pytest.mark.gpu

L, DT = 2, 600.0


def dot(a, b):
    return float(sum((x.ravel() * y.ravel()).sum() for x, y in zip(a, b)))


@pytest.mark.parametrize("configured", [False, True])
@pytest.mark.parametrize("T", [0, 1, 3])
def test_sw_step(T, configured):
    import mpaso.gpu as G
    mesh = mpaso.Mesh.icosa(0)
    f = fct_statics(mesh, L)
    h, u, tr = sw_state(mesh, 3, L, T)
    opts = dict(fct=T > 0, hmix=T > 0, kappa=1e6 if T else 0.0, nu=1e4)
    S = Oracle("restatement")
    want = S.sw_run(mesh, S.static(mesh, f), S.config(L, T, **opts), DT, 1, h, u, tr)
    dm = G.DeviceMesh(mesh, fct=f)
    st = G.State(dm, nlev=L, ntr=T, **opts)
    if configured:
        st.set_launch_config([1] * 3, [128] * 3)
    fields = (G.FIELD_H, G.FIELD_U, G.FIELD_TRACERS)[:3 if T else 2]
    for field, a in zip(fields, (h, u, tr)):
        st.set(field, a)
    st.step(DT, 1)
    for field, w in zip(fields, want):
        got = st.get(field)
        assert rel_max(got, np.asarray(w).reshape(got.shape)) < 1e-12


@pytest.mark.parametrize("T", [1, 3])
def test_ocean_step(T):
    import mpaso.gpu as G
    mesh = mpaso.Mesh.icosa(0)
    f = fct_statics(mesh, L)
    h, hE, u, tr = ocean_state(mesh, 4, L, T)
    opts = dict(fct=True, hmix=True, kappa=1e6)
    S = Oracle("restatement")
    want = S.ocean_run(mesh, S.static(mesh, f), S.config(L, T, **opts), DT, 2, h, hE, u, tr)
    dm = G.DeviceMesh(mesh, fct=f)
    st = G.State(dm, app=G.APP_OCEAN, nlev=L, ntr=T, **opts)
    for field, a in ((G.FIELD_H, h), (G.FIELD_LAYER_THICKNESS_EDGE, hE), (G.FIELD_U, u), (G.FIELD_TRACERS, tr)):
        st.set(field, a)
    st.step(DT, 2)
    got = st.get(G.FIELD_TRACERS)
    assert np.array_equal(got, np.asarray(want).reshape(got.shape))


@pytest.mark.parametrize("T,fct", [(0, False), (2, True), (1, False)])
def test_sw_gradient(T, fct):
    import mpaso.gpu as G
    from sw_complex import SwComplex
    mesh = mpaso.Mesh.icosa(0)
    f = fct_statics(mesh, L)
    h, u, tr = sw_state(mesh, 3, L, T)
    rng = np.random.default_rng(11)
    tr = 0.7 * tr + 0.3 * rng.uniform(0.0, 1.0, tr.shape)
    w = (rng.standard_normal(h.shape), rng.standard_normal(u.shape) * 100, rng.standard_normal(tr.shape) * 1e3)
    v = (rng.standard_normal(h.shape), rng.standard_normal(u.shape) * 1e-3, rng.standard_normal(tr.shape) * 1e-2)
    dm = G.DeviceMesh(mesh, fct=f)
    st = G.State(dm, nlev=L, ntr=T, fct=fct, nu=1e5)
    fields = (G.FIELD_H, G.FIELD_U, G.FIELD_TRACERS)[:3 if T else 2]
    for field, a in zip(fields, (h, u, tr)):
        st.set(field, a)
    st.forward(DT, 4, 2)
    C = SwComplex(mesh, L, fct=f, centred=not fct, T=T, nu=1e5)
    if T:
        g, jv = st.vjp_tracers(*w), C.jvp_tracers(h, u, tr, *v, DT, 4)
    else:
        g, jv = st.vjp(*w[:2]), C.jvp(h, u, *v[:2], DT, 4)
    scale = sum(np.abs(x.ravel() * y.ravel()).sum() for x, y in zip(w, jv))
    assert abs(dot(w, jv) - dot(g, v)) <= 1e-10 * scale


@pytest.mark.parametrize("T", [1, 2, 3])
def test_ocean_gradient(T):
    import mpaso.gpu as G
    from sw_complex import SwComplex
    mesh = mpaso.Mesh.icosa(0)
    f = fct_statics(mesh, L)
    h, hE, u, tr = ocean_state(mesh, 7, L, T, clip=False)
    rng = np.random.default_rng(3)
    tr = 0.7 * tr + 0.3 * tr.max() * rng.uniform(0.0, 1.0, tr.shape)
    w, v = rng.standard_normal(tr.shape), rng.standard_normal(tr.shape)
    dm = G.DeviceMesh(mesh, fct=f)
    opts = dict(fct=True, hmix=True, kappa=1e5)
    st = G.State(dm, app=G.APP_OCEAN, nlev=L, ntr=T, **opts)
    for field, a in ((G.FIELD_H, h), (G.FIELD_LAYER_THICKNESS_EDGE, hE), (G.FIELD_U, u), (G.FIELD_TRACERS, tr)):
        st.set(field, a)
    st.forward(DT, 4, 2)
    _, _, gt = st.vjp_tracers(np.zeros(h.shape), np.zeros(u.shape), w)
    C = SwComplex(mesh, L, fct=f, centred=False, T=T, hmix=True, kappa=1e5)
    jv = C.ocean_jvp(h, hE, u, tr, v, DT, 4)
    assert abs(float((w * jv).sum()) - float((gt * v).sum())) <= 1e-10 * np.abs(w * jv).sum()
