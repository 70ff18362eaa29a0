"""The ocean stage kernels' integer-pipe products at and outside their exponent
window (magnitudes 2^-256 .. 2^256), against the oracle value for value: zeros,
subnormals and factors on both sides of each end, one to three tracers, on
stencils of exactly ten cells and of run-time width."""
import numpy as np
import pytest

import mpaso
from mpaso.initial import ocean_state
from mpaso.setup import fct_statics
from oracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ntr", [1, 2, 3])
@pytest.mark.parametrize("spec", [("icosa", 2), ("hex", 9, 6)])
@pytest.mark.parametrize("exp2", [-1060, -300, -257, -250, 0, 240, 300])
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
