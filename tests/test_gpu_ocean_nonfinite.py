"""An infinite or NaN tracer in one cell of the ocean app: its high-order fluxes
reach the cells within two rings in each of the four stages, and a flux that is
no number makes a cell's tendency no number whatever its limiter factor (zero at
local extrema among them).  After a step exactly the cells within eight rings, in
that level and tracer, are not finite."""
import numpy as np
import pytest

import mpaso
from mpaso.initial import ocean_state
from mpaso.setup import fct_statics

pytestmark = pytest.mark.gpu


def _rings(mesh, c, n):
    off, idx = mesh.crs()["c2c"]
    seen = np.zeros(mesh.nCells, bool)
    seen[c] = True
    for _ in range(n):
        for k in np.flatnonzero(seen):
            seen[idx[off[k]:off[k + 1]]] = True
    return seen


@pytest.mark.parametrize("value", [np.nan, np.copysign(np.nan, -1.0), np.inf, -np.inf])
@pytest.mark.parametrize("spec,L,T", [(("icosa", 4), 2, 1), (("icosa", 4), 1, 3), (("hex", 24, 22), 2, 2)])
def test_what_is_no_number_spreads(spec, L, T, value):
    import mpaso.gpu as G
    mesh = mpaso.Mesh.icosa(spec[1]) if spec[0] == "icosa" else mpaso.Mesh.hex(spec[1], spec[2], 20e3, 1e-4)
    f = fct_statics(mesh, L)
    assert f["highOrderAdvMask"].all()
    h, hE, u, tr = ocean_state(mesh, 4, L, T)
    rng = np.random.default_rng(5)
    tr = tr * rng.uniform(0.5, 1.5, tr.shape)  # local extrema everywhere
    c, k, t = mesh.nCells // 2, L - 1, T - 1
    tr[c, k, t] = value
    dm = G.DeviceMesh(mesh, fct=f)
    st = G.State(dm, app=G.APP_OCEAN, nlev=L, ntr=T, fct=True)
    for field, a in ((G.FIELD_H, h), (G.FIELD_LAYER_THICKNESS_EDGE, hE), (G.FIELD_U, u), (G.FIELD_TRACERS, tr)):
        st.set(field, a)
    st.step(100.0, 1)
    bad = ~np.isfinite(st.get(G.FIELD_TRACERS))
    want = np.zeros_like(bad)
    want[:, k, t] = _rings(mesh, c, 8)
    assert np.array_equal(bad, want), (int(bad.sum()), int(want.sum()))
