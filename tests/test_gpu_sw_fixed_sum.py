"""The sw stage's integer-pipe flux sum (unrolled ten-slot stencils) against the
hardware sums of the run-time stencil loop: ordinary winds, still water, and
winds so small that the products reach the subnormals, on a uniform layer
(where the tendency is the Coriolis term the sum forms), sphere and plane.

Both sums carry at most ten roundings of a term, 1.1e-15 of the largest term;
the bar of 1e-13 of the largest velocity leaves two decades for the four
stages and for sums smaller than their terms."""
import numpy as np
import pytest

import mpaso
from mpaso.initial import sw_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spec", [("icosa", 3), ("hex", 12, 10)])
@pytest.mark.parametrize("exp2", [None, -1060, -960, -800, -770, -700, -300, 0])
@pytest.mark.parametrize("nlev", [1, 3])
def test_unrolled_step_equals_runtime_loops(spec, exp2, nlev):
    import mpaso.gpu as G
    mesh = mpaso.Mesh.icosa(spec[1]) if spec[0] == "icosa" else mpaso.Mesh.hex(spec[1], spec[2], 20e3, 1e-4)
    _, u, _ = sw_state(mesh, 3, nlev, 0)
    u = np.zeros_like(u) if exp2 is None else np.ldexp(u, exp2)
    u[::7] = 0.0
    h = np.full((mesh.nCells, nlev), 4096.0)
    got = []
    for unroll in (1, 0):
        dm = G.DeviceMesh(mesh)
        st = G.State(dm, nlev=nlev, ntr=0)
        st.set_launch_config([unroll] * 3, [64] * 3)
        st.set(G.FIELD_H, h)
        st.set(G.FIELD_U, u)
        st.step(50.0, 1)
        got.append((st.get(G.FIELD_H), st.get(G.FIELD_U)))
        st.close()
        dm.close()
    (h1, u1), (h0, u0) = got
    assert np.isfinite(u1).all() and np.isfinite(h1).all()
    assert np.abs(h1 - h0).max() <= 1e-13 * np.abs(h0).max()
    if exp2 is None:
        assert np.array_equal(u1, u0) and not u1.any()
    else:
        assert np.abs(u1 - u0).max() <= 1e-13 * np.abs(u0).max() + 2.0 ** -1070


@pytest.mark.parametrize("ntr", [0, 1, 2])
@pytest.mark.parametrize("exp2", [None, -960, -700, -512, -505, 0])
def test_gpu_filling_column_equals_its_levels(exp2, ntr):
    """A mesh that fills the GPU forms some products on the integer pipe that a
    smaller one leaves to the hardware, bit for bit the same: two levels of a
    level-5 sphere (61,440 edge-levels, above the line) against each level alone
    (30,720, below it)."""
    import mpaso.gpu as G
    mesh = mpaso.Mesh.icosa(5)
    h, u, tr = sw_state(mesh, 5, 2, ntr)
    tr[::13] = 0.0
    u = np.zeros_like(u) if exp2 is None else np.ldexp(u, exp2)
    u[::11] = 0.0
    dm = G.DeviceMesh(mesh)

    def run(lev):
        st = G.State(dm, nlev=h[:, lev].shape[1], ntr=ntr, hmix=ntr > 0, kappa=1e4, nu=1e4)
        fields = [(G.FIELD_H, h), (G.FIELD_U, u)] + ([(G.FIELD_TRACERS, tr)] if ntr else [])
        for f, a in fields:
            st.set(f, np.ascontiguousarray(a[:, lev]))
        st.step(100.0, 2)
        out = [st.get(f) for f, _ in fields] + [st.get(G.FIELD_VORTICITY), st.get(G.FIELD_PV_VERTEX)]
        st.close()
        return out

    both = run(slice(0, 2))
    for k in range(2):
        for a, b in zip(both, run(slice(k, k + 1))):
            assert np.array_equal(a[:, k:k + 1], b)


@pytest.mark.parametrize("spec", [("icosa", 2), ("icosa", 4), ("hex", 12, 10)])
@pytest.mark.parametrize("nlev", [1, 3])
def test_fused_launches_equal_separate_ones(spec, nlev):
    """Without tracers a small mesh runs the last kernel of a stage with the first
    of the next; a set launch configuration (here the default's block size) runs
    them one by one: bit for bit the same fields and diagnostics."""
    import mpaso.gpu as G
    mesh = mpaso.Mesh.icosa(spec[1]) if spec[0] == "icosa" else mpaso.Mesh.hex(spec[1], spec[2], 20e3, 1e-4)
    h, u, _ = sw_state(mesh, 9, nlev, 0)
    dm = G.DeviceMesh(mesh)
    got = []
    for configured in (False, True):
        st = G.State(dm, nlev=nlev, ntr=0, nu=1e4)
        if configured:
            st.set_launch_config([1] * 3, [64] * 3)
        assert st.launches_per_step() == (12 if configured else 9)
        st.set(G.FIELD_H, h)
        st.set(G.FIELD_U, u)
        st.step(50.0, 2)
        st.step_graph(50.0, 2)
        got.append([st.get(f) for f in (G.FIELD_H, G.FIELD_U, G.FIELD_VORTICITY, G.FIELD_PV_VERTEX)])
        st.close()
    for a, b in zip(*got):
        assert np.array_equal(a, b)
