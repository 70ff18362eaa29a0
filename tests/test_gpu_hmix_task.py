"""mpaso_oc_tracer_hmix_del2_tend keeps no array of its own between the call and
its launch: recorded into a graph as the first task call on a context, the graph
stays right after calls that make the context's scratch grow; and its values, on
columns of which a thread block holds many, a few or a part, equal the oracle's."""
import ctypes

import numpy as np
import pytest

import mpaso
from mpaso.setup import fct_statics
from oracle import Oracle

pytestmark = pytest.mark.gpu

KAPPA = 1e4


def _fields(mesh, L, T, seed):
    rng = np.random.default_rng(seed)
    return (rng.uniform(1.0, 2.0, (mesh.nEdges, L)), rng.uniform(-1.0, 1.0, (mesh.nCells, L, T)),
            rng.uniform(-1.0, 1.0, (mesh.nCells, L, T)))


def _want(mesh, f, L, T, hE, tr, tend, coef):
    S = Oracle("restatement")
    out = tend.copy()
    S.call("oc_hmix_del2", S.mesh(mesh), S.static(mesh, f), S.config(L, T), hE, tr, out, coef)
    return out


@pytest.mark.parametrize("L", [1, 2, 3, 7, 255, 256, 300])
@pytest.mark.parametrize("spec", [("icosa", 2), ("hex", 9, 6)])
def test_values(spec, L):
    import mpaso.gpu as G
    mesh = mpaso.Mesh.icosa(spec[1]) if spec[0] == "icosa" else mpaso.Mesh.hex(spec[1], spec[2], 20e3, 1e-4)
    f = fct_statics(mesh, L)
    dm = G.DeviceMesh(mesh, fct=f)
    hE, tr, tend = _fields(mesh, L, 2, 1)
    want = _want(mesh, f, L, 2, hE, tr, tend, KAPPA)
    dm.call("oc_tracer_hmix_del2_tend", L, 2, hE, tr, tend, KAPPA)
    assert np.array_equal(tend, want)


def test_recorded_as_the_first_call_and_replayed_after_the_scratch_grew():
    torch = pytest.importorskip("torch")
    import mpaso.gpu as G
    from mpaso._lib import check, lib
    mesh = mpaso.Mesh.icosa(3)
    L, T = 3, 2
    f = fct_statics(mesh, L)
    dm = G.DeviceMesh(mesh, fct=f)
    hE, tr, tend = _fields(mesh, L, T, 2)
    d = [torch.from_numpy(a).cuda() for a in (hE, tr, tend)]
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        check(lib().mpaso_oc_tracer_hmix_del2_tend(
            dm.handle, L, T, *[ctypes.c_void_p(x.data_ptr()) for x in d], ctypes.c_double(KAPPA),
            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    for n in (L, 16):  # host arrays: staged through scratch, twice grown
        e, c, t = _fields(mesh, n, T, 3)
        dm.call("oc_tracer_hmix_del2_tend", n, T, e, c, t, 7.0 * KAPPA)
    g.replay()
    torch.cuda.synchronize()
    want = _want(mesh, f, L, T, hE, tr, tend, KAPPA)
    assert np.array_equal(d[2].cpu().numpy(), want)
