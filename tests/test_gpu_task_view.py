"""The per-task entries on device arrays in the reference's numbering: every
context ordering gives what host arrays give (which the oracle pins), also for
arrays on an odd 8-byte offset and for an output that shares memory with an
input, and entries a task leaves untouched keep their values."""
import ctypes

import numpy as np
import pytest

import mpaso
from mpaso.setup import fct_statics

pytestmark = pytest.mark.gpu


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def _dev(torch, a, off):
    """Device copy of `a` starting `off` doubles into its allocation."""
    buf = torch.zeros(a.size + off, dtype=torch.float64, device="cuda")
    t = buf[off:].view(a.shape)
    t.copy_(torch.from_numpy(a))
    return t


@pytest.mark.parametrize("reorder", [0, 1, 2, 3])
@pytest.mark.parametrize("spec", [("icosa", 2), ("hex", 9, 6)])
@pytest.mark.parametrize("off", [0, 1])
def test_device_arrays_equal_host_arrays(spec, reorder, off):
    torch = pytest.importorskip("torch")
    import mpaso.gpu as G
    from mpaso._lib import check, lib
    mesh = mpaso.Mesh.icosa(spec[1]) if spec[0] == "icosa" else mpaso.Mesh.hex(spec[1], spec[2], 20e3, 1e-4)
    L, T, dt = 3, 2, 100.0
    maxlev = np.full(mesh.nCells, L, np.int32)
    maxlev[::5] = L - 1  # columns with untouched levels
    dm = G.DeviceMesh(mesh, fct=fct_statics(mesh, L, maxLevelCell=maxlev), reorder=reorder)
    nC, nE, nV = mesh.nCells, mesh.nEdges, mesh.nVertices
    rng = np.random.default_rng(5)
    c = lambda *s: rng.uniform(0.5, 1.5, (nC, L) + s)  # noqa: E731
    e = lambda *s: rng.standard_normal((nE, L) + s)  # noqa: E731
    v = lambda: rng.standard_normal((nV, L))  # noqa: E731
    ctd = ctypes.c_double
    calls = [
        ("sw_compute_solve_diagnostics", (c(), e(), e(), v(), v(), v(), c(), e(), v()), ()),
        ("sw_compute_tend", (e(), c(), e(), c(), e(), c(), e()), ()),
        ("sw_compute_scalar_tend", (T, e(), e(), c(T), c(T)), ()),
        ("oc_calc_provisional_layer_thicknesses", (c(), e(), c(), c(), c()), (dt,)),
        ("oc_calc_horiz_tracer_advection_flux_mono_low_order", (T, e(), c(T), e(T)), ()),
        ("oc_calc_horiz_tracer_advection_flux_mono_high_order", (T, e(), c(T), e(T)), ()),
        ("oc_correct_and_rescale_high_order_mono_horiz_flux",
         (T, c(), c(), e(), e(T), c(T), e(T), c(T), c(T), c(T), c(T), c(T)), (dt,)),
        ("oc_accumulate_horiz_tracer_advection_tend_mono_FCT", (T, c(), c(), e(T), c(T), c(T), c(T)), (dt,)),
        ("oc_tracer_hmix_del2_tend", (T, e(), c(T), c(T)), (1e4,)),
    ]
    for name, args, tail in calls:
        host = [a if isinstance(a, int) else a.copy() for a in args]
        dev = [a if isinstance(a, int) else _dev(torch, a, off) for a in args]
        torch.cuda.synchronize()
        for arrs in (host, dev):
            conv = [ctypes.c_int32(a) if isinstance(a, int) else
                    (a.ctypes.data_as(ctypes.c_void_p) if isinstance(a, np.ndarray) else _ptr(a)) for a in arrs]
            check(getattr(lib(), "mpaso_" + name)(dm.handle, ctypes.c_int32(L), *conv, *[ctd(x) for x in tail], None))
        torch.cuda.synchronize()
        for k, (a, b) in enumerate(zip(host, dev)):
            if not isinstance(a, int):
                assert np.array_equal(a, b.cpu().numpy()), (name, k)


def test_output_sharing_memory_with_an_input():
    torch = pytest.importorskip("torch")
    import mpaso.gpu as G
    from mpaso._lib import check, lib
    mesh = mpaso.Mesh.icosa(3)
    L, T = 2, 2
    dm = G.DeviceMesh(mesh)
    rng = np.random.default_rng(6)
    hE, u = rng.uniform(1, 2, (mesh.nEdges, L)), rng.standard_normal((mesh.nEdges, L))
    tr = rng.uniform(0, 1, (mesh.nCells, L, T))
    want = dm.sw_compute_scalar_tend(L, T, hE, u, tr)
    d = [_dev(torch, a, 0) for a in (hE, u, tr)]
    torch.cuda.synchronize()
    check(lib().mpaso_sw_compute_scalar_tend(dm.handle, L, T, _ptr(d[0]), _ptr(d[1]), _ptr(d[2]), _ptr(d[2]), None))
    torch.cuda.synchronize()
    assert np.array_equal(d[2].cpu().numpy(), want)


def test_first_task_call_on_a_mesh_recorded_into_a_graph():
    torch = pytest.importorskip("torch")
    import mpaso.gpu as G
    from mpaso._lib import check, lib
    mesh = mpaso.Mesh.icosa(2)
    L, T = 2, 2
    dm = G.DeviceMesh(mesh)
    rng = np.random.default_rng(7)
    hE, u = rng.uniform(1, 2, (mesh.nEdges, L)), rng.standard_normal((mesh.nEdges, L))
    tr = rng.uniform(0, 1, (mesh.nCells, L, T))
    d = [_dev(torch, a, 0) for a in (hE, u, tr, np.zeros_like(tr))]
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        check(lib().mpaso_sw_compute_scalar_tend(dm.handle, L, T, *[_ptr(x) for x in d],
                                                 ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    assert not d[3].any()
    g.replay()
    torch.cuda.synchronize()
    assert np.array_equal(d[3].cpu().numpy(), dm.sw_compute_scalar_tend(L, T, hE, u, tr))
