"""Each per-task entry that reads the FCT statics as the first task call on a mesh
context gives what it gives after other tasks ran there (the context makes what
the tasks share in whichever comes first), and still refuses a level count other
than the statics'."""
import numpy as np
import pytest

import mpaso
from mpaso.setup import fct_statics

pytestmark = pytest.mark.gpu

L, T = 3, 2


def _calls(mesh):
    rng = np.random.default_rng(11)
    c = lambda *s: rng.uniform(0.5, 1.5, (mesh.nCells, L) + s)  # noqa: E731
    e = lambda *s: rng.standard_normal((mesh.nEdges, L) + s)  # noqa: E731
    return {"oc_calc_horiz_tracer_advection_flux_mono_high_order": (T, e(), c(T), e(T)),
            "oc_correct_and_rescale_high_order_mono_horiz_flux":
                (T, c(), c(), e(), e(T), c(T), e(T), c(T), c(T), c(T), c(T), c(T), 100.0),
            "oc_accumulate_horiz_tracer_advection_tend_mono_FCT": (T, c(), c(), e(T), c(T), c(T), c(T), 100.0)}


@pytest.mark.parametrize("reorder", [0, 1])
@pytest.mark.parametrize("name", ["oc_calc_horiz_tracer_advection_flux_mono_high_order",
                                  "oc_correct_and_rescale_high_order_mono_horiz_flux",
                                  "oc_accumulate_horiz_tracer_advection_tend_mono_FCT"])
def test_fct_task_as_the_first_call_on_a_context(name, reorder):
    import mpaso.gpu as G
    from mpaso._lib import MpasoError
    mesh = mpaso.Mesh.icosa(2)
    f = fct_statics(mesh, L)
    args = _calls(mesh)[name]
    got = []
    for warm in (False, True):
        dm = G.DeviceMesh(mesh, fct=f, reorder=reorder)
        if warm:
            dm.sw_compute_scalar_tend(L, 1, np.ones((mesh.nEdges, L)), np.ones((mesh.nEdges, L)),
                                      np.ones((mesh.nCells, L, 1)))
        with pytest.raises(MpasoError, match="level count"):
            dm.call(name, L - 1, *args)
        a = [x.copy() if isinstance(x, np.ndarray) else x for x in args]
        dm.call(name, L, *a)
        got.append([x for x in a if isinstance(x, np.ndarray)])
        dm.close()
    for x, y in zip(*got):
        assert np.array_equal(x, y)
