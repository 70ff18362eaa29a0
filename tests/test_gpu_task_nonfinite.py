"""The flux-correction task on infinities, NaN of either sign and huge numbers in
each of its arguments, against the oracle value for value (NaN equal to NaN):
std::max / std::min and the products with a zero weight decide what becomes of
them, not the shortcuts the kernels take for finite numbers."""
import numpy as np
import pytest

import mpaso
from mpaso.setup import fct_statics
from oracle import Oracle

pytestmark = pytest.mark.gpu

VALUES = [np.nan, np.copysign(np.nan, -1.0), np.inf, -np.inf, 1e308, -1e308]
NAMES = ("hpi", "h", "ntf", "lo", "tr", "ho", "fi", "fo", "tend", "mx", "mn")


def _check(spec, T, arg, value, uneven):
    import mpaso.gpu as G
    mesh = mpaso.Mesh.icosa(spec[1]) if spec[0] == "icosa" else mpaso.Mesh.hex(spec[1], spec[2], 20e3, 1e-4)
    L, dt = 3, 100.0
    rng = np.random.default_rng(17)
    maxlev = rng.integers(1, L + 1, mesh.nCells).astype(np.int32) if uneven else np.full(mesh.nCells, L, np.int32)
    f = fct_statics(mesh, L, maxLevelCell=maxlev)
    c = lambda *s: rng.uniform(0.5, 1.5, (mesh.nCells, L) + s)  # noqa: E731
    e = lambda *s: rng.standard_normal((mesh.nEdges, L) + s)  # noqa: E731
    # thicknesses about 1 and fluxes about the cells' areas, so that limiter factors between 0 and 1 occur
    area = float(mesh.fields["areaCell"].mean())
    a = dict(hpi=c(), h=c(), ntf=e(), lo=e(T) * area * 1e-3, tr=c(T), ho=e(T) * area * 1e-3, fi=c(T), fo=-c(T),
             tend=e(T)[:mesh.nCells] * 1e-3, mx=c(T), mn=c(T))
    a[arg].reshape(-1)[rng.integers(0, a[arg].size, 12)] = value
    b = {k: v.copy() for k, v in a.items()}
    dm = G.DeviceMesh(mesh, fct=f)
    S = Oracle("restatement")
    with np.errstate(all="ignore"):
        S.call("oc_correct_and_rescale", S.mesh(mesh), S.static(mesh, f), S.config(L, T), *[b[k] for k in NAMES], dt)
    dm.call("oc_correct_and_rescale_high_order_mono_horiz_flux", L, T, *[a[k] for k in NAMES], dt)
    for k in NAMES:
        assert np.array_equal(a[k], b[k], equal_nan=True), k


@pytest.mark.parametrize("value", VALUES)
@pytest.mark.parametrize("arg", ["hpi", "h", "lo", "ho", "tend"])
@pytest.mark.parametrize("spec,T", [(("icosa", 2), 1), (("hex", 9, 6), 3)])
def test_limiter_factors(spec, T, arg, value):
    """A quotient that is no number counts as 0 (std::max(0, NaN) is 0)."""
    _check(spec, T, arg, value, uneven=False)


@pytest.mark.parametrize("value", VALUES)
@pytest.mark.parametrize("arg", ["ntf", "tr"])
@pytest.mark.parametrize("spec,T", [(("icosa", 2), 1), (("hex", 9, 6), 3)])
def test_centred_flux_of_weight_zero(spec, T, arg, value):
    """Edges with a high-order stencil add the centred flux with a weight of zero,
    and zero times an infinity or NaN is NaN."""
    _check(spec, T, arg, value, uneven=False)


@pytest.mark.parametrize("value", VALUES)
@pytest.mark.parametrize("arg", ["ho", "lo", "fi", "fo", "tr"])
@pytest.mark.parametrize("spec,T", [(("icosa", 2), 1), (("hex", 9, 6), 3)])
def test_levels_below_a_column(spec, T, arg, value):
    """An edge that goes deeper than one of its cells reads that cell's unlimited
    flxIn and flxOut, of which the one its flux does not use counts zero times."""
    _check(spec, T, arg, value, uneven=True)
