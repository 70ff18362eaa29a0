"""The configuration that a state begins with names the launch rules: reading it,
running another and setting it back returns to them, on this state and on others;
and the autotuner keeps them where they are faster than any configuration (a small
sphere without tracers: nine fused launches a step against twelve, by a sixth)."""
import numpy as np
import pytest

import mpaso
from mpaso.initial import sw_state

pytestmark = pytest.mark.gpu


def _state(level, T=0):
    import mpaso.gpu as G
    mesh = mpaso.Mesh.icosa(level)
    h, u, _ = sw_state(mesh, 3, 1, T)
    st = G.State(G.DeviceMesh(mesh), nlev=1, ntr=T, nu=1e4)
    st.set(G.FIELD_H, h)
    st.set(G.FIELD_U, u)
    return st


def test_first_configuration_set_again():
    st, other = _state(3), _state(2)
    first = st.launch_config()
    for s in (st, other):
        assert s.launches_per_step() == 9
        s.set_launch_config([1] * 3, [128] * 3)
        assert s.launches_per_step() == 12
        s.set_launch_config([1] * 3, [256] * 3, lanes=2)
        assert s.launches_per_step() == 12
        s.set_launch_config(**first)
        assert s.launch_config() == first and s.launches_per_step() == 9


@pytest.mark.parametrize("level", [3, 4])
def test_autotuner_keeps_the_faster_untuned_form(level):
    import mpaso.gpu as G
    st = _state(level)
    first, u = st.launch_config(), st.get(G.FIELD_U)
    assert st.autotune(60.0, 3) == first
    assert st.launch_config() == first and st.launches_per_step() == 9
    assert np.array_equal(st.get(G.FIELD_U), u)
    st.step_graph(60.0, 2)
    assert np.isfinite(st.get(G.FIELD_U)).all()
