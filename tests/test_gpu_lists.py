"""The two-group neighbour lists: results do not depend on how a list is held,
and reading the lists whole (sphgpu_nnps) between the method entries of a step
leaves the step as it was."""
import numpy as np
import pytest

import scenes
from checkers import ORC_JACOBI, ORC_POW_CR, STATE_FIELDS, Oracle

pytestmark = pytest.mark.gpu


def _three_phase():
    return scenes.rain_slope_3d(dx=0.5, H=2.0, crest=2.0, width=2.0, length=6.0, rows=1, steps=40)


SCENES = {
    "water": lambda: scenes.dam_break_2d(dx=0.04),
    "saturated soil": lambda: scenes.soil_column_3d(dx=0.1),
    "soil, air and rain": _three_phase,
    "soil and structure": lambda: scenes.footing(ndim=2, dx=0.05, ss_type=3),
}


@pytest.mark.parametrize("name", sorted(SCENES))
def test_lists_read_between_search_and_update(name):
    import sphgpu
    st = scenes.initialise(SCENES[name]())
    orc = Oracle(st.params, ORC_JACOBI, ORC_POW_CR)
    orc.load_state(st.fields, st.fluid, st.soil, st.rain)
    eng = sphgpu.Engine(st.params, device=0)
    eng.load_state(st.fields, st.fluid, st.soil, st.rain)
    for _ in range(3):
        assert eng.parttocell() == 0 and eng.partisearching() == 0
        n1, i1 = eng.nnps()
        assert eng.update() == 0
        err, n2, i2, _ = orc.nnps()
        assert err == 0 and np.array_equal(n1, n2)
        listed = (np.arange(100) >= 1) & (np.arange(100) <= n1[:, None])     # the oracle leaves the rest unset
        assert np.array_equal(np.where(listed, i1, 0), np.where(listed, i2, 0))
        assert orc.step(1) == 0
    for f in STATE_FIELDS:
        a, b = eng.get_field(f), orc.get_field(f)
        assert np.array_equal(a, b, equal_nan=a.dtype.kind == "f"), f
    eng.close()
