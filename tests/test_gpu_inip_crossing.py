"""Steps on both sides of inip: the passes that take the viscosity sums change
when the damping ends, whatever calls the steps come in."""
import numpy as np
import pytest

import scenes
from checkers import ORC_JACOBI, ORC_POW_CR, STATE_FIELDS, Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ndim", (2, 3))
@pytest.mark.parametrize("calls", ((8,), (1,) * 8, (3, 1, 4)))
def test_damped_then_free(ndim, calls):
    import sphgpu
    sc = scenes.slope_2d(H=1.0, dx=0.1) if ndim == 2 else scenes.soil_column_3d(dx=0.1)
    sc.problem["inip"] = 3
    st = scenes.initialise(sc)
    rng = np.random.default_rng(1)
    free = ((st.fields["type"] == 1) | (st.fields["type"] == 2))[:, None]
    st.fields["vxp"] = st.fields["vxp"] + np.where(free, 0.05 * rng.standard_normal((sc.n, 3)), 0.0) * \
        (1.0, 1.0, float(ndim == 3))
    st.fields["cd"] = np.where(free[:, 0], 0.5, 0.0)
    orc = Oracle(st.params, ORC_JACOBI, ORC_POW_CR)
    eng = sphgpu.Engine(st.params, device=0)
    for q in (orc, eng):
        q.load_state(st.fields, st.fluid, st.soil)
    assert orc.step(sum(calls)) == 0
    for n in calls:
        eng.step(n)
    for f in STATE_FIELDS:
        assert np.array_equal(eng.get_field(f), orc.get_field(f)), f
    eng.close()
