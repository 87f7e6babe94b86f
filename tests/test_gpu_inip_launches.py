"""A call whose steps cross inip launches past it what a call of its own would:
the own-type loop of the damped steps ends with them."""
import numpy as np
import pytest

import scenes
import sphgpu
from checkers import STATE_FIELDS

pytestmark = pytest.mark.gpu


def _engine(ndim, inip, precision):
    sc = scenes.slope_2d(H=1.0, dx=0.1) if ndim == 2 else scenes.soil_column_3d(dx=0.1)
    sc.problem["inip"] = inip
    st = scenes.initialise(sc)
    eng = sphgpu.Engine(st.params, device=0)
    eng.load_state(st.fields, st.fluid, st.soil)
    eng.set_precision(precision)
    return eng


@pytest.mark.parametrize("ndim", (2, 3))
@pytest.mark.parametrize("inip,steps", [(1, 2), (3, 8), (7, 8), (8, 8)])
@pytest.mark.parametrize("precision", (sphgpu.PREC_FP64, sphgpu.PREC_FP32_BULK))
def test_one_call_as_two(ndim, inip, steps, precision):
    one, two = _engine(ndim, inip, precision), _engine(ndim, inip, precision)
    one.step(steps)
    two.step(inip)
    launches = two.last_step_launches()
    if steps > inip:
        two.step(steps - inip)
        launches += two.last_step_launches()
    assert one.last_step_launches() == launches
    for f in STATE_FIELDS:
        assert np.array_equal(one.get_field(f), two.get_field(f), equal_nan=True), f
    # and the steps after it
    one.step(2)
    two.step(2)
    assert one.last_step_launches() == two.last_step_launches()
    assert np.array_equal(one.get_field("vxp"), two.get_field("vxp"))
    one.close()
    two.close()
