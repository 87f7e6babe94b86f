"""An expansion of more terms than shared memory holds is refused, and the
context goes on as if it had not been asked."""
import numpy as np
import pytest

import scenes
import sphgpu
from checkers import ORC_JACOBI, ORC_POW_CR, STATE_FIELDS, Oracle

pytestmark = pytest.mark.gpu


def test_too_many_terms():
    st = scenes.initialise(scenes.slope_2d(H=1.0, dx=0.1))
    orc = Oracle(st.params, ORC_JACOBI, ORC_POW_CR)
    eng = sphgpu.Engine(st.params, device=0)
    for q in (orc, eng):
        q.load_state(st.fields, st.fluid, st.soil)
    # a domain and lengths at which the bisection of all roots converges
    dom = sphgpu.kl_domain((0.0, 0.0, 0.0), (2000.0, 2000.0, 0.0), 2000.0, 2000.0)
    K = 16000
    with pytest.raises(sphgpu.SPHError):
        eng.kl_generate(dom, [sphgpu.kl_field(0, 1, 30.0, 3.0, [20.0, 20.0, 0.0], 0.0)], np.zeros((1, K)), K)
    eng.nnps()
    eng.step(2)
    eng.step_profiled(1)
    assert orc.step(3) == 0
    for f in STATE_FIELDS:
        assert np.array_equal(eng.get_field(f), orc.get_field(f)), f
    eng.close()
