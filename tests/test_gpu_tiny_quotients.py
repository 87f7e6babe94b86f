"""Velocities at the bottom of the FP64 range, as they stand ahead of a
disturbance that spreads by one support per step: the XSPH quotients there are
subnormal, and still the IEEE ones."""
import numpy as np
import pytest

import scenes
import sphgpu
from checkers import ORC_JACOBI, ORC_POW_CR, STATE_FIELDS, Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ndim", (2, 3))
def test_subnormal_velocities(ndim):
    sc = scenes.dam_break_2d(dx=0.04) if ndim == 2 else scenes.soil_column_3d(dx=0.1)
    sc.problem["g"] = (0.0, 0.0, 0.0)
    sc.problem["art_vis"] = ((0.0, 0.0),) * 3
    st = scenes.initialise(sc)
    rng = np.random.default_rng(7)
    free = ((st.fields["type"] == 1) | (st.fields["type"] == 2))[:, None]
    v = rng.standard_normal((sc.n, 3)) * 10.0 ** rng.uniform(-318, -304, (sc.n, 3))
    st.fields["vxp"] = np.where(free, v, 0.0) * (1.0, 1.0, float(ndim == 3))
    st.fields["prep"] = np.zeros(sc.n)
    orc = Oracle(st.params, ORC_JACOBI, ORC_POW_CR)
    eng = sphgpu.Engine(st.params, device=0)
    for q in (orc, eng):
        q.load_state(st.fields, st.fluid, st.soil)
    for _ in range(3):
        eng.step(1)
        assert orc.step(1) == 0
    vx = orc.get_field("vx")[free[:, 0]]
    tiny = (vx != 0.0) & (np.abs(vx) < 2.3e-308)
    assert tiny.mean() > 0.05
    for f in STATE_FIELDS:
        a, b = eng.get_field(f), orc.get_field(f)
        assert np.array_equal(a, b, equal_nan=a.dtype.kind == "f"), f
    eng.close()
