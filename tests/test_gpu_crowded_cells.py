"""Cells that hold hundreds to hundreds of thousands of particles out of the
calculation (type 7, as water that left the box becomes): the order within
them is still the reference's, and it costs in proportion to their number."""
import numpy as np
import pytest

import scenes
from checkers import ORC_JACOBI, ORC_POW_CR, Oracle

pytestmark = pytest.mark.gpu

DR = 0.1


def _state(ndim, xp, out):
    n = len(xp)
    sc = scenes.slope_2d(H=1.0, dx=DR) if ndim == 2 else scenes.soil_column_3d(dx=DR, with_water=False)
    sc.xp, sc.vxp = np.array(xp, dtype=np.float64), np.zeros((n, 3))
    sc.ptype, sc.matype = np.full(n, 2, np.int32), np.full(n, 2, np.int32)
    sc.permtype, sc.etype = np.zeros(n, np.int32), np.ones(n, np.int32)
    st = scenes.initialise(sc)
    st.fields["type"] = np.where(out, 7, 2).astype(np.int32)
    return st


def _cell_corner(ndim, k):
    """The lower corner of the k-th cell along each axis, for particles from 0 to 40 DR."""
    st = _state(ndim, [(0.0,) * 3, (40 * DR, 40 * DR, 40 * DR * (ndim == 3))], np.zeros(2, bool))
    lo = np.array([st.params[q] for q in ("xmin", "ymin", "zmin")])
    return np.where(np.arange(3) < ndim, lo + 2 * DR * k, 0.0)


@pytest.mark.parametrize("ndim", (2, 3))
@pytest.mark.parametrize("count", (257, 511, 512, 513, 700, 768, 3000, 70000))
def test_order_in_a_crowded_cell(ndim, count):
    """`count` particles in one cell, about 60 of them within reach of the live
    particles in the cell diagonally below, in shuffled order."""
    import sphgpu
    rng = np.random.default_rng(count)
    flat = np.array((1.0, 1.0, float(ndim == 3)))
    c = _cell_corner(ndim, 10)
    near = 60
    xp = c + flat * 2 * DR * np.concatenate([0.02 + 0.1 * rng.random((near, 3)),
                                             0.9 + 0.09 * rng.random((count - near, 3))])
    live = c - flat * 2 * DR * (0.05 + 0.3 * rng.random((20, 3)))
    ends = np.array([(0.0,) * 3, 40 * DR * flat])
    xp = np.concatenate([ends, xp, live])
    out = np.zeros(len(xp), bool)
    out[2:2 + count] = True
    order = rng.permutation(len(xp))
    st = _state(ndim, xp[order], out[order])
    orc = Oracle(st.params, ORC_JACOBI, ORC_POW_CR)
    orc.load_state(st.fields, st.fluid, st.soil)
    eng = sphgpu.Engine(st.params, device=0)
    eng.load_state(st.fields, st.fluid, st.soil)
    err, n2, i2, _ = orc.nnps()
    n1, i1 = eng.nnps()
    eng.close()
    assert err == 0
    alive = st.fields["type"] == 2
    listed = (np.arange(100) >= 1) & (np.arange(100) <= n2[:, None]) & alive[:, None]
    assert np.array_equal(n1[alive], n2[alive])
    assert np.array_equal(np.where(listed, i1, 0), np.where(listed, i2, 0))
    assert n1[alive].max() >= 40


def test_the_cost_is_in_proportion():
    import sphgpu
    t = {}
    for count in (100000, 400000):
        rng = np.random.default_rng(count)
        xp = np.concatenate([np.array([(0.0, 0.0, 0.0), (4.0, 4.0, 0.0)]),
                             _cell_corner(2, 10) + 2 * DR * rng.random((count, 3)) * (1.0, 1.0, 0.0)])
        out = np.arange(count + 2) >= 2
        st = _state(2, xp, out)
        eng = sphgpu.Engine(st.params, device=0)
        eng.load_state(st.fields, st.fluid, st.soil)
        t[count] = min(eng.step_profiled(1)["k_cellrange"] for _ in range(5))
        eng.close()
    print("k_cellrange: %.3f ms for 100,000 in one cell, %.3f for 400,000" % (t[100000], t[400000]))
    assert t[400000] < 7.0 * t[100000]          # in proportion 4, with the square 16
