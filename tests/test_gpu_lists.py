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


def _search_equal(xp, ndim, dr, h=None):
    """The engine's whole lists against the oracle's for soil particles at xp."""
    import sphgpu
    n = len(xp)
    sc = scenes.slope_2d(H=1.0, dx=dr) if ndim == 2 else scenes.soil_column_3d(dx=dr, with_water=False)
    sc.xp, sc.vxp = np.array(xp, dtype=np.float64), np.zeros((n, 3))
    sc.ptype, sc.matype = np.full(n, 2, np.int32), np.full(n, 2, np.int32)
    sc.permtype, sc.etype = np.zeros(n, np.int32), np.ones(n, np.int32)
    st = scenes.initialise(sc)
    if h is not None:
        st.fields["hl"] = np.asarray(h, dtype=np.float64)
    orc = Oracle(st.params, ORC_JACOBI, ORC_POW_CR)
    orc.load_state(st.fields, st.fluid, st.soil)
    err, n2, i2, _ = orc.nnps()
    eng = sphgpu.Engine(st.params, device=0)
    eng.load_state(st.fields, st.fluid, st.soil)
    if err:
        with pytest.raises(sphgpu.SPHError) as e:
            eng.nnps()
        assert e.value.code == err
        eng.close()
        return err
    n1, i1 = eng.nnps()
    eng.close()
    listed = (np.arange(100) >= 1) & (np.arange(100) <= n1[:, None])
    assert np.array_equal(n1, n2)
    assert np.array_equal(np.where(listed, i1, 0), np.where(listed, i2, 0))
    return int(n1.max())


@pytest.mark.parametrize("ndim", (2, 3))
@pytest.mark.parametrize("count", (1, 31, 33, 64, 65, 100, 101))
def test_crowded_cells(ndim, count):
    """Cells of one word of candidate bits and more; 99 neighbours and one too
    many (error 5)."""
    rng = np.random.default_rng(count)
    dr = 0.1
    xp = rng.random((count + 40, 3)) * 0.9 * dr + 5 * dr          # one cell, all within reach
    xp[count:] = 12 * dr + rng.random((40, 3)) * 9 * dr           # a few around
    if ndim == 2:
        xp[:, 2] = 0.0
    got = _search_equal(xp, ndim, dr)
    assert got == (5 if count > 100 else max(got, count - 1))


@pytest.mark.parametrize("ndim", (2, 3))
def test_unequal_h(ndim):
    rng = np.random.default_rng(3)
    dr, n = 0.1, 300
    xp = rng.random((n, 3)) * (1.5 if ndim == 2 else 0.9)
    if ndim == 2:
        xp[:, 2] = 0.0
    _search_equal(xp, ndim, dr, dr * rng.choice((0.4, 0.7, 1.0), n))


def test_far_from_the_grid_origin():
    """Coordinates so large against h that FP32 differences decide nothing."""
    rng = np.random.default_rng(4)
    dr = 0.1
    xp = rng.random((200, 3)) * 1.5
    xp[100:, 0] += 0.4e6 * dr
    xp[:, 2] = 0.0
    _search_equal(xp, 2, dr)


@pytest.mark.parametrize("cells", ((31, 33), (32, 32), (64, 64), (41, 75), (200, 3), (3, 5)))
def test_cell_counts_around_the_scan_blocks(cells):
    """Grids whose number of cells is at, one past and far from a multiple of
    what a block of the cell scan takes; particles at every corner."""
    rng = np.random.default_rng(sum(cells))
    dr = 0.1
    ext = [2 * dr * (c - 2.5) - 4 * dr for c in cells]           # celllist_ini1 then gives these counts
    xp = np.zeros((600, 3))
    for k in range(2):
        xp[:, k] = rng.random(600) * max(ext[k], 0.05)
        xp[:4, k] = (0.0, max(ext[k], 0.05)) * 2 if k else (0.0, 0.0, max(ext[0], 0.05), max(ext[0], 0.05))
    _search_equal(xp[:max(8, min(600, 4 * cells[0] * cells[1]))], 2, dr)
