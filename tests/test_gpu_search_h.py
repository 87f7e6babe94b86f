"""The neighbour search for smoothing lengths other than the spacing: the lists
are the oracle's, and a run whose particles all have another h is searched as
fast as one with h = dr (the FP32 test decides its candidates too)."""
import numpy as np
import pytest

import scenes
from test_gpu_lists import _search_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ndim", (2, 3))
@pytest.mark.parametrize("h", ("one smaller", "one larger", "two sizes", "an outlier", "zeros and NaN"))
def test_lists(ndim, h):
    rng = np.random.default_rng(5)
    dr, n = 0.1, 300
    xp = rng.random((n, 3)) * (2.5 if ndim == 2 else 0.9)
    if ndim == 2:
        xp[:, 2] = 0.0
    hl = {"one smaller": np.full(n, 0.7 * dr), "one larger": np.full(n, 1.02 * dr),
          "two sizes": dr * rng.choice((0.5, 1.0), n), "an outlier": np.where(np.arange(n) == 17, 0.01 * dr, 0.8 * dr),
          "zeros and NaN": np.where(np.arange(n) % 50 == 0, np.where(np.arange(n) % 100 == 0, np.nan, 0.0), 0.9 * dr)}[h]
    _search_equal(xp, ndim, dr, hl)


def test_one_other_h_is_searched_as_fast():
    import sphgpu
    sc = scenes.soil_column_3d(dx=0.02)
    rng = np.random.default_rng(6)
    sc.xp = sc.xp + 0.05 * sc.dr * rng.standard_normal((sc.n, 3)).clip(-2.5, 2.5)
    st = scenes.initialise(sc)
    engines = []
    for factor in (1.0, 0.98):
        e = sphgpu.Engine(st.params, device=0)
        e.load_state(dict(st.fields, hl=factor * st.fields["hl"]), st.fluid, st.soil)
        engines.append(e)
    t = [[], []]
    for _ in range(6):
        for k, e in enumerate(engines):
            t[k].append(e.step_profiled(3)["k_nnps"])
    for e in engines:
        e.close()
    same, other = min(t[0]), min(t[1])
    print("k_nnps, 3 steps: h = dr %.3f ms, h = 0.98 dr %.3f ms" % (same, other))
    assert other < 1.3 * same
