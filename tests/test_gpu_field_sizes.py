"""Random fields at the sizes where their kernels change: correlation matrices
around whole panels of the factorisation."""
import numpy as np
import pytest

import scenes
import sphgpu
from checkers import rf_oracle

pytestmark = pytest.mark.gpu

TOL = 1e-12        # of the field's magnitude, as the golden cases are held


def _engine(sc):
    st = scenes.initialise(sc)
    eng = sphgpu.Engine(st.params, device=0)
    eng.load_state(st.fields, st.fluid, st.soil)
    d = scenes.kl_domain(sc)
    return eng, d, sphgpu.kl_domain(d["nb_min"], d["nb_max"], d["soil_max"], d["water_max"])


def _close(a, b):
    assert np.array_equal(np.isnan(a), np.isnan(b))
    m = ~np.isnan(b)
    if m.any():
        assert np.abs(a[m] - b[m]).max() <= TOL * np.abs(b[m]).max()


# one panel of 64 columns, one more, two, three, four and a rest
@pytest.mark.parametrize("cells,crest,ndx", [(64, 3.2, 4.2368), (65, 1.3, 3.3947), (128, 0.6, 2.1516),
                                             (192, 2.0, 2.1316), (256, 3.4, 2.1216), (260, 1.5, 1.7206)])
def test_matrices_around_whole_panels(cells, crest, ndx):
    sc = scenes.slope_2d(H=1.5, dx=0.1, crest=crest)
    eng, d, dom = _engine(sc)
    f = {"no": 1, "type": 2, "mean": 10.0e3, "sd": 3.0e3, "rl": [3.0, 0.8, 0.0], "coe_depth": 100.0, "flag_auto": 1,
         "cell_ndx": ndx}
    fl = sphgpu.rf_flags(ndx, 1)
    assert eng.rf_cells(dom, fl) == cells
    z = np.random.default_rng(cells).standard_normal(cells)
    err, want, n = rf_oracle(2, sc.xp, sc.ptype, sc.dr, f, d, z)
    assert err == 0 and n == cells
    _close(eng.rf_generate(dom, [sphgpu.kl_field(1, 2, 10.0e3, 3.0e3, [3.0, 0.8, 0.0], 100.0)], fl, z[None])[0], want)
    eng.close()
