"""Correlation-matrix fields whose factor overflows: a rotated kernel grows
without bound across it, so short correlation lengths give infinite entries.
The reference then writes infinite values in the first cells and NaN (no value)
in the later ones; which is which is the same here."""
import numpy as np
import pytest

import scenes
import sphgpu
from checkers import rf_oracle

pytestmark = pytest.mark.gpu


# one panel of the factorisation, where the order of the sums is the reference's
@pytest.mark.parametrize("beta,rl", [(30.0, 0.0005), (30.0, 0.003), (60.0, 0.01), (60.0, 0.001), (90.0, 0.003)])
def test_infinite_entries(beta, rl):
    sc = scenes.slope_2d(H=1.5, dx=0.1, crest=3.2)
    st = scenes.initialise(sc)
    eng = sphgpu.Engine(st.params, device=0)
    eng.load_state(st.fields, st.fluid, st.soil)
    d = scenes.kl_domain(sc)
    dom = sphgpu.kl_domain(d["nb_min"], d["nb_max"], d["soil_max"], d["water_max"])
    f = {"no": 1, "type": 1, "mean": 10.0e3, "sd": 3.0e3, "rl": [3.0, rl, 1.0], "coe_depth": 100.0, "flag_auto": 3,
         "cell_ndx": 4.2368, "beta": beta}
    z = np.random.default_rng(1).standard_normal(64)
    err, want, n = rf_oracle(2, sc.xp, sc.ptype, sc.dr, f, d, z)
    assert err == 0 and n == 64 and np.isinf(want).any()
    fl = sphgpu.rf_flags(f["cell_ndx"], 3, beta)
    got = eng.rf_generate(dom, [sphgpu.kl_field(1, 1, 10.0e3, 3.0e3, f["rl"], 100.0)], fl, z[None])[0]
    eng.close()
    assert np.array_equal(np.isnan(got), np.isnan(want))
    assert np.array_equal(np.where(np.isinf(got), got, 0.0), np.where(np.isinf(want), want, 0.0))
