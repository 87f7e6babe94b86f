"""The rate of the correlation matrix's factorisation: its trailing updates are
nearly all of it at 13,248 cells, and ran a fifth slower on the FP64 tensor cores
than as multiply-adds on registers."""
import time

import numpy as np
import pytest

import scenes
import sphgpu

pytestmark = pytest.mark.gpu


def test_factor_of_many_cells_at_a_third_of_the_fp64_rate():
    sc = scenes.slope_2d(H=5.0, dx=0.1)
    st = scenes.initialise(sc)
    d = scenes.kl_domain(sc)
    dom = sphgpu.kl_domain(d["nb_min"], d["nb_max"], d["soil_max"], d["water_max"])
    ext = 1.2 * (np.array(d["nb_max"]) - np.array(d["nb_min"]))
    fl = sphgpu.rf_flags(1.03 * float(np.sqrt(ext[0] * ext[1] / 14000) / sc.dr), 1)
    eng = sphgpu.Engine(st.params, device=0)
    eng.load_state(st.fields, st.fluid, st.soil)
    n = eng.rf_cells(dom, fl)
    assert n > 13000
    # two fields of different lengths have a factor each: the difference from
    # one field's call leaves the material records out
    fields = [sphgpu.kl_field(1, 2, 10.0e3, 3.0e3, [lx, 1.5, 0.0], 100.0) for lx in (6.0, 5.0)]
    z = np.random.default_rng(3).standard_normal((2, n))
    best = {}
    for k in (1, 2):
        eng.rf_generate(dom, fields[:k], fl, z[:k])
        took = []
        for _ in range(5):
            t = time.perf_counter()
            eng.rf_generate(dom, fields[:k], fl, z[:k])
            took.append(time.perf_counter() - t)
        best[k] = min(took)
    eng.close()
    fp64, _ = sphgpu.pipe_peaks(0)
    assert n ** 3 / 3.0 / (best[2] - best[1]) / 1e12 > fp64 / 3.0
