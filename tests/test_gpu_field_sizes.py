"""Random fields at the sizes where their kernels change: correlation matrices
around whole panels of the factorisation, K-L expansions of few and of very
many distinct factors, and fields of a phase that few or no particles have."""
import numpy as np
import pytest

import scenes
import sphgpu
from checkers import kl_oracle, rf_oracle

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


@pytest.mark.parametrize("ndim,K,rl", [
    (2, 1, (6.0, 1.5, 0.0)), (2, 40, (1.0, 1.0, 0.0)), (2, 300, (0.05, 1.0, 0.0)),
    (3, 1, (0.5, 0.25, 0.25)), (3, 56, (0.3, 0.3, 0.3)), (3, 64, (0.1, 1.0, 1.0)),
])
def test_expansions_of_few_and_many_factors(ndim, K, rl):
    sc = scenes.slope_2d(H=1.0, dx=0.1) if ndim == 2 else scenes.soil_column_3d(dx=0.1)
    eng, d, dom = _engine(sc)
    xi = np.random.default_rng(K).standard_normal(K)
    f = {"no": 0, "type": 1, "mean": 30.0, "sd": 3.0, "rl": list(rl), "coe_depth": 0.5}
    want = kl_oracle(ndim, sc.xp, sc.ptype, f, d, xi, K)[0]
    got = eng.kl_generate(dom, [sphgpu.kl_field(0, 1, 30.0, 3.0, list(rl), 0.5)], xi[None], K)[0]
    _close(got, want)
    eng.close()


@pytest.mark.parametrize("no", (0, 4))
def test_synthesis_of_one_phase(no):
    """The tensor-core synthesis against the FP64 field, for a phase of part of
    the particles and for one of none (every value NaN)."""
    import torch
    sc = scenes.soil_column_3d(dx=0.0625, with_water=False)
    eng, d, dom = _engine(sc)
    K, R = 40, 16
    xi = np.random.default_rng(5).standard_normal((R, K))
    field = sphgpu.kl_field(no, 1, 30.0, 3.0, [0.5, 0.3, 0.2], 2.0)
    out = torch.full((R, eng.n), 7.0, dtype=torch.float32, device="cuda")
    eng.kl_synthesize(dom, field, xi, out.data_ptr(), K)
    got = out.cpu().numpy()
    phase = sc.ptype == (2 if no == 0 else 1)
    assert np.array_equal(np.isnan(got), np.broadcast_to(~phase, got.shape))
    if phase.any():
        for r in (0, R - 1):
            want = eng.kl_generate(dom, [field], xi[r:r + 1], K)[0]
            assert np.abs(got[r, phase] - want[phase]).max() <= 1e-5 * np.abs(want[phase]).max()
    eng.close()
