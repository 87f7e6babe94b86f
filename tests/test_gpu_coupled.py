"""coupled_Water_Soil_Structure (contact types 1-3 with acc_type 2): its pair
sums read whole lists and, in 2-D, records without a z component."""
import numpy as np
import pytest

import scenes
from checkers import ORC_JACOBI, ORC_POW_CR, STATE_FIELDS, Oracle

pytestmark = pytest.mark.gpu


def _coupled_footing(ndim):
    sc = scenes.footing(ndim=ndim, dx=0.04 if ndim == 2 else 0.1, bed=(1.2, 0.6, 0.5), width=0.4, height=0.2, gap=0.4,
                        ss_type=2, zeta=0.1, v=0.5)
    sc.problem["ss"] = (2, 0.3, 0.1, 2)      # deformable: the penalty form's forces leave the finite range here
    return sc


@pytest.mark.parametrize("ndim", (2, 3))
def test_switch_to_the_bulk_form(ndim, tmp_path):
    """FP64 steps, then FP32-bulk ones: the state is that of a context that
    never held FP64 records."""
    import sphgpu
    st = scenes.initialise(_coupled_footing(ndim))
    path = str(tmp_path / "state.bin")
    a = sphgpu.Engine(st.params, device=0)
    a.load_state(st.fields, st.fluid, st.soil)
    a.step(6)
    a.checkpoint_save(path)
    a.set_precision(sphgpu.PREC_FP32_BULK)
    b = sphgpu.Engine(st.params, device=0)
    b.checkpoint_load(path)
    b.set_precision(sphgpu.PREC_FP32_BULK)
    for e in (a, b):
        e.step(4)
    for f in STATE_FIELDS:
        x, y = a.get_field(f), b.get_field(f)
        assert np.array_equal(x, y, equal_nan=x.dtype.kind == "f"), f
    assert np.isfinite(a.get_field("vx")).all()
    a.close()
    b.close()


def _wet_footing(ndim, ss):
    """Soil with pore water, a footing and walls, all with stress and motion."""
    sc = _coupled_footing(ndim)
    soil = sc.ptype == 2
    m = int(soil.sum())
    for k, v in (("xp", sc.xp[soil]), ("vxp", np.zeros((m, 3))), ("ptype", np.full(m, 1, np.int32)),
                 ("matype", np.zeros(m, np.int32)), ("permtype", np.zeros(m, np.int32)), ("etype", np.ones(m, np.int32))):
        setattr(sc, k, np.concatenate([getattr(sc, k), v]))
    sc.flags["fli"] = 1
    sc.soils[2]["eps0"] = 0.6667             # porous: the water's porosity is the soil's
    sc.problem.update(interc=1.0, pers=1.0e-4, perl=1.0e-4, perm=1.0e-4, ss=ss)
    st = scenes.initialise(sc)
    rng = np.random.default_rng(ndim)
    solid = (st.fields["type"] == 2) | (st.fields["type"] == 4)
    flat = (1.0, 1.0, float(ndim == 3))
    st.fields["vxp"] = st.fields["vxp"] + 0.05 * (st.fields["type"] > 0)[:, None] * rng.standard_normal((sc.n, 3)) * flat
    sig = np.where(solid[:, None], -1.0e3 * rng.random((sc.n, 6)), 0.0)
    if ndim == 2:
        sig[:, 4:] = 0.0
    st.fields["sig"] = sig
    return st


@pytest.mark.parametrize("ndim", (2, 3))
@pytest.mark.parametrize("before,after", (((0, 0.0, 0.0, 0), (2, 0.3, 0.1, 2)), ((2, 0.3, 0.1, 2), (2, 0.3, 0.1, 0)),
                                          ((2, 0.3, 0.1, 0), (1, 0.3, 0.1, 2))))
def test_contact_set_between_search_and_update(ndim, before, after):
    """The contact form is read by update alone: setting it after the search
    of a step (as the reference's classes do in the first one) gives the step of
    a run that had it from the start."""
    import sphgpu
    st, want = _wet_footing(ndim, before), _wet_footing(ndim, after)
    orc = Oracle(want.params, ORC_JACOBI, ORC_POW_CR)
    orc.load_state(want.fields, want.fluid, want.soil)
    eng = sphgpu.Engine(st.params, device=0)
    eng.load_state(st.fields, st.fluid, st.soil)
    assert eng.parttocell() == 0 and eng.partisearching() == 0
    eng.update_params(want.params)
    assert eng.update() == 0
    eng.step(1)
    assert orc.step(2) == 0
    for f in STATE_FIELDS:
        a, b = eng.get_field(f), orc.get_field(f)
        assert np.array_equal(a, b, equal_nan=a.dtype.kind == "f"), f
    assert np.isfinite(orc.get_field("vx")).all()
    eng.close()


def test_precision_set_between_search_and_update():
    import sphgpu
    st = _wet_footing(2, (2, 0.3, 0.1, 2))
    out = []
    for late in (False, True):
        eng = sphgpu.Engine(st.params, device=0)
        eng.load_state(st.fields, st.fluid, st.soil)
        if not late:
            eng.set_precision(sphgpu.PREC_FP32_BULK)
        assert eng.parttocell() == 0 and eng.partisearching() == 0
        if late:
            eng.set_precision(sphgpu.PREC_FP32_BULK)
        assert eng.update() == 0
        out.append([eng.get_field(f) for f in STATE_FIELDS])
        eng.close()
    for f, a, b in zip(STATE_FIELDS, *out):
        assert np.array_equal(a, b, equal_nan=a.dtype.kind == "f"), f
