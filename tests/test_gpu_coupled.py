"""coupled_Water_Soil_Structure (contact types 1-3 with acc_type 2): its pair
sums read whole lists and, in 2-D, records without a z component."""
import numpy as np
import pytest

import scenes
from checkers import STATE_FIELDS

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
