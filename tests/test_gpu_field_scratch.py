"""The device memory of a random field is given back once the context steps."""
import numpy as np
import pytest

import scenes
import sphgpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("entry", ("step", "update", "step_profiled"))
def test_given_back(entry):
    import torch
    sc = scenes.slope_2d(H=3.0, dx=0.1)
    st = scenes.initialise(sc)
    eng = sphgpu.Engine(st.params, device=0)
    eng.load_state(st.fields, st.fluid, st.soil)
    d = scenes.kl_domain(sc)
    dom = sphgpu.kl_domain(d["nb_min"], d["nb_max"], d["soil_max"], d["water_max"])
    flags = sphgpu.rf_flags(1.1, 1)
    cells = eng.rf_cells(dom, flags)
    matrix = 8 * cells ** 2
    assert 60e6 < matrix < 250e6
    run = {"step": lambda: eng.step(1), "update": eng.update, "step_profiled": lambda: eng.step_profiled(1)}[entry]
    run()
    before = torch.cuda.mem_get_info()[0]
    field = [sphgpu.kl_field(1, 2, 10.0e3, 3.0e3, [6.0, 1.5, 0.0], 0.0)]
    eng.rf_generate(dom, field, flags, np.random.default_rng(1).standard_normal((1, cells)))
    run()
    after = torch.cuda.mem_get_info()[0]
    eng.close()
    assert before - after < matrix / 4, (before - after, matrix)
