"""A cached launch shape is applied only to the passes it was timed on."""
import numpy as np
import pytest

import scenes
import sphgpu

pytestmark = pytest.mark.gpu


def _engine(inip=0):
    sc = scenes.dam_break_2d(dx=0.04, steps=100)
    sc.problem["inip"] = inip
    st = scenes.initialise(sc)
    eng = sphgpu.Engine(st.params, device=0)
    eng.load_state(st.fields, st.fluid, st.soil)
    return eng


def _lines(path):
    return [line.split() for line in path.read_text().splitlines()]


def test_damped_and_free_steps_are_tuned_apart(tmp_path):
    cache = tmp_path / "tune.txt"
    eng = _engine(inip=20)
    assert (eng.autotune(1, str(cache)) > 0).any()            # damped: steps 1-4
    assert (eng.autotune(1, str(cache)) == 0).all()
    eng.step(20)
    assert (eng.autotune(1, str(cache)) > 0).any()            # free
    assert (eng.autotune(1, str(cache)) == 0).all()
    keys = [line[0] for line in _lines(cache)]
    assert len(keys) == 2 and keys[0] != keys[1]
    eng.close()


def test_tuned_across_the_change_is_not_kept(tmp_path):
    cache = tmp_path / "tune.txt"
    eng = _engine(inip=2)
    eng.autotune(1, str(cache))                               # steps 1-4: two damped, two free
    assert not cache.exists()
    eng.close()


def test_lines_of_other_passes_are_not_applied(tmp_path):
    """A line with the key as it was written before it named the passes."""
    import torch
    cache = tmp_path / "tune.txt"
    eng = _engine()
    p = eng.params
    old = "%s/ndim%d/n%d/flbndy%d/fli%d/ss%d/prec%d/inst%d" % (
        torch.cuda.get_device_name(0).replace(" ", "_"), 2, eng.n, p.flbndy, p.fli, p.ss_type, 0, 0)
    cache.write_text(old + " 32" * 10 + "\n")
    assert (eng.autotune(1, str(cache)) > 0).any()
    assert len(_lines(cache)) == 2
    eng.close()


def test_every_stage_is_a_pass():
    """The resolve pass is part of the pair records: no stage of its own, and
    its entry of the launch shape follows theirs."""
    eng = _engine()
    assert "k_nnps_resolve" not in eng.step_profiled(1)
    table, chosen = eng.autotune(1), eng.launch()
    resolve, pairw = (eng.TUNE_PASSES.index(k) for k in ("k_nnps_resolve", "k_pairw"))
    assert np.array_equal(table[:, resolve], table[:, pairw]) and chosen[resolve] == chosen[pairw]
    eng.close()
