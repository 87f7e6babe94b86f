"""Records downloaded at the sizes where the transfer divides its work: the
rest of a warp's 32 records, one thread's 2,048 particles and one more, and
counts that leave the last thread a short share or several pieces."""
import ctypes as C

import numpy as np
import pytest

import scenes
import sphgpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,stride", [(1, 1064), (31, 1064), (33, 1072), (2048, 1064), (2049, 1064),
                                      (16385, 1064), (100_003, 1096), (262_145, 1064)])
def test_every_member_of_every_record(n, stride):
    st = scenes.initialise(scenes.soil_column_3d(dx=0.2))
    p = st.params if isinstance(st.params, sphgpu.Params) else sphgpu.params_from_dict(st.params)
    p.ntotal = n
    eng = sphgpu.Engine(p, device=0)
    rng = np.random.default_rng(n)
    want = np.full((n, stride), 0xAB, np.uint8)
    for name, nc in sphgpu.FIELDS.items():
        off, k = C.c_size_t(), C.c_int()
        assert eng.lib.sphgpu_particle_layout(name.encode(), C.byref(off), C.byref(k)) == 0 and k.value == nc
        if name in sphgpu.INT_FIELDS:
            v = rng.integers(0, 5, (n, nc)).astype(np.int32)
        else:
            v = rng.standard_normal((n, nc))
        eng.set_field(name, v)
        want[:, off.value:off.value + v.itemsize * nc] = v.view(np.uint8).reshape(n, -1)
    for _ in range(2):
        got = np.full((n, stride), 0xAB, np.uint8)
        eng.download_particles(got, stride)
        assert np.array_equal(got, want)
    eng.close()
