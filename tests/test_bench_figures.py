"""bench.py's own figures on the CPU: the kernels whose traffic it adds up are
the ones the step launches, the committed traffic names them all, and the
download's bytes are those of the packed records."""
import os
import sys

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if REPO not in sys.path:
    sys.path.insert(0, REPO)

import bench  # noqa: E402

MOMENTUM = "stress divergence + viscosity + walls + velocity update"
STRAIN = "strain + stress + free surface + eigen"


def test_no_viscosity_loop_in_the_momentum_stage():
    names = bench.traffic_kernels(bench.PASS_KERNELS[MOMENTUM], {"k_accel_a": 1.7, "k_accel_b": 2.3})
    assert names == ["k_accel_a", "k_accel_b_drag", "k_accel_b_tail"]


def test_stages_that_did_not_run_add_no_traffic():
    assert bench.traffic_kernels(("k_strain", "k_regu_eps", "k_stress"),
                                 {"k_strain": 2.9, "k_regu_eps": 0.002, "k_stress": 1.2}) == ["k_strain", "k_stress"]


def test_committed_traffic_covers_the_heavy_passes():
    per_kernel = bench.ncu_traffic()
    for name in (MOMENTUM, STRAIN):
        ran = {k: 1.0 for k in ("k_strain", "k_stress", "k_accel_a", "k_accel_b")}
        for k in bench.traffic_kernels(bench.PASS_KERNELS[name], ran):
            assert per_kernel[k] > 0.0, k
    # kernels that are no longer launched
    assert not {"k_nnps_resolve", "k_accel_b"} & set(per_kernel)


def test_download_bytes_are_the_packed_records():
    # 73 doubles and four ints of Particle, without x
    assert bench.download_record_bytes() == 73 * 8 + 4 * 4
