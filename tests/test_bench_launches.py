"""bench.py's account of what a gate batch launches (kernel names of its line,
launch count, shared-memory roofline) against the launch rules of
csrc/bootstrap.cu: launch_auto_fp32, launch_low_latency, launch_ring_batched,
launch_auto_fp64 and blind_rotate_tail_start, on both sides of every line.
CPU only."""
import os
import sys

import pytest

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))

bench = pytest.importorskip("bench")

DUO = "k_blind_rotate_duo<3,%d,4,2>"
RING4 = "k_blind_rotate_ring<float,2,4,3,4,inline,nb3>"
RING3 = "k_blind_rotate_ring<float,2,3,%d,4,inline,nb%d>"
ONE, TWO = "k_blind_rotate_spread<%d>", "k_blind_rotate_spread2<%d>"
ONE_P, TWO_P = "k_blind_rotate_spread<%d,pair>", "k_blind_rotate_spread2<%d,pair>"


def _names(*parts):
    return ["%s x %d" % p for p in parts]


@pytest.mark.parametrize("batch,want", [
    (1, _names((TWO % 3, 1))), (76, _names((TWO % 3, 76))), (77, _names((ONE % 3, 77))),
    (152, _names((ONE % 3, 152))), (153, _names((ONE_P % 3, 152), (TWO_P % 3, 1))),
    (228, _names((ONE_P % 3, 152), (TWO_P % 3, 76))), (229, _names((ONE_P % 3, 229))),
    (304, _names((ONE_P % 3, 304))), (305, _names((RING3 % (3, 3), 305))), (456, _names((RING3 % (3, 3), 456))),
    (457, _names((RING4, 457))), (608, _names((RING4, 608))), (609, _names((RING4, 608), (TWO % 3, 1))),
    (684, _names((RING4, 608), (TWO % 3, 76))), (685, _names((RING4, 608), (ONE % 3, 77))),
    (760, _names((RING4, 608), (ONE % 3, 152))), (761, _names((DUO % 3, 761))), (912, _names((DUO % 3, 912))),
    (913, _names((DUO % 3, 912), (TWO % 3, 1))), (912 + 229, _names((DUO % 3, 912), (ONE_P % 3, 229))),
    (912 + 760, _names((DUO % 3, 912), (RING4, 608), (ONE % 3, 152))), (912 + 761, _names((DUO % 3, 912 + 761))),
    (4096, _names((DUO % 3, 3648), (RING3 % (3, 3), 448)))])
def test_automatic_split_fp32_launches(batch, want):
    assert bench.launched_blind_rotations("split_fp32", 0, batch) == want


@pytest.mark.parametrize("batch,want", [
    (228, _names((ONE_P % 2, 152), (TWO_P % 2, 76))), (229, _names(("k_blind_rotate_pair<float,2,2,2,4>", 229))),
    (304, _names(("k_blind_rotate_pair<float,2,2,2,4>", 304))), (305, _names((RING3 % (2, 2), 305))),
    (457, _names(("k_blind_rotate_duo<2,2,4,2>", 457))), (1100, _names((DUO % 2, 912), (ONE_P % 2, 152), (TWO_P % 2, 36)))])
def test_automatic_split_fp32_launches_with_two_levels(batch, want):
    assert bench.launched_blind_rotations("split_fp32", 0, batch, l=2) == want


def test_fixed_order_never_takes_the_pair_order():
    assert bench.launched_blind_rotations("split_fp32", 15, 200) == _names((ONE % 3, 152), (TWO % 3, 48))
    assert bench.launched_blind_rotations("split_fp32", 15, 300, l=2) == _names((ONE % 2, 300))
    assert bench.launched_blind_rotations("split_fp32", 15, 4096) == bench.launched_blind_rotations("split_fp32", 0, 4096)


@pytest.mark.parametrize("batch,want", [
    (48, _names(("k_blind_rotate_cluster8_f64<3>", 48))), (49, _names(("k_blind_rotate_spread2_f64<3>", 49))),
    (76, _names(("k_blind_rotate_spread2_f64<3>", 76))), (77, _names(("k_blind_rotate_spread_f64<3>", 77))),
    (304, _names(("k_blind_rotate_spread_f64<3>", 304))),
    (305, _names(("k_external_product<double,1,BlindRotate,3,3>", 305))),
    (457, _names(("k_external_product<double,1,BlindRotate,3,3>", 456), ("k_blind_rotate_cluster8_f64<3>", 1)))])
def test_automatic_fp64_launches(batch, want):
    assert bench.launched_blind_rotations("fp64", 0, batch) == want


@pytest.mark.parametrize("form,shape,batch,want", [
    ("split_fp32", 4, 9, "k_external_product<float,2,BlindRotate,4,3>"),
    ("split_fp32", 5, 9, "k_blind_rotate_ring<float,2,5,3,4,producer-warp>"),
    ("split_fp32", 6, 9, "k_blind_rotate_ring<float,2,6,3,4,inline>"), ("split_fp32", 9, 456, RING3 % (3, 3)),
    ("split_fp32", 9, 457, RING4), ("split_fp32", 10, 5, DUO % 3),
    ("split_fp32", 12, 5, "k_blind_rotate_pair<float,2,2,3,4>"), ("split_fp32", 14, 500, ONE % 3),
    ("split_fp32", 16, 500, TWO % 3), ("fp64", 3, 5, "k_external_product<double,1,BlindRotate,3,3>"),
    ("fp64", 4, 5, "k_blind_rotate_ring<double,1,4,3,4,inline>"), ("fp64", 16, 5, "k_blind_rotate_spread2_f64<3>")])
def test_explicit_shapes_launch_one_kernel(form, shape, batch, want):
    assert bench.launched_blind_rotations(form, shape, batch) == [want]


@pytest.mark.parametrize("form,shape,batch,want", [
    ("split_fp32", 0, 1, 3), ("split_fp32", 0, 912, 3), ("split_fp32", 0, 4096, 5), ("split_fp32", 0, 912 + 608, 5),
    ("split_fp32", 0, 912 + 609, 5),  # three rotations, one key switch
    ("split_fp32", 15, 913, 5), ("split_fp32", 10, 4096, 3), ("split_fp32", 9, 1000, 3),
    ("fp64", 0, 1000, 4), ("fp64", 3, 4096, 3)])
def test_kernels_of_an_eager_gate_batch(form, shape, batch, want):
    assert bench.eager_gate_launches(form, shape, batch) == want


def test_shared_memory_roofline_of_what_runs():
    layer = bench.launched_blind_rotations("split_fp32", 0, 4096)
    r = bench.smem_roofline(layer, 4096, 29.0, {"sm_mhz": 2000.0})
    assert abs(r["wavefronts_per_step"] - (3648 * 1.26e9 / 912 + 448 * 0.74e9 / 448)) < 1.0
    assert bench.smem_roofline(bench.launched_blind_rotations("split_fp32", 0, 700), 700, 6.0, None) is None
