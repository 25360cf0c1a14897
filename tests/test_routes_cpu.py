"""Dispatch rules (sc_lbm_b200/csrc/routes.h), compiled from the library's own
header: the kernel chosen is the faster one where both were timed on a B200."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
FP64, FP32, FP16, SMS = 0, 1, 2, 148


@pytest.fixture(scope="module")
def ask(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("routes") / "routes")
    subprocess.run(["g++", "-std=c++17", "-I" + os.path.join(ROOT, "include"),
                    "-I" + os.path.join(ROOT, "sc_lbm_b200", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "routes.cpp"), "-o", exe], check=True)

    def answers(questions):
        text = "\n".join(" ".join(map(str, q)) for q in questions)
        out = subprocess.run([exe], input=text, check=True, capture_output=True, text=True).stdout
        got = [tuple(map(int, line.split())) for line in out.splitlines()]
        assert len(got) == len(questions)
        return got
    return answers


# nx, ny, form: us per step of the depth, and by one node per thread (many
# steps a call; one step a call)
SINGLE = [
    ((200, 50, FP64), 6, True), ((64, 32, FP32), 6, True), ((300, 300, FP64), 3, True),
    ((400, 200, FP32), 5, True), ((400, 200, FP16), 5, True),
    ((1500, 600, FP64), 2, False),     # 18.5 / 28.9; 32.0 / 28.9
    ((2048, 2048, FP64), 2, False),    # 78 / 116; 135 / 116
    ((1024, 1024, FP32), 3, False),    # 12.7 / 18.7; 20.9 / 19.0
    ((2048, 2048, FP16), 3, False),    # 55 / 76; 99 / 76
    ((500, 500, FP64), 2, True),       # 6.0 / 9.3; 9.0 / 9.4
    ((500, 500, FP32), 3, True),       # 3.9 / 8.3; 6.7 / 8.4
    ((29, 40000, FP64), 2, False),     # 23 / 35; 39 / 35
    ((100000, 13, FP32), 3, False),    # 21.0 / 23.7; 38 / 24
    ((4, 100000, FP64), 1, False),     # 49 / 10.4
    ((4, 100000, FP32), 1, False),     # 31 / 9.7
    ((4, 100000, FP16), 1, False),     # 36 / 10.4
    ((29, 40000, FP32), 1, False),     # 25.5 / 20.6
    ((33, 30000, FP16), 1, False),     # 21.8 / 18.6
    ((200000, 4, FP64), 1, False),     # 32 / 25
    ((1, 10000, FP64), 1, False),      # 6.7 / 4.3
]


def test_single_component_depth(ask):
    got = ask([("single", *shape, SMS) for shape, _, _ in SINGLE])
    assert got == [(depth, int(one)) for _, depth, one in SINGLE]


def test_launch_counts(ask):
    """Enough launches, none without a step, and on demand of the steps' parity."""
    questions = [(n, K, keep) for n in range(0, 40) for K in (1, 2, 3, 5, 6) for keep in (0, 1)]
    for (n, K, keep), (launches,) in zip(questions, ask([("launches", *q) for q in questions])):
        least = -(-n // K)
        assert least <= launches <= min(n, least + keep)
        assert not keep or (launches - n) % 2 == 0


# nx, ny, form, solid nodes: whether one node per thread was faster than the
# register tile (us per step)
FLAT = [
    ((1021, 763, FP32, 0), True), ((1201, 1101, FP32, 0), True),    # 40.7 / 44.8
    ((1801, 1501, FP32, 0), True),                                  # 82.4 / 84.7
    ((1501, 1101, FP32, 0), False), ((1500, 1100, FP32, 0), False), # 53.2 / 50.2; 52.4 / 50.1
    ((2047, 2047, FP32, 0), False), ((4095, 4095, FP32, 0), False), # 123 / 118; 484 / 450
    ((2047, 2047, FP32, 1), True), ((2801, 2401, FP32, 1), True),   # 142 / 150; 226 / 233
    ((3501, 3001, FP32, 1), False), ((4095, 4095, FP32, 1), False), # 355 / 351; 546 / 534
    ((2801, 2401, FP16, 0), True), ((3001, 2701, FP16, 0), False),  # 145 / 155; 184 / 176
    ((4095, 4095, FP16, 1), True),                                  # 431 / 463
    ((1501, 1101, FP64, 0), True), ((4095, 4095, FP64, 1), True),   # 84 / 96; 967 / 1077
]


def test_single_steps_off_the_ring(ask):
    assert ask([("flat", *q) for q, _ in FLAT]) == [(int(want),) for _, want in FLAT]


def test_low_bands_take_single_steps(ask):
    """us per step, pairs / single steps: FP32 1024^2 3 rows 33.7 / 37.1, 2 rows 42 / 37,
    256^2 2 rows (384 units) 5.6 / 6.3; FP16 2048^2 5 rows 104 / 100, with solid nodes 126 /
    132, 1024^2 3 rows with solid nodes 42.3 / 39.1, 300^2 3 rows (300 units) 7.4 / 8.4."""
    least = {(FP32, 0): 3, (FP32, 1): 3, (FP16, 0): 6, (FP16, 1): 4}
    questions = [("rows", p, n, 3000, solid, SMS) for p, solid in least for n in (0, 1, 2, 3, 4, 5, 6, 7, 64)]
    assert ask(questions) == [(int(n == 0 or n >= least[p, solid]),) for _, p, n, _, solid, _ in questions]
    assert ask([("rows", FP32, 2, 384, 0, SMS), ("rows", FP16, 3, 300, 0, SMS)]) == [(1,), (1,)]


def test_narrow_fp16_domains_with_solid_nodes(ask):
    """us per step of a batch, pairs / one-warp tiles: 300 x (20 x 20) 20.0 / 12.2,
    300 x (60 x 60) 50 / 46, 300 x (90 x 60) 57 / 71, 300 x (12 x 8) 9.4 / 9.7, 60 x (20 x 20)
    6.2 / 9.8, 60 x (44 x 60) 12.6 / 14.0."""
    rows_full = [(6000, 163), (18000, 491), (18000, 737), (2400, 98), (1200, 163), (3600, 360)]
    assert ask([("warp", *q, SMS) for q in rows_full]) == [(0,), (0,), (1,), (1,), (1,), (1,)]


# thousand nodes, fill of the ring's strips and changes along rows in
# thousandths: whether one node per thread was faster than the ring (us per step)
BATCH64 = [
    ((262, 1000, 180), True),                             # 4 x 256^2 20 / 28
    ((979, 781, 180), True),                              # 8 x (400 x 306) 94 / 100
    ((1049, 500, 375), True), ((1049, 1000, 375), True),  # 256 x 64^2 97 / 143; 4 x 512^2 100 / 107
    ((2938, 781, 375), True), ((3840, 781, 375), False),  # 24 x (400 x 306) 280 / 288; 64 x (300 x 200) 401 / 371
    ((1311, 1000, 56), True), ((1311, 1000, 95), False),  # 5 x 512^2 100 / 106; 115 / 113
    ((2097, 1000, 52), True), ((2097, 1000, 79), False),  # 2 x 1024^2 155 / 163; 179 / 173
    ((2938, 781, 118), True),                             # 24 x (400 x 306) 255 / 276
    ((3840, 781, 94), True), ((3840, 781, 180), False),   # 64 x (300 x 200) 337 / 345; 377 / 362
    ((4194, 1000, 56), False),                            # 16 x 512^2 309 / 301
    ((4896, 781, 45), True), ((10240, 833, 55), False),   # 40 x (400 x 306) 369 / 401; the 512-domain ensemble 1685 / 1673
]


def test_fp64_batches_with_solid_nodes(ask):
    assert ask([("batch64", *q) for q, _ in BATCH64]) == [(int(want),) for _, want in BATCH64]
