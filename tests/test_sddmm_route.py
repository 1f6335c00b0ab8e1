"""The choice between the tensor cores and the gather kernels for SDDMM (csrc/sddmm_route.h, host code) against times
measured both ways on a B200: no call that it takes is slower for it, and the estimates it rests on hold."""
import os
import random
import shutil
import subprocess

import numpy as np
import pytest

SHAPES = [(64, 64), (256, 256), (512, 2048), (2048, 512), (1024, 4096)]
SPARSITIES = [0.5, 0.7, 0.8, 0.9, 0.95, 0.98]
INNER = [32, 128, 256]

# (M, K, inner dimension, density, with factors, us on the gather kernels, us on the tensor cores)
ALONE = [
    (400, 2048, 32, 0.1, 1, 3.6, 32.1), (400, 2048, 128, 0.3, 1, 19.1, 47.9), (400, 2048, 512, 0.3, 0, 56.7, 57.5),
    (400, 2048, 512, 0.05, 0, 11.4, 56.7), (510, 340, 608, 0.3, 0, 35.9, 27.9), (512, 512, 512, 0.5, 0, 23.2, 25.3),
    (512, 512, 512, 0.5, 1, 26.3, 28.7), (512, 2048, 512, 0.3, 0, 66.0, 57.9), (512, 2048, 512, 0.3, 1, 66.2, 62.0),
    (879, 253, 399, 0.2, 1, 40.4, 23.3), (941, 764, 928, 0.3, 1, 58.5, 55.1), (1024, 1024, 64, 0.5, 1, 10.7, 32.8),
    (1024, 1024, 128, 0.3, 0, 18.1, 27.8), (1024, 1024, 256, 0.5, 1, 36.8, 38.4), (1024, 1024, 256, 0.3, 1, 22.5, 32.2),
    (1024, 1024, 256, 0.3, 0, 26.1, 29.9), (1024, 1024, 512, 0.3, 0, 51.0, 35.9), (1024, 1024, 512, 0.5, 0, 80.1, 39.9),
    (1024, 1024, 512, 0.3, 1, 52.3, 38.3), (1024, 4096, 128, 0.5, 1, 83.6, 106.6), (1024, 4096, 256, 0.5, 1, 137.7, 115.5),
    (1024, 4096, 256, 0.3, 1, 86.7, 94.8), (1024, 4096, 512, 0.1, 0, 71.9, 100.2), (1038, 744, 64, 0.3, 1, 6.1, 27.5),
    (1234, 3987, 480, 0.5, 0, 269.2, 117.5), (1311, 802, 416, 0.3, 0, 38.0, 34.2), (2048, 512, 32, 0.1, 0, 3.8, 18.2),
    (2048, 512, 128, 0.1, 0, 6.3, 19.9), (2048, 512, 256, 0.5, 1, 30.2, 31.1), (2048, 512, 512, 0.05, 0, 18.0, 25.5),
    (2048, 512, 512, 0.1, 1, 17.9, 26.5), (2048, 512, 512, 0.5, 0, 76.6, 31.1), (2048, 512, 512, 0.5, 1, 66.0, 33.9),
    (4096, 4096, 32, 0.05, 0, 10.1, 72.0), (4096, 4096, 128, 0.1, 1, 87.7, 98.6), (4096, 4096, 128, 0.05, 1, 30.5, 97.9),
    (4096, 4096, 256, 0.3, 1, 250.4, 194.5), (4096, 4096, 256, 0.5, 0, 412.8, 175.8), (4096, 4096, 512, 0.05, 1, 103.7, 115.1),
    (4096, 4096, 512, 0.1, 1, 196.0, 116.4), (4096, 4096, 512, 0.3, 1, 570.0, 200.1), (7076, 7055, 796, 0.05, 1, 483.3, 528.9),
    (8192, 2048, 64, 0.3, 0, 126.9, 113.4), (8192, 2048, 128, 0.5, 1, 211.3, 260.1), (8192, 2048, 128, 0.1, 1, 76.8, 92.0),
    (8192, 2048, 128, 0.1, 0, 76.8, 73.6), (8192, 2048, 128, 0.3, 1, 130.9, 148.2), (8192, 2048, 512, 0.3, 0, 611.4, 154.4),
    (8192, 2048, 512, 0.3, 1, 613.7, 191.9), (8192, 2048, 512, 0.5, 1, 975.2, 355.0), (8448, 1335, 189, 0.1, 0, 79.1, 54.2),
    (16384, 1024, 64, 0.5, 0, 113.8, 153.1), (16384, 1024, 128, 0.3, 1, 156.2, 155.3), (16384, 1024, 128, 0.1, 0, 65.0, 78.5),
    (16384, 1024, 256, 0.5, 1, 324.7, 266.2), (16384, 1024, 512, 0.05, 0, 114.1, 107.1), (16384, 1024, 512, 0.05, 1, 96.7, 119.6),
    (573, 3711, 71, 0.5, 1, 42.6, 76.5), (10580, 403, 171, 0.1, 1, 38.3, 47.3), (1024, 4096, 128, 0.5, 0, 64.7, 80.3),
]
# (problems, seed of their sizes, spread of the row lengths, us of the gather kernels alone, us of the tensor-core part of
# a split call, us of the split call)
GROUPS = [
    (8, 764678, 0.4, 169, 104, 142), (10, 638438, 0.4, 153, 88, 160), (12, 726743, 0.4, 161, 118, 233),
    (18, 753158, 0.4, 369, 166, 201), (20, 831025, 0.4, 303, 121, 318), (27, 506830, 0.4, 754, 178, 322), (35, 674405, 0.4, 635, 301, 515),
    (40, 338656, 0.4, 416, 147, 379), (44, 150414, 0.4, 763, 216, 474), (55, 304060, 0.4, 648, 364, 597), (73, 136612, 0.4, 614, 176, 435),
    (87, 235201, 0.4, 591, 321, 529), (106, 681595, 0.4, 1077, 433, 709), (8, 334361, 0.0, 88, 59, 101), (11, 308055, 0.0, 52, 46, 72),
    (12, 106844, 0.0, 100, 106, 141), (15, 515561, 0.0, 197, 89, 214), (19, 1036956, 0.0, 244, 125, 175), (20, 845683, 0.0, 216, 84, 155),
    (22, 105970, 0.0, 402, 120, 238), (29, 330628, 0.0, 267, 154, 243), (31, 164413, 0.0, 427, 153, 312), (41, 907540, 0.0, 417, 183, 310),
    (57, 978582, 0.0, 598, 256, 531), (76, 144189, 0.0, 634, 330, 527), (91, 74792, 0.0, 678, 332, 583), (117, 922008, 0.0, 806, 456, 719),
]


def problems_of(count, seed):
    rng = random.Random(seed)
    out = []
    for _ in range(count):
        (M, K), N, sparsity = rng.choice(SHAPES), rng.choice(INNER), rng.choice(SPARSITIES)
        out.append((M, K, N, M * K * (1.0 - sparsity)))
    return out


@pytest.fixture(scope="module")
def route(pkg, tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("no g++")
    exe = str(tmp_path_factory.mktemp("route") / "route")
    header = os.path.join(pkg.PKG_DIR, "csrc", "sddmm_route.h")
    main = os.path.join(os.path.dirname(os.path.abspath(__file__)), "sddmm_route_main.cpp")
    subprocess.run(["g++", "-std=c++17", "-O1", f'-DROUTE_HEADER="{header}"', "-o", exe, main], check=True)

    def run(lines):
        text = subprocess.run([exe], input="\n".join(lines), check=True, capture_output=True, text=True).stdout
        return [(int(a), float(b)) for a, b in (line.split() for line in text.splitlines())]

    return run


def test_lone_calls(route):
    got = route([f"alone {M} {K} {N} {M * K * d} {masked} {int(N % 4 == 0)}" for (M, K, N, d, masked, gather, tensor) in ALONE])
    errors = [us / tensor - 1.0 for (taken, us), (M, K, N, d, masked, gather, tensor) in zip(got, ALONE)]
    assert np.sqrt(np.mean(np.square(errors))) < 0.2
    for (taken, us), case in zip(got, ALONE):
        gather, tensor = case[5:]
        assert not taken or tensor <= 1.02 * gather, case
        assert taken or tensor >= 0.55 * gather, case  # the clear cases are taken


def test_groups(route):
    lines = []
    for (count, seed, cov, gather, part, split) in GROUPS:
        lines.append(f"group {count} " + " ".join(f"{M} {K} {N} {nnz}" for (M, K, N, nnz) in problems_of(count, seed)))
    errors, taken_total = [], 0
    for (taken, us), case in zip(route(lines), GROUPS):
        gather, part, split = case[3:]
        if taken:
            assert split <= 1.02 * gather, case
            errors.append(us / part - 1.0)
            taken_total += 1
        else:
            assert split >= 0.5 * gather, case  # (uneven rows, which the sizes do not show)
    assert taken_total >= len(GROUPS) // 2
    assert np.sqrt(np.mean(np.square(errors))) < 0.15 and max(map(abs, errors)) < 0.25


def test_sizes_that_stay_with_the_gather_kernels(route):
    """Few rows, operands beyond 32-bit offsets, empty patterns; parts and strips of very large ones stay in range."""
    calls = [(384, 4096, 512, 0.5), (1 << 21, 64, 512, 0.5), (64, 1 << 21, 512, 0.5), (4096, 4096, 512, 0.0), (4096, 0, 512, 0.0)]
    assert all(taken == 0 for taken, us in route([f"alone {M} {K} {N} {M * K * d} 0 1" for (M, K, N, d) in calls]))
    many = [(1 << 20, 4096, 256, (1 << 20) * 4096 * 0.4)] * 3
    (taken, us), = route(["group 3 " + " ".join(f"{M} {K} {N} {nnz}" for (M, K, N, nnz) in many)])
    one, = route(["group 1 " + f"{many[0][0]} {many[0][1]} {many[0][2]} {many[0][3]}"])
    assert taken == 3 and one[0] == 1 and abs(us - 3 * one[1]) < 0.01 * us
