"""The layout a batch runs in (``interleaved_pays``) against measured times of an iteration on a B200 in
both layouts: grids of 48 to 400 columns a side, 32 to 256 situations, 8 to 44 swept levels, the three
models.  The picked layout is never more than a fifth slower than the other (the fit's residuals are
15 % and less on each side), and batches below 32 situations take the row chains.
"""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# model, nii, njj, situations, levels, ms on row chains, ms interleaved
MEASURED = [
    (1, 64, 64, 33, 8, 0.84, 2.871), (0, 64, 64, 33, 8, 1.257, 2.961), (0, 64, 64, 144, 8, 5.182, 3.256),
    (2, 64, 64, 33, 8, 1.808, 4.715), (1, 64, 64, 33, 16, 0.995, 3.768), (0, 64, 64, 33, 16, 1.387, 4.44),
    (2, 64, 64, 33, 16, 2.137, 7.184), (1, 64, 64, 33, 28, 1.257, 5.695), (0, 64, 64, 33, 28, 1.605, 6.882),
    (2, 64, 64, 33, 28, 2.608, 11.596), (1, 64, 64, 33, 44, 1.538, 7.998), (0, 64, 64, 33, 44, 1.826, 9.97),
    (2, 64, 64, 33, 44, 3.032, 16.777), (1, 200, 200, 33, 8, 7.679, 11.29), (1, 200, 200, 64, 8, 14.9, 11.532),
    (0, 200, 200, 64, 8, 21.416, 11.731), (1, 200, 200, 33, 16, 8.657, 13.925),
    (0, 200, 200, 64, 16, 23.214, 16.474), (1, 200, 200, 33, 28, 10.875, 20.133),
    (0, 200, 200, 64, 28, 26.203, 24.923), (1, 200, 200, 33, 44, 13.567, 27.781),
    (0, 200, 200, 64, 44, 29.9, 36.108), (1, 48, 48, 32, 10, 0.647, 2.326), (1, 48, 48, 256, 10, 4.313, 2.888),
    (0, 48, 48, 32, 10, 0.896, 2.624), (2, 48, 48, 32, 10, 1.299, 4.469), (1, 48, 48, 32, 22, 0.753, 3.357),
    (0, 48, 48, 32, 22, 0.976, 3.99), (2, 48, 48, 32, 22, 1.56, 6.368), (1, 48, 48, 32, 36, 0.914, 4.95),
    (0, 48, 48, 32, 36, 1.092, 6.042), (2, 48, 48, 32, 36, 1.778, 10.177), (1, 96, 300, 32, 10, 5.087, 11.34),
    (0, 96, 300, 32, 10, 6.892, 12.231), (2, 96, 300, 32, 10, 10.907, 20.384), (1, 96, 300, 32, 22, 6.323, 15.394),
    (0, 96, 300, 32, 22, 7.793, 18.382), (2, 96, 300, 32, 22, 13.376, 30.43), (1, 96, 300, 32, 36, 8.314, 21.679),
    (0, 96, 300, 32, 36, 9.329, 29.854), (0, 96, 300, 80, 36, 22.957, 28.95), (2, 96, 300, 32, 36, 16.716, 45.094),
    (1, 300, 96, 32, 10, 5.675, 11.381), (0, 300, 96, 32, 10, 7.815, 11.646), (2, 300, 96, 32, 10, 11.916, 20.406),
    (1, 300, 96, 32, 22, 6.931, 15.404), (0, 300, 96, 32, 22, 8.664, 18.234), (2, 300, 96, 32, 22, 14.333, 30.494),
    (1, 300, 96, 32, 36, 8.913, 21.716), (0, 300, 96, 32, 36, 10.176, 26.446), (2, 300, 96, 32, 36, 17.582, 45.352),
    (1, 400, 400, 32, 10, 29.205, 26.867), (0, 400, 400, 40, 10, 47.941, 29.062),
    (1, 400, 400, 32, 22, 36.361, 36.184), (0, 400, 400, 40, 22, 53.937, 48.174),
    (1, 400, 400, 32, 36, 47.363, 50.279), (0, 400, 400, 40, 36, 63.898, 77.368),
]


def picks(cases, tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    exe = str(tmp_path / "layout_check")
    subprocess.run([gxx, "-std=c++17", "-O1", "-I", os.path.join(ROOT, "gral_b200", "csrc"), "-o", exe,
                    os.path.join(ROOT, "tests", "native", "layout_check.cpp")], check=True)
    text = "\n".join(" ".join(str(x) for x in c) for c in cases)
    return [int(x) for x in subprocess.run([exe], input=text, capture_output=True, text=True, check=True).stdout.split()]


def test_the_picked_layout_is_the_faster_one(tmp_path):
    got = picks([m[:5] for m in MEASURED], tmp_path)
    assert len(got) == len(MEASURED)
    for m, il in zip(MEASURED, got):
        assert m[6 if il else 5] <= 1.2 * min(m[5:]), m


def test_small_batches_take_the_row_chains(tmp_path):
    cases = [(m, ni, ni, n, v) for m in range(3) for ni in (4, 400) for n in (1, 31) for v in (2, 60)]
    assert picks(cases, tmp_path) == [0] * len(cases)
