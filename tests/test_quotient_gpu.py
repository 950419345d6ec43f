"""The quotients that replace divisions in the sweeps (``gral_b200/csrc/prog_quot.cuh``) against plain
divisions on the device (``tests/native/quotient_check.cu``): the reciprocal over every divisor of its
range, quotients of 2^28 random operands inside their range, over all floats and doubles and around the
ends of the range, and of special values.  Every result must be the IEEE quotient."""
import os
import subprocess

import pytest

from gral_b200 import build

pytestmark = pytest.mark.gpu


def test_quotients_are_the_ieee_quotients(gpu_required, tmp_path):
    exe = str(tmp_path / "quotient_check")
    subprocess.run([build.nvcc()] + build.flags() + ["-o", exe, os.path.join(build.ROOT, "tests", "native",
                                                                             "quotient_check.cu")], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, check=True).stdout.split()
    got = {name: int(n) for name, n in zip(out[::2], out[1::2])}
    assert len(got) == 12
    assert got == {name: 0 for name in got}
