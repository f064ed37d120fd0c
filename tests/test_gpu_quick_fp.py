"""The branch-free division and square root of the projections (csrc/quick_fp.cuh)
against the plain operators, bit for bit: every mantissa of the reciprocal and the
square root, random, near-midpoint and end-of-range quotients, every arc cosine."""
import shutil
import subprocess
from pathlib import Path

import pytest

from solidcloth_b200 import build

pytestmark = pytest.mark.gpu

# values compared per form (quotients: both forms; near-midpoint ones with two neighbours)
COUNTS = {"recip": 10 << 23, "sqrt": 6 << 23, "quot_random": 2 << 30, "quot_midpoint": 6 << 28,
          "quot_ends": 64 << 23, "special": 8, "acos": 2 * 0x3f800000}


def test_bits_of_the_plain_operators(tmp_path):
    if not shutil.which(build.nvcc()):
        pytest.skip("no nvcc")
    exe = tmp_path / "quick_fp_check"
    src = Path(__file__).with_name("quick_fp_check.cu")
    subprocess.run([build.nvcc(), *build.ARCH, *build.FLAGS, "-I", str(build.CSRC), str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    rows = {f[0]: f[1:] for f in (line.split() for line in r.stdout.splitlines())}
    assert r.returncode == 0, r.stdout
    assert set(rows) == set(COUNTS)
    for name, want in COUNTS.items():
        assert int(rows[name][0]) == want and int(rows[name][2]) == 0, (name, rows[name])
