"""quotient_proven (fastdiv.cuh), on which the exactness of the acoustic substep's elimination rests:
it accepts the IEEE quotient and refuses the doubles beside it (tests/quotient_check.cu)."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


def test_accepts_the_quotient_and_refuses_its_neighbours(tmp_path):
    exe = str(tmp_path / "quotient_check")
    subprocess.run(["nvcc", "-O3", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "--fmad=false", "-o", exe,
                    os.path.join(HERE, "quotient_check.cu")], check=True)
    n = 1 << 30
    out = subprocess.run([exe, str(n), "9"], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout + out.stderr
    wrong, refused, _, accepted = map(int, out.stdout.split())
    assert (wrong, refused) == (0, 0) and accepted > n // 2
