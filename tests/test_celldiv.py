"""The branch-free divisions of the tracer cell (FastDiv, fastdiv.cuh) on the GPU against IEEE
division, bit for bit (tests/celldiv_check.cu): every numerator for denominators the model uses
and hard ones (significands of one and of all ones, the ends of the admitted range), every
denominator of the reciprocal, and random bit patterns in both types. No accepted quotient may
differ; denominators outside the prepared range must be refused for every numerator."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    exe = tmp_path_factory.mktemp("celldiv") / "celldiv_check"
    subprocess.run(["nvcc", "-O3", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a",
                    "--fmad=false", "-o", str(exe), os.path.join(HERE, "celldiv_check.cu")], check=True)
    return str(exe)


def run(checker, *args):
    out = subprocess.run([checker] + [str(a) for a in args], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout + out.stderr
    return [[int(x) for x in line.split()[1:]] for line in out.stdout.strip().splitlines()]


def test_every_numerator(checker):
    bs = ["250", "125", "100", "500", "2", "6", "1.1535", "0.8123", "0.3141", "102.5", "0x1.fffffep+6", "0x1.000002p+6",
          "0x1p-40", "0x1p40"]
    for b, (cdiv, quot, ratio, ratio_neg, bad) in zip(bs, run(checker, "cdiv", *bs)):
        assert (cdiv, quot, ratio, ratio_neg) == (0, 0, 0, 0), b
        assert bad < 2 ** 32 * 0.6, b  # NaN, infinities and the range the scaling leaves out
    for b, line in zip(("0x1p-41", "0x1p41"), run(checker, "cdiv", "0x1p-41", "0x1p41")):
        assert line[:4] == [0, 0, 0, 0] and line[4] == 2 ** 32, b


def test_every_denominator_of_the_reciprocal_and_sixths(checker):
    assert run(checker, "rcp") == [[0]]
    assert run(checker, "div6") == [[0]]


def test_random_bit_patterns(checker):
    ((cdiv, quot, ratio, accepted),) = run(checker, "random", 1 << 31, 5)
    assert (cdiv, quot, ratio) == (0, 0, 0) and accepted > 1 << 29
    ((cdiv, quot, ratio, div6, accepted),) = run(checker, "random64", 1 << 30, 6)
    assert (cdiv, quot, ratio, div6) == (0, 0, 0, 0) and accepted > 1 << 28
