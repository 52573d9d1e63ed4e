"""The bounded waits inside the tracer sweeps (tests/sweep_waits_check.cu). moist_set_wait_limit reaches
the tiled sweep's (test_wait_limit.py); the warps of the streaming sweep, which ensembles always run, wait
for their neighbours within a limit that the launch carries. One cycle makes these waits run out: the sweep
then ends by itself and sets the timeout word. With the default's two seconds it never does, and the
results are those of the wavefront sweep bit for bit. Likewise the tiled sweep's bound of passes: a sweep
that reaches it before its fixed point ends with the error word set."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))
LONG = 4 * 10 ** 9


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    exe = tmp_path_factory.mktemp("waits") / "sweep_waits_check"
    subprocess.run(["nvcc", "-O3", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "--fmad=false",
                    "-o", str(exe), os.path.join(HERE, "sweep_waits_check.cu")], check=True)
    return str(exe)


def run(checker, *args):
    out = subprocess.run([checker] + [str(a) for a in args], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0, out.stdout + out.stderr
    return [int(x) for x in out.stdout.split()]


@pytest.mark.parametrize("nx,nz", [(70, 17), (300, 48), (129, 250)])
def test_stream_waits(checker, nx, nz):
    timeout, _ = run(checker, "stream", nx, nz, 1)
    assert timeout == 1
    assert run(checker, "stream", nx, nz, LONG) == [0, 0]


@pytest.mark.parametrize("nx,nz", [(70, 17), (300, 48), (129, 250)])
def test_tiles_pass_bound(checker, nx, nz):
    error, mismatches = run(checker, "tiles", nx, nz, 1)
    assert error == 2 and mismatches > 0
    assert run(checker, "tiles", nx, nz, -(-nx // 32) + -(-nz // 16) + 2) == [0, 0]
