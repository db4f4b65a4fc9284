"""The arithmetic that deals a batch's rays to the traversal kernels' warps, on
the host: every ray once, up to the largest batch an int counts."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
INT_MAX = 2**31 - 1


@pytest.fixture(scope="module")
def deal(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("ray_range") / "ray_range_main")
    subprocess.run([os.environ.get("CXX", "g++"), "-std=c++17", "-O2", "-fsanitize=signed-integer-overflow",
                    "-fno-sanitize-recover", os.path.join(HERE, "ray_range_main.cpp"), "-o", exe], check=True, timeout=300)

    def run(*args):
        r = subprocess.run([exe, *map(str, args)], capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stdout + r.stderr
    return run


@pytest.mark.parametrize("own", [0, 1], ids=["counter", "own_first"])
@pytest.mark.parametrize("n", [1, 31, 33, 4863, 4864, 4865, 155647, 155648, 155649, 1000003])
def test_every_ray_once(deal, n, own):
    for warps in (32, 4864):
        deal(n, warps, own, 0)


@pytest.mark.parametrize("own", [0, 1], ids=["counter", "own_first"])
@pytest.mark.parametrize("n", [INT_MAX, INT_MAX - 31, 2**31 - 77824, 2**31 - 100000, 2**31 - 155648])
def test_largest_batches(deal, n, own):
    """From where the last million rays are left: the counter passes the
    largest int while the last warps look for more."""
    deal(n, 4864, own, n - 1000000 - (4864 * 32 if own else 0))
