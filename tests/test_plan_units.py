"""Work-unit tables on the host (CPU): plan_units.cpp prints what the library's
scheduling functions give."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.join(os.path.dirname(HERE), "chime-x_b200")
ONE_SM, SM_PAIR = 1, 2


@pytest.fixture(scope="module")
def units(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("units") / "plan_units")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(cuda, "include"), "-o", exe,
                    os.path.join(HERE, "plan_units.cpp"), "-L", PKG, "-lchimex", "-L",
                    os.path.join(cuda, "lib64"), "-lcudart", "-Wl,-rpath," + PKG], check=True)

    def run(*args):
        out = subprocess.run([exe] + [str(a) for a in args], check=True, capture_output=True,
                             text=True).stdout
        return [[float(w) for w in line.split()] for line in out.splitlines()]
    return run


@pytest.mark.parametrize("T", [1, 100, 128, 4096])
def test_one_tile_channel_beside_larger_ones(units, T):
    """On the one-SM tile a channel of one tile costs what a larger channel's last unit,
    one tile against itself too, costs: both run the same kernel."""
    small = units("costs", ONE_SM, 128, T)
    larger = units("costs", ONE_SM, 256, T)
    assert small == [u for u in larger if u[1] == 1]
