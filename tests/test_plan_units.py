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


def test_stages_within_a_budget(units):
    """unit_stages is the inverse of unit_cost."""
    assert units("inverse") == []


# The most time that a plan's two tables may take, as a multiple of what scheduling its
# units with one to eight equal ranges takes.  Half way (geometrically) between what a
# search for every piece's length (2.6, 1.20, 1.21, 1.30) and the tables now (1.08, 0.39,
# 0.38, 0.42) measured.
@pytest.mark.parametrize("E,F,T,limit", [
    (256, 16, 16384, 1.7), (96, 64, 4096, 0.7), (64, 65, 5616, 0.7), (32, 67, 11973, 0.7),
])
def test_balancing_is_cheap(units, E, F, T, limit):
    both, equal = min((units("times", E, F, T)[0] for _ in range(3)), key=lambda t: t[0] / t[1])
    assert both < limit * equal


@pytest.mark.parametrize("vblocks,ngroups", [
    (1, 1), (11, 1), (32, 1), (137, 2), (148, 7), (4096, 1), (4096, 15), (4096, 16), (1, 10000),
])
def test_offset_sums_use_every_sm(units, vblocks, ngroups):
    """No CTA takes a second vector block while another SM could, and short sums, which
    give few warps of a CTA anything to load, have the warps of an SM in several CTAs."""
    sms = 148
    warps, ctas = units("sums", vblocks, ngroups, sms)[0]
    assert min(vblocks, sms) <= ctas <= min(sms * 16 // warps, vblocks * ngroups)
    assert warps <= max(4, ngroups)


@pytest.mark.parametrize("T,rows", [(1, 3), (736, 3), (737, 2), (767, 2), (768, 2), (769, 2)])
def test_two_rows_from_24_steps(units, T, rows):
    """A last step of less than 32 samples counts as one."""
    assert units("rows", T) == [[rows]]


@pytest.mark.parametrize("E,F,T,storing,adding", [
    (256, 16, 16384, 1, 1), (1024, 9, 4096, 1, 1), (512, 30, 2048, 1, 1), (96, 64, 4096, 1, 1),
    (64, 1, 16384, 1, 1), (128, 3, 300001, 1, 1),
    (1024, 4, 1912, 0, 1),                      # zeroing the output would cost more than it gives
    (2048, 8, 16384, 0, 0), (256, 1, 256, 0, 0),  # whole waves; too short to cut
])
def test_which_plans_are_balanced(units, E, F, T, storing, adding):
    """Automatic plans cut units to equal shares per SM where that is worth it, and each
    of their tables covers every tile pair of every channel once, with the units of a
    cut range marked as adding."""
    for add, balanced in ((0, storing), (1, adding)):
        table = units("table", E, F, T, add)
        assert table[0] == [balanced]
        ranges = {}
        for chan, tyx, t0, t1, split, _ in table[1:]:
            ranges.setdefault((chan, tyx), []).append((t0, t1, split))
        assert len(ranges) % F == 0
        for r in ranges.values():
            r.sort()
            assert r[0][0] == 0 and r[-1][1] == T
            assert all(a[1] == b[0] for a, b in zip(r, r[1:]))
            assert all(s == (len(r) > 1) for _, _, s in r)
        if balanced:  # at most one cut per SM besides those of the longest unit
            assert len(ranges) < len(table) - 1 <= len(ranges) * -(-T // 262144) + 148


# us for one unit per SM of two x tiles and of one on the one-SM tile, at 1965 MHz.
ONE_SM_US = {2: {512: 18.7, 4096: 71.9, 16384: 249.7}, 1: {512: 14.4, 4096: 66.2, 16384: 242.0}}


@pytest.mark.parametrize("nx", [1, 2])
@pytest.mark.parametrize("T", [4096, 16384])
def test_one_sm_unit_costs_follow_the_measured_times(units, nx, T):
    """Cycles between two lengths, within 5 %, what a balanced plan has to gain at least.
    E = 256 has one unit with two x tiles and one with one."""
    cost = {t: dict((x, c) for c, x in units("costs", ONE_SM, 256, t))[nx] for t in (512, T)}
    cycles = 1965 * (ONE_SM_US[nx][T] - ONE_SM_US[nx][512])
    assert abs(cost[T] - cost[512] - cycles) < 0.05 * cycles
