"""The SM-pair kernel at the edges of its dispatch rules, word for word
against the CPU oracle (bit-exact integers: no tolerance)."""
import numpy as np
import pytest

import pyoracle as orc

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def cx():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import chimex
    return chimex


def pair_plan(cx, E, F, T, TA=256, ut=1, kb=0, tsplit=1):
    p = cx.Plan(E, F, T, TA, ut, kb, 0)
    p.set_option(cx.OPT_TILE, 2)
    p.set_option(cx.OPT_TSPLIT, tsplit)
    return p


@pytest.mark.parametrize("T", [32768, 32769, 65600])
def test_longest_scaled_unit(cx, T):
    """Up to 32768 samples per unit the y operand is scaled by 8; one more and
    it is not.  Extreme values (constant -8: |Re| = 128 T, the largest sum) in
    half the elements, random ones in the others."""
    E, F = 160, 1
    packed = orc.generate(T, F, E, 4, 300 + T, no_repeat=1).reshape(T, E)
    packed[:, :80] = 0
    packed = np.ascontiguousarray(packed.reshape(-1))
    p = pair_plan(cx, E, F, T)
    out = p.correlate(torch.from_numpy(packed).cuda())
    p.check_device()
    np.testing.assert_array_equal(out.cpu().numpy(), orc.correlate_channel(packed, T, F, E, 0, 1))


@pytest.mark.parametrize("kb", [0, 1])
@pytest.mark.parametrize("T", [32768, 33024])
def test_longest_scaled_unit_offset_maps(cx, kb, T):
    """The same edge for the reference partials (offset nibbles up to 15: both
    packed bytes 0xFF and 0xF0 reach the largest sums)."""
    E, F = 160, 1
    packed = orc.generate(T, F, E, 4, 400 + T, no_repeat=1).reshape(T, E)
    packed[:, :40] = 0xFF
    packed[:, 40:80] = 0xF0
    packed = np.ascontiguousarray(packed.reshape(-1))
    p = pair_plan(cx, E, F, T, 256, 1, kb)
    zero = torch.zeros(p.block_words, dtype=torch.int32, device="cuda")
    out = p.corr_compat(torch.from_numpy(packed).cuda(), zero)
    p.check_device()
    np.testing.assert_array_equal(out.cpu().numpy(), orc.corr_partials(packed, T, F, E, kb, 1))


@pytest.mark.parametrize("E,F,T", [
    (2048, 1, 1), (2048, 1, 33),          # fewer steps than the lanes' skew
    (256, 3, 384), (256, 3, 416),         # as many steps as the skew, one more
    (384, 2, 500), (1152, 1, 700),        # odd tile counts: one-lane units
    (160, 2, 64), (512, 9, 1000),         # few units: narrow ones
    (512, 40, 450), (384, 80, 450),       # several units per SM pair
])
@pytest.mark.parametrize("tsplit", [0, 1, 2])
def test_skewed_lanes(cx, E, F, T, tsplit):
    """Lane 1 trails lane 0 and wraps around the samples; every channel word
    for word, through the plan, then added once more."""
    packed = orc.generate(T, F, E, 4, 500 + E + T, no_repeat=1)
    ref = np.concatenate([orc.correlate_channel(packed, T, F, E, f, 1) for f in range(F)])
    p = pair_plan(cx, E, F, T, tsplit=tsplit)
    d = torch.from_numpy(packed).cuda()
    out = p.correlate(d)
    np.testing.assert_array_equal(out.cpu().numpy(), ref)
    p.correlate(d, out, accumulate=True)
    p.check_device()
    np.testing.assert_array_equal(out.cpu().numpy(), (ref.astype(np.int64) * 2).astype(np.int32))


@pytest.mark.parametrize("E,F,T", [(256, 1, 40), (384, 2, 70), (512, 8, 1024), (1152, 3, 100),
                                   (2048, 2, 64), (640, 40, 64)])
def test_noalloc_narrow_and_wide_units(cx, E, F, T):
    """The allocation-free entry point derives its units on the device: narrow
    (few units) and wide ones, odd and even tile counts."""
    packed = orc.generate(T, F, E, 4, 600 + E + T, no_repeat=1)
    ref = np.concatenate([orc.correlate_channel(packed, T, F, E, f, 1) for f in range(F)])
    out = torch.empty(ref.size, dtype=torch.int32, device="cuda")
    cx.correlate_noalloc(torch.from_numpy(packed).cuda(), out, E, F, T)
    cx.noalloc_check()
    np.testing.assert_array_equal(out.cpu().numpy(), ref)


@pytest.mark.parametrize("E,F,T", [(1024, 4, 1912), (1024, 4, 330), (256, 75, 200), (128, 150, 400),
                                   (96, 149, 70)])
def test_units_beyond_a_whole_wave(cx, E, F, T):
    """A few units more than the SMs (or SM pairs) take at once may be cut into
    pieces that add to their cells; others of the launch store theirs."""
    packed = orc.generate(T, F, E, 4, 1100 + E + T, no_repeat=1)
    ref = np.concatenate([orc.correlate_channel(packed, T, F, E, f, 0) for f in range(F)])
    p = cx.Plan(E, F, T, 256, 0)
    d = torch.from_numpy(packed).cuda()
    out = torch.full((p.block_words,), 12345, dtype=torch.int32, device="cuda")
    p.correlate(d, out)
    np.testing.assert_array_equal(out.cpu().numpy(), ref)
    p.correlate(d, out, accumulate=True)
    p.check_device()
    np.testing.assert_array_equal(out.cpu().numpy(), (ref.astype(np.int64) * 2).astype(np.int32))
