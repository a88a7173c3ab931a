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
