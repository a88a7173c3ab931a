"""Offset sums at the edges of the kernel's work split, against the CPU oracle
(integer sums: no tolerance)."""
import numpy as np
import pytest

import pyoracle as orc

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("E,F,T", [
    (32, 1, 1), (32, 1, 15), (32, 1, 17),         # one partial group, a group and one sample
    (96, 3, 127), (96, 3, 129),                   # the fewest groups per CTA, one more
    (512, 1, 2048), (544, 1, 2047),               # one vector block, a partial second one
    (2048, 2, 3000), (1120, 5, 1111),             # shares crossing vector blocks
])
def test_offset_sums(E, F, T):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import chimex as cx
    packed = orc.generate(T, F, E, 4, 50 + E + T, no_repeat=1)
    packed[:E * F] = 0xFF
    ref = orc.offset_accumulate(packed, T, F, E)
    p = cx.Plan(E, F, T)
    d = torch.from_numpy(packed).cuda()
    sums = torch.full((p.sum_words,), -1, dtype=torch.int32, device="cuda")
    for _ in range(3):  # each call zeroes first
        p.offset_accumulate(d, sums)
    np.testing.assert_array_equal(sums.cpu().numpy().view(np.uint32), ref)
    p.offset_accumulate(d, sums, accumulate=True)
    np.testing.assert_array_equal(sums.cpu().numpy().view(np.uint32), 2 * ref)


@pytest.mark.parametrize("E,F,T", [
    (96, 55, 1), (96, 55, 2),                     # less than a group in each vector block
    (2048, 8, 16), (2048, 8, 17),                 # one group, one sample of the next
    (2048, 300, 1), (2048, 150, 33),              # more vector blocks than CTAs
    (544, 3, 240), (544, 3, 241), (2048, 4, 255),  # the most groups in short CTAs, one more
])
@pytest.mark.parametrize("accumulate", [False, True])
def test_short_offset_sums(E, F, T, accumulate):
    """Few samples: CTAs of four warps, whole vector blocks."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import chimex as cx
    packed = np.random.default_rng(E + F + T).integers(0, 256, T * F * E, dtype=np.uint8)
    packed[:E * F] = 0xFF
    ref = orc.offset_accumulate(packed, T, F, E)
    p = cx.Plan(E, F, T)
    d = torch.from_numpy(packed).cuda()
    sums = torch.full((p.sum_words,), 5, dtype=torch.int32, device="cuda")
    for _ in range(2):
        p.offset_accumulate(d, sums, accumulate=accumulate)
    ref = ref * 2 + 5 if accumulate else ref
    np.testing.assert_array_equal(sums.cpu().numpy().view(np.uint32), ref)
