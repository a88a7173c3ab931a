"""The kernel for channels of at most 128 elements, word for word against the
CPU oracle (bit-exact integers: no tolerance)."""
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


@pytest.mark.parametrize("E", [32, 64, 96, 128])
@pytest.mark.parametrize("F,T,tsplit,ut", [
    (1, 1, 0, 1), (2, 31, 0, 0), (3, 33, 1, 1),   # one stage, its remainder
    (1, 2000, 0, 1), (5, 1000, 3, 0),             # split sample ranges
    (400, 100, 1, 1),                             # several units per SM: both buffers
    (160, 640, 2, 1),
])
def test_small_channels(cx, E, F, T, tsplit, ut):
    packed = orc.generate(T, F, E, 4, 700 + E + F + T, no_repeat=1)
    ref = orc.correlate_blocks(packed, T, F, E, ut)
    p = cx.Plan(E, F, T, 256, ut)
    p.set_option(cx.OPT_TSPLIT, tsplit)
    d = torch.from_numpy(packed).cuda()
    out = p.correlate(d)
    np.testing.assert_array_equal(out.cpu().numpy(), ref)
    p.correlate(d, out, accumulate=True)
    p.check_device()
    np.testing.assert_array_equal(out.cpu().numpy(), (ref.astype(np.int64) * 2).astype(np.int32))


@pytest.mark.parametrize("E", [32, 96, 128])
@pytest.mark.parametrize("kb,ut", [(0, 1), (0, 0), (1, 1), (1, 0)])
def test_small_channels_offset_maps(cx, E, kb, ut):
    T, F = 512, 1 if kb else 3
    packed = orc.generate(T, F, E, 4, 800 + E, no_repeat=1)
    packed[:E] = 0xFF
    p = cx.Plan(E, F, T, 256, ut, kb)
    zero = torch.zeros(p.block_words, dtype=torch.int32, device="cuda")
    out = p.corr_compat(torch.from_numpy(packed).cuda(), zero)
    p.check_device()
    np.testing.assert_array_equal(out.cpu().numpy(), orc.corr_partials(packed, T, F, E, kb, ut))


@pytest.mark.parametrize("T", [262144, 262145])
def test_small_channel_longest_unit(cx, T):
    """Constant -8 (the largest sums) up to the longest unit, and one sample more."""
    E = 64
    p = cx.Plan(E, 1, T)
    p.set_option(cx.OPT_TSPLIT, 1)
    out = p.correlate(torch.zeros(T * E, dtype=torch.uint8, device="cuda"))
    p.check_device()
    out = out.view(-1, 2)
    assert bool((out[:, 0] == 128 * T).all()) and bool((out[:, 1] == 0).all())


def test_ragged_batch_of_small_channels(cx):
    """Own element counts per launch: the MMA width follows the channel."""
    shapes = [(32, 100, 3), (128, 77, 2), (96, 500, 1), (64, 64, 4)]
    chans, refs = [], []
    for E, T, n in shapes:
        packed = orc.generate(n * T, 1, E, 4, 900 + E, no_repeat=1)
        refs.append(np.concatenate([orc.correlate_blocks(packed[i * T * E:(i + 1) * T * E], T, 1, E, 1)
                                    for i in range(n)]))
        out = torch.empty(refs[-1].size, dtype=torch.int32, device="cuda")
        chans.append((torch.from_numpy(packed).cuda(), out, E, T, n))
    b = cx.Batch(chans)
    b.run()
    b.check_device()
    for ch, ref in zip(chans, refs):
        np.testing.assert_array_equal(ch[1].cpu().numpy(), ref)


@pytest.mark.parametrize("E,F,T,tsplit", [(64, 3, 500, 1), (256, 2, 700, 2), (512, 1, 300, 1)])
def test_captured_launches_overlap_safely(cx, E, F, T, tsplit):
    """A user's own graph over several calls (zeroing, overwrite, add): the
    launches' set-up may overlap, their work may not."""
    packed = orc.generate(T, F, E, 4, 1000 + E, no_repeat=1)
    ref = np.concatenate([orc.correlate_channel(packed, T, F, E, f, 1) for f in range(F)])
    p = cx.Plan(E, F, T)
    p.set_option(cx.OPT_TSPLIT, tsplit)
    d = torch.zeros(packed.size, dtype=torch.uint8, device="cuda")
    out = p.correlate(d)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        p.correlate(d, out)
        p.correlate(d, out, accumulate=True)
        tri = p.blocks_to_triangle(out)
        p.correlate(d, out, accumulate=True)
    d.copy_(torch.from_numpy(packed))
    for _ in range(3):
        g.replay()
    p.check_device()
    np.testing.assert_array_equal(out.cpu().numpy(), (3 * ref.astype(np.int64)).astype(np.int32))
    np.testing.assert_array_equal(
        tri.cpu().numpy(), orc.blocks_to_triangle((2 * ref.astype(np.int64)).astype(np.int32), F, E))


@pytest.mark.parametrize("E", [32, 64, 96, 128])
@pytest.mark.parametrize("F,T,tsplit,ut", [
    (2, 736, 1, 1), (2, 737, 1, 0),     # 23 and 24 stages: below and at the two-row rule
    (2, 768, 1, 1), (1, 769, 1, 0),     # whole stages, one sample of the next
    (320, 800, 1, 1), (160, 1600, 2, 0),  # several units per SM, split
    (150, 1500, 0, 1),                  # balanced pieces, short ones among them
])
def test_two_row_units(cx, E, F, T, tsplit, ut):
    """Units whose imaginary part is K - K^T, storing and adding."""
    packed = np.random.default_rng(E + F + T).integers(0, 256, T * F * E, dtype=np.uint8)
    p = cx.Plan(E, F, T, 256, ut)
    p.set_option(cx.OPT_TSPLIT, tsplit)
    d = torch.from_numpy(packed).cuda()
    out = p.correlate(d)
    p.check_device()
    got = out.view(F, -1).cpu().numpy()
    for f in {0, F // 2, F - 1}:
        chan = np.ascontiguousarray(packed.reshape(T, F, E)[:, f]).reshape(-1)
        np.testing.assert_array_equal(got[f], orc.correlate_blocks(chan, T, 1, E, ut).reshape(-1))
    twice = p.correlate(d, out.clone(), accumulate=True)
    p.check_device()
    assert torch.equal(twice, out * 2)


@pytest.mark.parametrize("E", [32, 96, 128])
@pytest.mark.parametrize("kb,ut", [(0, 1), (0, 0), (1, 1), (1, 0)])
def test_two_row_offset_maps(cx, E, kb, ut):
    """The offset-domain maps at lengths where the first multiplies two rows."""
    T, F = 1024, 1 if kb else 3
    packed = orc.generate(T, F, E, 4, 810 + E, no_repeat=1)
    packed[:E] = 0xFF
    p = cx.Plan(E, F, T, 256, ut, kb)
    p.set_option(cx.OPT_TSPLIT, 1)
    zero = torch.zeros(p.block_words, dtype=torch.int32, device="cuda")
    out = p.corr_compat(torch.from_numpy(packed).cuda(), zero)
    p.check_device()
    np.testing.assert_array_equal(out.cpu().numpy(), orc.corr_partials(packed, T, F, E, kb, ut))
