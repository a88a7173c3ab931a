"""Plans whose sample ranges are cut to equal shares per SM against the same plan
unsplit, and against the CPU oracle on two channels, word for word (bit-exact
integers: no tolerance), storing and adding."""
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


@pytest.mark.parametrize("E,F,T,tile,ut", [
    (256, 16, 4096, 0, 1),    # fewer units than SM pairs
    (160, 100, 3000, 0, 0),   # ragged elements, a remainder of 24 samples
    (512, 30, 2048, 0, 1),    # a full wave and a half
    (384, 7, 1913, 0, 1),     # units of one lane among those of two
    (1024, 4, 1912, 0, 0),    # cut only where the output is added to
    (96, 64, 4096, 0, 1), (64, 1, 16384, 0, 0), (32, 300, 1024, 0, 1),
    (128, 3, 300001, 0, 1),   # longer than one unit may be
    (640, 3, 3000, 1, 1),     # one-SM tile
    (256, 75, 512, 0, 1), (256, 73, 257, 0, 1),  # next to a whole wave
    (256, 1, 8 * 32, 0, 1), (256, 1, 17 * 32 + 1, 0, 1),  # about the shortest pieces
])
def test_balanced_units(cx, E, F, T, tile, ut):
    packed = torch.from_numpy(np.random.default_rng(E + F + T).integers(
        0, 256, T * F * E, dtype=np.uint8)).cuda()
    one, p = cx.Plan(E, F, T, 256, ut), cx.Plan(E, F, T, 256, ut)
    one.set_option(cx.OPT_TILE, tile)
    one.set_option(cx.OPT_TSPLIT, 1)
    p.set_option(cx.OPT_TILE, tile)
    ref = one.correlate(packed)
    out = torch.full_like(ref, 7)
    p.correlate(packed, out)
    p.check_device()
    assert torch.equal(out, ref)
    p.correlate(packed, out, accumulate=True)
    p.check_device()
    assert torch.equal(out, ref * 2)
    for f in {0, F - 1}:
        chan = np.ascontiguousarray(packed.view(T, F, E)[:, f].cpu().numpy()).reshape(-1)
        np.testing.assert_array_equal(ref.view(F, -1)[f].cpu().numpy().reshape(-1),
                                      orc.correlate_blocks(chan, T, 1, E, ut).reshape(-1))
