"""Block layout to packed triangle and full matrix: block rows of every parity
and length, pairs of blocks crossing rows and an odd last block, against the
oracle's reorganisation (integers moved, bit for bit)."""
import numpy as np
import pytest

import pyoracle as orc

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("E,F", [(32, 1), (32, 3), (64, 2), (96, 5), (160, 3), (224, 1), (1888, 1),
                                 (2048, 2)])
def test_triangle_and_full(E, F):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import chimex as cx
    rng = np.random.default_rng(E + F)
    blocks = rng.integers(-2**31, 2**31, F * orc.num_blocks(E) * 2048, dtype=np.int64).astype(np.int32)
    p = cx.Plan(E, F, 64)
    d = torch.from_numpy(blocks).cuda()
    guard = 64  # words behind the triangle stay untouched
    buf = torch.full((p.triangle_words + guard,), 77, dtype=torch.int32, device="cuda")
    p.blocks_to_triangle(d, buf[:p.triangle_words])
    np.testing.assert_array_equal(buf[:p.triangle_words].cpu().numpy(),
                                  orc.blocks_to_triangle(blocks, F, E))
    assert bool((buf[p.triangle_words:] == 77).all())
    np.testing.assert_array_equal(p.blocks_to_full(d).cpu().numpy(), orc.blocks_to_full(blocks, F, E))
