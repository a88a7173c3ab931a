"""Work of one stream beside launches of another that leave SMs idle: a launch
that waits for its predecessor must not hold the SMs that are left."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def cx():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import chimex
    return chimex


# Two such calls together need every SM of the GPU, one of them at most 100.
@pytest.mark.parametrize("E,F,tile", [
    (128, 37, 2),   # 37 SM pairs
    (64, 100, 0),   # 100 SMs (one tile per channel)
])
def test_second_stream_runs_beside_waiting_launch(cx, E, F, tile):
    T = 262144  # one unit per channel, at least a millisecond
    a, b = cx.Plan(E, F, T), cx.Plan(256, 16, 512)
    a.set_option(cx.OPT_TILE, tile)
    a.set_option(cx.OPT_TSPLIT, 1)
    da = torch.zeros(a.input_bytes, dtype=torch.uint8, device="cuda")
    db = torch.zeros(b.input_bytes, dtype=torch.uint8, device="cuda")
    oa, ob = a.correlate(da), b.correlate(db)
    sa, sb = torch.cuda.Stream(), torch.cuda.Stream()
    start, a_end, b_end = (torch.cuda.Event(enable_timing=True) for _ in range(3))
    shares = []
    for _ in range(5):
        torch.cuda.synchronize()
        with torch.cuda.stream(sa):
            start.record()
            a.correlate(da, oa)
            a.correlate(da, oa)
            a_end.record()
        with torch.cuda.stream(sb):
            b.correlate(db, ob)
            b_end.record()
        torch.cuda.synchronize()
        shares.append(start.elapsed_time(b_end) / start.elapsed_time(a_end))
    a.check_device()
    b.check_device()
    # Behind the first of A's calls it would end after half of A's time at the
    # earliest; it needs about 20 us of SM time.
    assert sorted(shares)[2] < 0.25, shares
