"""Calls whose kernels load their input ahead of the wait for the previous kernel (split
correlations and offset sums, behind the kernel that zeroes their output), directly after
a kernel that writes this input: what they read is what that kernel wrote.  Each result
against the same call after a synchronisation, word for word."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SHAPES = [
    (256, 16, 4096),   # SM pair, balanced ranges
    (96, 64, 4096),    # small channels, balanced ranges
    (1024, 2, 4096),   # SM pair
]


@pytest.fixture(scope="module")
def cx():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import chimex
    return chimex


def inputs(n, seed):
    """64 MiB before the packed samples, so that a kernel writing all of it reaches them
    last, and the samples themselves."""
    lead = 64 << 20
    g = torch.Generator(device="cuda").manual_seed(seed)
    noise = torch.randint(0, 256, (lead + n,), dtype=torch.uint8, device="cuda", generator=g)
    buf = torch.empty_like(noise)
    return noise, buf, buf[lead:]


@pytest.mark.parametrize("E,F,T", SHAPES)
@pytest.mark.parametrize("op", ["correlate", "offset_accumulate"])
def test_input_written_by_the_previous_kernel(cx, E, F, T, op):
    p = cx.Plan(E, F, T)
    noise, buf, packed = inputs(p.input_bytes, E + F)
    call = getattr(p, op)
    keys = [3 + 31 * i for i in range(8)]
    ref = []
    for k in keys:
        torch.bitwise_xor(noise, k, out=buf)
        torch.cuda.synchronize()
        ref.append(call(packed))
        torch.cuda.synchronize()
    got = [torch.full_like(ref[0], -1) for _ in keys]
    torch.cuda.synchronize()
    for k, out in zip(keys, got):
        torch.bitwise_xor(noise, k, out=buf)
        call(packed, out)
    p.check_device()
    for a, b in zip(got, ref):
        assert torch.equal(a, b)
    assert not torch.equal(ref[0], ref[1])


@pytest.mark.parametrize("E,F,T", SHAPES)
def test_captured_fork_and_join(cx, E, F, T):
    """One graph: a kernel writes the input, two streams correlate it and sum its
    offsets, and what they wrote is used after they join."""
    p = cx.Plan(E, F, T)
    noise, buf, packed = inputs(p.input_bytes, E + F + 1)
    torch.bitwise_xor(noise, 77, out=buf)
    blocks, sums = p.correlate(packed), p.offset_accumulate(packed)
    seeds = p.preseed(sums)
    want = p.correlate(packed, seeds.clone(), accumulate=True)
    tri = p.blocks_to_triangle(want)
    out, out2 = torch.zeros_like(blocks), torch.zeros_like(blocks)
    osums, otri = torch.zeros_like(sums), torch.zeros_like(tri)
    side = torch.cuda.Stream()
    g = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(g):
        main = torch.cuda.current_stream()
        torch.bitwise_xor(noise, 77, out=buf)
        side.wait_stream(main)
        p.correlate(packed, out)
        with torch.cuda.stream(side):
            p.offset_accumulate(packed, osums)
            p.preseed(osums, out2)
        main.wait_stream(side)
        p.correlate(packed, out2, accumulate=True)
        p.blocks_to_triangle(out2, otri)
    for _ in range(3):
        for t in (buf, out, out2, osums, otri):
            t.zero_()
        g.replay()
        p.check_device()
        assert torch.equal(out, blocks) and torch.equal(osums, sums)
        assert torch.equal(out2, want) and torch.equal(otri, tri)
