"""Representative calls of the correlator's public entry points, for timing.

Each case is one call pattern of a program that uses this library, with the
sizes such a program has: element counts from a small array (32) to the full
telescope (2048), one to many frequency channels, integrations from a few
hundred samples to 16384.  listed() names the fixed ones, draw() gives more of
the same ranges, run() makes the calls and exact() computes the same outputs
with 64-bit torch arithmetic.
"""
import os
import sys

import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "chime-x_b200"))

import chimex as cx  # noqa: E402

DEV = torch.device("cuda", 0)


def listed():
    return [
        # Smallest call: one channel of a 256-element array, one 256-sample
        # integration per call.  Latency of a single launch.
        {"name": "plain_e256_f1_t256", "kind": "plain", "E": 256, "F": 1, "T": 256, "ut": 1},
        # One compute node of a 256-element array: many samples, few blocks.
        {"name": "plain_e256_f16_t16384", "kind": "plain", "E": 256, "F": 16, "T": 16384,
         "ut": 1},
        # The full telescope: the bench's headline workload.
        {"name": "plain_e2048_f8_t16384", "kind": "plain", "E": 2048, "F": 8, "T": 16384,
         "ut": 1},
        # An array whose elements do not fill the tiles, a sample count that
        # is no multiple of a stage, and the other triangle convention.
        {"name": "plain_e1888_f4_t10001", "kind": "plain", "E": 1888, "F": 4, "T": 10001,
         "ut": 0},
        # A small test array (less than one tile) with many channels.
        {"name": "plain_e96_f64_t4096", "kind": "plain", "E": 96, "F": 64, "T": 4096, "ut": 1},
        # A long integration arriving in parts: the first call overwrites the
        # blocks, the others add to them (time_accum 1912 of the overflow test).
        {"name": "integrate_e1024_f4_t1912x4", "kind": "integrate", "E": 1024, "F": 4,
         "T": 1912, "parts": 4, "ut": 1},
        # The per-frame loop of a real-time correlator that may not allocate.
        {"name": "noalloc_e512_f8_t1024", "kind": "noalloc", "E": 512, "F": 8, "T": 1024,
         "ut": 1},
        # 64 channels with their own element counts and integration lengths in
        # one graph launch, four integrations each: the bench's batched workload.
        {"name": "batch_64ch", "kind": "batch", "channels": 64, "integrations": 4, "shapes": 42,
         "ut": 1},
        # Streaming: four frame ticks complete one integration of every channel
        # (70 % E=2048, 30 % E=1024, 256-sample frames, as the bench's stream
        # workload, 48 channels).
        {"name": "stream_48ch_t1024", "kind": "stream", "channels": 48, "frame": 256,
         "ticks": 4, "shapes": 42, "ut": 1},
        # The reference's own pipeline: offset sums, preseed, corr.
        {"name": "pipeline_e2048_f4_t8192", "kind": "pipeline", "E": 2048, "F": 4, "T": 8192,
         "time_accum": 256, "packed_kernel": False, "ut": 1},
        # Offset sums of one full buffer on their own.
        {"name": "offsets_e2048_f8_t16384", "kind": "offsets", "E": 2048, "F": 8, "T": 16384,
         "ut": 1},
        # Handing the visibilities on as a packed triangle.
        {"name": "triangle_e2048_f8", "kind": "reorg", "E": 2048, "F": 8, "to": "triangle",
         "ut": 1},
    ]


# No drawn case does more padded work than the listed full-telescope one:
# tensor work counted in whole 256-element tiles, and bytes.
MAX_TILE_SAMPLES = 36 * 8 * 16384 // 2
MAX_BYTES = 256 << 20


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def _elements(rng, lo=32, hi=2048):
    return max(lo, min(hi, 32 * round(_log(rng, lo, hi) / 32)))


def _tiles(E):
    n = (E + 255) // 256
    return n * (n + 1) // 2


def _sized(rng, E, f_max, t_lo, t_hi):
    """(F, T) whose work and bytes stay below the caps."""
    while True:
        F, T = _log(rng, 1, f_max), _log(rng, t_lo, t_hi)
        if (_tiles(E) * F * T <= MAX_TILE_SAMPLES and F * T * E <= MAX_BYTES
                and F * cx.num_blocks(E) * 8192 <= MAX_BYTES):
            return F, T


def draw(rng):
    kind = rng.choice(["plain"] * 6 + ["integrate", "noalloc", "noalloc", "batch", "batch",
                                       "stream", "pipeline", "offsets", "reorg", "reorg"])
    ut = rng.choice([1, 1, 0])
    if kind == "batch":
        return {"kind": kind, "channels": _log(rng, 4, 64), "integrations": rng.randint(1, 4),
                "shapes": rng.randrange(1 << 20), "ut": ut}
    if kind == "stream":
        ticks = rng.choice([1, 2, 4])
        return {"kind": kind, "channels": _log(rng, 4, 48), "frame": 32 * rng.randint(4, 32 // ticks),
                "ticks": ticks, "shapes": rng.randrange(1 << 20), "ut": ut}
    E = _elements(rng)
    if kind == "plain":
        F, T = _sized(rng, E, 64, 64, 16384)
        return {"kind": kind, "E": E, "F": F, "T": T, "ut": ut}
    if kind == "integrate":
        F, T = _sized(rng, E, 16, 64, 1912)
        return {"kind": kind, "E": E, "F": F, "T": T, "parts": rng.randint(2, 4), "ut": ut}
    if kind == "noalloc":
        F, T = _sized(rng, E, 32, 64, 4096)
        return {"kind": kind, "E": E, "F": F, "T": T, "ut": ut}
    if kind == "pipeline":
        packed = rng.random() < 0.3
        F, T = _sized(rng, E, 8, 256, 8192)
        return {"kind": kind, "E": E, "F": 1 if packed else F, "T": 256 * (T // 256),
                "time_accum": 256, "packed_kernel": packed, "ut": ut}
    if kind == "offsets":
        F, T = _sized(rng, E, 64, 256, 16384)
        return {"kind": kind, "E": E, "F": F, "T": T, "ut": ut}
    while True:
        F = _log(rng, 1, 64)
        to = rng.choice(["triangle", "full"])
        if F * cx.num_blocks(E) * (8192 if to == "triangle" else 16384) <= MAX_BYTES:
            return {"kind": kind, "E": E, "F": F, "to": to, "ut": ut}


def _batch_shapes(case):
    """(E, time_accum) of every channel."""
    import numpy as np
    rng = np.random.default_rng(case["shapes"])
    n = case["channels"]
    Es = [int(e) for e in rng.choice([256, 512, 1024, 1536, 2048], size=n)]
    Ts = [int(t) for t in rng.integers(64, 1913, size=n)]
    return list(zip(Es, Ts))


def _stream_shapes(case):
    """Element counts: 70 % 2048, 30 % 1024."""
    import numpy as np
    n = case["channels"]
    n_big = (7 * n + 9) // 10
    Es = [2048] * n_big + [1024] * (n - n_big)
    np.random.default_rng(case["shapes"]).shuffle(Es)
    return [int(e) for e in Es]


def _samples(n, seed):
    """n packed samples, both nibbles uniform (re, im uniform in [-8, 7])."""
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    return torch.randint(0, 256, (n,), dtype=torch.uint8, device=DEV, generator=gen)


def _empty(n):
    return torch.empty(n, dtype=torch.int32, device=DEV)


def prepare(case, seed):
    kind, ut = case["kind"], case["ut"]
    st = {"case": case, "kind": kind}
    if kind == "batch":
        shapes = _batch_shapes(case)
        nint = case["integrations"]
        packed = _samples(sum(nint * T * E for E, T in shapes), seed)
        st["blocks"] = _empty(sum(nint * cx.num_blocks(E) * 2048 for E, _ in shapes))
        chans, i, o = [], 0, 0
        for E, T in shapes:
            ni, no = nint * T * E, nint * cx.num_blocks(E) * 2048
            chans.append((packed[i:i + ni], st["blocks"][o:o + no], E, T, nint))
            i, o = i + ni, o + no
        st["batch"] = cx.Batch(chans, ut, DEV.index)
        return st
    if kind == "stream":
        Es = _stream_shapes(case)
        st["stream"] = cx.Stream(len(Es), case["frame"], ut, 0, DEV.index)
        st["ids"] = [st["stream"].admit(E, case["frame"] * case["ticks"]) for E in Es]
        st["packed"] = _samples(case["ticks"] * case["frame"] * sum(Es), seed)
        at, st["frames"] = st["packed"].data_ptr(), []
        for _ in range(case["ticks"]):  # one list of frame addresses per tick
            st["frames"].append([])
            for E in Es:
                st["frames"][-1].append(at)
                at += case["frame"] * E
        return st
    E, F = case["E"], case["F"]
    T = case.get("T", 256)
    kb = cx.KERNEL_PACKED if case.get("packed_kernel") else cx.KERNEL_CONFERENCE
    if kind != "noalloc":
        st["plan"] = cx.Plan(E, F, T, case.get("time_accum", 256), ut, kb, DEV.index)
    n_blocks = F * cx.num_blocks(E) * 2048
    if kind == "reorg":
        gen = torch.Generator(device=DEV)
        gen.manual_seed(seed)
        st["blocks"] = torch.randint(-128 * 16384, 128 * 16384, (n_blocks,), dtype=torch.int32,
                                     device=DEV, generator=gen)
        st["out"] = _empty(F * E * (E + 1) if case["to"] == "triangle" else F * E * E * 2)
        return st
    parts = case.get("parts", 1)
    st["packed"] = list(_samples(parts * T * F * E, seed).view(parts, -1))
    if kind == "offsets":
        st["sums"] = _empty(F * E * 2)
    else:
        st["blocks"] = _empty(n_blocks)
    if kind == "pipeline":
        st["sums"] = _empty(F * E * 2)
    return st


def run(st):
    kind = st["kind"]
    if kind == "plain":
        return st["plan"].correlate(st["packed"][0], st["blocks"])
    if kind == "integrate":
        for i, part in enumerate(st["packed"]):
            st["plan"].correlate(part, st["blocks"], accumulate=i > 0)
        return st["blocks"]
    if kind == "noalloc":
        c = st["case"]
        return cx.correlate_noalloc(st["packed"][0], st["blocks"], c["E"], c["F"], c["T"], c["ut"])
    if kind == "batch":
        st["batch"].run()
        return st["blocks"]
    if kind == "stream":
        s = st["stream"]
        for frames in st["frames"]:
            s.submit(st["ids"], frames)
        s.sync()  # a program reads a dump once it is published
        dumps = []
        for cid in st["ids"]:
            dump = s.last_dump_tensor(cid)[0]
            dump.stream = s  # the view's memory belongs to the stream
            dumps.append(dump)
        return dumps
    if kind == "pipeline":
        plan, packed = st["plan"], st["packed"][0]
        plan.offset_accumulate(packed, st["sums"])
        plan.preseed(st["sums"], st["blocks"])
        plan.corr_compat(packed, st["blocks"])
        return {"sums": st["sums"], "blocks": st["blocks"]}
    if kind == "offsets":
        return st["plan"].offset_accumulate(st["packed"][0], st["sums"])
    if st["case"]["to"] == "triangle":
        return st["plan"].blocks_to_triangle(st["blocks"], st["out"])
    return st["plan"].blocks_to_full(st["blocks"], st["out"])


def _channels(case):
    """(E, samples per integration, integrations) of every correlated channel."""
    kind = case["kind"]
    if kind == "batch":
        return [(E, T, case["integrations"]) for E, T in _batch_shapes(case)]
    if kind == "stream":
        return [(E, case["frame"] * case["ticks"], 1) for E in _stream_shapes(case)]
    return [(case["E"], case["T"] * case.get("parts", 1), 1)] * case["F"]


def work(case):
    """Input read once, output written once; 8 operations per visibility and
    sample (a complex multiply-add) over the upper triangle."""
    if case["kind"] == "reorg":
        E, F = case["E"], case["F"]
        out = F * E * (E + 1) * 4 if case["to"] == "triangle" else F * E * E * 8
        return {"bytes": float(F * cx.num_blocks(E) * 8192 + out), "flops": 0.0}
    if case["kind"] == "offsets":
        n = case["F"] * case["E"]
        return {"bytes": float(n * case["T"] + 8 * n), "flops": 2.0 * n * case["T"]}
    b = f = 0.0
    for E, T, nint in _channels(case):
        b += nint * (E * T + cx.num_blocks(E) * 8192)
        f += nint * 8.0 * E * (E + 1) / 2 * T
    if case["kind"] == "pipeline":
        b += 8.0 * case["F"] * case["E"]
    return {"bytes": b, "flops": f}


def _unpack(packed):
    """(re, im) of packed samples as float64."""
    return (packed >> 4).double() - 8, (packed & 15).double() - 8


def _blocks64(packed, E, ut):
    """Block layout [NB * 2048] int64 of one channel's samples [T, E]."""
    re = torch.zeros(E, E, dtype=torch.float64, device=packed.device)
    im = torch.zeros_like(re)
    for part in packed.split(8192):
        r, i = _unpack(part)
        re += r.T @ r + i.T @ i
        im += i.T @ r - r.T @ i
    if not ut:
        im = -im
    n = E // 32
    v = torch.stack([re, im], -1).round().long().view(n, 32, n, 32, 2)
    by, bx = torch.triu_indices(n, n, device=packed.device)
    return v[by, :, bx].reshape(-1)


def exact(case, seed):
    kind, ut = case["kind"], case["ut"]
    if kind == "reorg":
        E, F, n = case["E"], case["F"], case["E"] // 32
        blocks = prepare(case, seed)["blocks"].long().view(F, -1, 32, 32, 2)
        by, bx = torch.triu_indices(n, n, device=DEV)
        outs = []
        y, x = torch.triu_indices(E, E, device=DEV)
        for f in range(F):
            m = torch.zeros(n, 32, n, 32, 2, dtype=torch.int64, device=DEV)
            m[by, :, bx] = blocks[f]
            m = m.view(E, E, 2)
            if case["to"] == "triangle":
                outs.append(m[y, x].reshape(-1))
            else:
                re, im = m[..., 0].triu(), m[..., 1].triu()
                re = re + re.triu(1).T
                im = im - im.triu(1).T
                outs.append(torch.stack([re, im], -1).reshape(-1))
        return torch.cat(outs)
    if kind == "batch":
        shapes, nint = _batch_shapes(case), case["integrations"]
        packed = _samples(sum(nint * T * E for E, T in shapes), seed)
        outs, at = [], 0
        for E, T in shapes:
            for _ in range(nint):
                outs.append(_blocks64(packed[at:at + T * E].view(T, E), E, ut))
                at += T * E
        return torch.cat(outs)
    if kind == "stream":
        Es, ticks, frame = _stream_shapes(case), case["ticks"], case["frame"]
        packed = _samples(ticks * frame * sum(Es), seed).view(ticks, -1)
        outs, at = [], 0
        for E in Es:
            outs.append(_blocks64(packed[:, at:at + frame * E].reshape(-1, E), E, ut))
            at += frame * E
        return outs
    E, F, T = case["E"], case["F"], case["T"] * case.get("parts", 1)
    packed = _samples(T * F * E, seed).view(T, F, E)
    sums = None
    if kind in ("offsets", "pipeline"):
        hi = (packed >> 4).long().sum(0)
        lo = (packed & 15).long().sum(0)
        sums = torch.stack([hi, lo], -1).reshape(-1)
        if kind == "offsets":
            return sums
    blocks = torch.cat([_blocks64(packed[:, f], E, ut) for f in range(F)])
    return blocks if sums is None else {"sums": sums, "blocks": blocks}
