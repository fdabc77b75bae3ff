"""The slot sort (one array per block) where its counters, maps and limits
change form: slots of 15 and 16 keys, counter bytes that pass 255, ranges at
the edge of the direct map, 64-bit keys with few high words, the extremes of
the key range, sizes at the edges of the classes.  Sorting is exact, so every
output is compared bit by bit with torch.sort."""
import pytest

pytestmark = pytest.mark.gpu

SIZES = (257, 300, 1023, 1024, 1025, 2047, 2048, 2049, 4095, 4097, 8191, 8193, 16383, 16384)


def _inputs(n, dtype, seed):
    """(name, n keys) for every shape of spread."""
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    bits = 31 if dtype == torch.int32 else 63

    def rnd(lo, hi, m=n):
        return torch.randint(lo, hi, (m,), dtype=dtype, device="cuda", generator=g)

    full = rnd(-(1 << bits), (1 << bits) - 1)
    yield "uniform", full
    for dup in (2, 14, 15, 16, 17, 255, 256, 257):  # keys equal to one key
        t = full.clone()
        t[torch.randperm(n, device="cuda", generator=g)[:min(dup, n)]] = t[0].clone()
        yield f"dup{dup}", t
    cap = 4 * next(c for c in (1024, 2048, 4096, 8192, 16384) if c >= n)  # slots of the block
    for r in (1, 2, 3, cap - 1, cap, cap + 1):  # range at the edge of one slot per value
        t = rnd(-5, r - 4)
        t[0], t[-1] = -5, r - 5
        yield f"range{r}", t
    t = full.clone()
    t[0], t[1] = -(1 << bits), (1 << bits) - 1
    yield "extremes", t
    t = rnd(0, n)
    t[0] = (1 << bits) - 1
    yield "outlier", t
    yield "cluster", torch.where(full > 0, full >> (bits - 16), full)
    yield "ascending", torch.sort(full).values
    for share in (3, 20):  # some values repeat, among spread ones, and one has a few close neighbours
        t = full.clone()
        hot = full[:8][torch.randint(0, 8, (n,), device="cuda", generator=g)]
        t = torch.where(rnd(0, share) == 0, hot, t)
        t[:12] = hot[0] + torch.arange(-6, 6, dtype=dtype, device="cuda")
        yield f"hot{share}", t
    yield "equal", torch.full((n,), -7, dtype=dtype, device="cuda")
    if dtype == torch.int64:
        for hi in (1, 2, 4095, 4096, 4097):  # distinct high words
            yield f"high{hi}", (rnd(0, hi) << 32) + rnd(0, 1 << 32)
            yield f"high{hi}low", (rnd(0, hi) << 32) + rnd(0, 3)


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("dt", ["int32", "int64"])
def test_one_block_arrays(s512, cuda, n, dt):
    import torch
    for name, t0 in _inputs(n, getattr(torch, dt), n):
        t = t0.clone()
        s512.sort(t)
        assert torch.equal(t, torch.sort(t0).values), (name, n)


@pytest.mark.parametrize("n", SIZES)
def test_one_block_doubles(s512, cuda, n):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    u = torch.rand(n, dtype=torch.float64, device="cuda", generator=g)
    z = torch.randn(n, dtype=torch.float64, device="cuda", generator=g)
    for t0 in (u, z, torch.exp(2 * z), u * 1e-300, torch.round(8 * z), torch.round(64 * u) + 1e-9 * z):
        t = t0.clone()
        s512.sort(t)
        assert torch.equal(t, torch.sort(t0).values)


@pytest.mark.parametrize("dt", ["int32", "kv"])
def test_segments_of_every_spread(s512, cuda, dt):
    """The same inputs as the segments of one batch."""
    import torch
    parts = [t for n in SIZES for _, t in _inputs(n, torch.int32, n + 1)]
    keys0 = torch.cat(parts)
    off = torch.zeros(len(parts) + 1, dtype=torch.int64, device="cuda")
    off[1:] = torch.cumsum(torch.tensor([p.numel() for p in parts], device="cuda"), 0)
    k = keys0.clone()
    if dt == "int32":
        s512.segsort(k, off)
        assert torch.equal(k, torch.cat([torch.sort(p).values for p in parts]))
        return
    vals0 = torch.randint(-100, 100, (keys0.numel(),), dtype=torch.int32, device="cuda")
    v = vals0.clone()
    s512.segsort_kv(k, v, off)

    def pack(a, b):  # (key, value) order as one word
        return (a.to(torch.int64) << 32) | (b.to(torch.int64) + (1 << 31))

    word = pack(keys0, vals0)
    want = torch.cat([torch.sort(word[off[i]:off[i + 1]]).values for i in range(len(parts))])
    assert torch.equal(pack(k, v), want)


@pytest.mark.parametrize("n", [4300003, 6000011, 9000001, 14000029])
def test_uneven_leaves_of_large_arrays(s512, cuda, n):
    """Levels large enough for a launch per leaf class, with buckets that the
    slot counts turn away: values that repeat some 18 times, crowded pairs."""
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    for t0 in (torch.randint(0, n // 18, (n,), dtype=torch.int32, device="cuda", generator=g) * 97,
               torch.randint(0, n // 18, (n,), dtype=torch.int64, device="cuda", generator=g) << 33,
               torch.randn(n, dtype=torch.float64, device="cuda", generator=g).mul_(1e4).round_()):
        t = t0.clone()
        s512.sort(t)
        assert torch.equal(t, torch.sort(t0).values)
    k0 = torch.randint(0, n // 60, (n,), dtype=torch.int32, device="cuda", generator=g) * 9973
    v0 = torch.arange(n, dtype=torch.int32, device="cuda")
    k, v = k0.clone(), v0.clone()
    s512.sort_kv(k, v)
    want = torch.sort((k0.to(torch.int64) << 32) | v0.to(torch.int64)).values
    assert torch.equal((k.to(torch.int64) << 32) | v.to(torch.int64), want)
