"""Partition levels whose segments are split at slot boundaries (a bucket from
one table byte) next to those split between keys: keys outside the sample's
range, ranges of just under and over the table's slots, 64-bit ranges of one,
two and many high words, clusters and repeats that must take the other route,
and the exact-count redo, which searches the same boundaries as keys.  Sorting
is exact, so every output is compared bit by bit with torch.sort."""
import pytest

pytestmark = pytest.mark.gpu

SIZES = (16385, 70001, 300007, 1 << 20)
SLOTS = 16384


def _inputs(n, dtype):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    bits = 31 if dtype == torch.int32 else 63

    def rnd(lo, hi):
        return torch.randint(lo, hi, (n,), dtype=dtype, device="cuda", generator=g)

    full = rnd(-(1 << bits), (1 << bits) - 1)
    yield "uniform", full
    t = full >> 3  # a few keys far outside the rest, hardly ever sampled
    t[0], t[1], t[2], t[3] = -(1 << bits), (1 << bits) - 1, -(1 << bits) + 1, (1 << bits) - 2
    yield "outside", t
    for r in (SLOTS - 1, SLOTS, SLOTS + 1, 3 * SLOTS, 1 << 20):
        yield f"range{r}", rnd(-7, r - 7)
    yield "half dense", torch.where(full > 0, full >> 8, full)
    yield "cluster", torch.where(full > 0, full >> (bits - 12), full)
    yield "few", rnd(0, 40) * 1000003
    t = full.clone()
    t[::3] = 12345  # a third of the keys equal
    yield "heavy", t
    yield "ascending", torch.sort(full).values
    yield "descending", torch.sort(full, descending=True).values
    if dtype == torch.int64:
        for hi in (1, 2, 3, 4095, 4097, 1 << 20):
            yield f"high{hi}", (rnd(0, hi) << 32) + rnd(0, 1 << 32)


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("dt", ["int32", "int64"])
@pytest.mark.parametrize("redo", [False, True])
def test_both_routes(s512, cuda, n, dt, redo):
    import torch
    try:
        s512.set_config(fault_inject=s512.FAULT_OVERFLOW if redo else 0)
        for name, t0 in _inputs(n, getattr(torch, dt)):
            t = t0.clone()
            s512.sort(t)
            assert torch.equal(t, torch.sort(t0).values), (name, n)
    finally:
        s512.set_config(fault_inject=0)
