"""The merge path at the edges of its tiles and of the co-rank search: every
split of small arrays, lopsided splits, ties (a stable merge takes the left run
first: seen on signed zeros), more pairs than travel with a launch.  Merging is
exact, so outputs are compared bit by bit."""
import pytest

pytestmark = pytest.mark.gpu

TILE = 4096


def _runs(torch, n, mid, dt, g, lo, hi):
    x = torch.randint(lo, hi, (n,), dtype=torch.int32, device="cuda", generator=g).to(dt)
    x[:mid] = torch.sort(x[:mid]).values
    x[mid:] = torch.sort(x[mid:]).values
    return x


@pytest.mark.parametrize("dt", ["int32", "float64"])
@pytest.mark.parametrize("n", [2, 3, 17, 255, TILE - 1, TILE, TILE + 1, 3 * TILE + 5, 300007])
def test_merge_splits(s512, cuda, n, dt):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    dtype = getattr(torch, dt)
    for mid in sorted({1, 2, n // 3, n // 2, n - 2, n - 1, min(n - 1, TILE), min(n - 1, 8), min(n - 1, 9), min(n - 1, 10)}):
        if not 0 < mid < n:
            continue
        for lo, hi in ((-(1 << 31), (1 << 31) - 1), (0, 3), (5, 6)):
            x = _runs(torch, n, mid, dtype, g, lo, hi)
            want = torch.sort(x).values
            s512.merge(x, mid)
            assert torch.equal(x, want), (n, mid, lo)
    for first in (True, False):  # disjoint runs, either order
        x = torch.arange(n, device="cuda").to(dtype)
        if not first:
            x = torch.roll(x, n // 2)
            mid = n // 2
        else:
            mid = n // 3
        if 0 < mid < n:
            s512.merge(x, mid)
            assert torch.equal(x, torch.arange(n, device="cuda").to(dtype))


def test_merge_takes_the_left_run_first(s512, cuda):
    import torch
    for n, mid in ((6000, 2500), (9001, 8000)):
        x = torch.zeros(n, dtype=torch.float64, device="cuda")
        x[:mid] = -0.0  # equal to +0.0: the left run's come first
        s512.merge(x, mid)
        neg = torch.signbit(x)
        assert bool(neg[:mid].all()) and not bool(neg[mid:].any())


@pytest.mark.parametrize("parts", [2, 3, 31, 32, 33, 34, 100])
def test_sort_omp_merge_many_parts(s512, cuda, parts):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(parts)
    for n in (parts, 50021, 400009):
        x0 = torch.randint(-1000, 1 << 30, (n,), dtype=torch.int32, device="cuda", generator=g)
        x = x0.clone()
        s512.sort_omp_merge(x, parts)
        assert torch.equal(x, torch.sort(x0).values)
