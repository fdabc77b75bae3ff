"""The two-way partition at the edges of its rows, runs and blocks, on ranges that
start at odd places: lows in input order, then highs in reverse input order,
exactly, and nothing written outside the range."""
import pytest

pytestmark = pytest.mark.gpu

# rows are 32 elements, a warp's smallest run 256, a block's 2048; the grid
# stops growing at 1184 blocks (2424832 elements)
SIZES = (1, 31, 32, 33, 255, 256, 257, 2047, 2048, 2049, 65537, 1048575, 1048577, 2424831, 2424832, 2424833, 6000011)


def _want(k, pivot, *more):
    import torch
    low = k <= pivot
    return [torch.cat((t[low], t[~low].flip(0))) for t in (k, *more)], int(low.sum())


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("dt", ["int32", "float64"])
def test_arrangement(s512, cuda, n, dt):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    for left in (0, 3):
        if dt == "int32":
            base = torch.randint(-1000, 1000, (n + 5,), dtype=torch.int32, device=cuda, generator=g)
            pivots = (-2000, -1000, 0, 7, 999, 2000)
        else:
            base = torch.randn(n + 5, dtype=torch.float64, device=cuda, generator=g)
            base[::7] = float("nan")  # NaN is never <= pivot
            pivots = (float("-inf"), -0.5, 0.0, 1.0, float("inf"))
        for pivot in pivots:
            a = base.clone()
            lim = s512.partition(a, left, left + n - 1, pivot)
            (want,), low = _want(base[left:left + n], pivot)
            assert lim == left + low
            assert torch.equal(a[left:left + n].nan_to_num(nan=9e9), want.nan_to_num(nan=9e9)) if dt == "float64" \
                else torch.equal(a[left:left + n], want)
            for part in (slice(0, left), slice(left + n, n + 5)):
                assert torch.equal(a[part].nan_to_num(), base[part].nan_to_num()) if dt == "float64" \
                    else torch.equal(a[part], base[part])


@pytest.mark.parametrize("n", SIZES)
def test_arrangement_kv(s512, cuda, n):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    k0 = torch.randint(-50, 50, (n,), dtype=torch.int32, device=cuda, generator=g)
    v0 = torch.arange(n, dtype=torch.int32, device=cuda)
    for pivot in (-51, 0, 30, 49):
        k, v = k0.clone(), v0.clone()
        lim = s512.partition_kv(k, v, 0, n - 1, pivot)
        (wk, wv), low = _want(k0, pivot, v0)
        assert lim == low and torch.equal(k, wk) and torch.equal(v, wv)
