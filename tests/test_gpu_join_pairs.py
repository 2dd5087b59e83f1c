"""Joins on two columns whose windows of right keys do not fit shared memory
(5632 pairs): the bounds are found between samples of the window, at every
distance of the samples, with runs of equal keys inside, over and across them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
W = 5632


def check(ctx, lk, rk):
    """lk, rk: sorted 64-bit keys."""
    import vedas_gb300 as vg

    cols = [[(k >> np.uint64(32)).astype(np.uint32), k.astype(np.uint32),
             np.arange(k.shape[0], dtype=np.uint32) * np.uint32(3) + np.uint32(s)] for s, k in enumerate((lk, rk))]
    l, r = (vg.Relation.from_host(ctx, c) for c in cols)
    out = vg.join2(ctx, l, r)
    lo, hi = np.searchsorted(rk, lk, "left"), np.searchsorted(rk, lk, "right")
    n = hi - lo
    li = np.repeat(np.arange(lk.shape[0]), n)
    ri = np.arange(n.sum()) - np.repeat(np.cumsum(n) - n, n) + np.repeat(lo, n)
    assert out.nrows == li.shape[0]
    for a, b in zip(out.to_host(), [cols[0][0][li], cols[0][1][li], cols[0][2][li], cols[1][2][ri]]):
        assert np.array_equal(a, b)
    for x in (l, r, out):
        x.free()


@pytest.mark.parametrize("window", [W - 1, W, W + 1, 2 * W - 1, 2 * W, 2 * W + 1, 3 * W + 1, 100_000, 1_000_003])
@pytest.mark.parametrize("nl", [2, 7, 255, 2047, 2048, 2049, 5000])
def test_windows(ctx, window, nl):
    """The tile's right keys are all of `window` keys, a few on either side outside it."""
    rng = np.random.default_rng(window + nl)
    rk = np.sort(rng.integers(1 << 33, 1 << 34, size=window, dtype=np.uint64))
    rk = np.concatenate([np.arange(3, dtype=np.uint64), rk, np.full(2, (1 << 63) + 1, dtype=np.uint64)])
    pick = rng.choice(rk[3:-2], size=max(0, nl // 2 - 2))
    other = rng.integers(1 << 33, 1 << 34, size=nl - pick.shape[0] - 2, dtype=np.uint64) if nl > pick.shape[0] + 2 else pick[:0]
    lk = np.sort(np.concatenate([pick, other, rk[3:4], rk[-3:-2]]))
    check(ctx, lk, rk)


@pytest.mark.parametrize("run", [1, 2, 17, 18, 19, 177, 178, 179, 400, 9000])
@pytest.mark.parametrize("shift", [0, 1, 5])
def test_runs_of_equal_keys(ctx, run, shift):
    """A million right keys in runs: samples are 178 keys apart."""
    rk = np.sort(np.concatenate([np.zeros(shift, dtype=np.uint64),
                                 np.arange(1_000_000, dtype=np.uint64) // np.uint64(run) * np.uint64(1 << 20) + np.uint64(7)]))
    keys = np.unique(rk)
    rng = np.random.default_rng(run)
    near = rng.choice(keys, size=min(200, keys.shape[0]))
    check(ctx, np.sort(np.concatenate([near, near + np.uint64(1), near - np.minimum(near, np.uint64(1)), keys[:1], keys[-1:]])), rk)


def test_random_draws(ctx):
    rng = np.random.default_rng(11)
    for _ in range(25):
        nl, nr = int(rng.integers(1, 40_000)), int(rng.integers(10_000, 1_500_000))
        k0 = int(10 ** rng.uniform(0, 5))
        k1 = int(10 ** rng.uniform(0, 6))
        if nl * nr / (k0 * k1) > 2e7:
            k1 = max(k1, 1 + nl * nr // (k0 * 20_000_000))
        two = lambda n: np.sort(rng.integers(0, k0, size=n, dtype=np.uint64) << np.uint64(32) |
                                rng.integers(0, k1, size=n, dtype=np.uint64))
        check(ctx, two(nl), two(nr))
