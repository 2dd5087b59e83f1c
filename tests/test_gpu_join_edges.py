"""Joins of two relations against numpy where the kernels' parts meet: left
tiles of 2048 rows, right windows that fit shared memory or not (11264 keys,
5632 pairs), outputs that are guessed (up to 2^20 left rows: twice the rows,
at least 1024), written again because they are larger, or written after the
count; output tiles of 512 and 2048 rows fed by more left rows than are staged;
row counts above which windows and ranges get kernels of their own."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def pairs(lk, rk):
    """(left row, right row) of every match, in order."""
    lo, hi = np.searchsorted(rk, lk, "left"), np.searchsorted(rk, lk, "right")
    n = hi - lo
    li = np.repeat(np.arange(lk.shape[0]), n)
    ri = np.arange(n.sum()) - np.repeat(np.cumsum(n) - n, n) + np.repeat(lo, n)
    return li, ri


def check_one(ctx, lcols, rcols):
    import vedas_gb300 as vg

    l, r = vg.Relation.from_host(ctx, lcols), vg.Relation.from_host(ctx, rcols)
    out, ends = vg.join(ctx, l, r)
    li, ri = pairs(lcols[0], rcols[0])
    want = [c[li] for c in lcols] + [c[ri] for c in rcols[1:]]
    assert out.nrows == li.shape[0]
    got = out.to_host()
    for a, b in zip(got, want):
        assert np.array_equal(a, b)
    if li.shape[0]:
        assert ends == (int(want[0][0]), int(want[0][-1]))
    for x in (l, r, out):
        x.free()


def side(rng, n, keys, cols):
    return [np.sort(rng.integers(0, keys, size=n, dtype=np.uint32))] + \
        [rng.integers(0, 1 << 32, size=n, dtype=np.uint32) for _ in range(cols - 1)]


@pytest.mark.parametrize("nl,nr,keys", [
    (1, 1, 1), (1, 5000, 3), (255, 256, 100), (2047, 2049, 1500), (2048, 2048, 2000), (2049, 70_000, 30_000),
    (4097, 4095, 100), (3000, 200, 50_000_000), (60_000, 60_000, 4_000_000_000), (100_003, 7, 1 << 20),
    (5, 1_000_000, 100), (1 << 20, 300_000, 900_000), ((1 << 20) + 1, 300_000, 900_000),
    (1_245_184, 40_000, 70_000), (1_245_185, 1_900_000, 2_000_000), (3_000_000, 50, 3_000_000),
])
@pytest.mark.parametrize("lc,rc", [(1, 1), (2, 3), (5, 5)])
def test_join(ctx, nl, nr, keys, lc, rc):
    rng = np.random.default_rng(nl * 3 + nr)
    check_one(ctx, side(rng, nl, keys, lc), side(rng, nr, keys, rc))


@pytest.mark.parametrize("rows", [0, 1, 2, 3, 99, 100, 101, 511, 512, 513, 1023, 1024, 1025, 2048, 6000, 6001])
def test_output_sizes(ctx, rows):
    """3000 left rows, one of which (or the last few) has all the matches."""
    lk = np.arange(1, 3001, dtype=np.uint32)
    for at in (1, 1500, 3000):
        rk = np.full(rows, at, dtype=np.uint32)
        if rows == 0:
            rk = np.array([0, 3001], dtype=np.uint32)
        check_one(ctx, [lk, lk * 7], [rk, np.arange(rk.shape[0], dtype=np.uint32)])


@pytest.mark.parametrize("window", [11263, 11264, 11265, 11266, 50_000])
@pytest.mark.parametrize("shift", [0, 1, 2, 3])
def test_windows(ctx, window, shift):
    """A tile whose right window has `window` keys, starting at any alignment."""
    lk = np.concatenate([np.arange(shift + 1), np.arange(1000, 3000)]).astype(np.uint32)
    rk = np.sort(np.concatenate([np.arange(shift), np.full(window, 1500), [900, 5000]])).astype(np.uint32)
    check_one(ctx, [lk, lk + 1], [rk, np.arange(rk.shape[0], dtype=np.uint32)])


def test_heavy_keys_both_sides(ctx):
    rng = np.random.default_rng(5)
    lk = np.sort(np.concatenate([rng.integers(0, 50_000, 30_000), np.full(4000, 777), np.full(100, 40_000)]))
    rk = np.sort(np.concatenate([rng.integers(0, 50_000, 20_000), np.full(3000, 777), np.full(9000, 40_000)]))
    check_one(ctx, [lk.astype(np.uint32), np.arange(lk.shape[0], dtype=np.uint32)],
              [rk.astype(np.uint32), np.arange(rk.shape[0], dtype=np.uint32)])


@pytest.mark.parametrize("nl,nr,k0,k1", [
    (1, 1, 1, 1), (2047, 3000, 40, 50), (2049, 2048, 2000, 2), (50_000, 20_000, 300, 1 << 31), (3000, 9000, 1, 1500),
    (10, 400_000, 2, 5), (1_300_000, 1_000_000, 4000, 300), (4096, 5632, 1, 1),
])
def test_join_on_two_columns(ctx, nl, nr, k0, k1):
    import vedas_gb300 as vg

    rng = np.random.default_rng(nl + nr)

    def two(n):
        k = np.sort((rng.integers(0, k0, size=n, dtype=np.uint64) << np.uint64(32)) |
                    rng.integers(0, k1, size=n, dtype=np.uint64))
        return k, [(k >> np.uint64(32)).astype(np.uint32), k.astype(np.uint32),
                   rng.integers(0, 1 << 32, size=n, dtype=np.uint32)]

    lk, lcols = two(min(nl, 3000) if k0 == 1 and k1 == 1 else nl)
    rk, rcols = two(nr)
    l, r = vg.Relation.from_host(ctx, lcols), vg.Relation.from_host(ctx, rcols)
    out = vg.join2(ctx, l, r)
    li, ri = pairs(lk, rk)
    for a, b in zip(out.to_host(), [c[li] for c in lcols] + [rcols[2][ri]]):
        assert np.array_equal(a, b)
    for x in (l, r, out):
        x.free()


def test_a_guess_that_does_not_fit_the_arena():
    """The output is guessed at twice the left rows where that fits; a join
    whose own output fits goes through in an arena where the guess does not."""
    import vedas_gb300 as vg

    with vg.Context(0, arena_bytes=64 << 20) as c:
        n = 1_000_000
        lk = np.arange(n, dtype=np.uint32)
        rk = np.arange(0, n, 1000, dtype=np.uint32)
        l, r = vg.Relation.from_host(c, [lk] * 6), vg.Relation.from_host(c, [rk])
        out, _ = vg.join(c, l, r)
        assert out.nrows == rk.shape[0]
        for col in out.to_host():
            assert np.array_equal(col, rk)


@pytest.mark.parametrize("gap", [0, 7, 8, 9, 2047, 2048, 4097, 32_760, 32_767, 32_768, 32_769, 32_784, 300_001])
@pytest.mark.parametrize("nl", [400_000, (1 << 20) + 700_003])
def test_left_rows_without_matches(ctx, nl, gap):
    """Output tiles whose left rows lie far apart: runs of `gap` rows without
    matches between rows with one or a few, and a hub at either end."""
    lk = np.arange(nl, dtype=np.uint32)
    at = np.arange(3, nl - 1, gap + 1, dtype=np.uint32)
    times = np.ones(at.shape[0], dtype=np.int64)
    times[::5] = 3
    times[0] = times[-1] = 5000
    rk = np.repeat(at, times)
    check_one(ctx, [lk, lk ^ np.uint32(0x5555)], [rk, np.arange(rk.shape[0], dtype=np.uint32)])


@pytest.mark.parametrize("nl,times", [(1 << 18, 2), (1 << 18, 3), ((1 << 18) + 1, 2), ((1 << 18) + 1, 7),
                                      ((1 << 18) + 1, 8), ((1 << 18) + 1, 9), (1 << 20, 8)])
def test_outputs_around_the_guess(ctx, nl, times):
    """Every left row matches `times` rows: room is taken for 2 (up to 2^18
    left rows) or 8 times the left rows; one more output row than that."""
    lk = np.arange(nl, dtype=np.uint32)
    rk = np.repeat(lk, times)
    check_one(ctx, [lk], [rk, np.arange(rk.shape[0], dtype=np.uint32)])
    rk = np.append(rk, rk[-1])
    check_one(ctx, [lk, lk], [rk])
