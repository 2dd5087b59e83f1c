"""Row sorts and repeated-row removal against numpy at the edges of their
rules: packed rows of up to 64 bits and wider ones, columns of zeros, one to
nine columns, tiles of 2048 rows, relations with nothing, something or nearly
everything to drop."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
SIZES = [2, 7, 2047, 2048, 2049, 10_001, 650_000]


def lexsorted(cols):
    order = np.lexsort(cols[::-1])
    return [c[order] for c in cols]


def adjacent_unique(cols):
    keep = np.zeros(cols[0].shape[0], dtype=bool)
    keep[:1] = True
    for c in cols:
        keep[1:] |= c[1:] != c[:-1]
    return [c[keep] for c in cols]


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("tops", [
    (3, 3), (0, 5), (0, 0), ((1 << 32) - 1, (1 << 32) - 1), ((1 << 32) - 1, (1 << 31) - 1, 1),
    ((1 << 32) - 1, (1 << 32) - 1, 1), (9,) * 9, ((1 << 32) - 1,) * 9, ((1 << 20) - 1, 0, (1 << 20) - 1, 7),
], ids=str)
def test_sort_rows(ctx, n, tops):
    import vedas_gb300 as vg

    rng = np.random.default_rng(n + len(tops))
    cols = [rng.integers(0, t, size=n, endpoint=True, dtype=np.uint32) for t in tops]
    for c, t in zip(cols, tops):
        c[n // 2] = t
    rel = vg.Relation.from_host(ctx, cols)
    vg.sort_rows(ctx, rel)
    want = lexsorted(cols)
    for a, b in zip(rel.to_host(), want):
        assert np.array_equal(a, b)
    vg.unique(ctx, rel)
    want = adjacent_unique(want)
    assert rel.nrows == want[0].shape[0]
    for a, b in zip(rel.to_host(), want):
        assert np.array_equal(a, b)
    rel.free()


@pytest.mark.parametrize("n", [1, 2, 8, 9, 2047, 2048, 2049, 4096, 100_003, 1_300_001])
@pytest.mark.parametrize("ncols", [1, 2, 3, 9])
@pytest.mark.parametrize("share", [0.0, 0.001, 0.5, 1.0])
def test_unique(ctx, n, ncols, share):
    """Rows that repeat the one before them with the given probability; the
    others differ from it in one column only, any of them."""
    import vedas_gb300 as vg

    rng = np.random.default_rng(n * 10 + ncols)
    new = rng.random(n) >= share
    which = rng.integers(0, ncols, size=n)
    cols = [np.cumsum(new & (which == c)).astype(np.uint32) for c in range(ncols)]
    rel = vg.Relation.from_host(ctx, cols)
    vg.unique(ctx, rel)
    want = adjacent_unique(cols)
    assert rel.nrows == want[0].shape[0]
    for a, b in zip(rel.to_host(), want):
        assert np.array_equal(a, b)
    rel.free()


@pytest.mark.parametrize("n", [1000, 700_001])
@pytest.mark.parametrize("ncols", [1, 2, 3, 9])
def test_swap(ctx, n, ncols):
    import vedas_gb300 as vg

    rng = np.random.default_rng(n + ncols)
    cols = [rng.integers(0, 50_000, size=n, dtype=np.uint32) for _ in range(ncols)]
    for col in range(ncols):
        rel = vg.Relation.from_host(ctx, cols)
        vg.swap(ctx, rel, col)
        want = list(cols)
        want[0], want[col] = want[col], want[0]
        order = np.argsort(want[0], kind="stable")
        for a, b in zip(rel.to_host(), want):
            assert np.array_equal(a, b[order])
        rel.free()


def test_swap_of_many_columns_in_a_full_arena():
    """New columns that do not fit all at once are made one after the other."""
    import vedas_gb300 as vg

    n = 2_600_000                        # 10.4 MB a column
    with vg.Context(0, arena_bytes=160 << 20) as c:
        rng = np.random.default_rng(3)
        cols = [rng.integers(0, 1 << 30, size=n, dtype=np.uint32) for _ in range(9)]
        rel = vg.Relation.from_host(c, cols)
        vg.swap(c, rel, 0)
        order = np.argsort(cols[0], kind="stable")
        for a, b in zip(rel.to_host(), cols):
            assert np.array_equal(a, b[order])


@pytest.mark.parametrize("n", [3000, 2048 * 5 + 1, 300_007])
@pytest.mark.parametrize("size", [1, 2, 63, 64, 65, 200, 5000])
def test_rows_that_agree_in_their_top_bits(ctx, n, size):
    """Wide rows in groups of `size` that differ in the last column only (the
    first columns tell the groups apart), across tiles of 2048 rows."""
    import vedas_gb300 as vg

    rng = np.random.default_rng(n + size)
    group = np.arange(n) // size
    a = (rng.permutation(group.max() + 1) * 3)[group].astype(np.uint32)
    cols = [a, np.full(n, 1 << 20, dtype=np.uint32), rng.integers(0, 1 << 22, size=n, dtype=np.uint32)]
    order = rng.permutation(n)
    cols = [c[order] for c in cols]
    rel = vg.Relation.from_host(ctx, cols)
    vg.sort_rows(ctx, rel)
    for x, y in zip(rel.to_host(), lexsorted(cols)):
        assert np.array_equal(x, y)
    rel.free()
