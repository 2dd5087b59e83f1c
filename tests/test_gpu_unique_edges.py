"""Repeated-row removal where its parts meet: relations of one tile of 2048
rows (one launch) and more, of up to 2^19 rows (the rows go to one of three
rooms) and more, more tiles than one pass of the scan over them takes (2048),
rows that repeat in whole tiles or none; results hold what their rows take."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
SMALL_MAX = 8 << 20


def block(rows):
    need = max(1, -(-rows * 4 // 256)) * 256
    return need if need > SMALL_MAX else max(256, 1 << (need - 1).bit_length())


@pytest.fixture(scope="module")
def own_ctx(built):
    import vedas_gb300 as vg

    c = vg.Context(0, arena_bytes=3 << 30)
    yield c
    c.close()


def check(c, new, ncols):
    """Rows that differ from the one before where `new` is set, in the last column or all."""
    import vedas_gb300 as vg

    key = np.cumsum(new).astype(np.uint32)
    for cols in ([key * np.uint32(3)] * ncols, [np.full_like(key, 7)] * (ncols - 1) + [key]):
        before = c.memory()[0]
        rel = vg.Relation.from_host(c, cols)
        vg.unique(c, rel)
        keep = np.array(new)
        keep[0] = True
        kept = int(keep.sum())
        assert rel.nrows == kept
        for a, b in zip(rel.to_host(), cols):
            assert np.array_equal(a, b[keep])
        assert c.memory()[0] - before == ncols * (block(kept) if kept < len(key) else block(len(key)))
        rel.free()


@pytest.mark.parametrize("n", [2, 63, 64, 65, 256, 257, 1024, 1025, 2047, 2048, 2049, 4097, 100_003, 1 << 19, (1 << 19) + 1])
@pytest.mark.parametrize("ncols", [1, 3, 9])
def test_kept_rows_around_the_rooms(own_ctx, n, ncols):
    for kept in sorted({1, 2, 3, n // 8, n // 4, n // 4 + 1, n // 2, n // 2 + 1, n - 1, n, 64, 65, 128, 129, 512, 513, 1 << 17, 1 << 18, 1 << 20, (1 << 20) + 1} & set(range(1, n + 1))):
        new = np.zeros(n, dtype=bool)
        new[np.linspace(0, n - 1, kept).astype(int)] = True
        check(own_ctx, new, ncols)


@pytest.mark.parametrize("n", [2048 * 2048, 2048 * 2048 + 1, 9_000_001])
@pytest.mark.parametrize("kind", ["none", "all", "one at the end", "first tiles", "last tiles", "some"])
def test_many_tiles(own_ctx, n, kind):
    new = np.ones(n, dtype=bool)
    if kind == "all":
        new[:] = False
    elif kind == "one at the end":
        new[-1] = False
    elif kind == "first tiles":
        new[: 2048 * 1500 + 3] = False
    elif kind == "last tiles":
        new[2048 * 1500 + 3:] = False
    elif kind == "some":
        new = np.random.default_rng(n).random(n) < 0.6
    check(own_ctx, new, 2)
