"""Radix sorts hold half a byte a key for their passes' look-back words (1 MiB
in small sorts), however many passes they have, and passes that use the same
words again give the same order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
SLACK = 256 << 10   # digit counts, flags and the like


def words(n):
    """The arena's block for half a byte a key, of whole tiles of 4096 keys."""
    need = max(-(-n // 4096) * 2048, 1 << 20)
    return need if need > 8 << 20 else 1 << (need - 1).bit_length()


def held(c, work):
    """Bytes that `work` took of the arena at its peak, above what was in use."""
    used, peak, _ = c.memory()
    assert used == peak
    work()
    return c.memory()[1] - used


# rows whose columns are blocks of their own size (above 8 MiB)
@pytest.mark.parametrize("n", [2_200_001, 4_194_304, 9_000_001])
def test_swap_scratch(built, n):
    """32-bit keys in four passes, the second column as values."""
    import vedas_gb300 as vg

    rng = np.random.default_rng(n)
    key, val = rng.integers(0, 1 << 32, size=n, dtype=np.uint32), np.arange(n, dtype=np.uint32)
    with vg.Context(0, arena_bytes=1 << 30) as c:
        rel = vg.Relation.from_host(c, [key, val])
        assert held(c, lambda: vg.swap(c, rel, 0)) <= 8 * n + words(n) + SLACK
        order = np.argsort(key, kind="stable")
        for a, b in zip(rel.to_host(), (key, val)):
            assert np.array_equal(a, b[order])


@pytest.mark.parametrize("n", [2_200_001, 4_194_304, 9_000_001])
def test_row_sort_scratch(built, n):
    """Rows of 64 bits of which a few values of the first column start thousands
    each: every bit is sorted by, in eight passes."""
    import vedas_gb300 as vg

    rng = np.random.default_rng(n)
    cols = [rng.choice(rng.integers(1 << 31, 1 << 32, size=9, dtype=np.uint32), size=n),
            rng.integers(0, 1 << 32, size=n, dtype=np.uint32)]
    with vg.Context(0, arena_bytes=1 << 30) as c:
        rel = vg.Relation.from_host(c, cols)
        assert held(c, lambda: vg.sort_rows(c, rel)) <= 16 * n + words(n) + SLACK
        key = np.sort(cols[0].astype(np.uint64) << np.uint64(32) | cols[1])
        got = rel.to_host()
        assert np.array_equal(got[0].astype(np.uint64) << np.uint64(32) | got[1], key)


@pytest.mark.parametrize("n", [70_001, 300_000, 622_591])
def test_small_sorts_use_their_words_again(ctx, n):
    """Sorts of so few rows that tiles have 1024, whose words of all passes are
    more than 1 MiB."""
    import vedas_gb300 as vg

    rng = np.random.default_rng(n)
    cols = [rng.choice(rng.integers(1 << 31, 1 << 32, size=9, dtype=np.uint32), size=n),
            rng.integers(0, 1 << 32, size=n, dtype=np.uint32)]
    rel = vg.Relation.from_host(ctx, cols)
    vg.sort_rows(ctx, rel)
    key = np.sort(cols[0].astype(np.uint64) << np.uint64(32) | cols[1])
    got = rel.to_host()
    rel.free()
    assert np.array_equal(got[0].astype(np.uint64) << np.uint64(32) | got[1], key)
