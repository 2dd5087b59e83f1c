"""Joins of a few output rows of many left rows: output tiles whose left rows
lie so far apart that every row's is searched for (more than 4096 groups of
eight left rows a tile), and tiles just below that."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
FAR = 4096 * 8   # left rows


def sides(nl, at, times):
    """Left rows 0 .. nl - 1 of which `at` match `times` right rows each."""
    lk = np.arange(nl, dtype=np.uint32)
    rk = np.repeat(np.asarray(at, dtype=np.uint32), times)
    return [lk, lk ^ np.uint32(0x5555)], [rk, np.arange(rk.shape[0], dtype=np.uint32)]


def expected(l, r):
    return [r[0], l[1][r[0]], r[1]]   # (left row i has key i)


def at_and_times(nl, kind, rng):
    if kind == "ends":        # one output tile over all left rows
        return [0, nl - 1], [1, 1]
    if kind == "one":
        return [nl // 2], [1]
    if kind == "full":        # tiles of 2048 (and 512) rows and one more row
        return [0, nl // 3, nl - 1], [1, 2046, 2]
    if kind == "group":       # several rows of one group, and hubs over many tiles
        return [0, 8, 9, 11, 15, nl // 2, nl - 8, nl - 1], [3, 1, 2, 1, 5000, 7, 1, 6000]
    at = np.sort(rng.choice(nl, size=900, replace=False))
    return at, rng.integers(1, 6, size=900)


NLS = [FAR - 8, FAR, FAR + 1, FAR + 8, FAR + 2048, 100_001, 262_144, 300_001, 1 << 20, (1 << 20) + 77, 2_097_152]
KINDS = ["ends", "one", "full", "group", "random"]


@pytest.mark.parametrize("nl", NLS + [5_000_003])
@pytest.mark.parametrize("kind", KINDS)
def test_join(ctx, nl, kind):
    import vedas_gb300 as vg

    lh, rh = sides(nl, *at_and_times(nl, kind, np.random.default_rng(nl)))
    l, r = vg.Relation.from_host(ctx, lh), vg.Relation.from_host(ctx, rh)
    out, ends = vg.join(ctx, l, r)
    want = expected(lh, rh)
    assert out.nrows == want[0].shape[0] and ends == (int(want[0][0]), int(want[0][-1]))
    for a, b in zip(out.to_host(), want):
        assert np.array_equal(a, b)
    for x in (l, r, out):
        x.free()


@pytest.mark.parametrize("nl", NLS)
@pytest.mark.parametrize("kind", KINDS)
def test_join_into_given_buffers(ctx, nl, kind):
    """The same with 64-bit offsets."""
    import vedas_gb300 as vg

    lh, rh = sides(nl, *at_and_times(nl, kind, np.random.default_rng(nl)))
    want = expected(lh, rh)
    l, r = vg.Relation.from_host(ctx, lh), vg.Relation.from_host(ctx, rh)
    out = vg.Relation.from_host(ctx, [np.zeros_like(w) for w in want])

    def ptrs(rel):
        return (ctypes.c_void_p * rel.ncols)(*[rel.ir.cols[c] for c in range(rel.ncols)])

    pp = ctypes.POINTER(ctypes.c_void_p)
    fn = vg.lib().vg_join_noalloc
    fn.restype = ctypes.c_int
    fn.argtypes = [pp, ctypes.c_uint32, ctypes.c_uint64, pp, ctypes.c_uint32, ctypes.c_uint64, pp, ctypes.c_uint64,
                   ctypes.POINTER(ctypes.c_uint64), ctypes.c_void_p]
    rows = ctypes.c_uint64()
    ctx.sync()
    assert fn(ptrs(l), 2, nl, ptrs(r), 2, rh[0].shape[0], ptrs(out), want[0].shape[0], ctypes.byref(rows), None) == 0
    assert rows.value == want[0].shape[0]
    for a, b in zip(out.to_host(), want):
        assert np.array_equal(a, b)
    for x in (l, r, out):
        x.free()


@pytest.mark.parametrize("n", [FAR + 2048, 700_001])
def test_batch(ctx, n):
    """Two patterns of n subjects each that meet in a few (a batch's joins)."""
    import vedas_gb300 as vg

    rng = np.random.default_rng(n)
    odd, even = np.arange(n, dtype=np.uint32) * 2 + 1, np.arange(n, dtype=np.uint32) * 2 + 2
    at = rng.choice(n, size=300, replace=False)
    even[at] -= 1
    s = np.concatenate([odd, even, [1, 1]]).astype(np.uint32)   # and two more predicates
    p = np.concatenate([np.repeat([1, 2], n), [3, 4]]).astype(np.uint32)
    o = rng.integers(1, 1 << 20, size=2 * n + 2, dtype=np.uint32)
    x = np.sort(odd[at])
    y, z = o[:n][(x - 1) // 2], o[n:2 * n][(x - 1) // 2]
    ix = vg.Index(ctx, s, p, o)
    b = vg.Batch(ix, ["SELECT * WHERE { ?x <1> ?y . ?x <2> ?z . }"] * 3)
    for q in range(3):
        assert b.status(q) == 0, b.error(q)
        got = dict(zip(b.headers(q), b.columns(q)))
        for name, want in (("?x", x), ("?y", y), ("?z", z)):
            assert np.array_equal(got[name], want)
    b.close()
    ix.close()
