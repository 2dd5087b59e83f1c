"""Calls that run out of arena halfway: they say so, give back all that they
took, and leave their relations as they were; in an arena with room they go
through.  What is left of the arena is swept, so that each of a call's
allocations fails in turn."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
OOM = 2
N = 2_200_001   # columns of 8.8 MB, blocks of their own size


def used(c):
    return c.memory()[0]


class Filler:
    """Takes all but `left` bytes of a context's largest free block."""

    def __init__(self, vg, c, left):
        self.irs, self.vg, self.c = [], vg, c
        lo, hi = 0, c.memory()[2] >> 18   # the most rows / 65536 that fit
        while lo < hi:
            mid = (lo + hi + 1) // 2
            ir = vg.vg_ir()
            if vg.lib().vg_ir_alloc(c.h, 1, mid << 16, ctypes.byref(ir)) == 0:
                vg.check(vg.lib().vg_ir_free(c.h, ctypes.byref(ir)))
                lo = mid
            else:
                hi = mid - 1
        rows = (lo << 16) - left // 4
        if rows > 9 << 18:   # (a large block)
            ir = vg.vg_ir()
            vg.check(vg.lib().vg_ir_alloc(c.h, 1, rows, ctypes.byref(ir)))
            self.irs.append(ir)

    def free(self):
        for ir in self.irs:
            self.vg.check(self.vg.lib().vg_ir_free(self.c.h, ctypes.byref(ir)))


def sweep(vg, c, lefts, call, unchanged):
    """call() with each of `lefts` bytes free: how often it failed and passed."""
    failed = passed = 0
    for left in lefts:
        f = Filler(vg, c, left)
        before = used(c)
        try:
            call()
            passed += 1
        except vg.VgError as e:
            assert e.status == OOM
            assert used(c) == before, left
            failed += 1
            unchanged()
        f.free()
    return failed, passed


@pytest.mark.parametrize("ncols", [1, 2, 3, 6])
def test_swap(built, ncols):
    import vedas_gb300 as vg

    rng = np.random.default_rng(ncols)
    cols = [rng.integers(0, 1 << 32, size=N, dtype=np.uint32) for _ in range(ncols)]
    with vg.Context(0, arena_bytes=400 << 20) as c:
        rel = vg.Relation.from_host(c, cols)
        now = [cols]

        def call():
            vg.swap(c, rel, ncols - 1)
            w = list(now[0])
            w[0], w[-1] = w[-1], w[0]
            order = np.argsort(w[0], kind="stable")
            now[0] = [x[order] for x in w]
            unchanged()

        def unchanged():
            for a, b in zip(rel.to_host(), now[0]):
                assert np.array_equal(a, b)

        failed, passed = sweep(vg, c, [m << 20 for m in range(4, 64, 4)], call, unchanged)
        assert failed >= 2 and passed >= 2


@pytest.mark.parametrize("top", [(1 << 32) - 1, 255])   # rows too wide to pack, and packed ones
def test_sort_rows_and_unique(built, top):
    import vedas_gb300 as vg

    rng = np.random.default_rng(top)
    cols = [rng.integers(0, top, size=N, endpoint=True, dtype=np.uint32) for _ in range(3)]
    order = np.lexsort(cols[::-1])
    want = [x[order] for x in cols]
    keep = np.zeros(N, dtype=bool)
    keep[0] = True
    for x in want:
        keep[1:] |= x[1:] != x[:-1]
    with vg.Context(0, arena_bytes=400 << 20) as c:
        def call():
            rel = vg.Relation.from_host(c, cols)
            before = used(c)
            try:
                vg.sort_rows(c, rel)
                for a, b in zip(rel.to_host(), want):
                    assert np.array_equal(a, b)
                vg.unique(c, rel)
                for a, b in zip(rel.to_host(), want):
                    assert np.array_equal(a, b[keep])
            except vg.VgError:
                assert used(c) == before
                raise
            finally:
                rel.free()

        failed, passed = sweep(vg, c, [m << 20 for m in range(28, 120, 4)], call, lambda: None)
        assert failed >= 2 and passed >= 2


@pytest.mark.parametrize("full", [False, True])
@pytest.mark.parametrize("n", [20_011, 400_003])
def test_index_build(built, full, n):
    import vedas_gb300 as vg

    rng = np.random.default_rng(n)
    s, o = (rng.integers(1, n, size=n, dtype=np.uint32) for _ in range(2))
    p = rng.integers(1, 30, size=n, dtype=np.uint32)
    with vg.Context(0, arena_bytes=400 << 20) as c:
        def call():
            vg.Index(c, s, p, o, full=full).close()

        failed, passed = sweep(vg, c, [m << 18 for m in range(0, 8 + n // 2500, 1 + n // 30_000)] +
                               [200 << 20, 300 << 20], call, lambda: None)
        assert failed >= 1 and passed >= 1


@pytest.mark.parametrize("which", ["star", "chain"])
def test_query(built, which):
    """Queries whose relations take megabytes, each in a new context (the size
    classes of one that ran before stay carved out)."""
    import vedas_gb300 as vg
    from vedas_gb300 import workloads

    g = workloads.graph_chain(n=2_000_000, n_entities=40_000, seed=5)
    text = workloads.star_query(1, 2) if which == "star" else workloads.chain_query_open()
    want, count = None, [0, 0]
    for left in [1 << 30] + [m << 20 for m in range(2, 130, 6)]:
        with vg.Context(0, arena_bytes=2 << 30) as c:
            ix = vg.Index(c, g.s, g.p, g.o)

            def call():
                nonlocal want
                r = ix.query(text)
                got = r.columns()
                r.close()
                want = want or got
                for a, b in zip(got, want):
                    assert np.array_equal(a, b)

            for k, v in enumerate(sweep(vg, c, [left], call, lambda: None)):
                count[k] += v
            ix.close()
    assert count[0] >= 1 and count[1] >= 1
