"""What results hold of the arena: a join's output takes the blocks that its
rows ask for, whatever room was taken before its size was known, so a program
can keep thousands of small results of large left sides."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
SMALL_MAX = 8 << 20


def block(rows):
    """Bytes of the arena's block for a column of so many rows."""
    need = max(1, -(-rows * 4 // 256)) * 256
    return need if need > SMALL_MAX else max(256, 1 << (need - 1).bit_length())


@pytest.fixture(scope="module")
def own_ctx(built):
    import vedas_gb300 as vg

    c = vg.Context(0, arena_bytes=6 << 30)
    yield c
    c.close()


def used(c):
    return c.memory()[0]


def check_join(vg, c, nl, rows, tight=False):
    """Left rows 0 .. nl - 1, `rows` output rows spread over them; returns the output.
    tight: an arena without room for another chunk of a size class gives blocks
    that are no larger than asked for."""
    lk = np.arange(nl, dtype=np.uint32)
    rk = np.sort(np.resize(lk, rows)) if rows else np.array([nl], dtype=np.uint32)
    l, r = vg.Relation.from_host(c, [lk, lk ^ np.uint32(5)]), vg.Relation.from_host(c, [rk, rk + np.uint32(7)])
    before = used(c)
    out, ends = vg.join(c, l, r)
    assert out.nrows == rows
    assert used(c) - before <= 3 * block(rows) if tight else used(c) - before == 3 * block(rows)
    if rows:
        for a, b in zip(out.to_host(), [rk, rk ^ np.uint32(5), rk + np.uint32(7)]):
            assert np.array_equal(a, b)
        assert ends == (int(rk[0]), int(rk[-1]))
    l.free()
    r.free()
    return out


# left rows around the rules (twice, eight times the rows or no room at all);
# output rows per left row, around each of the rooms
@pytest.mark.parametrize("nl", [1, 10, 700, 3001, 100_000, 1 << 18, (1 << 18) + 1, 600_001, 1 << 20, (1 << 20) + 1])
@pytest.mark.parametrize("part", [0, 1e-9, 1 / 64, 0.26, 0.5, 0.6, 1.0, 1.4, 2.0, 2.01, 3.7, 8.0, 8.2])
def test_an_output_holds_what_its_rows_take(own_ctx, nl, part):
    import vedas_gb300 as vg

    check_join(vg, own_ctx, nl, int(np.ceil(nl * part))).free()


@pytest.mark.parametrize("rows", [1, 64, 65, 128, 129, 1024, 1025, 2048, 2049, 4096, 4097, 8192, 8193])
def test_outputs_at_the_edges_of_the_rooms(own_ctx, rows):
    import vedas_gb300 as vg

    check_join(vg, own_ctx, 3001, rows).free()


def test_many_small_results_are_kept(built):
    import vedas_gb300 as vg

    with vg.Context(0, arena_bytes=512 << 20) as c:
        kept = [check_join(vg, c, 200_000, 10) for _ in range(600)]
        assert all(k.nrows == 10 for k in kept)


def test_many_small_results_on_two_columns_are_kept(built):
    import vedas_gb300 as vg

    n = 200_000
    with vg.Context(0, arena_bytes=512 << 20) as c:
        k = np.arange(n, dtype=np.uint32)
        l = vg.Relation.from_host(c, [k // 7, k, k + np.uint32(1)])
        at = np.array([0, 7, 63, n - 1], dtype=np.uint32)
        r = vg.Relation.from_host(c, [at // 7, at, at * np.uint32(3)])
        before = used(c)
        kept = [vg.join2(c, l, r) for _ in range(600)]
        assert used(c) - before == 600 * 4 * 256
        for x in kept[::100]:
            for a, b in zip(x.to_host(), [at // 7, at, at + np.uint32(1), at * np.uint32(3)]):
                assert np.array_equal(a, b)


def test_many_small_query_results_are_kept(built):
    """Two patterns of 200,000 rows each that meet in a few subjects."""
    import vedas_gb300 as vg

    n, both = 200_000, 9
    odd, even = np.arange(n, dtype=np.uint32) * 2 + 1, np.arange(n, dtype=np.uint32) * 2 + 2
    even[n // 20::n // both] -= 1   # a few subjects of the other pattern
    both = len(even[n // 20::n // both])
    s = np.concatenate([odd, even, [1, 1]]).astype(np.uint32)   # and two more predicates
    p = np.concatenate([np.repeat([1, 2], n), [3, 4]]).astype(np.uint32)
    o = (np.arange(2 * n + 2) % 1000 + 1).astype(np.uint32)
    with vg.Context(0, arena_bytes=512 << 20) as c:
        ix = vg.Index(c, s, p, o)
        text = "SELECT * WHERE { ?x <1> ?y . ?x <2> ?z . }"
        kept = [ix.query(text)]
        before = used(c)
        kept += [ix.query(text) for _ in range(400)]
        held = used(c) - before
        rows = [k.nrows for k in kept]
        cols = [k.columns() for k in kept[::50]]
        for k in kept:
            k.close()
        ix.close()
        assert rows == [both] * 401
        assert held == 400 * 3 * block(both)
        for k in cols:
            for a, b in zip(k, cols[0]):
                assert np.array_equal(a, b)


@pytest.mark.parametrize("mb", [24, 40, 64, 96, 160, 320, 1000])
@pytest.mark.parametrize("nl", [200_000, 300_000, 700_000])
def test_joins_in_arenas_with_little_room(built, nl, mb):
    """Arenas in which all, some or none of the rooms fit: the same output in
    the same blocks."""
    import vedas_gb300 as vg

    with vg.Context(0, arena_bytes=mb << 20) as c:
        for rows in (3, nl // 2, nl):
            try:
                out = check_join(vg, c, nl, rows, tight=True)
            except vg.VgError as e:   # the relations themselves do not fit
                assert e.status == 2 and mb <= 40
                return
            out.free()
