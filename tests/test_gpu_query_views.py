"""Results of one pattern, which are views of the index until they are handed
out: of no row, one, two, as many as are copied before repeated rows are looked
for, and more; they stay what they are when the index is gone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 2, 3, 2048, 2049, 32_768, 32_769, 65_536, 65_537, 200_000])
def test_results_of_one_pattern(ctx, rows):
    import vedas_gb300 as vg

    rng = np.random.default_rng(rows)
    s = np.arange(1, rows + 1, dtype=np.uint32)
    o = rng.integers(1, 1000, size=rows, dtype=np.uint32)
    more = 4   # three more predicates of one triple each
    ix = vg.Index(ctx, np.concatenate([s, s[:1], s[:1], s[:1]]),
                  np.concatenate([np.full(rows, 2), [1, 3, 4]]).astype(np.uint32),
                  np.concatenate([o, np.full(more - 1, 7, dtype=np.uint32)]))
    both = ix.query("SELECT * WHERE { ?x <2> ?y . }")
    of = ix.query(f"SELECT ?x WHERE {{ ?x <2> <{o[0]}> . }}")
    one = ix.query("SELECT ?y WHERE { <1> <2> ?y . }")
    none = ix.query("SELECT ?x WHERE { ?x <2> <1001> . }")
    ix.close()
    vg.Index(ctx, s[::-1].copy(), np.full(rows, 5, dtype=np.uint32), o).close()   # the memory is another's
    got = dict(zip(both.headers, both.columns()))
    assert np.array_equal(got["?x"], s) and np.array_equal(got["?y"], o)
    assert np.array_equal(of.columns()[0], s[o == o[0]])
    assert one.columns()[0].tolist() == [o[0]]
    assert none.nrows == 0
    for r in (both, of, one, none):
        r.close()
