"""Index build against plain numpy sorts where its parts meet: (p, s) groups
of up to 64, of 65 and of many more objects, across the unpack kernel's tiles
of 2048 rows; ids with and without literals; field widths that share digits."""
import numpy as np
import pytest

import vedas_gb300 as vg

pytestmark = pytest.mark.gpu
LIT = 50_000_000


def runs(*keys):
    d = np.zeros(keys[0].shape[0], dtype=bool)
    d[:1] = True
    for k in keys:
        d[1:] |= k[1:] != k[:-1]
    return np.nonzero(d)[0].astype(np.uint32)


def expected(s, p, o, full):
    def perm(x, y, z):
        q = np.lexsort((z, y, x))
        return x[q], y[q], z[q]

    out = {}
    a, b, c = perm(p, s, o)
    h = runs(a)
    out["p_idx_values"], out["p_idx_offsets"] = a[h], h
    h = runs(a, b)
    out["ps_s_idx_values"], out["ps_idx_offsets"], out["ps_data"], out["pso_data"] = b[h], h, b, c
    a, b, c = perm(p, o, s)
    h = runs(a, b)
    out["po_o_idx_values"], out["po_idx_offsets"], out["po_data"], out["pos_data"] = b[h], h, b, c
    if full:
        for cols, val, off, data in (((s, p, o), "sp_p_idx_values", "sp_idx_offsets", "spo_data"),
                                     ((s, o, p), "so_o_idx_values", "so_idx_offsets", "sop_data"),
                                     ((o, p, s), "op_p_idx_values", "op_idx_offsets", "ops_data")):
            a, b, c = perm(*cols)
            h = runs(a, b)
            out[val], out[off], out[data] = b[h], h, c
        a, b, c = perm(o, s, p)
        h = runs(a)
        out["o_idx_values"], out["o_idx_offsets"], out["os_data"], out["osp_data"] = a[h], h, b, c
    return out


def check(ctx, s, p, o, full):
    ix = vg.Index(ctx, s, p, o, full=full)
    try:
        for name, want in expected(s, p, o, full).items():
            assert np.array_equal(ix.array(name), want), name
    finally:
        ix.close()


def grouped(sizes, rng, top):
    """Triples with (p, s) groups of the given sizes, shuffled."""
    s = np.repeat(np.arange(1, len(sizes) + 1, dtype=np.uint32), sizes)
    p = np.repeat(rng.integers(1, 4, size=len(sizes), dtype=np.uint32), sizes)
    o = rng.integers(1, top, size=s.shape[0], dtype=np.uint32)
    at = rng.permutation(s.shape[0])
    return s[at], p[at], o[at]


@pytest.mark.parametrize("full", [False, True])
@pytest.mark.parametrize("sizes", [
    [1], [64], [65], [63, 64, 1, 64], [2047, 2], [1] * 2047 + [64, 64], [64] * 40, [65] * 40,
    [3] * 700 + [5000] + [2] * 100, [60_000], [1, 300, 64, 2, 90] * 50, [64, 65] * 100,
], ids=lambda z: f"{len(z)}x{max(z)}")
def test_groups(ctx, sizes, full):
    rng = np.random.default_rng(len(sizes) * 31 + max(sizes))
    check(ctx, *grouped(sizes, rng, 1 + max(4, sum(sizes) // 3)), full)      # with repeated triples
    s, p, o = grouped(sizes, rng, 1 << 20)
    lit = rng.random(o.shape[0]) < 0.4
    check(ctx, s, p, np.where(lit, o + LIT, o).astype(np.uint32), full)


@pytest.mark.parametrize("ids", [
    (1, 1, 1), (255, 255, 255), (256, 3, 70_000), (70_000, 3, 256), (1 << 16, 86, 1 << 17), (1 << 17, 200, 1 << 16),
    ((1 << 25) - 1, (1 << 25) - 1, (1 << 14) - 1), ((1 << 32) - 1, 2, 5), (5, 2, (1 << 32) - 1),
    (9, 9, LIT - 1), (9, 9, LIT), (9, 9, LIT + 9),
])
def test_field_widths(ctx, ids):
    n = 5003
    rng = np.random.default_rng(sum(ids) % 9973)
    cols = [rng.integers(0, top, size=n, endpoint=True, dtype=np.uint32) for top in ids]
    for c, top in zip(cols, ids):
        c[rng.integers(0, n)] = top
    check(ctx, *cols, True)
    only_literals = (LIT + cols[2] % 1000).astype(np.uint32)
    # (literal ids take 26 bits; the build refuses more than 64 in all)
    if ids[2] <= LIT and int(ids[0]).bit_length() + int(ids[1]).bit_length() + 26 <= 64:
        check(ctx, cols[0], cols[1], only_literals, False)


def test_too_wide_ids_are_refused(ctx):
    big = np.full(3, (1 << 32) - 1, dtype=np.uint32)
    with pytest.raises(vg.VgError) as e:
        vg.Index(ctx, big, np.ones(3, dtype=np.uint32), big)
    assert e.value.status == 5
