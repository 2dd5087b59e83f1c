"""Radix sort passes at the edges of their tiles and dispatch rules: tiles of
1024, 2048, 3072 and 4096 keys (chosen by row count and launch parameter),
digits of 7 and 8 bits, 32- and 64-bit look-back words (2^30 rows and more)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# one tile and its neighbours, and the row counts where the tile size changes
# on a 152-SM GPU (two tiles per SM: 622592 and 1245184 rows)
SIZES = [2, 31, 33, 255, 1023, 1024, 1025, 4095, 4097, 8193, 622591, 622592, 1245183, 1245184, 1249281]


@pytest.fixture(scope="module")
def ctx():
    import vedas_gb300 as vg

    c = vg.Context(0, arena_bytes=2 << 30)
    yield c
    c.close()


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("top", [1, 127, 1 << 21, (1 << 32) - 1])
def test_swap_is_a_stable_sort(ctx, n, top):
    import vedas_gb300 as vg

    rng = np.random.default_rng(n * 7 + top % 1009)
    key = rng.integers(0, top, size=n, endpoint=True, dtype=np.uint32)
    first, tag = rng.integers(0, 1 << 32, size=n, dtype=np.uint32), np.arange(n, dtype=np.uint32)
    rel = vg.Relation.from_host(ctx, [first, key, tag])
    vg.swap(ctx, rel, 1)
    order = np.argsort(key, kind="stable")
    got = rel.to_host()
    rel.free()
    for a, b in zip(got, (key[order], first[order], tag[order])):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("items", [8, 12, 16])
@pytest.mark.parametrize("look", [1, 4])
def test_every_tile_choice(ctx, items, look):
    import vedas_gb300 as vg

    rng = np.random.default_rng(items + look)
    n = 1_500_011
    key, tag = rng.integers(0, 1 << 24, size=n, dtype=np.uint32), np.arange(n, dtype=np.uint32)
    ctx.tune_set("sort_items", items)
    ctx.tune_set("sort_lookback", look)
    try:
        rel = vg.Relation.from_host(ctx, [key, tag])
        vg.swap(ctx, rel, 0)
        got = rel.to_host()
        rel.free()
    finally:
        ctx.tune_set("sort_items", 16)
        ctx.tune_set("sort_lookback", 4)
    order = np.argsort(key, kind="stable")
    assert np.array_equal(got[0], key[order]) and np.array_equal(got[1], tag[order])


def test_wide_look_back_words():
    import ctypes

    import torch

    import vedas_gb300 as vg

    class View:
        def __init__(self, ptr, n):
            self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<i4", "data": (ptr, False), "version": 3}

    n = (1 << 30) + 4099
    with vg.Context(0, arena_bytes=14 << 30) as c:
        ir = vg.vg_ir()
        vg.check(vg.lib().vg_ir_alloc(c.h, 1, n, ctypes.byref(ir)))
        rel = vg.Relation(c, ir)
        g = torch.Generator(device="cuda")
        g.manual_seed(5)
        want = torch.randint(0, 1 << 15, (n,), generator=g, device="cuda", dtype=torch.int32)
        torch.as_tensor(View(rel.ir.cols[0], n), device="cuda").copy_(want)
        torch.cuda.synchronize()
        vg.swap(c, rel, 0)
        counts = torch.bincount(want, minlength=1 << 15)
        got = torch.as_tensor(View(rel.ir.cols[0], n), device="cuda")
        assert bool((got[1:] >= got[:-1]).all())
        assert torch.equal(torch.bincount(got, minlength=1 << 15), counts)
        del got
        rel.free()
