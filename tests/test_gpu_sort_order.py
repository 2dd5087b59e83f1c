"""Rows of equal digits keep their order in a radix sort pass where the lane
that places a digit's rows changes from one row of a thread to the next: few
digits, their rows spread over the lanes differently in every 32 rows."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [4096, 4097 * 3, 650_003, 1_310_720])   # tiles of 1024, 2048 and 4096 rows
@pytest.mark.parametrize("digits,lane_step,row_step", [(1, 0, 0), (2, 1, 1), (2, 0, 1), (3, 1, 1), (5, 2, 1), (31, 1, 7),
                                                       (33, 1, 1), (64, 31, 33)])
def test_equal_digits_keep_their_order(ctx, n, digits, lane_step, row_step):
    import vedas_gb300 as vg

    i = np.arange(n, dtype=np.uint64)
    key = ((i % 32 * lane_step + i // 32 * row_step) % digits * 0x01010101).astype(np.uint32)   # the digit in every pass
    tag = np.arange(n, dtype=np.uint32)
    order = np.argsort(key, kind="stable")
    for cols in ([key, tag], [key, tag, tag ^ np.uint32(0x2a)]):   # values that travel, and row numbers
        rel = vg.Relation.from_host(ctx, cols)
        vg.swap(ctx, rel, 0)
        got = rel.to_host()
        rel.free()
        for a, b in zip(got, cols):
            assert np.array_equal(a, b[order])
