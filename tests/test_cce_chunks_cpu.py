"""The chunk rule of the fused linear cross-entropy's backward."""
import time

import pytest

from chronicals_b200 import ops


@pytest.mark.parametrize("M", [1, 64, 1000, 4096, 8192, 70000])
@pytest.mark.parametrize("V", [1, 520, 5000, 32000, 151936])
def test_chunk_width(M, V):
    w = ops._cce_chunk(M, 896, V, 148)
    assert w % 8 == 0 and 0 < w <= (V + 7) // 8 * 8
    assert w % 256 == 0 or w == (V + 7) // 8 * 8                   # whole tiles, or everything
    assert M * w <= max(ops.CCE_BWD_ELEMENTS, M * ops.CCE_BWD_CHUNK)   # no more scratch than the fixed width took at 8192


def test_a_new_token_count_costs_no_search():
    """A data set without padding brings another token count almost every step."""
    ops._cce_chunk(7, 896, 151936, 148)
    t = time.perf_counter()
    for M in range(1, 501):
        ops._cce_chunk(M, 896, 151936, 148)
    assert time.perf_counter() - t < 0.1                           # a fifth of a millisecond each, forty times what it takes
