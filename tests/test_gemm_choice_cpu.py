"""The choice between the GEMM kernels, which is a function of the sizes alone."""
import random

from chronicals_b200.ops import _ext


def test_one_round_of_narrow_tiles_is_not_widened():
    choice, rng = _ext.lib().cb_gemm_choice, random.Random(1)
    sizes = [(896, 896, 128), (1152, 896, 128), (896, 896, 64), (1, 1, 8), (128, 148 * 128, 64)]
    sizes += [tuple(int(2 ** rng.uniform(3, 14)) for _ in range(3)) for _ in range(3000)]
    seen = set()
    for M, N, K in sizes:
        for a_mn, b_mn in ((0, 0), (0, 1), (1, 1)):
            got = choice(M, N, K, a_mn, b_mn, 2, 148)
            seen.add(got)
            if -(-M // 128) * -(-N // 128) <= 148:
                assert got != 256, (M, N, K)
    assert seen == {0, 128, 256}
