"""The choice between the GEMM kernels, which is a function of the sizes alone."""
import random

from chronicals_b200.ops import _ext


def test_one_round_of_narrow_tiles():
    """Never widened on single CTAs; to CTA pairs only with K-major operands and a long K, or at an adapter's width."""
    choice, rng = _ext.lib().cb_gemm_choice, random.Random(1)
    sizes = [(896, 896, 128), (1152, 896, 128), (896, 896, 64), (1, 1, 8), (128, 148 * 128, 64), (696, 120, 18944), (32, 9728, 6000)]
    sizes += [tuple(int(2 ** rng.uniform(3, 14)) for _ in range(3)) for _ in range(3000)]
    seen = set()
    for M, N, K in sizes:
        for a_mn, b_mn in ((0, 0), (0, 1), (1, 1)):
            got = choice(M, N, K, a_mn, b_mn, 2, 148)
            seen.add(got)
            if -(-M // 128) * -(-N // 128) <= 148:
                assert got == 128 or (got == 0 and not a_mn and (N <= 64 or (not b_mn and K > 71 * 64))), (M, N, K)
    assert seen == {0, 128, 256}
    # measured on either side: us of pairs / single CTAs
    assert choice(2048, 1152, 18944, 0, 0, 2, 148) == 0            # 76 / 86
    assert choice(128, 552, 8960, 0, 0, 2, 148) == 0               # 36 / 39
    assert choice(128, 9728, 8960, 0, 0, 2, 148) == 128            # 45 / 42
    assert choice(1024, 896, 3584, 0, 0, 2, 148) == 128            # 20.4 / 20.2


# sizes measured on either side of the line (tokens, intermediate size, width); ties left out
def test_fused_gate_gradient_only_where_it_is_faster():
    pays = _ext.lib().cb_glu_bwd_fused_pays
    apart = [(16, 4864, 896), (64, 4864, 896), (256, 4864, 896), (64, 8960, 1536), (256, 8960, 1536), (128, 11008, 2048),
             (64, 18944, 3584), (128, 18944, 3584), (128, 13824, 5120)]
    fused = [(2624, 4864, 896), (8192, 4864, 896), (16384, 4864, 896), (1000, 8960, 1536), (8192, 8960, 1536), (1000, 11008, 2048),
             (8192, 11008, 2048), (512, 18944, 3584), (8192, 18944, 3584), (1000, 13824, 5120), (8192, 13824, 5120)]
    assert not any(pays(*s, 148) for s in apart)
    assert all(pays(*s, 148) for s in fused)
