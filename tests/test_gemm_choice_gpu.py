"""Products on either side of the lines between the GEMM kernels and tile widths, against fp64."""
import pytest
import torch

from chronicals_b200 import ops
from chronicals_b200.ops import _ext

pytestmark = pytest.mark.gpu
DEV = "cuda"


# 128-wide single-CTA tiles, 256-wide ones, pairs of 256, 224 and 192, tiles cut along K; ragged last tiles in M and N, K that
# is no multiple of the k-block
@pytest.mark.parametrize("M,N,K", [(1000, 896, 1152), (512, 1152, 896), (128, 896, 4864), (2624, 2048, 1096), (4096, 1536, 1000),
                                   (3000, 1800, 520), (1500, 3584, 1024), (1008, 200, 2056), (9728, 896, 4104), (304, 5120, 328),
                                   # outputs as narrow as an adapter's rank
                                   (8192, 32, 2056), (300, 48, 896), (1000, 64, 520), (256, 16, 4104), (136, 8, 72)])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True)])
@pytest.mark.parametrize("fp32", [False, True])
def test_chosen_kernel(M, N, K, a_mn, b_mn, fp32):
    if (a_mn and M % 8) or (b_mn and N % 8):
        pytest.skip("operand pitch")
    g = torch.Generator(device=DEV).manual_seed(M + N + K)
    a = torch.randn(*((K, M) if a_mn else (M, K)), device=DEV, generator=g).to(torch.bfloat16)
    b = torch.randn(*((K, N) if b_mn else (N, K)), device=DEV, generator=g).to(torch.bfloat16)
    out = torch.full((M, N), 7.0, device=DEV, dtype=torch.float32 if fp32 else torch.bfloat16)
    ops.gemm(a, b, a_mn=a_mn, b_mn=b_mn, out=out)
    _ext.check_status()
    want = (a.t() if a_mn else a).double() @ (b if b_mn else b.t()).double()
    # fp32 sums of K products of order one, one rounding of the result
    slack = K ** 0.5 * 2e-6 * 8 + (0 if fp32 else 1e-6)
    assert ((out.double() - want).abs() <= (1e-6 if fp32 else 2.0 ** -8) * want.abs() + slack * 4).all()


# one row, ragged row tiles, a last tile of 128 activation columns, frozen weights; with and without bias and residual
@pytest.mark.parametrize("T,H,I", [(1, 64, 128), (300, 896, 640), (513, 256, 1408), (130, 72, 256)])
@pytest.mark.parametrize("extras,frozen", [(False, False), (True, False), (True, True)])
def test_swiglu_mlp_gradients(T, H, I, extras, frozen):
    g = torch.Generator(device=DEV).manual_seed(T + I)

    def r(*shape, scale=1.0):
        return (scale * torch.randn(*shape, device=DEV, generator=g)).to(torch.bfloat16)
    x, wg, wd, dy = r(T, H), r(2 * I, H, scale=H ** -0.5), r(H, I, scale=I ** -0.5), r(T, H)
    b, res = (r(2 * I, scale=0.1), r(T, H)) if extras else (None, None)
    leaves = [t for t in (x, b, res) if t is not None] + ([] if frozen else [wg, wd])
    for t in leaves:
        t.requires_grad_()
    y = ops.swiglu_mlp(x, wg, wd, b, res)
    y.backward(dy)
    _ext.check_status()
    got = [y] + [t.grad for t in leaves]
    up = {id(t): t.detach().double().requires_grad_() for t in (x, wg, wd, b, res) if t is not None}
    gate, lin = (up[id(x)] @ up[id(wg)].t() + (up[id(b)] if extras else 0)).chunk(2, dim=1)
    want = (torch.nn.functional.silu(gate) * lin) @ up[id(wd)].t() + (up[id(res)] if extras else 0)
    want.backward(dy.double())
    for a, w in zip(got, [want] + [up[id(t)].grad for t in leaves]):
        # gate | up, the activation (by tanh.approx, 2^-11) and d(gate) | d(up) are rounded to bf16 on the way
        assert ((a.double() - w).norm() <= 2.0 ** -7 * w.norm() + 1e-6).item()
    assert frozen is False or (wg.grad is None and wd.grad is None)


# both ways of the backward, whichever the sizes would take
@pytest.mark.parametrize("T,H,I", [(1, 64, 128), (300, 896, 640), (513, 256, 1408), (130, 72, 256)])
@pytest.mark.parametrize("fused", [True, False])
def test_swiglu_mlp_gradients_either_way(T, H, I, fused, monkeypatch):
    monkeypatch.setattr(ops, "_glu_bwd_fused", lambda *a: fused)
    test_swiglu_mlp_gradients(T, H, I, True, False)
