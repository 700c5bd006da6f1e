"""The attention backward entry point writes its gradient into any buffer whose rows start on 8-byte boundaries."""
import pytest
import torch

from chronicals_b200 import ops
from chronicals_b200.ops import _ext

pytestmark = pytest.mark.gpu
DEV = "cuda"


# one document of one tile and one query head per key head: every value of the gradient is one sum, the same each time
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("shift,gap", [(0, 0), (4, 0), (0, 4), (4, 12), (8, 8)])
def test_rows_of_the_gradient(d, shift, gap):
    T, h = 100, 2
    n = 3 * h * d
    g = torch.Generator(device=DEV).manual_seed(d)
    qkv = torch.randn(T, n, device=DEV, generator=g).to(torch.bfloat16).requires_grad_()
    do = torch.randn(T, h * d, device=DEV, generator=g).to(torch.bfloat16)
    cu = torch.tensor([0, T], dtype=torch.int32, device=DEV)
    o = ops.attention_qkv_packed(qkv, cu, h, h, d)
    lse = o.grad_fn.saved_tensors[2]
    o.backward(do)
    x, at, f32 = qkv.detach(), qkv.element_size() * h * d, dict(dtype=torch.float32, device=DEV)
    delta, acc = torch.empty(h, T, **f32), torch.empty(3, T, h * d, **f32)
    buf = torch.full((shift + T * (n + gap),), 7.0, dtype=torch.bfloat16, device=DEV)
    dqkv = buf[shift:].view(T, n + gap)
    code = _ext.lib().cb_attn_bwd(
        x.data_ptr(), x.data_ptr() + at, x.data_ptr() + 2 * at, o.data_ptr(), do.data_ptr(), lse.data_ptr(), cu.data_ptr(), 1, T,
        h, h, d, n, n, n, h * d, h * d, d ** -0.5, delta.data_ptr(), acc[0].data_ptr(), acc[1].data_ptr(), acc[2].data_ptr(),
        dqkv.data_ptr(), dqkv.stride(0), _ext.status_buffer(qkv.device).data_ptr(), _ext.stream_ptr(), 0)
    assert code == 0
    _ext.check_status()
    assert torch.equal(dqkv[:, :n], qkv.grad)
    assert (dqkv[:, n:] == 7).all() and (buf[:shift] == 7).all()
