"""Attention gradients on both backward kernels against 64-bit attention, document by document."""
import math

import pytest
import torch

from chronicals_b200 import ops
from chronicals_b200.ops import _ext

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _grad64(qkv, do, lens, hq, hk, d):
    x = qkv.detach().double().requires_grad_()
    q, k, v = (t.reshape(x.shape[0], -1, d) for t in x.split([hq * d, hk * d, hk * d], dim=1))
    out, at = [], 0
    for n in lens:
        mask = torch.ones(n, n, dtype=torch.bool, device=DEV).triu_(1)
        heads = []
        for h in range(hq):
            s = (q[at:at + n, h] @ k[at:at + n, h // (hq // hk)].t() / math.sqrt(d)).masked_fill(mask, -math.inf)
            heads.append(torch.softmax(s, -1) @ v[at:at + n, h // (hq // hk)])
        out.append(torch.cat(heads, dim=1))
        at += n
    if at < x.shape[0]:
        out.append(torch.zeros(x.shape[0] - at, hq * d, dtype=torch.float64, device=DEV))
    torch.cat(out).backward(do.double())
    return x.grad


# head size 128: one block short of, at and past a tile; one to five query blocks in a loop (the rings wrap at two); more
# than 32 documents; padding behind the last one.  Head size 64: the pipelined kernel (few tiles, 4096 tokens and more a
# document) and the phase-by-phase one on either side of the line between them
@pytest.mark.parametrize("hq,hk,d,lens,pad", [
    (2, 1, 128, [1], 0), (3, 3, 128, [127, 128, 129], 0), (4, 2, 128, [31, 33, 64, 257, 600, 2], 5), (2, 1, 128, [3] * 40 + [130], 200),
    (1, 1, 128, [1023], 1), (7, 1, 128, [385, 512], 0),
    (4, 2, 64, [1], 0), (4, 4, 64, [513], 0), (3, 1, 64, [640, 511, 513], 3), (2, 2, 64, [1300], 0), (2, 1, 64, [4100], 0),
    (14, 2, 64, [511, 512], 0), (14, 2, 64, [512, 512], 0), (32, 8, 64, [700, 700], 0)])
def test_attention_gradients(hq, hk, d, lens, pad):
    g = torch.Generator(device=DEV).manual_seed(sum(lens) + hq)
    T = sum(lens) + pad
    qkv = torch.randn(T, (hq + 2 * hk) * d, device=DEV, generator=g).to(torch.bfloat16).requires_grad_()
    do = torch.randn(T, hq * d, device=DEV, generator=g).to(torch.bfloat16)
    cu = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32, device=DEV)
    ops.attention_qkv_packed(qkv, cu, hq, hk, d).backward(do)
    _ext.check_status()
    want = _grad64(qkv, do, lens, hq, hk, d)
    valid = sum(lens)
    assert pad == 0 or qkv.grad[valid:].abs().max().item() == 0
    # P and dS are rounded to bf16 (relative 2^-9 each) before the second products, the result once more; delta comes from
    # the rounded output: below 2^-7 of the norm together
    for a, b in ((0, hq * d), (hq * d, (hq + hk) * d), ((hq + hk) * d, (hq + 2 * hk) * d)):
        got, ref = qkv.grad[:valid, a:b].double(), want[:valid, a:b]
        assert ((got - ref).norm() <= 2.0 ** -7 * ref.norm() + 1e-3).item(), ((got - ref).norm() / ref.norm()).item()


# A document's last query block is loaded with the first rows of the next one, whose probabilities are zero: finite rows of any
# size take no part.  NaN there is not covered, since 0 x NaN is NaN; towards the rows behind it a document never spreads.
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("value", [1e30, math.nan])
def test_attention_gradients_stay_within_their_document(d, value):
    lens, hq, hk = [600, 70, 650], 4, 2
    T, a, b = sum(lens), lens[0], lens[0] + lens[1]
    g = torch.Generator(device=DEV).manual_seed(1)
    qkv = torch.randn(T, (hq + 2 * hk) * d, device=DEV, generator=g).to(torch.bfloat16)
    do = torch.randn(T, hq * d, device=DEV, generator=g).to(torch.bfloat16)
    want = _grad64(qkv, do, lens, hq, hk, d)
    do[a:b] = value                                               # the gradient of one document's output
    cu = torch.tensor([0, a, b, T], dtype=torch.int32, device=DEV)
    x = qkv.requires_grad_()
    ops.attention_qkv_packed(x, cu, hq, hk, d).backward(do)
    for rows in ([slice(b, T)] if math.isnan(value) else [slice(0, a), slice(b, T)]):
        got, ref = x.grad[rows].double(), want[rows]
        assert ((got - ref).norm() <= 2.0 ** -7 * ref.norm()).item()      # the bound of the test above
