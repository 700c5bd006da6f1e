"""Reductions over rows, runs and columns at the sizes where their splits can go wrong, against 64-bit formulas."""
import math
import threading

import pytest
import torch

from chronicals_b200 import ops

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


# vocabularies below one vector, odd ones (every row starts elsewhere within 16 bytes), rows shared by 2, 4 and 8 blocks,
# more rows than fit at once; `gap` elements between the rows, `shift` before the first one
@pytest.mark.parametrize("rows,V,gap,shift", [(1, 3, 0, 0), (2, 4099, 0, 1), (5, 8192, 0, 0), (7, 33001, 3, 0), (2, 70000, 0, 0),
                                              (2500, 1031, 0, 0), (40, 12288, 8, 8)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_logits_cross_entropy_rows(rows, V, gap, shift, dtype):
    g = _gen(rows + V)
    buf = (3 * torch.randn(shift + rows * (V + gap), device=DEV, generator=g)).to(dtype)
    lg = buf[shift:].view(rows, V + gap)[:, :V]
    if V > 100:
        lg[0, : V // 2] = -math.inf                               # a masked vocabulary: whole batches of -inf
    y = torch.randint(V // 2, V, (rows,), device=DEV, generator=g)
    y[1::3] = -100
    if rows > 4:
        y[4] = V                                                  # no row of the vocabulary: takes no part either
    x = lg.detach().requires_grad_()
    loss = ops.cross_entropy_logits(x, y, -100, 0.0, 1e-3, reduction="none")
    gr = torch.rand(rows, device=DEV, generator=g) + 0.5
    loss.backward(gr)
    ok = (y >= 0) & (y < V)
    xr = lg.detach().double().requires_grad_()
    lse = torch.logsumexp(xr, -1)
    want = torch.where(ok, lse - xr.gather(1, y.clamp(0, V - 1)[:, None])[:, 0] + 1e-3 * lse.square(), torch.zeros_like(lse))
    want.backward(gr.double())
    # fp32 arithmetic on values of order 10: a few ulp of the largest intermediate
    assert (loss.double() - want).abs().max().item() < 2e-5
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 1e-5          # rounding of the stored gradient
    assert ((x.grad.double() - xr.grad).abs() <= eps * xr.grad.abs() + 1e-6).all()
    assert (x.grad[~ok] == 0).all()
    if gap:                                                       # nothing outside the rows was written
        assert torch.equal(buf[shift:].view(rows, V + gap)[:, :V], lg)


# a warp, two and eight a row with a batch that is just full, short of it and past it; rows on either side of the line between
# one vector and four a thread; rows shared by clusters in pieces of either kind
@pytest.mark.parametrize("rows,V,gap,shift", [(593, 128, 0, 0), (592, 1023, 1, 1), (593, 1023, 1, 1), (593, 1024, 0, 0), (600, 1025, 0, 0),
                                              (593, 8192, 0, 0), (593, 8200, 0, 0), (40, 24576, 0, 0), (74, 24584, 0, 0),
                                              (75, 24584, 0, 0), (300, 33001, 0, 1)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_logits_cross_entropy_row_layouts(rows, V, gap, shift, dtype):
    test_logits_cross_entropy_rows(rows, V, gap, shift, dtype)


# chunk and tile edges of the sort by counting, several tiles of ids, the range sorted by the library; one id only, ids
# outside the table
@pytest.mark.parametrize("T,V,N", [(1, 5, 8), (31, 40, 64), (32, 3, 896), (33, 1, 8), (64, 1000, 1032), (65, 7, 256),
                                   (4097, 151, 896), (9000, 32000, 64), (33000, 500, 64)])
def test_embedding_backward_runs(T, V, N):
    g = _gen(T + V)
    table = torch.randn(V, N, device=DEV, generator=g).to(torch.bfloat16).requires_grad_()
    ids = (torch.exp(torch.rand(T, device=DEV, generator=g) * math.log(V + 1)) - 1).long().clamp_(0, V - 1)
    if T > 64:
        ids[40:60], ids[62] = V + 5, -1                           # read row 0 forward, take no part backward
    dy = torch.randn(T, N, device=DEV, generator=g).to(torch.bfloat16)
    y = ops.embedding(ids, table)
    y.backward(dy)
    ok = (ids >= 0) & (ids < V)
    assert torch.equal(y, table.detach()[torch.where(ok, ids, torch.zeros_like(ids))])
    want = torch.zeros(V, N, dtype=torch.float64, device=DEV).index_add_(0, ids[ok], dy[ok].double())
    size = torch.zeros(V, N, dtype=torch.float64, device=DEV).index_add_(0, ids[ok], dy[ok].double().abs())
    # one rounding to bf16, and T fp32 additions of at most `size`
    assert ((table.grad.double() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -23 * 40 * size).all()
    first = table.grad.clone()
    table.grad = None
    ops.embedding(ids, table).backward(dy)
    assert torch.equal(first, table.grad)


# one vector, a warp's row at its widest, the narrowest and the widest block with two vectors a thread (with a ragged last
# vector), the first and the last width with four; fewer rows than the ring, rows that wrap it, more rows than blocks
@pytest.mark.parametrize("M,N", [(1, 8), (3, 1024), (5, 1032), (700, 2056), (2, 5120), (301, 5120), (1, 5128), (613, 6664), (299, 8192),
                                 (5000, 264)])
@pytest.mark.parametrize("residual", [False, True])
def test_rmsnorm_layouts(M, N, residual):
    g = _gen(M + N)
    x, dy, dh = (torch.randn(M, N, device=DEV, generator=g).to(torch.bfloat16) for _ in range(3))
    w = (1 + 0.1 * torch.randn(N, device=DEV, generator=g)).to(torch.bfloat16)
    xr, wr = x.double().requires_grad_(), w.double().requires_grad_()
    yr = xr * torch.rsqrt(xr.square().mean(-1, keepdim=True) + 1e-6) * wr
    x.requires_grad_(), w.requires_grad_()
    if residual:
        y, h = ops.rmsnorm_residual(x, w)
        torch.autograd.backward((y, h), (dy, dh))
        torch.autograd.backward((yr, xr * 1.0), (dy.double(), dh.double()))
    else:
        y = ops.rmsnorm(x, w)
        y.backward(dy)
        yr.backward(dy.double())
    size = (dy.double() * yr.detach()).abs().sum(0)               # of the terms that a column of dw adds up
    for got, want, slack in ((y, yr, 1e-5), (x.grad, xr.grad, 2e-5), (w.grad, wr.grad, 1e-5 * size + 1e-5)):
        # one rounding to bf16 and fp32 sums (dx of a residual cancels: its terms are of order one)
        assert ((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + slack).all()


def test_rmsnorm_backward_from_two_threads():
    """Calls that need more and calls that need less shared memory of the same kernel, at the same time."""
    M, N, calls = 4, 5120, 4000                                   # 90 KB a block with a residual's gradient, 60 KB without
    L = ops._ext.lib()
    g = _gen(1)
    dy, h, res = (torch.randn(M, N, device=DEV, generator=g).to(torch.bfloat16) for _ in range(3))
    w, rstd = torch.ones(N, device=DEV, dtype=torch.bfloat16), torch.ones(M, device=DEV)
    failed, ended = [], []

    def run(dres):
        s = torch.cuda.Stream()
        dx, dw = torch.empty_like(h), torch.empty_like(w)
        part = torch.empty(L.cb_rmsnorm_bwd_blocks(M, N) * N, device=DEV)
        s.wait_stream(torch.cuda.default_stream())
        for _ in range(calls):
            code = L.cb_rmsnorm_bwd(dy.data_ptr(), h.data_ptr(), w.data_ptr(), rstd.data_ptr(), dres, dx.data_ptr(), dw.data_ptr(),
                                    part.data_ptr(), M, N, 0.0, 0, s.cuda_stream)
            if code != 0:
                failed.append(code)
        s.synchronize()
        ended.append(dres)

    threads = [threading.Thread(target=run, args=(d,)) for d in (res.data_ptr(), None)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed and len(ended) == 2


# one block of 32, ragged tiles of 128 in either direction, a pitch, a base off the 16-byte boundary, either copy alone
@pytest.mark.parametrize("R,C,pitch,shift", [(32, 32, 32, 0), (160, 224, 224, 0), (96, 416, 424, 0), (416, 96, 96, 3), (1024, 640, 640, 8)])
@pytest.mark.parametrize("fmt", ["e4m3", "e5m2"])
@pytest.mark.parametrize("rows,cols", [(True, True), (True, False), (False, True)])
def test_mxfp8_copies_of_a_matrix_and_its_transpose(R, C, pitch, shift, fmt, rows, cols):
    from chronicals_b200.ops import ref
    from chronicals_b200.utils import fp8_utils as F8
    g = _gen(R + C)
    buf = (torch.randn(shift + R * pitch, device=DEV, generator=g) * 4).to(torch.bfloat16)
    x = buf[shift:].view(R, pitch)[:, :C]
    x[0, :32], x[:32, C - 1] = 0, 0                               # whole blocks of zeros
    q, s, qt, st = F8.mxfp8_quantize_dual(x, fmt, 128, 192, rows, cols)
    for got, scales, m, want, tile in ((q, s, x, rows, 128), (qt, st, x.t(), cols, 192)):
        assert (got is not None) == want
        if want:
            qr, sr = ref.mxfp8_quantize(m.float().contiguous(), fmt)
            assert torch.equal(got, qr.view(torch.uint8)) and torch.equal(scales, F8.pack_mx_scales(sr, tile))


def test_the_copy_along_the_rows_alone_needs_no_transposing_kernel(monkeypatch):
    from chronicals_b200.ops import ref
    from chronicals_b200.utils import fp8_utils as F8

    def refuse(*a):
        raise AssertionError("kernel of both copies")
    monkeypatch.setattr(ops._ext.lib(), "cb_mxfp8_quant_dual", refuse, raising=False)
    x = torch.randn(96, 416, device=DEV, generator=_gen(5)).to(torch.bfloat16)
    q, s, qt, st = F8.mxfp8_quantize_dual(x, "e4m3", 128, 192, True, False)
    qr, sr = ref.mxfp8_quantize(x.float(), "e4m3")
    assert torch.equal(q, qr.view(torch.uint8)) and torch.equal(s, F8.pack_mx_scales(sr, 128)) and qt is None and st is None


# one chunk and several, a last chunk narrower than a tile, a vocabulary that is no multiple of 8
@pytest.mark.parametrize("T,V,chunk", [(130, 5000, None), (130, 5000, 2048), (64, 4099, 1024), (257, 2056, 2048)])
def test_linear_cross_entropy_chunks(T, V, chunk, monkeypatch):
    if chunk is not None:
        monkeypatch.setattr(ops, "_cce_chunk", lambda *a: chunk)
    g = _gen(T + V)
    h = torch.randn(T, 256, device=DEV, generator=g).to(torch.bfloat16).requires_grad_()
    w = (0.05 * torch.randn(V, 256, device=DEV, generator=g)).to(torch.bfloat16).requires_grad_()
    y = torch.randint(0, V, (T,), device=DEV, generator=g)
    ops.linear_cross_entropy(h, w, y).backward()
    hr, wr = h.detach().double().requires_grad_(), w.detach().double().requires_grad_()
    torch.nn.functional.cross_entropy(hr @ wr.t(), y).backward()
    # d(logits) is rounded to bf16 (2^-9) and so is either gradient
    for got, want in ((h.grad, hr.grad), (w.grad, wr.grad)):
        assert ((got.double() - want).norm() <= 2.0 ** -7 * want.norm()).item()


# one item in all, runs of one tile, a last run shorter than the others, several rounds
@pytest.mark.parametrize("T,V", [(1, 8), (64, 256), (130, 5000), (300, 40000), (3000, 4099)])
@pytest.mark.parametrize("smoothing", [0.0, 0.1])
def test_linear_cross_entropy_splits(T, V, smoothing):
    g = _gen(T + V)
    h = torch.randn(T, 128, device=DEV, generator=g).to(torch.bfloat16)
    w = (0.1 * torch.randn(V, 128, device=DEV, generator=g)).to(torch.bfloat16)
    y = torch.randint(0, V, (T,), device=DEV, generator=g)
    rows = ops.linear_cross_entropy(h, w, y, label_smoothing=smoothing, reduction="none")
    want = torch.nn.functional.cross_entropy(h.double() @ w.double().t(), y, label_smoothing=smoothing, reduction="none")
    assert (rows.double() - want).abs().max().item() < 2e-5 * max(1.0, want.abs().max().item())      # fp32 sums throughout


# less than a load, less than and just past the four loads in flight, a chunk and one value more, a base off the 16-byte boundary
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("master", [False, True])
def test_adamw_norm_and_update_at_the_edges_of_a_chunk(dtype, master):
    from chronicals_b200.optimizers.fused_adamw import FusedAdamW
    g = _gen(3)
    sizes = [1, 3, 7, 2048, 4095, 6151, 8191, 8192, 8193, 20000, 9 * 8192 + 5]
    params = [torch.nn.Parameter(torch.randn(n, device=DEV, generator=g).to(dtype)) for n in sizes]
    for i, p in enumerate(params):
        grad = torch.randn(sizes[i] + 1, device=DEV, generator=g).to(dtype)
        p.grad = grad[1:] if i % 2 else grad[:-1]
    opt = FusedAdamW(params, lr=1e-2, weight_decay=0.1, max_grad_norm=1.0, master_weights=master)
    before = [p.detach().double() for p in params]
    opt.step()
    norm = sum(p.grad.double().square().sum() for p in params).sqrt()
    assert abs(opt.last_grad_norm.double() - norm).item() < 1e-5 * norm.item()       # fp32 sums of 8192 squares, fp64 beyond
    clip = 1.0 / (norm + 1e-6)
    for p, b in zip(params, before):
        gr = p.grad.double() * clip
        want = b * (1 - 1e-3) - 1e-2 * gr / (gr.abs() + 1e-8)                        # first step: m / bc1 = g, v / bc2 = g^2
        eps = 2.0 ** -8 if dtype == torch.bfloat16 else 1e-6
        assert ((p.detach().double() - want).abs() <= eps * want.abs() + 2e-6).all()
