"""Numerics of each hand-written sm_100a kernel against a plain PyTorch fp32 reference of the same op."""
import math
import time

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"


@pytest.fixture(scope="module")
def ext():
    from surogate_b200.ops import ext as load

    return load()


def _rel_err(a, b):
    return ((a.float() - b.float()).norm() / (b.float().norm() + 1e-12)).item()


def _check_flag():
    from surogate_b200.ops import check_device_errors

    check_device_errors()


# ----------------------------------------------------------------------------- GEMM
GEMM_SHAPES = [(256, 256, 128), (128, 128, 64), (384, 512, 320), (300, 264, 200), (1024, 1536, 1024), (136, 8, 64), (4096, 512, 2048)]


@pytest.mark.parametrize("M,N,K", GEMM_SHAPES)
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True), (True, False)])
def test_gemm_bf16(ext, M, N, K, a_mn, b_mn):
    from surogate_b200.runtime.ops_cuda import gemm

    if (a_mn and M % 8) or (b_mn and N % 8) or K % 8:
        pytest.skip("row stride must be a multiple of 16 bytes")
    torch.manual_seed(M + N + K)
    A = torch.randn(M, K, device=DEV)
    B = torch.randn(N, K, device=DEV)
    a = (A.t().contiguous() if a_mn else A).bfloat16()
    b = (B.t().contiguous() if b_mn else B).bfloat16()
    ref = (a.t() if a_mn else a).float() @ (b.t() if b_mn else b).float().t()
    out = gemm(a, b, a_mn=a_mn, b_mn=b_mn)
    torch.cuda.synchronize()
    _check_flag()
    assert _rel_err(out, ref) < 6e-3, _rel_err(out, ref)


PAIR_SHAPES = [(256, 256, 128), (512, 768, 320), (300, 264, 200), (1024, 1536, 1024), (2048, 1000, 4096), (4096, 512, 2048), (128, 520, 64)]


@pytest.mark.parametrize("M,N,K", PAIR_SHAPES)
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True), (True, False)])
@pytest.mark.parametrize("fp8", [False, True])
def test_gemm_cta_pair(ext, M, N, K, a_mn, b_mn, fp8):
    """The cta_group::2 kernel (256 x 256 tile per two-CTA cluster, TMA-store epilogue), forced with tile_n=512: every operand
    layout, bf16 and FP8, ragged edges in M, N and K, bf16 and fp32 outputs, fp32 accumulation (TMA add) and bf16 accumulation."""
    from surogate_b200.runtime.ops_cuda import gemm

    es = 1 if fp8 else 2
    if (a_mn and M * es % 16) or (b_mn and N * es % 16) or K * es % 16 or N % 8:
        pytest.skip("row stride must be a multiple of 16 bytes")
    torch.manual_seed(M + N + K)
    A = torch.randn(M, K, device=DEV)
    B = torch.randn(N, K, device=DEV)
    dt = torch.float8_e4m3fn if fp8 else torch.bfloat16
    a = (A.t().contiguous() if a_mn else A).to(dt)
    b = (B.t().contiguous() if b_mn else B).to(dt)
    ref = (a.float().t() if a_mn else a.float()) @ (b.float().t() if b_mn else b.float()).t()
    kw = dict(scale_a=torch.tensor([0.5], device=DEV), scale_b=torch.tensor([2.0], device=DEV)) if fp8 else {}
    amax = torch.zeros(1, device=DEV)
    out = gemm(a, b, a_mn=a_mn, b_mn=b_mn, tile_n=512, amax_out=amax, **kw)
    torch.cuda.synchronize()
    _check_flag()
    assert _rel_err(out, ref) < 6e-3, _rel_err(out, ref)
    assert abs(amax.item() - out.float().abs().max().item()) <= 0.01 * amax.item()
    out32 = gemm(a, b, a_mn=a_mn, b_mn=b_mn, tile_n=512, out_dtype=torch.float32, **kw)
    assert _rel_err(out32, ref) < 1e-4 if not fp8 else _rel_err(out32, ref) < 1e-4
    base = torch.randn(M, N, device=DEV)
    acc32 = base.clone()
    gemm(a, b, acc32, a_mn=a_mn, b_mn=b_mn, tile_n=512, accumulate=True, alpha=0.5, **kw)
    assert _rel_err(acc32, base + 0.5 * ref) < 1e-4
    acc16 = base.bfloat16()
    ref16 = acc16.float() + ref
    gemm(a, b, acc16, a_mn=a_mn, b_mn=b_mn, tile_n=512, accumulate=True, **kw)
    assert _rel_err(acc16, ref16) < 6e-3
    # a view into a wider buffer: the store must not touch the columns next to it
    wide = torch.zeros(M, N + 64, device=DEV, dtype=torch.bfloat16)
    gemm(a, b, wide[:, 32:32 + N], a_mn=a_mn, b_mn=b_mn, tile_n=512, **kw)
    assert _rel_err(wide[:, 32:32 + N], ref) < 6e-3
    assert wide[:, :32].abs().max() == 0 and wide[:, 32 + N:].abs().max() == 0
    torch.cuda.synchronize()
    _check_flag()


# M, N, K, tile_n, whole tiles before the cut ones
SPLIT_SHAPES = [(16, 5120, 16384, 0, False), (1024, 16, 16384, 0, False), (136, 200, 16400, 0, False),      # single CTAs, every tile cut
                (640, 4104, 16400, 0, True),                                                                # single CTAs, a wave of whole tiles first
                (1024, 1024, 16384, 512, False), (2000, 1000, 16400, 512, False),                           # CTA pairs, every tile cut, ragged edges
                (2560, 2048, 8192, 512, True), (5376, 1032, 16400, 512, True), (5000, 2056, 16400, 0, True)]  # CTA pairs, whole waves first


@pytest.mark.parametrize("M,N,K,tile_n,whole", SPLIT_SHAPES)
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True)])
@pytest.mark.parametrize("fp8", [False, True])
def test_gemm_with_a_split_contraction(ext, M, N, K, tile_n, whole, a_mn, b_mn, fp8):
    """Shapes whose tiles leave SMs idle are cut along the contraction (the plan is asked, so that other constants cannot empty this test).  bf16 and fp32 outputs, plain and accumulated, against fp32
    PyTorch: the error is the rounding of the output (2^-9 per element, twice with accumulation) and of fp32 sums; and the same bits twice,
    since the pieces are added in a fixed order."""
    from surogate_b200.runtime.ops_cuda import gemm

    es = 1 if fp8 else 2
    if (a_mn and M * es % 16) or (b_mn and N * es % 16) or K * es % 16:
        pytest.skip("row stride must be a multiple of 16 bytes")
    for out_fp32, accumulate in ((False, False), (False, True), (True, True)):
        pair, pieces, first_cut, _ = ext.gemm_plan(M, N, K, es, a_mn, b_mn, out_fp32, accumulate, tile_n, 148)
        assert pieces > 1 and (first_cut > 0) == whole and (pair or tile_n != 512)
    torch.manual_seed(M + N + K)
    dt = torch.float8_e4m3fn if fp8 else torch.bfloat16
    a = torch.randn(*((K, M) if a_mn else (M, K)), device=DEV).to(dt)
    b = torch.randn(*((K, N) if b_mn else (N, K)), device=DEV).to(dt)
    ref = (a.float().t() if a_mn else a.float()) @ (b.float() if b_mn else b.float().t())
    D0 = torch.randn(M, N, device=DEV) * K ** 0.5
    wide = torch.zeros(M, N + 24, device=DEV, dtype=torch.bfloat16)      # a strided output: nothing outside it may change
    out = wide[:, 8:8 + N]
    gemm(a, b, out, a_mn=a_mn, b_mn=b_mn, tile_n=tile_n)
    again = gemm(a, b, a_mn=a_mn, b_mn=b_mn, tile_n=tile_n)
    acc = D0.bfloat16()
    amax = torch.zeros(1, device=DEV)
    gemm(a, b, acc, a_mn=a_mn, b_mn=b_mn, tile_n=tile_n, accumulate=True, alpha=0.5, amax_out=amax)
    acc32 = D0.clone()
    gemm(a, b, acc32, a_mn=a_mn, b_mn=b_mn, tile_n=tile_n, accumulate=True, alpha=0.5)
    torch.cuda.synchronize()
    _check_flag()
    assert torch.equal(out, again) and not wide[:, :8].any() and not wide[:, 8 + N:].any()
    assert _rel_err(out, ref) < 2.5e-3
    want = D0.bfloat16().float() + 0.5 * ref
    assert _rel_err(acc, want) < 2.5e-3
    assert abs(amax.item() - acc.float().abs().max().item()) <= 2 ** -8 * amax.item()
    assert _rel_err(acc32, D0 + 0.5 * ref) < 2e-5


def test_gemm_runs_unsplit_when_the_workspace_does_not_fit(ext):
    """A split contraction takes up to 58 MB of workspace; a device with less to spare still multiplies.  (The allocator is limited, not the
    device filled.)"""
    from surogate_b200.runtime.ops_cuda import gemm

    torch.manual_seed(0)
    M, N, K = 1024, 3072, 16384
    a, b = torch.randn(K, M, device=DEV).bfloat16(), torch.randn(K, N, device=DEV).bfloat16()
    assert ext.gemm_plan(M, N, K, 2, True, True, False, False, 0, 148)[3] > 20 << 20
    want, out = gemm(a, b, a_mn=True, b_mn=True), torch.empty(M, N, device=DEV, dtype=torch.bfloat16)
    ref = a.float().t() @ b.float()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    try:
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (1 << 20)) / total)
        gemm(a, b, out, a_mn=True, b_mn=True)
        torch.cuda.synchronize()
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    _check_flag()
    assert _rel_err(out, ref) < 2.5e-3 and _rel_err(want, ref) < 2.5e-3


def test_gemm_bf16_accumulation_with_a_short_contraction(ext):
    """D += A.B^T where D is the traffic (adapter updates, gradient accumulation): its tiles travel through shared memory both ways."""
    from surogate_b200.runtime.ops_cuda import gemm

    torch.manual_seed(3)
    for M, N, K in [(8192, 4096, 16), (4000, 5128, 48), (2600, 2056, 72)]:
        h = torch.randn(M, 3 * K, device=DEV).bfloat16()
        a, b = h[:, K:2 * K], torch.randn(N, K, device=DEV).bfloat16()
        wide = torch.randn(M, N + 64, device=DEV).bfloat16()
        before = wide.clone()
        gemm(a, b, wide[:, 32:32 + N], accumulate=True, alpha=2.0)
        torch.cuda.synchronize()
        _check_flag()
        want = before[:, 32:32 + N].float() + 2.0 * (a.float() @ b.float().t())
        assert (wide[:, 32:32 + N].float() - want).abs().max() <= 2 ** -8 * want.abs().max()
        assert _rel_err(wide[:, 32:32 + N], want) < 2.5e-3
        assert torch.equal(wide[:, :32], before[:, :32]) and torch.equal(wide[:, 32 + N:], before[:, 32 + N:])


def test_gemm_accumulate_fp32_and_alpha(ext):
    from surogate_b200.runtime.ops_cuda import gemm

    M, N, K = 512, 384, 256
    a = torch.randn(M, K, device=DEV).bfloat16()
    b = torch.randn(N, K, device=DEV).bfloat16()
    base = torch.randn(M, N, device=DEV)
    out = base.clone()
    gemm(a, b, out, accumulate=True, alpha=0.5)
    ref = base + 0.5 * (a.float() @ b.float().t())
    assert _rel_err(out, ref) < 1e-4
    out16 = base.bfloat16()
    ref16 = out16.float() + a.float() @ b.float().t()
    gemm(a, b, out16, accumulate=True)
    assert _rel_err(out16, ref16) < 6e-3
    # strided output / strided inputs (views into wider buffers)
    wide = torch.zeros(M, N + 64, device=DEV, dtype=torch.bfloat16)
    gemm(a, b, wide[:, 32:32 + N])
    assert _rel_err(wide[:, 32:32 + N], a.float() @ b.float().t()) < 6e-3
    assert wide[:, :32].abs().max() == 0 and wide[:, 32 + N:].abs().max() == 0
    _check_flag()


@pytest.mark.parametrize("M,N,K", [(256, 256, 256), (384, 512, 384), (1024, 768, 2048), (272, 264, 144)])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True)])
@pytest.mark.parametrize("a_e5m2", [False, True])
def test_gemm_fp8(ext, M, N, K, a_mn, b_mn, a_e5m2):
    from surogate_b200.runtime.ops_cuda import gemm

    if (a_mn and M % 16) or (b_mn and N % 16) or K % 16:
        pytest.skip("row stride must be a multiple of 16 bytes")
    torch.manual_seed(1)
    A = torch.randn(M, K, device=DEV)
    B = torch.randn(N, K, device=DEV)
    a = (A.t().contiguous() if a_mn else A).to(torch.float8_e5m2 if a_e5m2 else torch.float8_e4m3fn)
    b = (B.t().contiguous() if b_mn else B).to(torch.float8_e4m3fn)
    sa = torch.tensor([0.5], device=DEV)
    sb = torch.tensor([2.5], device=DEV)
    ref = 1.25 * ((a.float().t() if a_mn else a.float()) @ (b.float().t() if b_mn else b.float()).t())
    amax = torch.zeros(1, device=DEV)
    out = gemm(a, b, a_mn=a_mn, b_mn=b_mn, scale_a=sa, scale_b=sb, amax_out=amax)
    torch.cuda.synchronize()
    _check_flag()
    assert _rel_err(out, ref) < 6e-3, _rel_err(out, ref)
    assert abs(amax.item() - out.float().abs().max().item()) <= 0.01 * amax.item()


# ----------------------------------------------------------------------------- norms
@pytest.mark.parametrize("C", [1024, 4096, 5120])
def test_rmsnorm_fwd_bwd(ext, C):
    rows = 333
    x = torch.randn(rows, C, device=DEV).bfloat16()
    r = torch.randn(rows, C, device=DEV).bfloat16()
    w = (1 + 0.1 * torch.randn(C, device=DEV)).bfloat16()
    res, y, rstd, _ = ext.rmsnorm_fwd(x, r, w, 1e-6, True, None, None, False)
    rf = (x.float() + r.float()).bfloat16().float()
    ref_rstd = torch.rsqrt(rf.pow(2).mean(-1) + 1e-6)
    assert torch.equal(res, rf.bfloat16())
    assert torch.allclose(rstd, ref_rstd, rtol=1e-4)
    assert _rel_err(y, rf * ref_rstd[:, None] * w.float()) < 5e-3
    dy = torch.randn(rows, C, device=DEV).bfloat16()
    dres = torch.randn(rows, C, device=DEV).bfloat16()
    dx, dw = ext.rmsnorm_bwd(dy, res, w, rstd, dres)
    xhat = rf * ref_rstd[:, None]
    dn = dy.float() * w.float()
    ref_dx = ref_rstd[:, None] * (dn - xhat * (dn * xhat).mean(-1, keepdim=True)) + dres.float()
    assert _rel_err(dx, ref_dx) < 5e-3
    assert _rel_err(dw, (dy.float() * xhat).sum(0)) < 1e-4
    # fp8 output with scale and abs-max
    scale = torch.tensor([3.0], device=DEV)
    amax = torch.zeros(1, device=DEV)
    _, _, _, y8 = ext.rmsnorm_fwd(x, r, w, 1e-6, False, scale, amax, True)
    yref = rf * ref_rstd[:, None] * w.float()
    assert _rel_err(y8.float() / 3.0, yref) < 0.05
    assert abs(amax.item() - yref.abs().max().item()) < 0.02 * amax.item()


@pytest.mark.parametrize("rows,C", [(5, 24), (300, 1000), (3000, 1024), (257, 4104), (40, 16384)])
def test_rmsnorm_weight_gradient_sums(ext, rows, C):
    """The column sums behind dw: widths that are no multiple of a CTA's 16 columns, fewer partial rows than a CTA reads side by side, and
    many.  fp32 sums of `rows` products against fp64: a few 2^-24 of the largest column sum of magnitudes."""
    torch.manual_seed(rows + C)
    dy, x, w = (torch.randn(*s, device=DEV).bfloat16() for s in ((rows, C), (rows, C), (C,)))
    rstd = torch.rand(rows, device=DEV) + 0.5
    _, dw = ext.rmsnorm_bwd(dy, x, w, rstd, None)
    terms = dy.double() * x.double() * rstd.double()[:, None]
    assert ((dw.double() - terms.sum(0)).abs() <= 16 * 2.0 ** -24 * terms.abs().sum(0)).all()
    assert torch.equal(dw, ext.rmsnorm_bwd(dy, x, w, rstd, None)[1])


@pytest.mark.parametrize("rows,C", [(1, 8), (3, 256), (5, 2048), (4, 2056), (3, 4096), (2, 8192), (2, 8200)])
def test_rmsnorm_forward_widths(ext, rows, C):
    """Widths around those at which the row is kept in one, two or four vectors per thread, and beyond."""
    torch.manual_seed(C)
    x, res, w = (torch.randn(*s, device=DEV).bfloat16() for s in ((rows, C), (rows, C), (C,)))
    r, y, rstd, _ = ext.rmsnorm_fwd(x, res, w, 1e-6, True, None, None, False)
    scale, amax = torch.tensor([3.0], device=DEV), torch.zeros(1, device=DEV)
    _, _, _, y8 = ext.rmsnorm_fwd(x, res, w, 1e-6, False, scale, amax, True)
    want_r = x + res
    want = want_r.float() * torch.rsqrt(want_r.float().pow(2).mean(-1, keepdim=True) + 1e-6) * w.float()
    assert torch.equal(r, want_r) and _rel_err(y, want) < 3e-3          # one bf16 rounding
    assert _rel_err(y8.float() / 3.0, want) < 4e-2                      # one E4M3 rounding
    assert abs(amax.item() - want.abs().max().item()) < 1e-4 * amax.item()
    y0 = ext.rmsnorm_fwd(x, None, w, 1e-6, True, None, None, False)[1]
    want0 = x.float() * torch.rsqrt(x.float().pow(2).mean(-1, keepdim=True) + 1e-6) * w.float()
    assert _rel_err(y0, want0) < 3e-3


@pytest.mark.parametrize("rows,M", [(1, 8), (3, 264), (2, 12288), (8193, 768), (1025, 2056)])
def test_swiglu_row_counts(ext, rows, M):
    """One row, row counts off the grid's stride, and widths of one to many vectors."""
    torch.manual_seed(rows + M)
    x, dy = torch.randn(rows, 2 * M, device=DEV).bfloat16(), torch.randn(rows, M, device=DEV).bfloat16()
    xr = x.float().requires_grad_(True)
    ref = torch.nn.functional.silu(xr[:, M:]) * xr[:, :M]
    ref.backward(dy.float())
    scale, amax = torch.tensor([2.0], device=DEV), torch.zeros(1, device=DEV)
    y, y8 = ext.swiglu_fwd(x, True, scale, amax, True)
    assert _rel_err(y, ref.detach()) < 3e-3 and _rel_err(y8.float() / 2.0, ref.detach()) < 4e-2
    assert abs(amax.item() - ref.abs().max().item()) < 1e-3 * amax.item()
    assert _rel_err(ext.swiglu_bwd(dy, x), xr.grad) < 3e-3
    d8 = ext.swiglu_bwd_fp8(dy, x, scale, torch.zeros(1, device=DEV))
    assert _rel_err(d8.float() / 2.0, xr.grad) < 8e-2                   # one E5M2 rounding
    limit = torch.tensor([rows // 2], device=DEV, dtype=torch.int32)
    half = ext.swiglu_fwd(x, True, None, None, False, limit)[0]
    assert torch.equal(half[:rows // 2], y[:rows // 2])


@pytest.mark.parametrize("V", [8, 4096, 8200, 32000, 151936])
def test_cross_entropy_fp8_gradient(ext, V):
    """The E5M2 gradient bit for bit against quantising the bf16 one, the same losses, untouched logits; rows with -inf logits and ignored
    rows, and a row stride."""
    torch.manual_seed(V)
    rows = 6
    wide = (3 * torch.randn(rows, V + 16, device=DEV)).bfloat16()
    logits = wide[:, 8:8 + V] if V % 16 else wide[:, :V]
    logits[1, : V // 2] = float("-inf")
    logits[2] = 0
    tgt = torch.randint(0, V, (rows,), device=DEV, dtype=torch.int32)
    tgt[1] = V - 1
    tgt[4] = -100
    before = logits.clone()
    ref_loss = torch.nn.functional.cross_entropy(logits.float(), tgt.long(), ignore_index=-100, reduction="none")
    scale, q_scale = torch.tensor([0.5], device=DEV), torch.tensor([57344.0 * 0.5 / 0.25], device=DEV)
    loss8, d8 = ext.cross_entropy_fwd_bwd_fp8(logits, tgt, scale, 0.5, q_scale)
    assert torch.equal(logits, before)
    loss = ext.cross_entropy_fwd_bwd(logits, tgt, scale, 0.5, True)
    assert torch.allclose(loss, ref_loss, rtol=1e-4, atol=1e-4) and torch.equal(loss8, loss)
    assert torch.equal(d8.view(torch.uint8), ext.quantize_fp8(logits.contiguous(), q_scale, None, True).view(torch.uint8)) and not logits[4].any()


@pytest.mark.parametrize("n,V,C", [(1, 4, 8), (7, 3, 512), (64, 2, 520), (1000, 50, 1032), (300, 7, 6), (257, 1, 24)])
@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float32])
def test_embedding_gradient_runs(ext, n, V, C, dt):
    """Runs of equal ids of one, around the eight rows in flight, and hundreds; column counts around a CTA's 512 and one that is not a
    multiple of 8; ids outside the table; accumulation into a table, twice the same bits."""
    torch.manual_seed(n + C)
    ids = torch.randint(0, V + 1, (n,), device=DEV, dtype=torch.int32)        # V itself is outside: skipped
    if V == 1:
        ids[:] = 0
    d = torch.randn(n, C, device=DEV).bfloat16()
    start = torch.randn(V, C, device=DEV).to(dt)
    a, b = start.clone(), start.clone()
    ext.embedding_bwd(ids, d, a)
    ext.embedding_bwd(ids, d, b)
    keep = ids < V
    want = start.double().index_add(0, ids[keep].long(), d[keep].double())
    assert torch.equal(a, b)
    scale = start.double().abs().index_add(0, ids[keep].long(), d[keep].double().abs())
    assert ((a.double() - want).abs() <= (2.0 ** -8 if dt == torch.bfloat16 else 0.0) * want.abs() + n * 2.0 ** -24 * scale).all()
    t = torch.randn(V, C, device=DEV).to(dt)
    ext.zero_fill(t)
    assert not t.any()


@pytest.mark.parametrize("C,shift", [(1022, 0), (510, 0), (512, 1), (520, 2), (6, 0)])
@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float32])
def test_embedding_gradient_of_narrow_rows_needs_no_copy_of_the_table(ext, C, shift, dt):
    """Rows that are not whole 16-byte vectors (even widths, views off the boundary) are summed in place: the bits of the aligned case, and
    no allocation that grows with the table."""
    torch.manual_seed(C)
    n, V = 300, 20000
    ids = torch.randint(0, 40, (n,), device=DEV, dtype=torch.int32)
    d0 = torch.randn(n, C, device=DEV).bfloat16()
    d = torch.empty(n * C + 8, device=DEV, dtype=torch.bfloat16)[shift:shift + n * C].view(n, C).copy_(d0)
    start = torch.randn(V, C, device=DEV).to(dt)
    pad = (C + 7) // 8 * 8 - C
    want, rows = torch.nn.functional.pad(start, (0, pad)), torch.nn.functional.pad(d0, (0, pad))
    ext.embedding_bwd(ids, rows, want)
    got = torch.empty(V * C + 8, device=DEV, dtype=dt)[shift:shift + V * C].view(V, C).copy_(start)
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    ext.embedding_bwd(ids, d, got)
    torch.cuda.synchronize()
    grown = torch.cuda.max_memory_allocated() - before
    assert torch.equal(got, want[:, :C])
    assert grown < min(V * C, 1 << 20)       # the sort of the ids: a few KB for each


@pytest.mark.parametrize("n", [8, 2048, 148 * 8 * 256 * 8, 148 * 8 * 256 * 8 + 24, 3 * 148 * 8 * 256 * 8 + 8])
@pytest.mark.parametrize("e5m2", [False, True])
def test_quantize_fp8_counts(ext, n, e5m2):
    """Counts of one vector, one block, one whole trip of the grid (148 SMs x 8 blocks x 256 threads x 8 values), a few vectors more, and
    several trips: the bits of PyTorch's conversion (saturating), and the abs-max."""
    torch.manual_seed(n % 1000)
    x = (torch.randn(n, device=DEV) * 200).bfloat16()
    x[-1] = -3000.0
    scale, amax, amax2 = torch.tensor([1.7], device=DEV), torch.zeros(1, device=DEV), torch.zeros(1, device=DEV)
    q = ext.quantize_fp8(x, scale, amax, e5m2)
    dt, top = (torch.float8_e5m2, 57344.0) if e5m2 else (torch.float8_e4m3fn, 448.0)
    want = (x.float() * scale).clamp(-top, top).to(dt)
    assert torch.equal(q.view(torch.uint8), want.view(torch.uint8)) and amax.item() == x.float().abs().max().item()
    ext.amax(x, amax2)
    assert amax2.item() == amax.item()


def test_swiglu(ext):
    rows, M = 517, 3072
    x = torch.randn(rows, 2 * M, device=DEV).bfloat16()
    y = ext.swiglu_fwd(x, True, None, None, False)[0]
    up, gate = x[:, :M].float(), x[:, M:].float()
    assert _rel_err(y, torch.nn.functional.silu(gate) * up) < 5e-3
    dy = torch.randn(rows, M, device=DEV).bfloat16()
    dx = ext.swiglu_bwd(dy, x)
    s = torch.sigmoid(gate)
    ref = torch.cat([dy.float() * gate * s, dy.float() * up * s * (1 + gate * (1 - s))], -1)
    assert _rel_err(dx, ref) < 5e-3


@pytest.mark.parametrize("B,T,Hq,Hkv", [(2, 96, 8, 2), (1, 50, 3, 1), (1, 300, 32, 8), (2, 33, 5, 5)])
def test_qk_norm_rope(ext, B, T, Hq, Hkv):
    """Even and odd head counts (a half-warp without a head of its own still takes part in the shuffles), the benchmark's 32 / 8."""
    from surogate_b200.dsl.ir import OpNode
    from surogate_b200.runtime.ops_ref import RefOps

    D = 128
    qkv = torch.randn(B, T, (Hq + 2 * Hkv) * D, device=DEV).bfloat16()
    qw = (1 + 0.1 * torch.randn(D, device=DEV)).bfloat16()
    kw = (1 + 0.1 * torch.randn(D, device=DEV)).bfloat16()
    pos = torch.arange(T, device=DEV, dtype=torch.int32)[None].repeat(B, 1).contiguous()
    attrs = dict(num_q_heads=Hq, num_kv_heads=Hkv, head_dim=D, eps=1e-6, rope_theta=1e6, rotary_dim=D)
    ref = RefOps()
    op = OpNode("qkv_qk_norm_rope", [], [], attrs)
    r_out, r_q, r_k = ref.qkv_qk_norm_rope(None, op, qkv.float(), qw.float(), kw.float(), pos)
    out, q_rstd, k_rstd = ext.qk_norm_rope_fwd(qkv, qw, kw, pos, Hq, Hkv, D, 1e-6, 1e6)
    assert _rel_err(out, r_out) < 5e-3
    assert torch.allclose(q_rstd, r_q, rtol=1e-4) and torch.allclose(k_rstd, r_k, rtol=1e-4)
    dy = torch.randn_like(qkv)
    r_dx, r_dq, r_dk = ref.qkv_qk_norm_rope_backward(None, op, dy.float(), qkv.float(), qw.float(), kw.float(), r_q, r_k, pos)
    dx, dqw, dkw = ext.qk_norm_rope_bwd(dy, qkv, qw, kw, q_rstd, k_rstd, pos, Hq, Hkv, D, 1e-6, 1e6)
    assert _rel_err(dx, r_dx) < 5e-3
    assert _rel_err(dqw, r_dq) < 2e-3 and _rel_err(dkw, r_dk) < 2e-3
    # without qk-norm (Llama-style)
    out2, _, _ = ext.qk_norm_rope_fwd(qkv, None, None, pos, Hq, Hkv, D, 1e-6, 1e4)
    attrs2 = dict(attrs, rope_theta=1e4)
    r2, _, _ = ref.qkv_qk_norm_rope(None, OpNode("x", [], [], attrs2), qkv.float(), None, None, pos)
    assert _rel_err(out2, r2) < 5e-3


@pytest.mark.parametrize("Hq,Hkv", [(1, 1), (5, 1), (8, 4), (9, 4), (16, 1), (13, 6), (32, 8)])
@pytest.mark.parametrize("tokens", [1, 4, 5, 13])
def test_qk_norm_rope_forward_head_counts(ext, Hq, Hkv, tokens):
    """Up to 16 heads a warp takes a token, from 17 on two warps share it (3, 7, 16, 17, 18, 25 and 48 here), with token counts around a block's four
    and eight: fp64 on the same bf16 inputs, one bf16 rounding."""
    torch.manual_seed(Hq * tokens)
    H, Dh = Hq + 2 * Hkv, 128
    qkv = torch.randn(1, tokens, H * Dh, device=DEV).bfloat16()
    qw, kw = (1 + 0.1 * torch.randn(Dh, device=DEV)).bfloat16(), (1 + 0.1 * torch.randn(Dh, device=DEV)).bfloat16()
    pos = torch.randint(0, 500, (1, tokens), device=DEV, dtype=torch.int32)
    out, q_rstd, k_rstd = ext.qk_norm_rope_fwd(qkv, qw, kw, pos, Hq, Hkv, Dh, 1e-6, 1e4)
    x = qkv.double().view(tokens, H, Dh)
    rstd = torch.rsqrt(x.pow(2).mean(-1) + 1e-6)
    n = x * rstd[..., None] * torch.cat([qw.double().expand(Hq, Dh), kw.double().expand(Hkv, Dh), torch.ones(Hkv, Dh, device=DEV, dtype=torch.double)])
    ang = pos[0].double()[:, None, None] * 1e4 ** (-torch.arange(64, device=DEV).double() / 64)
    rot = torch.cat([n[..., :64] * ang.cos() - n[..., 64:] * ang.sin(), n[..., 64:] * ang.cos() + n[..., :64] * ang.sin()], -1)
    got = out.view(tokens, H, Dh)
    assert torch.equal(got[:, Hq + Hkv:], qkv.view(tokens, H, Dh)[:, Hq + Hkv:])
    assert _rel_err(got[:, :Hq + Hkv], rot[:, :Hq + Hkv].float()) < 3e-3
    assert torch.allclose(q_rstd.view(tokens, Hq).double(), rstd[:, :Hq], rtol=1e-5) and torch.allclose(k_rstd.view(tokens, Hkv).double(), rstd[:, Hq:Hq + Hkv], rtol=1e-5)


def test_qk_norm_rope_multi_axis_positions(ext):
    """(t, h, w) rotary positions: frequency j reads the height row if j % 3 == 1 and j < 3 * sec_h, the width row if
    j % 3 == 2 and j < 3 * sec_w, else the temporal row; forward and backward against the PyTorch op."""
    from types import SimpleNamespace

    from surogate_b200.dsl.ir import OpNode
    from surogate_b200.runtime.ops_ref import RefOps

    B, T, Hq, Hkv, D = 2, 64, 4, 2, 128
    qkv = torch.randn(B, T, (Hq + 2 * Hkv) * D, device=DEV).bfloat16()
    qw = (1 + 0.1 * torch.randn(D, device=DEV)).bfloat16()
    kw = (1 + 0.1 * torch.randn(D, device=DEV)).bfloat16()
    pos3 = torch.stack([torch.arange(T, device=DEV)[None].repeat(B, 1), torch.randint(0, 40, (B, T), device=DEV), torch.randint(0, 40, (B, T), device=DEV)]).to(torch.int32)
    attrs = dict(num_q_heads=Hq, num_kv_heads=Hkv, head_dim=D, eps=1e-6, rope_theta=5e6, rotary_dim=D, mrope_section=[24, 20, 20])
    ctx = SimpleNamespace(extras={"mrope_position_ids": pos3})
    op = OpNode("qkv_qk_norm_rope", [], [], attrs)
    ref = RefOps()
    r_out, r_q, r_k = ref.qkv_qk_norm_rope(ctx, op, qkv.float(), qw.float(), kw.float(), pos3[0])
    out, q_rstd, k_rstd = ext.qk_norm_rope_fwd(qkv, qw, kw, pos3.contiguous(), Hq, Hkv, D, 1e-6, 5e6, 20, 20)
    assert _rel_err(out, r_out) < 5e-3
    plain, _, _ = ext.qk_norm_rope_fwd(qkv, qw, kw, pos3[0].contiguous(), Hq, Hkv, D, 1e-6, 5e6)
    assert _rel_err(plain, r_out) > 0.05  # the height / width rows matter
    dy = torch.randn_like(qkv)
    r_dx, r_dq, r_dk = ref.qkv_qk_norm_rope_backward(ctx, op, dy.float(), qkv.float(), qw.float(), kw.float(), r_q, r_k, pos3[0])
    dx, dqw, dkw = ext.qk_norm_rope_bwd(dy, qkv, qw, kw, q_rstd, k_rstd, pos3.contiguous(), Hq, Hkv, D, 1e-6, 5e6, 20, 20)
    assert _rel_err(dx, r_dx) < 5e-3 and _rel_err(dqw, r_dq) < 2e-3 and _rel_err(dkw, r_dk) < 2e-3


def test_embedding(ext):
    V, C, n = 1000, 512, 4096
    table = torch.randn(V, C, device=DEV).bfloat16()
    tok = torch.randint(0, V, (4, n // 4), device=DEV, dtype=torch.int32)
    out = ext.embedding_fwd(tok, table)
    assert torch.equal(out, table[tok.long()])
    dout = torch.randn(4, n // 4, C, device=DEV).bfloat16()
    g = torch.zeros(V, C, device=DEV, dtype=torch.float32)
    ext.embedding_bwd(tok, dout, g)
    ref = torch.zeros(V, C, device=DEV).index_add_(0, tok.reshape(-1).long(), dout.reshape(-1, C).float())
    assert _rel_err(g, ref) < 1e-5
    # the default (sorted, no atomics) is bit-reproducible, also into a bf16 table and with a heavily repeated id; the atomic variant agrees
    tok[0, :700] = 7
    ref = torch.zeros(V, C, device=DEV).index_add_(0, tok.reshape(-1).long(), dout.reshape(-1, C).float())
    runs = []
    for _ in range(2):
        gb = torch.zeros(V, C, device=DEV, dtype=torch.bfloat16)
        ext.embedding_bwd(tok, dout, gb)
        runs.append(gb)
    assert torch.equal(runs[0], runs[1]) and _rel_err(runs[0], ref) < 4e-3
    ga = torch.zeros(V, C, device=DEV, dtype=torch.float32)
    ext.embedding_bwd(tok, dout, ga, False)
    assert _rel_err(ga, ref) < 1e-5


def test_cross_entropy(ext):
    rows, V = 257, 151936 // 8
    logits = (3 * torch.randn(rows, V, device=DEV)).bfloat16()
    tgt = torch.randint(0, V, (rows,), device=DEV, dtype=torch.int32)
    tgt[::7] = -100
    ref_logits = logits.float().requires_grad_(True)
    ref_loss = torch.nn.functional.cross_entropy(ref_logits, tgt.long(), ignore_index=-100, reduction="none")
    (ref_loss.sum() * 0.25).backward()
    scale = torch.tensor([0.5], device=DEV)
    work = logits.clone()
    loss = ext.cross_entropy_fwd_bwd(work, tgt, scale, 0.5, True)
    assert torch.allclose(loss, ref_loss.detach(), rtol=1e-3, atol=1e-3)
    assert _rel_err(work, ref_logits.grad) < 1e-2
    assert work[::7].abs().max() == 0


def test_quantize_fp8_and_sumsq(ext):
    x = (5 * torch.randn(1 << 20, device=DEV)).bfloat16()
    scale = torch.tensor([4.0], device=DEV)
    amax = torch.zeros(1, device=DEV)
    q = ext.quantize_fp8(x, scale, amax, False)
    assert torch.equal(q.view(torch.uint8), (x.float() * 4).clamp(-448, 448).to(torch.float8_e4m3fn).view(torch.uint8))
    assert amax.item() == x.float().abs().max().item()
    q2 = ext.quantize_fp8(x, scale, None, True)
    assert torch.equal(q2.view(torch.uint8), (x.float() * 4).to(torch.float8_e5m2).view(torch.uint8))
    assert abs(ext.sumsq(x).item() / x.float().pow(2).sum().item() - 1) < 1e-4
    xf = torch.randn(12345, device=DEV)
    assert abs(ext.sumsq(xf).item() / xf.pow(2).sum().item() - 1) < 1e-5


@pytest.mark.parametrize("shape", [(1, 8), (3, 40), (129, 1000), (2, 3, 48), (4096, 272)])
@pytest.mark.parametrize("dt", [torch.float8_e4m3fn, torch.float8_e5m2])
def test_dequantize_fp8(ext, shape, dt):
    """Counts below, at and off the 16 values of a thread: the fp32 product rounded once, so the bits are PyTorch's."""
    torch.manual_seed(sum(shape))
    q = (torch.randn(*shape, device=DEV) * 20).to(dt)
    scale = torch.tensor([0.0371], device=DEV)
    out = ext.dequantize_fp8(q, scale)
    assert out.shape == q.shape and torch.equal(out, (q.float() * scale).bfloat16())


@pytest.mark.parametrize("n", [1, 31, 1024, 5000])
def test_step_scalars(ext, n):
    """Target count and loss scale, squared norms, clip factor (also without a limit and for a norm that is not finite) and the step's record."""
    torch.manual_seed(n)
    tgt = torch.randint(0, 50, (n,), device=DEV, dtype=torch.int32)
    tgt[torch.rand(n, device=DEV) < 0.3] = -100
    valid = int((tgt != -100).sum())
    c = ext.count_targets(tgt, -100)
    assert c[0].item() == valid and abs(c[1].item() - 1 / max(valid, 1)) < 1e-7
    assert ext.count_targets(torch.full((n,), -100, device=DEV, dtype=torch.int32), -100).tolist() == [0.0, 1.0]
    a, b, e = torch.randn(8 * n, device=DEV).bfloat16(), torch.randn(n, device=DEV), torch.randn(4096, device=DEV).bfloat16()
    hp = torch.zeros(8, device=DEV)
    sq = ext.sumsq_groups([a, b], [e], hp)
    assert abs(sq[0].item() / (a.double().pow(2).sum() + b.double().pow(2).sum()).item() - 1) < 1e-5
    assert abs(sq[1].item() / e.double().pow(2).sum().item() - 1) < 1e-5
    assert ext.sumsq_groups([], [], hp).tolist() == [0.0, 0.0]
    host = [1e-3, 0.9, 0.99, 1e-8, 0.1, 0.19, 0.02]
    for total, limit, clip in [(16.0, 1.0, 1.0 / (4.0 + 1e-6)), (0.25, 1.0, 1.0), (16.0, 0.0, 1.0), (float("inf"), 1.0, 0.0), (float("nan"), 0.0, 0.0)]:
        norm = ext.step_hyper(hp, torch.tensor(total, device=DEV), host, limit)
        torch.testing.assert_close(hp.cpu(), torch.tensor(host + [clip]))
        assert norm.shape == () and (norm.item() == total ** 0.5 or total != total)
    out = ext.step_report(torch.tensor(6.0, device=DEV), c[0], torch.tensor(0.5, device=DEV), torch.tensor(2.0, device=DEV))
    torch.testing.assert_close(out.cpu(), torch.tensor([6.0 / max(valid, 1) + 0.5, 2.0, 0.5, 0.0]))


def test_adamw_kernels(ext):
    n = 100000 - 100000 % 32
    p = torch.randn(n, device=DEV)
    g = torch.randn(n, device=DEV) * 0.1
    mask = (torch.arange(n, device=DEV) % 3 != 0).to(torch.uint8)
    lr, b1, b2, eps, wd = 1e-2, 0.9, 0.95, 1e-8, 0.1
    p_ref, m_ref, v_ref = p.clone(), torch.zeros(n, device=DEV), torch.zeros(n, device=DEV)
    p32, m, v = p.clone(), torch.zeros(n, device=DEV), torch.zeros(n, device=DEV)
    p8 = p.clone()
    m8, v8 = torch.zeros(n, dtype=torch.int8, device=DEV), torch.zeros(n, dtype=torch.uint8, device=DEV)
    ng = (n + 31) // 32
    ms, vs = torch.zeros(ng, dtype=torch.float16, device=DEV), torch.zeros(ng, dtype=torch.float16, device=DEV)
    for step in range(1, 6):
        gs = g * (1 + 0.1 * step)
        hp = torch.tensor([lr, b1, b2, eps, wd, 1 - b1 ** step, 1 - b2 ** step, 1.0], device=DEV)
        m_ref = b1 * m_ref + (1 - b1) * gs
        v_ref = b2 * v_ref + (1 - b2) * gs * gs
        p_ref = p_ref * (1 - lr * wd * mask) - lr * (m_ref / (1 - b1 ** step)) / ((v_ref / (1 - b2 ** step)).sqrt() + eps)
        ext.adamw_step(p32, gs, m, v, mask, hp)
        ext.adamw8_step(p8, gs, m8, v8, ms, vs, mask, hp)
    assert _rel_err(p32, p_ref) < 1e-5
    # 8-bit state: updates stay close to the fp32-state trajectory
    assert _rel_err(p8 - p, p_ref - p) < 0.1
    # bf16 params / grads variant
    pb = p.bfloat16()
    ext.adamw_step(pb, g.bfloat16(), torch.zeros(n, device=DEV), torch.zeros(n, device=DEV), None,
                   torch.tensor([lr, b1, b2, eps, 0.0, 1 - b1, 1 - b2, 1.0], device=DEV))
    assert torch.isfinite(pb.float()).all()


def test_adamw_8bit_kernel_matches_the_pytorch_twin_code_for_code(ext):
    """Three steps of the 8-bit kernel against the PyTorch statement of the same state encoding (optim/adamw.py): the parameters
    agree to fp32 rounding of the approximated divisions, the int8 / uint8 codes are equal except for values that sit on a rounding
    boundary (off by one at most), the fp16 group scales are equal or one fp16 step apart."""
    from surogate_b200.optim.adamw import _softsign_dequant_reference, _softsign_quant_reference

    torch.manual_seed(3)
    n = 32 * 4096
    lr, b1, b2, eps, wd = 3e-3, 0.9, 0.95, 1e-8, 0.1
    for pdt, gdt in ((torch.float32, torch.float32), (torch.bfloat16, torch.bfloat16)):
        p = torch.randn(n, device=DEV).to(pdt)
        blocks = (torch.arange(n // 128, device=DEV) % 2 == 0).to(torch.uint8)
        mask = blocks.repeat_interleave(128).float()
        m8, v8 = torch.zeros(n, dtype=torch.int8, device=DEV), torch.zeros(n, dtype=torch.uint8, device=DEV)
        ms, vs = torch.zeros(n // 32, dtype=torch.float16, device=DEV), torch.zeros(n // 32, dtype=torch.float16, device=DEV)
        rm8, rv8, rms, rvs, rp = m8.clone(), v8.clone(), ms.clone(), vs.clone(), p.clone()
        for step in range(1, 4):
            g = (torch.randn(n, device=DEV) * 0.05 * torch.rand(n, device=DEV).pow(4)).to(gdt)
            bc1, bc2 = 1 - b1 ** step, 1 - b2 ** step
            hp = torch.tensor([lr, b1, b2, eps, wd, bc1, bc2, 0.7], device=DEV)
            ext.adamw8_step(p, g, m8, v8, ms, vs, blocks, hp)
            m, v = _softsign_dequant_reference(rm8, rv8, rms, rvs)
            gf = g.float() * 0.7
            m = b1 * m + (1 - b1) * gf
            v = b2 * v + (1 - b2) * gf * gf
            pn = rp.float() * (1 - lr * wd * mask) - lr * (m / bc1) / ((v / bc2).sqrt() + eps)
            upd_ref, upd = pn - rp.float(), p.float() - rp.float()
            rp = pn.to(pdt)
            rm8, rv8, rms, rvs = _softsign_quant_reference(m, v)
            if pdt == torch.float32:
                assert _rel_err(upd, upd_ref) < 2e-3, (step, _rel_err(upd, upd_ref))
            else:
                assert (p.float() - rp.float()).abs().max() <= 2 * 2 ** -7 * rp.float().abs().max()
            dm = (m8.int() - rm8.int()).abs()
            dv = (v8.int() - rv8.int()).abs()
            assert int(dm.max()) <= 1 and int(dv.max()) <= 1, (int(dm.max()), int(dv.max()))
            assert float((dm > 0).float().mean()) < 0.03 and float((dv > 0).float().mean()) < 0.03
            assert float((ms.float() - rms.float()).abs().max() / rms.float().abs().max()) < 2e-3
            # the next step starts from the kernel's own state on both sides, so differences do not accumulate
            rm8, rv8, rms, rvs, rp = m8.clone(), v8.clone(), ms.clone(), vs.clone(), p.clone()
    _check_flag()


# ----------------------------------------------------------------------------- MoE
@pytest.mark.parametrize("n", [32, 2048, 2080, 148 * 3 * 256 * 8 + 32, 148 * 3 * 256 * 8 * 5 + 160])
@pytest.mark.parametrize("pdt,gdt", [(torch.bfloat16, torch.bfloat16), (torch.float32, torch.float32), (torch.float32, torch.bfloat16)])
def test_adamw_8bit_counts(ext, n, pdt, gdt):
    """Counts from part of a warp to several trips around the shared-memory ring: every element is updated once, as when the same values
    are stepped in pieces of 32 (groups of 32 share a scale, so the pieces do not interact)."""
    torch.manual_seed(n % 997)
    hp = torch.tensor([1e-2, 0.9, 0.99, 1e-8, 0.1, 0.1, 0.01, 0.5], device=DEV)
    p, g = torch.randn(n, device=DEV).to(pdt), torch.randn(n, device=DEV).to(gdt)

    def state(k):
        return [torch.zeros(k, dtype=torch.int8, device=DEV), torch.zeros(k, dtype=torch.uint8, device=DEV),
                torch.zeros(k // 32, dtype=torch.float16, device=DEV), torch.zeros(k // 32, dtype=torch.float16, device=DEV)]

    full, st = p.clone(), state(n)
    for _ in range(2):
        ext.adamw8_step(full, g, *st, None, hp)
    for lo in sorted({0, n // 64 * 32, n - 32}):
        part, ps = p[lo:lo + 32].clone(), state(32)
        for _ in range(2):
            ext.adamw8_step(part, g[lo:lo + 32].clone(), *ps, None, hp)
        assert torch.equal(full[lo:lo + 32], part) and torch.equal(st[0][lo:lo + 32], ps[0]) and torch.equal(st[3][lo // 32:lo // 32 + 1], ps[3])
    assert not torch.equal(full, p) and (full != p).float().mean().item() > 0.9


def test_moe_softmax_topk(ext):
    tokens, E, K = 1000, 128, 8
    logits = torch.randn(tokens, E, device=DEV)
    counts = torch.zeros(E, dtype=torch.int32, device=DEV)
    psum = torch.zeros(E, device=DEV)
    lse = torch.zeros(1, device=DEV)
    w, idx, probs = ext.moe_softmax_topk(logits, K, True, counts, psum, lse, True)
    ref_p = torch.softmax(logits, -1)
    rw, ri = torch.topk(ref_p, K, -1)
    assert torch.equal(idx.long(), ri)
    assert torch.allclose(w, rw / rw.sum(-1, keepdim=True), rtol=1e-4, atol=1e-6)
    assert torch.allclose(probs, ref_p, rtol=1e-4, atol=1e-7)
    assert torch.equal(counts.long(), torch.bincount(ri.reshape(-1), minlength=E))
    assert torch.allclose(psum, ref_p.sum(0), rtol=1e-3)
    assert abs(lse.item() - torch.logsumexp(logits, -1).pow(2).sum().item()) < 1e-2 * lse.item()


@pytest.mark.parametrize("E,K,renorm,z", [(128, 8, True, 0.0), (16, 4, False, 1e-3), (60, 2, True, 1e-3), (256, 8, True, 0.0)])
def test_moe_router_backward_kernel(ext, E, K, renorm, z):
    """The fused router-backward kernel against the same formulas written with PyTorch ops in fp32."""
    torch.manual_seed(E + K)
    N, aux_coef = 777, 1e-2
    logits = (torch.randn(N, E, device=DEV) * 2).contiguous()
    probs = torch.softmax(logits, -1)
    ti = torch.topk(probs, K, -1).indices.to(torch.int32).contiguous()
    g = torch.randn(N, K, device=DEV)
    counts = torch.bincount(ti.reshape(-1).long(), minlength=E).to(torch.int32)
    da = torch.tensor([0.37], device=DEV)
    dl = ext.moe_router_bwd(logits, ti, g, counts, da, renorm, aux_coef, z)
    til = ti.long()
    sel = probs.gather(1, til)
    if renorm:
        S = sel.sum(-1, keepdim=True)
        d_sel = g / S - (g * sel).sum(-1, keepdim=True) / (S * S)
    else:
        d_sel = g
    d_probs = torch.zeros_like(probs).scatter_add_(1, til, d_sel) + da * aux_coef * E * (counts.float() / N) / N
    ref = probs * (d_probs - (d_probs * probs).sum(-1, keepdim=True))
    ref = ref + da * z * 2 * torch.logsumexp(logits, -1, keepdim=True) / N * probs
    assert _rel_err(dl, ref) < 6e-3, _rel_err(dl, ref)
    # without the auxiliary term and without top-k gradients the pieces are independent
    dl2 = ext.moe_router_bwd(logits, ti, g, None, None, renorm, aux_coef, z)
    ref2 = probs * (torch.zeros_like(probs).scatter_add_(1, til, d_sel) - (torch.zeros_like(probs).scatter_add_(1, til, d_sel) * probs).sum(-1, keepdim=True))
    assert _rel_err(dl2, ref2) < 6e-3
    _check_flag()


def test_moe_permute_grouped_gemm_unpermute(ext):
    torch.manual_seed(0)
    tokens, C, E, K, Nout = 700, 256, 16, 4, 384
    x = torch.randn(tokens, C, device=DEV).bfloat16()
    ti = torch.stack([torch.randperm(E, device=DEV)[:K] for _ in range(tokens)]).to(torch.int32)
    ti[:, 0] = torch.where(ti[:, 0] == 5, (ti[:, 0] + 1) % E, ti[:, 0])  # leave expert 5 under-used
    counts = torch.bincount(ti.reshape(-1).long(), minlength=E).to(torch.int32)
    cap = tokens * K + E * 128
    offsets = torch.empty(E + 1, dtype=torch.int32, device=DEV)
    cursors = torch.empty(E, dtype=torch.int32, device=DEV)
    err = ext.error_flag_tensor()
    ext.moe_offsets(counts, offsets, cursors, cap, err)
    ref_off = torch.cat([torch.zeros(1, device=DEV), torch.cumsum((counts + 127) // 128 * 128, 0)]).int()
    assert torch.equal(offsets, ref_off)
    row_map = torch.empty(tokens * K, dtype=torch.int32, device=DEV)
    xp = torch.zeros(cap, C, dtype=torch.bfloat16, device=DEV)
    ext.moe_permute(x, ti, offsets, cursors, row_map, xp, 0, E)
    rm = row_map.view(tokens, K).long()
    assert torch.equal(xp[rm.reshape(-1)], x.repeat_interleave(K, 0))
    e_of_row = torch.bucketize(rm, offsets[1:].long(), right=True)
    assert torch.equal(e_of_row, ti.long())
    assert len(torch.unique(rm)) == tokens * K
    # grouped forward
    w = torch.randn(E, Nout, C, device=DEV).bfloat16() * 0.1
    y = torch.zeros(cap, Nout, dtype=torch.bfloat16, device=DEV)
    ext.gemm_grouped(xp, w, y, offsets, 1, False, False, 1.0, None, None, err)
    ref_y = torch.einsum("rc,rnc->rn", x.repeat_interleave(K, 0).float(), w[ti.reshape(-1).long()].float())
    assert _rel_err(y[rm.reshape(-1)], ref_y) < 6e-3
    # grouped dgrad: dy [R, Nout] . W[g]
    dy = torch.zeros(cap, Nout, dtype=torch.bfloat16, device=DEV)
    dy_rows = torch.randn(tokens * K, Nout, device=DEV).bfloat16()
    dy[rm.reshape(-1)] = dy_rows
    dx = torch.zeros(cap, C, dtype=torch.bfloat16, device=DEV)
    ext.gemm_grouped(dy, w, dx, offsets, 1, True, False, 1.0, None, None, err)
    ref_dx = torch.einsum("rn,rnc->rc", dy_rows.float(), w[ti.reshape(-1).long()].float())
    assert _rel_err(dx[rm.reshape(-1)], ref_dx) < 6e-3
    # grouped wgrad: dW[g] = dy_g^T x_g
    dw = torch.zeros(E, Nout, C, dtype=torch.float32, device=DEV)
    ext.gemm_grouped(dy, xp, dw, offsets, 2, True, True, 1.0, None, None, err)
    ref_dw = torch.zeros_like(dw)
    ref_dw.index_add_(0, ti.reshape(-1).long(), torch.einsum("rn,rc->rnc", dy_rows.float(), x.repeat_interleave(K, 0).float()))
    assert _rel_err(dw, ref_dw) < 6e-3
    # weighted combine + backward
    tw = torch.rand(tokens, K, device=DEV)
    out = ext.moe_unpermute(y, tw, row_map, tokens, K)
    ref_out = (y[rm].float() * tw[..., None]).sum(1)
    assert _rel_err(out, ref_out) < 5e-3
    dout = torch.randn(tokens, Nout, device=DEV).bfloat16()
    d_yp, d_tw = ext.moe_unpermute_bwd(dout, y, tw, row_map)
    assert _rel_err(d_yp[rm.reshape(-1)], (dout.float()[:, None] * tw[..., None]).reshape(-1, Nout)) < 5e-3
    assert _rel_err(d_tw, (y[rm].float() * dout.float()[:, None]).sum(-1)) < 5e-3
    _check_flag()


@pytest.mark.parametrize("E,cap,C,pads", [(1, 128, 8, True), (8, 4096, 64, True), (128, 40000, 24, True), (8, 2048, 256, False), (4, 512, 16, True)])
def test_moe_zero_rows(ext, E, cap, C, pads):
    """Exactly the rows that no token owns are cleared: the padding of each group (with counts) and the tail; empty groups, full groups and a
    buffer with no tail."""
    g = torch.Generator().manual_seed(E + cap)
    counts = torch.randint(0, 400, (E,), generator=g)
    counts[0] = 128
    if E > 2:
        counts[2] = 0
    if E == 4:
        counts[:] = 128
    padded = (counts + 127) // 128 * 128
    offsets = torch.cat([torch.zeros(1, dtype=torch.long), padded.cumsum(0)])
    cap = max(cap, int(offsets[-1])) if E != 4 else int(offsets[-1])
    buf = torch.full((cap, C), 7.0, device=DEV, dtype=torch.bfloat16)
    ext.moe_zero_rows(buf, offsets.int().to(DEV), counts.int().to(DEV) if pads else None)
    want = torch.full((cap, C), 7.0)
    want[int(offsets[-1]):] = 0
    if pads:
        for e in range(E):
            want[int(offsets[e] + counts[e]):int(offsets[e + 1])] = 0
    assert torch.equal(buf.float().cpu(), want)


def test_moe_buffers_start_unwritten(ext):
    """The expert buffers of a training step are not cleared as a whole: every row is written by the permutation, the grouped GEMM, the
    un-permutation's backward or the clear of the rows without a token.  With NaN in all of them beforehand (and in the block that the
    allocator hands out again), no NaN is left, rows without a token are zero, and the weight gradient, which contracts over them, is right."""
    torch.manual_seed(1)
    tokens, C, E, K, Nout = 500, 256, 16, 4, 384
    nan = float("nan")
    x = torch.randn(tokens, C, device=DEV).bfloat16()
    ti = torch.stack([torch.randperm(E - 1, device=DEV)[:K] for _ in range(tokens)]).to(torch.int32)      # the last expert gets nothing
    counts = torch.bincount(ti.reshape(-1).long(), minlength=E).to(torch.int32)
    cap = tokens * K + E * 128
    offsets, cursors = torch.empty(E + 1, dtype=torch.int32, device=DEV), torch.empty(E, dtype=torch.int32, device=DEV)
    err = ext.error_flag_tensor()
    ext.moe_offsets(counts, offsets, cursors, cap, err)
    xp = torch.full((cap, C), nan, dtype=torch.bfloat16, device=DEV)
    ext.moe_zero_rows(xp, offsets, counts)
    row_map = torch.empty(tokens * K, dtype=torch.int32, device=DEV)
    ext.moe_permute(x, ti, offsets, cursors, row_map, xp, 0, E)
    empty = torch.ones(cap, dtype=torch.bool, device=DEV)
    empty[row_map.long()] = False
    assert not xp[empty].any() and torch.equal(xp[row_map.long()], x.repeat_interleave(K, 0))
    w = torch.randn(E, Nout, C, device=DEV).bfloat16() * 0.1
    y = torch.full((cap, Nout), nan, dtype=torch.bfloat16, device=DEV)
    ext.moe_zero_rows(y, offsets)
    ext.gemm_grouped(xp, w, y, offsets, 1, False, False, 1.0, None, None, err)
    ref_y = torch.einsum("rc,rnc->rn", x.repeat_interleave(K, 0).float(), w[ti.reshape(-1).long()].float())
    assert not y[empty].any() and _rel_err(y[row_map.long()], ref_y) < 6e-3
    tw, dout = torch.rand(tokens, K, device=DEV), torch.randn(tokens, Nout, device=DEV).bfloat16()
    torch.full((cap, Nout), nan, dtype=torch.bfloat16, device=DEV)           # freed at once
    d_yp, d_tw = ext.moe_unpermute_bwd(dout, y, tw, row_map, offsets, counts)
    want_d, want_w = ext.moe_unpermute_bwd(dout, y, tw, row_map)
    assert torch.equal(d_yp, want_d) and torch.equal(d_tw, want_w) and not d_yp[empty].any()
    dx = torch.full((cap, C), nan, dtype=torch.bfloat16, device=DEV)
    ext.moe_zero_rows(dx, offsets)
    ext.gemm_grouped(d_yp, w, dx, offsets, 1, True, False, 1.0, None, None, err)
    assert not dx[empty].any() and not dx.isnan().any()
    dw = torch.zeros(E, Nout, C, dtype=torch.float32, device=DEV)
    ext.gemm_grouped(d_yp, xp, dw, offsets, 2, True, True, 1.0, None, None, err)
    ref_dw = torch.zeros_like(dw)
    ref_dw.index_add_(0, ti.reshape(-1).long(), torch.einsum("rn,rc->rnc", d_yp[row_map.long()].float(), x.repeat_interleave(K, 0).float()))
    assert _rel_err(dw, ref_dw) < 6e-3
    _check_flag()


def test_embedding_rejects_out_of_range_token_ids():
    """An invalid token id must not read outside the table: the row is zero-filled and the error flag is raised."""
    from surogate_b200.ops import check_device_errors, ext

    e = ext()
    check_device_errors()
    table = torch.randn(64, 128, device="cuda", dtype=torch.bfloat16)
    tok = torch.tensor([[3, -100, 63, 64]], device="cuda", dtype=torch.int32)
    out = e.embedding_fwd(tok, table)
    assert torch.equal(out[0, 0], table[3]) and torch.equal(out[0, 2], table[63])
    assert out[0, 1].abs().sum() == 0 and out[0, 3].abs().sum() == 0
    with pytest.raises(RuntimeError, match="token id"):
        check_device_errors()
    check_device_errors()  # the flag was reset by the failed check


def test_cross_entropy_row_weights_and_topk_distillation():
    """The CE kernel's per-row weights (DPO / GRPO) and top-K KD term against an fp32 autograd reference."""
    from surogate_b200.ops import ext

    e = ext()
    torch.manual_seed(0)
    rows, V, K = 48, 4096, 16
    logits = (torch.randn(rows, V, device="cuda") * 3).bfloat16()
    tgt = torch.randint(0, V, (rows,), device="cuda", dtype=torch.int32)
    tgt[5] = -100
    rw = torch.randn(rows, device="cuda")
    teacher = torch.log_softmax(torch.randn(rows, V, device="cuda") * 2, -1)
    kl, ki = teacher.topk(K, -1)
    scale = torch.tensor([0.5], device="cuda")
    ref = logits.float().clone().requires_grad_(True)
    lp = torch.log_softmax(ref, -1)
    valid = (tgt >= 0).float()
    ce = -lp.gather(1, tgt.clamp_min(0).long()[:, None]).squeeze(1) * valid
    kd = (kl.exp() * (kl - lp.gather(1, ki))).sum(1) * valid
    (0.5 * ((ce * rw).sum() + 0.25 * kd.sum())).backward()
    work = logits.clone()
    kd_out = torch.empty(rows, device="cuda")
    loss = e.cross_entropy_fwd_bwd(work, tgt, scale, 1.0, True, rw, ki.to(torch.int32).contiguous(), kl.contiguous(), 0.25, kd_out)
    torch.testing.assert_close(loss, ce.detach(), rtol=2e-3, atol=2e-3)
    torch.testing.assert_close(kd_out, kd.detach(), rtol=5e-3, atol=5e-3)
    err = (work.float() - ref.grad).abs().max().item()
    assert err < 2e-2 * ref.grad.abs().max().item() + 1e-3, err
    assert work[5].abs().sum() == 0


def test_barrier_wait_runs_out_and_reports_instead_of_hanging():
    """A peer that never arrives: the barrier kernel gives up after its cycle budget, raises the error word and returns; the
    context stays usable.  (Two local signal pads stand in for two ranks; nothing ever writes the absent rank's arrival.)"""
    from surogate_b200.ops import check_device_errors, ext

    e = ext()
    check_device_errors()
    pads = [torch.zeros(64, dtype=torch.int32, device="cuda") for _ in range(2)]
    err = e.error_flag_tensor()
    t0 = time.time()
    e.symm_barrier([p.data_ptr() for p in pads], 0, 1, 0, err, 0.05)   # I am rank 0 of 2; rank 1 never signals
    torch.cuda.synchronize()
    assert time.time() - t0 < 5.0
    with pytest.raises(RuntimeError, match="wait timed out|error flag"):
        check_device_errors()
    x = torch.ones(8, device="cuda")
    assert float((x * 2).sum()) == 16.0  # the context survived
    check_device_errors()


@pytest.mark.parametrize("dtype,K,silu,packed", [(torch.bfloat16, 4, True, False), (torch.float32, 3, False, False), (torch.float32, 4, True, True),
                                                  (torch.bfloat16, 2, False, True)])
def test_causal_conv1d_forward_and_backward(ext, dtype, K, silu, packed):
    """Depth-wise causal convolution kernels against the PyTorch statement in fp32: tiles that need a halo (T > 64), a channel count that
    is not a multiple of the block, packed documents, the activation folded into backward."""
    from surogate_b200.ops.conv1d import causal_conv1d, causal_conv1d_reference

    torch.manual_seed(1)
    B, T, C = 3, 150, 264
    x = torch.randn(B, T, C, device=DEV).to(dtype).requires_grad_(True)
    w = (torch.randn(C, K, device=DEV) * 0.5).requires_grad_(True)
    b = torch.randn(C, device=DEV).requires_grad_(True)
    ids = None
    if packed:
        ids = torch.zeros(B, T, dtype=torch.int32, device=DEV)
        ids[:, 63:] = 1          # boundaries next to and inside tile edges
        ids[:, 64:] = 2
        ids[:, 130:] = 3
    y = causal_conv1d(x, w, b, "silu" if silu else None, ids)
    dy = torch.randn_like(y)
    y.backward(dy)
    got = (y.detach(), x.grad.clone(), w.grad.clone(), b.grad.clone())
    xr, wr, br = x.detach().float().requires_grad_(True), w.detach().clone().requires_grad_(True), b.detach().clone().requires_grad_(True)
    yr = causal_conv1d_reference(xr, wr, br, "silu" if silu else None, ids)
    yr.backward(dy.float())
    tol = 2e-2 if dtype == torch.bfloat16 else 1e-4
    for name, a, r in zip(("y", "dx", "dw", "db"), got, (yr.detach(), xr.grad, wr.grad, br.grad)):
        assert _rel_err(a, r) < tol, (name, _rel_err(a, r))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_runtime_compiled_elementwise_ops(dtype):
    """Kernels compiled at run time (nvcc -> cubin -> driver API) against their PyTorch statements, forward and backward, and through
    the model-family functions that use them."""
    from surogate_b200.ops import jit
    from surogate_b200.runtime import torch_fns

    torch.manual_seed(0)
    tol = 2e-2 if dtype == torch.bfloat16 else 2e-5
    x = torch.randn(3, 1000, 264, device=DEV).to(dtype)
    for op, ref, kw in ((jit.RELU2, jit._relu2_ref, {}), (jit.SOFTCAP, jit._softcap_ref, {"cap": 2.5})):
        a = x.clone().requires_grad_(True)
        b = x.clone().float().requires_grad_(True)
        y, yr = op(a, **kw), ref(b, **kw)
        dy = torch.randn_like(y)
        y.backward(dy)
        yr.backward(dy.float())
        assert _rel_err(y.detach(), yr.detach()) < tol and _rel_err(a.grad, b.grad) < tol, op.name
    g, u = torch.randn(2, 500, 512, device=DEV).to(dtype), torch.randn(2, 500, 512, device=DEV).to(dtype)
    ga, ua = g.clone().requires_grad_(True), u.clone().requires_grad_(True)
    gb, ub = g.clone().float().requires_grad_(True), u.clone().float().requires_grad_(True)
    y, yr = jit.GEGLU_TANH(ga, ua), jit._geglu_ref(gb, ub)
    dy = torch.randn_like(y)
    y.backward(dy)
    yr.backward(dy.float())
    assert _rel_err(y.detach(), yr.detach()) < tol and _rel_err(ga.grad, gb.grad) < tol and _rel_err(ua.grad, ub.grad) < tol
    packed = torch.cat([u, g], -1)            # [up | gate]
    assert _rel_err(torch_fns.geglu(packed), yr.detach()) < tol
    odd = torch.randn(7, 3, device=DEV).to(dtype)      # not a multiple of the vector width: the PyTorch statement answers
    assert torch.equal(torch_fns.relu2(odd), torch.relu(odd) ** 2)
