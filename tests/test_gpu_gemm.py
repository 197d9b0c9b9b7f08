"""GPU parity tests of the tcgen05 FP8 GEMMs (dense and grouped) against the CPU oracle and the
fixtures generated by the reference's Triton kernels."""
import pytest
import torch

from oracle import moe_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda"
FP8 = torch.float8_e4m3fn


def _status_ok():
    from dlblas_b200 import _C
    _C.check_status()


def test_fp8_gemm_golden(golden):
    from dlblas_b200 import ops
    g = golden("fp8_gemm.pt")
    c = ops.fp8_gemm(g["a"].to(DEV), g["b"].to(DEV), g["a_s"].to(DEV), g["b_s"].to(DEV), torch.float32)
    _status_ok()
    torch.testing.assert_close(c.cpu(), g["c_fp32"], rtol=1e-4, atol=2e-3)


def test_fp8_gemm_reference_test_case():
    """tests/kernels/test_fp8_gemm.py of the reference: 512^3, random (also negative) scales,
    output in the default dtype, atol 1e-1."""
    from dlblas_b200.kernels.fp8_gemm import fp8_gemm
    g = torch.Generator().manual_seed(0)
    a = torch.randn(512, 512, generator=g).to(FP8)
    b = torch.randn(512, 512, generator=g).to(FP8)
    a_s = torch.randn(512, 4, generator=g)
    b_s = torch.randn(4, 4, generator=g)
    out = fp8_gemm(a.to(DEV), b.to(DEV), a_s.to(DEV), b_s.to(DEV))
    _status_ok()
    assert out.dtype == torch.get_default_dtype()
    torch.testing.assert_close(out.cpu(), O.fp8_gemm(a, b, a_s, b_s, torch.float32), atol=1e-1, rtol=0)
    old = torch.get_default_dtype()
    torch.set_default_dtype(torch.bfloat16)
    try:
        out = fp8_gemm(a.to(DEV), b.to(DEV), a_s.to(DEV), b_s.to(DEV))
    finally:
        torch.set_default_dtype(old)
    assert out.dtype == torch.bfloat16
    assert O.rel_frobenius(out.cpu(), O.fp8_gemm(a, b, a_s, b_s, torch.float32)) < 4e-3


@pytest.mark.parametrize("m,n,k", [(1, 128, 128), (7, 256, 256), (128, 128, 512), (129, 384, 384), (300, 1024, 1024),
                                   (1000, 2048, 512), (4096, 512, 256), (64, 24, 128), (257, 4096, 7168)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_fp8_gemm_shapes(m, n, k, dtype):
    from dlblas_b200 import ops
    if dtype == torch.float32 and k > 2048:
        pytest.skip("covered by the bf16 case")
    g = torch.Generator().manual_seed(m * 7 + n + k)
    a, a_s = O.quant_fp8(torch.randn(m, k, generator=g).to(torch.bfloat16), 128)
    b = torch.randn(n, k, generator=g).to(FP8)
    b_s = torch.rand((n + 127) // 128, k // 128, generator=g) + 0.5
    c = ops.fp8_gemm(a.to(DEV), b.to(DEV), a_s.to(DEV), b_s.to(DEV), dtype)
    _status_ok()
    ref = O.fp8_gemm(a, b, a_s, b_s, torch.float32)
    assert c.shape == (m, n) and c.dtype == dtype
    tol = 1e-5 if dtype == torch.float32 else 4e-3
    assert O.rel_frobenius(c.cpu(), ref) < tol
    if dtype == torch.float32:
        torch.testing.assert_close(c.cpu(), ref, rtol=1e-4, atol=1e-3 * float(ref.abs().max()))


def test_fp8_gemm_leading_dims_and_empty():
    from dlblas_b200 import ops
    g = torch.Generator().manual_seed(1)
    a = torch.randn(3, 5, 256, generator=g).to(FP8)
    b = torch.randn(128, 256, generator=g).to(FP8)
    a_s = torch.rand(3, 5, 2, generator=g)
    b_s = torch.rand(1, 2, generator=g)
    c = ops.fp8_gemm(a.to(DEV), b.to(DEV), a_s.to(DEV), b_s.to(DEV))
    _status_ok()
    assert c.shape == (3, 5, 128)
    assert O.rel_frobenius(c.cpu(), O.fp8_gemm(a, b, a_s, b_s, torch.float32)) < 4e-3
    c = ops.fp8_gemm(a[:0].to(DEV), b.to(DEV), a_s[:0].to(DEV), b_s.to(DEV))
    assert c.shape == (0, 5, 128)
    with pytest.raises(AssertionError):
        ops.fp8_gemm(a[..., :100].contiguous().to(DEV), b[:, :100].contiguous().to(DEV), a_s.to(DEV), b_s.to(DEV))


def test_fp8_gemm_linearity_at_full_size():
    """Config-2 sized problem (M 4096, N 7168, K 2048): rows checked against the oracle, plus
    the scale-linearity property C(2 a_s) == 2 C(a_s) exactly."""
    from dlblas_b200 import ops
    g = torch.Generator().manual_seed(2)
    m, n, k = 4096, 7168, 2048
    a, a_s = O.quant_fp8(torch.randn(m, k, generator=g).to(torch.bfloat16), 128)
    b = torch.randn(n, k, generator=g).to(FP8)
    b_s = torch.rand(n // 128, k // 128, generator=g) + 0.5
    ad, bd, asd, bsd = a.to(DEV), b.to(DEV), a_s.to(DEV), b_s.to(DEV)
    c = ops.fp8_gemm(ad, bd, asd, bsd, torch.float32)
    c2 = ops.fp8_gemm(ad, bd, asd * 2, bsd, torch.float32)
    _status_ok()
    assert torch.equal(c2, c * 2)
    rows = torch.tensor([0, 1, 127, 128, 2047, 4095])
    ref = O.fp8_gemm(a[rows], b, a_s[rows], b_s, torch.float32)
    assert O.rel_frobenius(c.cpu()[rows], ref) < 1e-5
    cb = ops.fp8_gemm(ad, bd, asd, bsd, torch.bfloat16)
    assert torch.equal(cb, c.to(torch.bfloat16))          # one rounding, at the very end


def test_grouped_gemm_golden(golden):
    from dlblas_b200.layers.moe.kernels.blocked_fp8_fused_moe import fused_moe_blocked_fp8_kernel_launcher
    g = golden("grouped_gemm.pt")
    d = {k_: (v.to(DEV) if torch.is_tensor(v) else v) for k_, v in g.items()}
    t, k = g["ids"].shape
    c1 = torch.zeros(t * k, g["w"].shape[1], dtype=torch.float32, device=DEV)
    fused_moe_blocked_fp8_kernel_launcher(d["xq"], d["xs"], d["w"], d["ws"], c1, d["sorted_idx"], d["exp_start"],
                                          d["exp_end"], d["wts"], enable_weights=False, top_k=k, num_tokens=t,
                                          reindex_a=True, reindex_c=False)
    _status_ok()
    torch.testing.assert_close(c1.cpu(), g["c1_fp32"], rtol=1e-4, atol=2e-3)
    c2 = torch.zeros(t * k, g["w"].shape[1], dtype=torch.float32, device=DEV)
    fused_moe_blocked_fp8_kernel_launcher(d["aq"], d["as_"], d["w"], d["ws"], c2, d["sorted_idx"], d["exp_start"],
                                          d["exp_end"], d["wts"], enable_weights=True, top_k=1, num_tokens=t,
                                          reindex_a=False, reindex_c=True)
    _status_ok()
    torch.testing.assert_close(c2.cpu(), g["c2_fp32"], rtol=1e-4, atol=2e-3)


@pytest.mark.parametrize("t,k,e,h,n", [(64, 2, 8, 512, 2048), (500, 4, 16, 256, 512), (3000, 8, 64, 1024, 768)])
def test_grouped_gemm_random(t, k, e, h, n):
    from dlblas_b200 import _C, ops
    g = torch.Generator().manual_seed(t)
    ids = torch.stack([torch.randperm(e, generator=g)[:k] for _ in range(t)])
    ids[ids == 1] = 0                                              # an empty expert, a crowded one
    xq, xs = O.quant_fp8(torch.randn(t, h, generator=g).to(torch.bfloat16), 128)
    w = torch.randn(e, n, h, generator=g).to(FP8)
    ws = torch.rand(e, n // 128, h // 128, generator=g) + 0.5
    wts = torch.rand(t, k, generator=g)
    sidx, st, en, pos = ops.sort_by_expert(ids.to(DEV), e, want_pos=True)
    mt = ops.max_tiles_for(t * k, e)
    tiles = ops.build_tiles(st, en, 0, e, mt)
    a, a_s = ops.permute_rows(xq.to(DEV), xs.to(DEV), pos, k, t * k)
    c1 = torch.zeros(t * k, n, dtype=torch.bfloat16, device=DEV)
    ops.grouped_gemm(a, a_s, w.to(DEV), ws.to(DEV), tiles, mt, _C.EPI_STORE, c1)
    _status_ok()
    o_sidx, o_st, o_en = O.stable_sort_by_expert(ids, e)
    ref1 = O.grouped_gemm(xq, xs, w, ws, o_sidx, o_st, o_en, None, top_k=k, reindex_a=True, reindex_c=False,
                          out_dtype=torch.float32)
    assert O.rel_frobenius(c1.cpu(), ref1) < 4e-3
    c2 = torch.zeros(t * k, n, dtype=torch.bfloat16, device=DEV)
    ops.grouped_gemm(a, a_s, w.to(DEV), ws.to(DEV), tiles, mt, _C.EPI_SCATTER_WEIGHT, c2, sorted_idx=sidx,
                     weights=wts.to(DEV))
    _status_ok()
    ref2 = O.grouped_gemm(a.cpu(), a_s.cpu(), w, ws, o_sidx, o_st, o_en, wts, top_k=1, reindex_a=False, reindex_c=True,
                          out_dtype=torch.float32)
    assert O.rel_frobenius(c2.cpu(), ref2) < 4e-3


def test_grouped_gemm_swiglu_epilogue_matches_unfused():
    from dlblas_b200 import _C, ops
    g = torch.Generator().manual_seed(4)
    t, k, e, h, inter = 700, 4, 16, 512, 768
    ids = torch.stack([torch.randperm(e, generator=g)[:k] for _ in range(t)])
    xq, xs = O.quant_fp8(torch.randn(t, h, generator=g).to(torch.bfloat16), 128)
    w = (torch.randn(e, 2 * inter, h, generator=g) * 0.05)
    wq, wsc = O.quantize_weight_blocks(w)
    sidx, st, en, pos = ops.sort_by_expert(ids.to(DEV), e, want_pos=True)
    mt = ops.max_tiles_for(t * k, e)
    tiles = ops.build_tiles(st, en, 0, e, mt)
    a, a_s = ops.permute_rows(xq.to(DEV), xs.to(DEV), pos, k, t * k)
    c1 = torch.zeros(t * k, 2 * inter, dtype=torch.bfloat16, device=DEV)
    ops.grouped_gemm(a, a_s, wq.to(DEV), wsc.to(DEV), tiles, mt, _C.EPI_STORE, c1)
    for mode in (_C.QUANT_DIV_EPS, _C.QUANT_RECIP_MUL):          # both scale formulas of the reference
        hq = torch.zeros(t * k, inter, dtype=FP8, device=DEV)
        hs = torch.zeros(t * k, inter // 128, dtype=torch.float32, device=DEV)
        ops.grouped_gemm(a, a_s, wq.to(DEV), wsc.to(DEV), tiles, mt, _C.EPI_SWIGLU_QUANT, hq, q_scale=hs,
                         round_dtype=torch.bfloat16, quant_mode=mode, quant_eps=1e-10)
        _status_ok()
        hq2, hs2 = ops.silu_mul_quant(c1, mode, 1e-10)
        _status_ok()
        assert torch.equal(hs, hs2)
        assert torch.equal(hq.view(torch.uint8), hq2.view(torch.uint8))
    # and against the oracle
    o_sidx, o_st, o_en = O.stable_sort_by_expert(ids, e)
    ref1 = O.grouped_gemm(xq, xs, wq, wsc, o_sidx, o_st, o_en, None, top_k=k, reindex_a=True, reindex_c=False,
                          out_dtype=torch.bfloat16)
    oq, os_ = O.quant_fp8(O.silu_and_mul(ref1), 128)
    deq = hq.cpu().float() * hs.cpu().repeat_interleave(128, dim=1)
    assert O.rel_frobenius(deq, oq.float() * os_.repeat_interleave(128, dim=1)) < 1e-2


@pytest.mark.parametrize("rows_per_expert", [20, 90, 300, 1100])
def test_pairs_of_ctas_match_single_cta_tiles(rows_per_expert):
    """256-row tiles on pairs of CTAs (tcgen05 cta_group::2) run the same arithmetic in the same order as
    128-row tiles on single CTAs: every epilogue bit for bit, dense and grouped, ragged segments included."""
    from dlblas_b200 import _C, ops
    g = torch.Generator().manual_seed(rows_per_expert)
    e, k, h, inter = 6, 2, 512, 256
    t = rows_per_expert * e // k
    ids = torch.stack([torch.randperm(e, generator=g)[:k] for _ in range(t)])
    ids[ids == 4] = 3                                              # an empty expert, a crowded one
    xq, xs = O.quant_fp8(torch.randn(t, h, generator=g).to(torch.bfloat16), 128)
    wq, wsc = O.quantize_weight_blocks(torch.randn(e, 2 * inter, h, generator=g) * 0.05)
    w2q, w2s = O.quantize_weight_blocks(torch.randn(e, h, inter, generator=g) * 0.05)
    wts = torch.rand(t, k, generator=g).to(DEV)
    sidx, st, en, pos = ops.sort_by_expert(ids.to(DEV), e, want_pos=True)
    a, a_s = ops.permute_rows(xq.to(DEV), xs.to(DEV), pos, k, t * k)
    wq, wsc, w2q, w2s = wq.to(DEV), wsc.to(DEV), w2q.to(DEV), w2s.to(DEV)
    res = {}
    for rows in (128, 256):
        mt = ops.max_tiles_for(t * k, e, rows)
        tiles = ops.build_tiles(st, en, 0, e, mt, rows)
        c1 = torch.zeros(t * k, 2 * inter, dtype=torch.bfloat16, device=DEV)
        ops.grouped_gemm(a, a_s, wq, wsc, tiles, mt, _C.EPI_STORE, c1, tile_rows=rows)
        hq = torch.zeros(t * k, inter, dtype=FP8, device=DEV)
        hs = torch.zeros(t * k, inter // 128, dtype=torch.float32, device=DEV)
        ops.grouped_gemm(a, a_s, wq, wsc, tiles, mt, _C.EPI_SWIGLU_QUANT, hq, q_scale=hs, round_dtype=torch.bfloat16,
                         tile_rows=rows)
        y = torch.zeros(t * k, h, dtype=torch.bfloat16, device=DEV)
        ops.grouped_gemm(hq, hs, w2q, w2s, tiles, mt, _C.EPI_SCATTER_WEIGHT, y, sorted_idx=sidx, weights=wts.flatten(),
                         tile_rows=rows)
        d = ops.fp8_gemm(a, wq[0], a_s, wsc[0], torch.bfloat16, tile_rows=rows)
        _status_ok()
        res[rows] = (c1, hq.view(torch.uint8), hs, y, d)
    for x128, x256 in zip(res[128], res[256]):
        assert torch.equal(x128, x256)
    # and the single-CTA result is the oracle's
    o_sidx, o_st, o_en = O.stable_sort_by_expert(ids, e)
    ref1 = O.grouped_gemm(xq, xs, wq.cpu(), wsc.cpu(), o_sidx, o_st, o_en, None, top_k=k, reindex_a=True,
                          reindex_c=False, out_dtype=torch.float32)
    assert O.rel_frobenius(res[256][0].cpu(), ref1) < 4e-3


@pytest.mark.parametrize("m", [1, 100, 128, 130, 300])
def test_pairs_of_ctas_with_an_empty_second_half(m):
    """256-row tiles whose second CTA holds no row at all (m <= 128, or a last tile of <= 128 rows): that CTA
    still runs the main loop for its partner and must read nothing beyond the end of A's scales.  The inputs are
    carved so that the scale tensor ends exactly where its allocation ends."""
    from dlblas_b200 import ops
    g = torch.Generator().manual_seed(m)
    n, k = 384, 512
    a = torch.randn(m, k, generator=g).to(FP8)
    b = torch.randn(n, k, generator=g).to(FP8)
    a_s = torch.rand(m, k // 128, generator=g)
    b_s = torch.rand(n // 128, k // 128, generator=g)
    pool = torch.empty(4096 + m * (k // 128), dtype=torch.float32, device=DEV)
    a_s_dev = pool[4096:].view(m, k // 128)
    a_s_dev.copy_(a_s)
    c2 = ops.fp8_gemm(a.to(DEV), b.to(DEV), a_s_dev, b_s.to(DEV), torch.bfloat16, tile_rows=256)
    c1 = ops.fp8_gemm(a.to(DEV), b.to(DEV), a_s_dev, b_s.to(DEV), torch.bfloat16, tile_rows=128)
    _status_ok()
    assert torch.equal(c1, c2)
    assert O.rel_frobenius(c2.cpu(), O.fp8_gemm(a, b, a_s, b_s, out_dtype=torch.float32)) < 4e-3


def test_barrier_waits_run_out_report_and_leave_the_gpu_usable():
    """The time-out path of the GEMM kernels: with the loader switched off nothing ever fills a stage, every
    role's first wait runs into the (shortened) limit, the kernel hands back its tensor memory and returns, the
    status word says so, and the next ordinary launch is correct.  Nothing traps and no wait is unbounded."""
    from dlblas_b200 import _C, ops
    g = torch.Generator().manual_seed(5)
    m, n, k = 300, 512, 1024
    a = torch.randn(m, k, generator=g).to(FP8)
    b = torch.randn(n, k, generator=g).to(FP8)
    a_s = torch.rand(m, k // 128, generator=g)
    b_s = torch.rand(n // 128, k // 128, generator=g)
    dev = [t.to(DEV) for t in (a, b, a_s, b_s)]
    ref = O.fp8_gemm(a, b, a_s, b_s, out_dtype=torch.float32)
    _status_ok()
    _C.set_wait_policy(2_000_000, withhold_loads=True)          # about a millisecond per wait
    try:
        ops.fp8_gemm(dev[0], dev[1], dev[2], dev[3], torch.bfloat16)
        with pytest.raises(RuntimeError, match="gave up waiting"):
            _C.check_status()
        # the grouped kernel with the fused epilogue (its epilogue warps wait on a barrier of their own)
        e, t, h, inter = 2, 64, 512, 256
        xq, xs = O.quant_fp8(torch.randn(t, h, generator=g).to(torch.bfloat16), 128)
        wq, wsc = O.quantize_weight_blocks(torch.randn(e, 2 * inter, h, generator=g) * 0.05)
        ids = torch.randint(0, e, (t, 1), generator=g)
        sidx, st, en, pos = ops.sort_by_expert(ids.to(DEV), e, want_pos=True)
        aq, aqs = ops.permute_rows(xq.to(DEV), xs.to(DEV), pos, 1, t)
        mt = ops.max_tiles_for(t, e)
        tiles = ops.build_tiles(st, en, 0, e, mt)
        hq = torch.zeros(t, inter, dtype=FP8, device=DEV)
        hs = torch.zeros(t, inter // 128, dtype=torch.float32, device=DEV)
        ops.grouped_gemm(aq, aqs, wq.to(DEV), wsc.to(DEV), tiles, mt, _C.EPI_SWIGLU_QUANT, hq, q_scale=hs,
                         round_dtype=torch.bfloat16)
        with pytest.raises(RuntimeError, match="gave up waiting"):
            _C.check_status()
    finally:
        _C.set_wait_policy(0, withhold_loads=False)
    c = ops.fp8_gemm(dev[0], dev[1], dev[2], dev[3], torch.bfloat16)
    _status_ok()
    assert O.rel_frobenius(c.cpu(), ref) < 4e-3


def test_grouped_gemm_over_column_windows_equals_one_launch():
    """Two launches over halves of the output columns, the second on fewer CTAs, write what one launch writes."""
    from dlblas_b200 import _C, ops
    g = torch.Generator().manual_seed(3)
    e, k, n = 6, 512, 1536
    sizes = [130, 0, 257, 64, 5, 300]
    rows = sum(sizes)
    a = torch.randn(rows, k, generator=g).to(FP8).to(DEV)
    a_s = (torch.rand(rows, k // 128, generator=g) + 0.5).to(DEV)
    b = torch.randn(e, n, k, generator=g).to(FP8).to(DEV)
    b_s = (torch.rand(e, n // 128, k // 128, generator=g) + 0.5).to(DEV)
    ends = torch.tensor(sizes, dtype=torch.int64).cumsum(0).to(DEV)
    starts = ends - torch.tensor(sizes, dtype=torch.int64, device=DEV)
    mt = ops.max_tiles_for(rows, e)
    tiles = ops.build_tiles(starts, ends, 0, e, mt)
    whole = torch.empty(rows, n, dtype=torch.bfloat16, device=DEV)
    ops.grouped_gemm(a, a_s, b, b_s, tiles, mt, _C.EPI_STORE, whole)
    halves = torch.zeros(rows, n, dtype=torch.bfloat16, device=DEV)
    ops.grouped_gemm(a, a_s, b, b_s, tiles, mt, _C.EPI_STORE, halves, n_begin=0, n_count=768)
    assert not halves[:, 768:].any()                             # the first launch leaves the other window alone
    ops.grouped_gemm(a, a_s, b, b_s, tiles, mt, _C.EPI_STORE, halves, n_begin=768, n_count=768, sm_margin=16)
    _C.check_status()
    assert torch.equal(whole, halves)
    with pytest.raises(AssertionError):
        ops.grouped_gemm(a, a_s, b, b_s, tiles, mt, _C.EPI_STORE, halves, n_begin=128, n_count=256)


@pytest.mark.parametrize("m,n", [(4096 + 133, 4360), (4096, 4352), (100, 4360), (1, 8192)])
def test_fp8_gemm_tile_bands(m, n):
    """More than 16 tiles of columns: the tiles are walked in bands of 32 tiles of rows, the last band may be lower."""
    from dlblas_b200 import ops
    g = torch.Generator().manual_seed(m + n)
    a, a_s = O.quant_fp8(torch.randn(m, 128, generator=g).to(torch.bfloat16), 128)
    b = torch.randn(n, 128, generator=g).to(FP8)
    b_s = torch.rand((n + 127) // 128, 1, generator=g) + 0.5
    c = ops.fp8_gemm(a.to(DEV), b.to(DEV), a_s.to(DEV), b_s.to(DEV), torch.bfloat16)
    _status_ok()
    assert O.rel_frobenius(c.cpu(), O.fp8_gemm(a, b, a_s, b_s, torch.float32)) < 4e-3   # one rounding to bf16: 2^-8


def test_layer_tile_bands():
    """The same over ragged experts: 18 tiles of columns in the first GEMM, more than 32 tiles of rows."""
    from dlblas_b200.layers.moe.ep_moe import DlblasTritonFusedMoEBlockedF8Impl
    x, logits, w13, w13s, w2, w2s = O.make_layer_inputs(600, 256, 2304, 40, seed=9)
    w, ids = O.softmax_topk(logits, 2, True)
    layer = DlblasTritonFusedMoEBlockedF8Impl(top_k=2, num_experts=40, out_dtype=torch.bfloat16)
    out = layer.forward(*(t.to(DEV) for t in (x, w, ids, w13, w13s, w2, w2s)))
    _status_ok()
    assert O.rel_frobenius(out.cpu(), O.moe_layer(x, w, ids, w13, w13s, w2, w2s, top_k=2)) < 2e-2


@pytest.mark.parametrize("m,n,k", [(100, 7168, 256), (1, 64, 128), (33, 72, 384), (128, 9472, 128), (129, 4736, 128), (97, 136, 1152)])
def test_fp8_gemm_narrow_tiles(m, n, k):
    """Tiles of 64 columns where they make one wave (148 tiles at most), ragged columns."""
    from dlblas_b200 import ops
    g = torch.Generator().manual_seed(m + n)
    a, a_s = O.quant_fp8(torch.randn(m, k, generator=g).to(torch.bfloat16), 128)
    b = torch.randn(n, k, generator=g).to(FP8)
    b_s = torch.rand((n + 127) // 128, k // 128, generator=g) + 0.5
    for dtype in (torch.bfloat16, torch.float16):
        c = ops.fp8_gemm(a.to(DEV), b.to(DEV), a_s.to(DEV), b_s.to(DEV), dtype)
        _status_ok()
        assert O.rel_frobenius(c.cpu(), O.fp8_gemm(a, b, a_s, b_s, torch.float32)) < 4e-3


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("fuse", [True, False])
def test_layer_tiles_of_few_rows(dtype, fuse):
    """At most 32 rows per expert on average.  Segments around the 16-row chunks, the 32-row line and whole tiles, every expert
    with one row, and both sides of the line of the rule.  The first GEMM of the fused layer exchanges the operands of tiles
    of at most 32 rows here; the other launches take narrower tiles, except with 160 experts (for them see
    test_exchanged_operands_give_the_same_bits)."""
    from dlblas_b200.layers.moe.kernels.blocked_fp8_fused_moe import moe_expert_forward
    g = torch.Generator().manual_seed(41)
    for counts in ([1, 0, 15, 16, 17, 31, 32, 33, 49, 63, 64, 65, 127, 128, 129, 192, 193, 0, 2] + [0] * 20, [1] * 160, [32, 32],
                   [32, 33], [0, 5, 0]):
        e, t, h, inter = len(counts), sum(counts), 384, 256
        x, _, w13, w13s, w2, w2s = O.make_layer_inputs(t, h, inter, e, seed=e)
        x = x.to(dtype)
        ids = torch.repeat_interleave(torch.arange(e), torch.tensor(counts))[torch.randperm(t, generator=g)].view(t, 1)
        w = torch.rand(t, 1, generator=g) + 0.5
        out = moe_expert_forward(x.to(DEV), None, None, *(v.to(DEV) for v in (w13, w13s, w2, w2s, w, ids)), 1, dtype,
                                 fuse_swiglu=fuse).cpu()
        _status_ok()
        ref = O.moe_layer(x, w, ids, w13, w13s, w2, w2s, top_k=1)
        for k in range(e):
            rows = ids[:, 0] == k
            if bool(rows.any()):
                assert O.rel_frobenius(out[rows], ref[rows]) < 2e-2, (e, k)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("epilogue", ["store", "scatter", "swiglu"])
def test_exchanged_operands_give_the_same_bits(epilogue, dtype):
    """Enough tiles for 256 columns each (148) and at most 32 rows per expert on average: tiles of at most 32 rows exchange
    the operands, the others between them do not.  Tiles of 256 rows never do, and products and sums keep their order."""
    from dlblas_b200 import _C, ops
    counts = [1, 0, 15, 16, 17, 31, 32, 33, 49, 63, 64, 65, 127, 128, 129, 160, 161, 193, 2] + [0, 5, 30, 24] * 10
    e, rows, k, n = len(counts), sum(counts), 384, 1024 if epilogue == "swiglu" else 1152
    assert rows <= 32 * e and (rows // 128 + e) * -(-n // 256) >= 148
    g = torch.Generator().manual_seed(17)
    a, a_s = O.quant_fp8(torch.randn(rows, k, generator=g).to(torch.bfloat16), 128)
    b = torch.randn(e, n, k, generator=g).to(FP8)
    b_s = torch.rand(e, n // 128, k // 128, generator=g) * 0.01 + 0.01
    a, a_s, b, b_s = (t.to(DEV) for t in (a, a_s, b, b_s))
    ends = torch.tensor(counts, dtype=torch.int64).cumsum(0)
    starts = (ends - torch.tensor(counts)).to(DEV)
    order = torch.randperm(rows, generator=g).to(DEV)
    weights = (torch.rand(rows, generator=g) + 0.5).to(DEV)
    out = []
    for tile_rows in (128, 256):
        mt = ops.max_tiles_for(rows, e, tile_rows)
        tiles = ops.build_tiles(starts, ends.to(DEV), 0, e, mt, tile_rows)
        if epilogue == "swiglu":
            c, s = torch.zeros(rows, n // 2, device=DEV).to(FP8), torch.zeros(rows, n // 256, device=DEV)
            ops.grouped_gemm(a, a_s, b, b_s, tiles, mt, _C.EPI_SWIGLU_QUANT, c, q_scale=s, round_dtype=dtype, tile_rows=tile_rows)
            out.append((c.view(torch.uint8), s))
        else:
            c = torch.zeros(rows, n, dtype=dtype, device=DEV)
            extra = {"sorted_idx": order, "weights": weights} if epilogue == "scatter" else {}
            ops.grouped_gemm(a, a_s, b, b_s, tiles, mt, _C.EPI_SCATTER_WEIGHT if extra else _C.EPI_STORE, c,
                             tile_rows=tile_rows, **extra)
            out.append((c,))
    _status_ok()
    assert all(torch.equal(x, y) for x, y in zip(*out)) and bool(out[0][0].any())


def test_decode_step_of_few_rows_per_expert():
    """128 tokens over 256 experts, skewed: the direct step's GEMMs exchange the operands, those on the masked layout, which a
    replaced step leads to, do not.  Same bits."""
    from dlblas_b200.layers.moe.ep_moe import FusedMoELowLatency
    x, logits, *weights = (t.to(DEV) for t in O.make_layer_inputs(128, 512, 256, 256, seed=12))
    g = torch.Generator().manual_seed(12)
    p = torch.arange(1, 257).float().pow(-1.2)
    ids = torch.stack([torch.multinomial(p, 8, generator=g) for _ in range(128)]).to(DEV)
    w = torch.rand(128, 8, generator=g).to(DEV)
    layer = FusedMoELowLatency(1, None, 256, 512, 0)
    out = layer.forward(x, w, ids, *weights)
    layer.token_dispatcher.dispatch = layer.token_dispatcher.dispatch
    ref = layer.forward(x, w, ids, *weights)
    _status_ok()
    assert torch.equal(out, ref) and bool(out.any())


@pytest.mark.parametrize("k", [128, 256, 384])
@pytest.mark.parametrize("per_sm,extra", [(64, 0), (64, 8), (128, 0), (128, 8), (256, 0), (256, 8)])
def test_fp8_gemm_where_the_tile_width_changes(per_sm, extra, k):
    """One tile per SM of 64, 128 and 256 columns, and one tile more; one, two and three K blocks (the hand-over of the
    accumulators starts and ends differently)."""
    from dlblas_b200 import ops
    m, n = 3, torch.cuda.get_device_properties(DEV).multi_processor_count * per_sm + extra
    g = torch.Generator().manual_seed(per_sm + extra + k)
    a, a_s = O.quant_fp8(torch.randn(m, k, generator=g).to(torch.bfloat16), 128)
    b = torch.randn(n, k, generator=g).to(FP8)
    b_s = torch.rand((n + 127) // 128, k // 128, generator=g) + 0.5
    c = ops.fp8_gemm(a.to(DEV), b.to(DEV), a_s.to(DEV), b_s.to(DEV), torch.float32)
    cb = ops.fp8_gemm(a.to(DEV), b.to(DEV), a_s.to(DEV), b_s.to(DEV), torch.bfloat16)
    _status_ok()
    ref = O.fp8_gemm(a, b, a_s, b_s, torch.float32)
    assert O.rel_frobenius(c.cpu(), ref) < 1e-5
    # the same products in the same order at every width: one rounding apart
    assert torch.equal(cb, c.to(torch.bfloat16))


@pytest.mark.parametrize("kblocks", [1, 4, 7, 8, 9, 17])
@pytest.mark.parametrize("m,n", [(1, 8), (33, 72), (100, 200), (128, 64), (129, 1032)])
def test_narrow_tiles_leave_whole(m, n, kblocks):
    """Tiles of 64 columns, which the promotion warps store themselves: ragged rows and columns, K blocks around the number of
    stages and accumulators (8).  The fp32 output goes another way, through 128 columns and no staging tile."""
    from dlblas_b200 import ops
    k = 128 * kblocks
    g = torch.Generator().manual_seed(m + n + k)
    a, a_s = O.quant_fp8(torch.randn(m, k, generator=g).to(torch.bfloat16), 128)
    b = torch.randn(n, k, generator=g).to(FP8)
    b_s = torch.rand((n + 127) // 128, k // 128, generator=g) + 0.5
    args = (a.to(DEV), b.to(DEV), a_s.to(DEV), b_s.to(DEV))
    c = ops.fp8_gemm(*args, torch.float32)
    assert O.rel_frobenius(c.cpu(), O.fp8_gemm(a, b, a_s, b_s, torch.float32)) < 1e-5
    for dtype in (torch.bfloat16, torch.float16):
        assert torch.equal(ops.fp8_gemm(*args, dtype), c.to(dtype))
    _status_ok()


@pytest.mark.parametrize("m,n,k,tile_rows,dtype", [
    (100, 2048, 2176, 128, torch.bfloat16),      # 64 columns
    (128, 12288, 1152, 128, torch.bfloat16),     # 128
    (1000, 12288, 1152, 128, torch.bfloat16),    # 256, several tiles per CTA
    (1000, 4096, 1152, 128, torch.float32),      # stored by the promotion warps
    (1000, 12288, 1152, 256, torch.bfloat16),    # pairs of CTAs
])
def test_gemm_beside_copies(m, n, k, tile_rows, dtype):
    """A copy on another stream takes memory and SM time, so that the kernel's early questions for its barriers are answered
    now with yes, now with no.  Same bits as alone, every time."""
    from dlblas_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(m + n)
    a, b = (torch.randn(*s, generator=g, device=DEV).to(FP8) for s in ((m, k), (n, k)))
    a_s, b_s = torch.rand(m, k // 128, generator=g, device=DEV), torch.rand((n + 127) // 128, k // 128, generator=g, device=DEV)
    alone = ops.fp8_gemm(a, b, a_s, b_s, dtype, tile_rows=tile_rows)
    assert O.rel_frobenius(alone[:8].float().cpu(), O.fp8_gemm(a[:8].cpu(), b.cpu(), a_s[:8].cpu(), b_s.cpu(),
                                                               torch.float32)) < 4e-3
    src = torch.randn(32 << 20, device=DEV)
    dst, side, out = torch.empty_like(src), torch.cuda.Stream(), []
    torch.cuda.synchronize()
    for _ in range(20):
        with torch.cuda.stream(side):
            dst.copy_(src)
        for _ in range(3):
            out.append(ops.fp8_gemm(a, b, a_s, b_s, dtype, tile_rows=tile_rows))
    torch.cuda.synchronize()
    _status_ok()
    assert all(torch.equal(alone, c) for c in out)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("epilogue", ["store", "scatter"])
def test_more_tiles_than_expected(epilogue, dtype):
    """Tiles of 128 columns are chosen for the likely number of tiles, 8 x 16; here there are as many as there can be, 11 x 16, so
    that some CTAs have two, and the staging tile is filled and emptied more than once.  The bits are those of 256-row tiles."""
    from dlblas_b200 import _C, ops
    counts = [1, 129, 3, 129, 1, 129, 5, 1]
    e, rows, k, n = len(counts), sum(counts), 1152, 2048
    sms = torch.cuda.get_device_properties(DEV).multi_processor_count
    assert sum(-(-c // 128) for c in counts) == rows // 128 + e and (rows // 128 + e) * n // 128 > sms >= e * n // 128
    g = torch.Generator().manual_seed(23)
    a, a_s = O.quant_fp8(torch.randn(rows, k, generator=g).to(torch.bfloat16), 128)
    b = torch.randn(e, n, k, generator=g).to(FP8)
    b_s = torch.rand(e, n // 128, k // 128, generator=g) * 0.01 + 0.01
    ends = torch.tensor(counts).cumsum(0)
    order = torch.randperm(rows, generator=g)
    weights = torch.rand(rows, generator=g) + 0.5
    extra = {"sorted_idx": order.to(DEV), "weights": weights.to(DEV)} if epilogue == "scatter" else {}
    out = []
    for tile_rows in (128,) if dtype == torch.float32 else (128, 256):
        most = ops.max_tiles_for(rows, e, tile_rows)
        tiles = ops.build_tiles((ends - torch.tensor(counts)).to(DEV), ends.to(DEV), 0, e, most, tile_rows)
        c = torch.zeros(rows, n, dtype=dtype, device=DEV)
        ops.grouped_gemm(a.to(DEV), a_s.to(DEV), b.to(DEV), b_s.to(DEV), tiles, most,
                         _C.EPI_SCATTER_WEIGHT if extra else _C.EPI_STORE, c, tile_rows=tile_rows, **extra)
        out.append(c)
    _status_ok()
    assert torch.equal(out[0], out[-1])
    for i in range(e):
        sl = slice(int(ends[i]) - counts[i], int(ends[i]))
        ref = O.fp8_gemm(a[sl], b[i], a_s[sl], b_s[i], torch.float32)
        got = out[0].cpu().float()
        got = got[order[sl]] / weights[order[sl], None] if extra else got[sl]
        assert O.rel_frobenius(got, ref) < (1e-5 if dtype == torch.float32 else 4e-3), i
