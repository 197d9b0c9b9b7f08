"""16-bit grouped GEMM (tcgen05 kind::f16) against the oracle."""
import pytest
import torch

from oracle import moe_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("trans_b", [True, False])
@pytest.mark.parametrize("tile_rows", [128, 256])      # one CTA per tile / pairs of CTAs (cta_group::2)
def test_m_grouped_gemm(dtype, trans_b, tile_rows, monkeypatch):
    monkeypatch.setenv("DLBLAS_GEMM16_TILE_ROWS", str(tile_rows))
    from dlblas_b200 import _C
    from dlblas_b200.kernels.grouped_gemm.BF16 import m_grouped_gemm
    g = torch.Generator().manual_seed(13)
    for (sizes, n, k) in [([5, 0, 130, 64, 257], 264, 200), ([128, 128], 512, 256), ([1], 8, 8), ([300, 211], 1000, 1096)]:
        sz = torch.tensor(sizes, dtype=torch.int64)
        m = int(sz.sum())
        a = (torch.randn(m, k, generator=g) * 0.5).to(dtype)
        b = (torch.randn(len(sizes), n, k, generator=g) * 0.5).to(dtype)
        b_in = b if trans_b else b.transpose(1, 2).contiguous()
        out = m_grouped_gemm(a.to(DEV), b_in.to(DEV), sz.to(DEV), trans_b=trans_b)
        _C.check_status()
        ref = O.m_grouped_gemm(a, b, sz, trans_b=True)
        assert out.shape == (m, n) and out.dtype == dtype
        assert O.rel_frobenius(out.cpu(), ref) < 2e-3
        assert float((out.cpu().float() - ref.float()).abs().max()) <= 2 ** -6 * float(ref.float().abs().max())


def test_m_grouped_gemm_large_and_empty():
    from dlblas_b200 import _C
    from dlblas_b200.kernels.grouped_gemm.BF16 import m_grouped_gemm, utils
    g = torch.Generator(device=DEV).manual_seed(1)
    sizes = torch.tensor([1000, 3000, 17, 4175], device=DEV)
    a = torch.randn(8192, 2048, generator=g, device=DEV, dtype=torch.bfloat16)
    b = torch.randn(4, 1024, 2048, generator=g, device=DEV, dtype=torch.bfloat16) * 0.05
    ref = utils.gmm(a.float(), b.float(), sizes.cpu(), trans_b=True)
    out = m_grouped_gemm(a, b, sizes, trans_b=True)              # 2048 rows per group on average: the pair kernel
    _C.check_status()
    assert float((out.float() - ref).norm() / ref.norm()) < 3e-3
    import os
    os.environ["DLBLAS_GEMM16_TILE_ROWS"] = "128"
    try:
        out1 = m_grouped_gemm(a, b, sizes, trans_b=True)
    finally:
        del os.environ["DLBLAS_GEMM16_TILE_ROWS"]
    _C.check_status()
    assert torch.equal(out, out1)                                # same sums in the same order
    b_kn = b.transpose(1, 2).contiguous()                        # [G, K, N]: read as an MN-major operand, no transposition
    for tile_rows in ("128", "256"):
        os.environ["DLBLAS_GEMM16_TILE_ROWS"] = tile_rows
        try:
            out2 = m_grouped_gemm(a, b_kn, sizes, trans_b=False)
        finally:
            del os.environ["DLBLAS_GEMM16_TILE_ROWS"]
        _C.check_status()
        assert torch.equal(out, out2)
    empty = m_grouped_gemm(a[:0], b, torch.zeros(4, dtype=torch.int64, device=DEV), trans_b=True)
    assert empty.shape == (0, 1024)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("tile_rows", [128, 256])
def test_k_grouped_gemm(dtype, tile_rows, monkeypatch):
    monkeypatch.setenv("DLBLAS_GEMM16_TILE_ROWS", str(tile_rows))
    from dlblas_b200 import _C
    from dlblas_b200.kernels.grouped_gemm.BF16 import k_grouped_gemm
    g = torch.Generator().manual_seed(17)
    # ragged K ranges (not multiples of the 64-element K block), empty groups first / in the middle / last,
    # m and n that are not multiples of the tile, a single group
    for (sizes, m, n) in [([5, 0, 130, 64, 257], 264, 200), ([128, 128], 512, 256), ([1], 8, 8), ([0, 300, 211, 0], 136, 1096),
                          ([0], 16, 24)]:
        sz = torch.tensor(sizes, dtype=torch.int64)
        k = int(sz.sum())
        a = (torch.randn(k, m, generator=g) * 0.5).to(dtype)
        b = (torch.randn(k, n, generator=g) * 0.5).to(dtype)
        out = k_grouped_gemm(a.to(DEV), b.to(DEV), sz.to(DEV))
        _C.check_status()
        ref = O.k_grouped_gemm(a, b, sz)
        assert out.shape == (len(sizes), m, n) and out.dtype == dtype
        assert O.rel_frobenius(out.cpu(), ref) < 2e-3
        assert float((out.cpu().float() - ref.float()).abs().max()) <= 2 ** -6 * max(float(ref.float().abs().max()), 1e-6)
        for i, size in enumerate(sizes):
            if size == 0:
                assert not out[i].any()                          # an empty group writes zeros


def test_k_grouped_gemm_like_the_reference_test():
    # tests/kernels/grouped_gemm/BF16/test_k_grouped_gemm.py of the reference at a sixteenth of its K: random group
    # sizes, row-max normalisation, rtol = atol = 0.01
    import random
    from dlblas_b200 import _C
    from dlblas_b200.kernels.grouped_gemm.BF16 import k_grouped_gemm, utils
    random.seed(3)
    groups = 16
    raw = [random.randint(0, 2 * 2560) for _ in range(groups)]
    sizes = torch.tensor(raw, dtype=torch.int64, device=DEV)
    k = int(sizes.sum())
    g = torch.Generator(device=DEV).manual_seed(2)
    for (m, n) in ((1536, 2048), (2048, 768)):
        a = torch.randn(k, m, generator=g, device=DEV, dtype=torch.bfloat16)
        b = torch.randn(k, n, generator=g, device=DEV, dtype=torch.bfloat16)
        out = k_grouped_gemm(a, b, sizes)
        _C.check_status()
        ref = utils.gmm_dw(a, b, sizes.cpu())
        torch.testing.assert_close(utils.row_max_normalization(out.float()), utils.row_max_normalization(ref.float()),
                                   rtol=0.01, atol=0.01)


def test_k_grouped_gemm_sizes_that_do_not_add_up():
    """Group sizes that stop short of the operands' rows leave the rest unused; sizes that run past them are clipped
    (the last groups shrink, down to empty), as the entry point documents."""
    from dlblas_b200 import _C
    from dlblas_b200.kernels.grouped_gemm.BF16 import k_grouped_gemm
    g = torch.Generator().manual_seed(23)
    k, m, n = 300, 256, 136
    a = (torch.randn(k, m, generator=g) * 0.5).to(torch.bfloat16)
    b = (torch.randn(k, n, generator=g) * 0.5).to(torch.bfloat16)
    for sizes, clipped in (([100, 50], [100, 50]), ([200, 150, 70], [200, 100, 0])):
        out = k_grouped_gemm(a.to(DEV), b.to(DEV), torch.tensor(sizes, dtype=torch.int64, device=DEV))
        _C.check_status()
        ref = O.k_grouped_gemm(a, b, torch.tensor(clipped, dtype=torch.int64))
        assert O.rel_frobenius(out.cpu(), ref) < 2e-3
        assert not out[-1].any() or clipped[-1] > 0


@pytest.mark.parametrize("tile_rows", [128, 256])
@pytest.mark.parametrize("trans_b", [True, False])
def test_m_grouped_gemm_tile_bands(tile_rows, trans_b, monkeypatch):
    """More than 16 tiles of columns: bands of 4096 rows of tiles, the last one lower; groups end inside a band."""
    monkeypatch.setenv("DLBLAS_GEMM16_TILE_ROWS", str(tile_rows))
    from dlblas_b200 import _C
    from dlblas_b200.kernels.grouped_gemm.BF16 import m_grouped_gemm, utils
    g = torch.Generator(device=DEV).manual_seed(29)
    sizes = torch.tensor([1000, 0, 3300, 17, 513], device=DEV)
    a = torch.randn(4830, 64, generator=g, device=DEV, dtype=torch.bfloat16)
    b = torch.randn(5, 4360, 64, generator=g, device=DEV, dtype=torch.bfloat16)
    out = m_grouped_gemm(a, b if trans_b else b.transpose(1, 2).contiguous(), sizes, trans_b=trans_b)
    _C.check_status()
    ref = utils.gmm(a.float(), b.float(), sizes.cpu(), trans_b=True)
    assert float((out.float() - ref).norm() / ref.norm()) < 3e-3


@pytest.mark.parametrize("groups,m,n", [(1100, 8, 8), (1025, 264, 520), (40, 1536, 2048), (3, 8, 8), (2, 2560, 4096)])
@pytest.mark.parametrize("tile_rows", [128, 256])
def test_k_grouped_gemm_plan(groups, m, n, tile_rows, monkeypatch):
    """Fewer tiles than workers, many more, whole numbers of tiles per worker, and more groups than the plan takes at a time."""
    monkeypatch.setenv("DLBLAS_GEMM16_TILE_ROWS", str(tile_rows))
    from dlblas_b200 import _C
    from dlblas_b200.kernels.grouped_gemm.BF16 import k_grouped_gemm, utils
    g = torch.Generator().manual_seed(groups)
    sizes = torch.randint(0, 8 if groups > 1000 else 700, (groups,), generator=g)
    k = int(sizes.sum())
    a = torch.randn(k, m, generator=g).to(torch.bfloat16).to(DEV)
    b = torch.randn(k, n, generator=g).to(torch.bfloat16).to(DEV)
    out = k_grouped_gemm(a, b, sizes.to(DEV))
    _C.check_status()
    ref = utils.gmm_dw(a.float(), b.float(), sizes)
    assert float((out.float() - ref.float()).norm() / ref.float().norm()) < 3e-3


@pytest.mark.parametrize("groups,n", [(5, 8), (5, 120), (5, 128), (5, 136), (5, 392), (73, 256), (73, 264), (147, 256), (148, 256)])
def test_m_grouped_gemm_narrow_tiles(groups, n):
    """Tiles of 128 columns where there are fewer tiles of 256 than SMs (148): both sides of the line, ragged columns."""
    from dlblas_b200 import _C
    from dlblas_b200.kernels.grouped_gemm.BF16 import m_grouped_gemm, utils
    g = torch.Generator(device=DEV).manual_seed(31)
    sizes = torch.tensor([1, 130, 0, 257, 128] if groups == 5 else [1] * groups, device=DEV)
    m, k = int(sizes.sum()), 192
    a = torch.randn(m, k, generator=g, device=DEV, dtype=torch.float16)
    for trans_b in (True, False):
        b = torch.randn(groups, n, k, generator=g, device=DEV, dtype=torch.float16)
        out = m_grouped_gemm(a, b if trans_b else b.transpose(1, 2).contiguous(), sizes, trans_b=trans_b)
        _C.check_status()
        ref = utils.gmm(a.float(), b.float(), sizes.cpu(), trans_b=True)
        assert float((out.float() - ref).norm() / ref.norm()) < 1e-3     # one rounding to fp16


@pytest.mark.parametrize("tile_rows", [128, 256])
def test_m_grouped_gemm_beside_copies(tile_rows, monkeypatch):
    """Several tiles per CTA or pair, so that accumulators are handed back and used again, beside a copy on another stream:
    same bits as alone, every time."""
    monkeypatch.setenv("DLBLAS_GEMM16_TILE_ROWS", str(tile_rows))
    from dlblas_b200 import _C
    from dlblas_b200.kernels.grouped_gemm.BF16 import m_grouped_gemm, utils
    g = torch.Generator(device=DEV).manual_seed(6)
    sizes = torch.tensor([1500, 0, 700, 2300, 1], device=DEV)
    m, n, k = int(sizes.sum()), 6144, 192
    a = torch.randn(m, k, generator=g, device=DEV, dtype=torch.bfloat16)
    b = torch.randn(5, n, k, generator=g, device=DEV, dtype=torch.bfloat16)
    alone = m_grouped_gemm(a, b, sizes, trans_b=True)
    ref = utils.gmm(a.float(), b.float(), sizes.cpu(), trans_b=True)
    assert float((alone.float() - ref).norm() / ref.norm()) < 3e-3
    src = torch.randn(32 << 20, device=DEV)
    dst, side, out = torch.empty_like(src), torch.cuda.Stream(), []
    torch.cuda.synchronize()
    for _ in range(20):
        with torch.cuda.stream(side):
            dst.copy_(src)
        for _ in range(3):
            out.append(m_grouped_gemm(a, b, sizes, trans_b=True))
    torch.cuda.synchronize()
    _C.check_status()
    assert all(torch.equal(alone, c) for c in out)
