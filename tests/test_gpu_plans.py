"""Sizes at which the planning and row-moving kernels change their path: one block or several, lanes or chunks left over,
rows in flight, more experts than the first sort assumes."""
import pytest
import torch

from oracle import moe_oracle as O
from test_gpu_kernels import _check_sort

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("n", [1, 1024, 1025, 2049, 4096, 4097, 8193, 16385, 327680, 327681])
@pytest.mark.parametrize("experts", [1, 256, 1000])
def test_sort_at_the_edges_of_its_paths(n, experts):
    g = torch.Generator().manual_seed(n + experts)
    _check_sort(torch.randint(-1, experts, (n, 1), generator=g), experts)


@pytest.mark.parametrize("slots,experts,block", [(1, 3, 16), (4096, 64, 32), (4097, 160, 16), (20000, 256, 64), (9, 256, 1)])
@pytest.mark.parametrize("pad", [False, True])
def test_align_at_the_edges_of_the_sort(slots, experts, block, pad):
    from dlblas_b200.kernels.moe_align_block_size import moe_align_block_size
    g = torch.Generator().manual_seed(slots)
    ids = torch.randint(0, experts, (slots, 1), generator=g, dtype=torch.int32)
    got = moe_align_block_size(ids.to(DEV), block, experts, experts, None, pad)
    want = O.moe_align_block_size(ids, block, experts, pad)
    blocks = int(want[2]) // block
    assert torch.equal(got[2].cpu(), want[2].view(1)) and torch.equal(got[0].cpu(), want[0])
    assert torch.equal(got[1].cpu()[:blocks], want[1][:blocks])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
def test_quantiser_bytes_over_the_range(dtype):
    """The quotient comes from a reciprocal and corrections: same bytes as the division, also for tiny and huge groups."""
    from dlblas_b200 import ops
    g = torch.Generator().manual_seed(3)
    span = 12 if dtype == torch.float16 else 100
    x = torch.randn(512, 1024, generator=g) * torch.exp2(torch.randint(-span, span, (512, 8), generator=g).float()
                                                         .repeat_interleave(128, 1))
    x = (x * torch.exp2(-torch.randint(0, 12, x.shape, generator=g).float())).to(dtype)
    x[::3, ::5] = 0.0
    x[1::3, ::7] = -0.0                                          # the sign of a zero is a bit of its byte
    q, s = ops.quant_fp8(x.to(DEV), 128)
    oq, os_ = O.quant_fp8(x)
    assert torch.equal(s.cpu(), os_) and torch.equal(q.cpu().view(torch.uint8), oq.view(torch.uint8))


@pytest.mark.parametrize("tokens,top_k,hidden,experts", [(1, 1, 8, 4), (513, 8, 264, 64), (1025, 4, 8, 1500), (37, 9, 520, 1024)])
def test_permute_and_back(tokens, top_k, hidden, experts):
    from dlblas_b200.kernels.permute import permute, unpermute
    g = torch.Generator().manual_seed(tokens)
    ids = torch.stack([torch.randperm(experts, generator=g)[:top_k] if top_k <= experts else torch.arange(top_k)
                       for _ in range(tokens)]).int()
    ids[torch.rand(tokens, top_k, generator=g) < 0.2] = -1
    ids[0, 0] = experts - 1
    x = torch.randn(tokens, hidden, generator=g).to(torch.bfloat16)
    probs = torch.rand(tokens, top_k, generator=g)
    grad = torch.randn(tokens, hidden, generator=g).to(torch.bfloat16)
    xd, pd = x.to(DEV).requires_grad_(True), probs.to(DEV).requires_grad_(True)
    rows, rmap = permute(xd, ids.to(DEV))
    o_rows, o_rmap, _ = O.permute_topk(x, ids)
    assert torch.equal(rows.detach().cpu(), o_rows) and torch.equal(rmap.cpu(), o_rmap)
    y = unpermute(rows, rmap, pd)
    assert torch.equal(y.detach().cpu(), O.unpermute_topk(o_rows, o_rmap, probs, tokens, top_k))
    y.backward(grad.to(DEV))
    act, pg = O.unpermute_topk_bwd(grad, o_rows, o_rmap, probs)
    # sums of `hidden` products in fp32, in another order: hidden * 2^-24 of the sum of their magnitudes
    bound = hidden * 2.0 ** -24 * float(grad.float().abs().sum(1).max() * x.float().abs().max())
    assert float((pd.grad.cpu() - pg).abs().max()) <= bound
    gx = O.unpermute_topk(act.to(torch.bfloat16), o_rmap, None, tokens, top_k)
    assert torch.equal(xd.grad.cpu(), gx)


@pytest.mark.parametrize("tokens,experts,top_k", [(2, 8, 1), (33, 40, 2), (129, 256, 8)])
def test_gating_at_odd_sizes(tokens, experts, top_k):
    import dlblas_b200
    x = torch.randn(tokens, experts, generator=torch.Generator().manual_seed(tokens))
    got = dlblas_b200.topk_gating(x.to(DEV), top_k, 1.5, 2)
    want = O.topk_gating(x, top_k, 1.5, 2)
    for a, b in zip(got, want):
        if a.dtype.is_floating_point:
            torch.testing.assert_close(a.cpu(), b, rtol=1e-5, atol=1e-6)
        else:
            assert torch.equal(a.cpu(), b.to(a.dtype))
