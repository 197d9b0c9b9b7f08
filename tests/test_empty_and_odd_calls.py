"""Calls at the far ends of what the entry points take: no slots or tokens, rows without a finite score, 16-bit routing
weights, expert counts at the edge of the default shared-memory limit, shapes that do not fit together."""
import subprocess
import sys

import pytest
import torch

from oracle import moe_oracle as O

DEV = "cuda"


def _child(code):
    """A process of its own: for calls that would end it, and for limits that an earlier call would have raised."""
    return subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)


# ---- no slots ----------------------------------------------------------------------------------------------------
@pytest.mark.parametrize("block", [1, 16])
def test_align_without_slots_reaches_the_launch(block):
    """Without a device the call ends in a CUDA error; it must not end the process before that."""
    r = _child(f"""
from dlblas_b200 import _C
import ctypes
out = (ctypes.c_int32 * 64)()
p = ctypes.addressof(out)
n = 4 * ({block} - 1)
rc = _C.lib().dlb_moe_align_block_size(p, _C.DLB_I32, 0, 4, 4, {block}, p if n else None, n, p if n else None,
                                       -(-n // {block}), p, None, 0, None) if not __import__('torch').cuda.is_available() else 0
print('rc', rc)
""")
    assert r.returncode == 0 and "rc" in r.stdout, (r.returncode, r.stderr[-500:])
    assert "rc -1" not in r.stdout                                             # nor be refused


@pytest.mark.gpu
@pytest.mark.parametrize("experts,block", [(3, 1), (3, 16), (256, 64), (9000, 2)])
@pytest.mark.parametrize("pad", [False, True])
def test_align_without_slots(experts, block, pad):
    from dlblas_b200.kernels.moe_align_block_size import moe_align_block_size
    ids = torch.empty(0, 2, dtype=torch.int64, device=DEV)
    slots, owner, total = moe_align_block_size(ids, block, experts, experts, None, pad)
    n = experts * (block - 1)
    n = -(-n // block) * block if pad else n
    assert slots.shape == (n,) and owner.shape == (-(-n // block),)
    assert not slots.any() and not owner.any() and total.tolist() == [0]      # the filling is the number of slots


@pytest.mark.gpu
def test_permute_plan_without_tokens():
    from dlblas_b200.kernels.permute.moe_triton_kernels import moe_permute_topk_op_triton
    x = torch.empty(0, 64, dtype=torch.bfloat16, device=DEV)
    rmap = torch.empty(0, dtype=torch.int32, device=DEV)
    for ids in (torch.empty(0, 2, dtype=t, device=DEV) for t in (torch.int32, torch.int64)):
        out, got, order, _ = moe_permute_topk_op_triton(x, ids, 0, [], 0, 0, torch.empty_like(x), rmap)
        assert out.shape == (0, 64) and got.shape == (0,) and order.shape == (0,) and order.dtype == torch.int64


class _NoGradient(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x):
        return x.sum()

    @staticmethod
    def backward(ctx, grad):
        return None


@pytest.mark.gpu
def test_permute_whose_rows_get_no_gradient():
    from dlblas_b200.kernels.permute import permute
    x = torch.ones(5, 64, dtype=torch.bfloat16, device=DEV, requires_grad=True)
    rows, _ = permute(x, torch.zeros(5, 2, dtype=torch.int32, device=DEV))
    (grad,) = torch.autograd.grad(_NoGradient.apply(rows), x)
    assert grad.shape == x.shape and grad.dtype == x.dtype and not grad.any()


@pytest.mark.gpu
def test_errors_of_saved_tensor_hooks_come_through():
    import dlblas_b200
    from dlblas_b200.kernels.permute import permute, unpermute

    def pack(t):
        raise KeyError("packed")

    x = torch.ones(5, 64, dtype=torch.bfloat16, device=DEV, requires_grad=True)
    ids = torch.zeros(5, 2, dtype=torch.int32, device=DEV)
    rows, rmap = permute(x, ids)
    logits = torch.ones(5, 8, device=DEV, requires_grad=True)
    for call in (lambda: permute(x, ids), lambda: unpermute(rows, rmap, torch.ones(5, 2, device=DEV)),
                 lambda: dlblas_b200.topk_gating(logits, 2)):
        with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t), pytest.raises(KeyError, match="packed"):
            call()


# ---- one-rank decode layer ---------------------------------------------------------------------------------------
@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float64])
def test_decode_takes_weights_of_any_type(dtype):
    from dlblas_b200.layers.moe.ep_moe import FusedMoELowLatency
    x, logits, w13, w13s, w2, w2s = (t.to(DEV) for t in O.make_layer_inputs(24, 256, 256, 8, seed=5))
    w, ids = O.softmax_topk(logits.cpu(), 2, True)
    layer = FusedMoELowLatency(1, None, 8, 256, 0)
    w = w.to(DEV).to(dtype)
    out = layer.forward(x, w, ids.to(DEV), w13, w13s, w2, w2s)
    assert torch.equal(out, layer.forward(x, w.float(), ids.to(DEV), w13, w13s, w2, w2s))


def _decode_layer(dispatcher_class, layer_class=None):
    """A one-rank layer without its device buffers."""
    from dlblas_b200.layers.moe.ep_moe import FusedMoELowLatency
    layer_class = layer_class or FusedMoELowLatency
    d = dispatcher_class.__new__(dispatcher_class)
    d.world_size, d.num_max_dispatch_tokens_per_rank, d.max_top_k, d.handle = 1, 128, 8, None
    layer = layer_class.__new__(layer_class)
    layer.num_experts, layer.layer_index, layer.out_dtype, layer.token_dispatcher = 4, 0, torch.bfloat16, d
    return layer


def test_decode_calls_replaced_steps(monkeypatch):
    from dlblas_b200.layers.moe.ep_moe import FusedMoELowLatency
    from dlblas_b200.layers.moe.token_dispatcher import TokenDispatcherLowLatencyP2P as P2P
    called = []
    x, w, ids = torch.zeros(2, 128), torch.ones(2, 2), torch.zeros(2, 2, dtype=torch.int64)
    steps = {n: (lambda *a, n=n, r=r, **k: called.append(n) or r)
             for n, r in (("dispatch", (None,) * 5), ("experts", None), ("combine", x))}
    layer = _decode_layer(type("Exchange", (P2P,), {n: steps[n] for n in ("dispatch", "combine")}),
                          type("Layer", (FusedMoELowLatency,), {"experts": steps["experts"]}))
    layer.forward(x, w, ids, torch.zeros(4, 256, 128), None, None, None)
    assert called == ["dispatch", "experts", "combine"]


@pytest.mark.parametrize("name", ["experts", "dispatch", "dispatch_async", "combine", "combine_async"])
@pytest.mark.parametrize("where", ["object", "class", "subclass"])
def test_decode_is_direct_with_its_own_steps_only(name, where, monkeypatch):
    from dlblas_b200.layers.moe.ep_moe import FusedMoELowLatency
    from dlblas_b200.layers.moe.token_dispatcher import TokenDispatcherLowLatencyP2P as P2P
    assert _decode_layer(P2P)._direct()
    hook = lambda *a, **k: None  # noqa: E731
    if where == "subclass":
        kinds = (P2P, type("L", (FusedMoELowLatency,), {name: hook})) if name == "experts" else (type("D", (P2P,), {name: hook}),)
        layer = _decode_layer(*kinds)
    else:
        layer = _decode_layer(P2P)
        owner = layer if name == "experts" else layer.token_dispatcher
        monkeypatch.setattr(owner if where == "object" else type(owner), name, hook, raising=False)
    assert not layer._direct()


@pytest.mark.gpu
def test_decode_direct_and_step_by_step_agree():
    """Ids of no expert among them; a method on the object sends the call through the three steps."""
    from dlblas_b200.layers.moe.ep_moe import FusedMoELowLatency
    x, logits, w13, w13s, w2, w2s = (t.to(DEV) for t in O.make_layer_inputs(100, 384, 256, 16, seed=6))
    w, ids = (t.to(DEV) for t in O.softmax_topk(logits.cpu(), 4, True))
    ids[::7, 1] = -1
    ids[5] = -1
    layer = FusedMoELowLatency(1, None, 16, 384, 0)
    out = layer.forward(x, w, ids, w13, w13s, w2, w2s)
    layer.token_dispatcher.dispatch = layer.token_dispatcher.dispatch
    assert torch.equal(out, layer.forward(x, w, ids, w13, w13s, w2, w2s)) and layer.token_dispatcher.handle is not None


# ---- expert counts whose histograms just fill the default shared memory -------------------------------------------
@pytest.mark.gpu
def test_sort_at_the_default_shared_memory_limit():
    """32 warps' histograms and the bucket tables come within 272 bytes of 48 KB.  In a process of its own: a call that needs
    more would raise the limit for the ones after it."""
    r = _child("""
import sys
sys.path[:0] = ["tests", "."]
import torch
from test_gpu_kernels import _check_sort
g = torch.Generator().manual_seed(1)
for n, experts in ((1024, 640), (2048, 641), (4096, 642), (4097, 609)):
    ids = torch.randint(-1, experts, (n, 1), generator=g)
    _check_sort(ids, experts)
    _check_sort(ids, experts, torch.int32)
print("done")
""")
    assert r.returncode == 0 and "done" in r.stdout, r.stderr[-800:]


# ---- gating rows without a finite gate ----------------------------------------------------------------------------
@pytest.mark.gpu
@pytest.mark.parametrize("experts", [32, 40])             # whole lanes, and lanes with filling
@pytest.mark.parametrize("bad", [-200.0, float("nan")])   # every exp is 0, so 0 / 0; or a NaN to begin with
def test_gating_drops_rows_without_a_gate(experts, bad):
    import dlblas_b200
    good, top_k, capacity = 64, 2, 6                      # the capacity is the least one, whatever the number of tokens
    x = torch.randn(good, experts, generator=torch.Generator().manual_seed(experts))
    rows = torch.arange(good + 2)
    keep = (rows != 3) & (rows != good + 1)
    full = torch.full((good + 2, experts), bad)
    full[keep] = x
    logits = full.to(DEV).requires_grad_(True)
    l_aux, ec_idx, weights, select = dlblas_b200.topk_gating(logits, top_k, 1.0, capacity, True)
    _, want_idx, want_w, _ = O.topk_gating(x, top_k, 1.0, capacity)
    idx, w = ec_idx.cpu().view(top_k, -1), weights.detach().cpu().view(top_k, -1)
    assert torch.equal(idx[:, keep], want_idx.view(top_k, -1))
    torch.testing.assert_close(w[:, keep], want_w.view(top_k, -1), rtol=1e-5, atol=1e-6)
    assert not idx[:, ~keep].any() and not w[:, ~keep].any()
    place, live = idx[:, keep].flatten().long(), w[:, keep].flatten() > 0
    assert torch.equal(select.cpu()[place[live]], rows[keep].repeat(top_k)[live])
    assert int(select.min()) >= 0 and int(select.max()) < good + 2
    grad = torch.rand(top_k, good + 2, generator=torch.Generator().manual_seed(1))
    weights.backward(grad.flatten().to(DEV))
    ref = O.topk_gating_grad(x, top_k, 1.0, capacity, 0.0, grad[:, keep])
    torch.testing.assert_close(logits.grad.cpu()[keep], ref, rtol=1e-4, atol=1e-6)


# ---- shapes that do not fit together: the kernels would read or write past the smaller tensor -----------------------
@pytest.mark.gpu
def test_shapes_that_do_not_fit_are_refused():
    from dlblas_b200 import ops
    from dlblas_b200.kernels.permute.moe_triton_kernels import (moe_recover_topk_bwd_op_triton, moe_recover_topk_op_triton,
                                                                unpermute)
    rows = torch.zeros(12, 64, dtype=torch.bfloat16, device=DEV)
    rmap = torch.arange(12, dtype=torch.int32, device=DEV)
    probs, grad = torch.ones(6, 2, device=DEV), torch.zeros(6, 64, dtype=torch.bfloat16, device=DEV)
    unpermute(rows, rmap, probs)
    moe_recover_topk_bwd_op_triton(grad, rows, rmap, probs)
    for bad in (torch.ones(7, 2, device=DEV), torch.ones(6, 3, device=DEV)):
        with pytest.raises(AssertionError):
            unpermute(rows, rmap, bad)
        with pytest.raises(AssertionError):
            moe_recover_topk_bwd_op_triton(grad, rows, rmap, bad)
    with pytest.raises(AssertionError):
        moe_recover_topk_op_triton(rows, rmap, probs[:5], 6, 2)
    with pytest.raises(AssertionError):
        moe_recover_topk_op_triton(rows, rmap[:11], None, 6, 2)
    for bad in (grad[:5], grad[:, :32], torch.zeros(6, 128, dtype=torch.bfloat16, device=DEV)):
        with pytest.raises(AssertionError):
            moe_recover_topk_bwd_op_triton(bad, rows, rmap, probs)
    x = torch.zeros(4, 128, dtype=torch.bfloat16, device=DEV)
    pos = torch.arange(8, dtype=torch.int32, device=DEV)
    ops.quant_fp8(x, 128, dst_pos=pos, fanout=2, rows_out=8)
    with pytest.raises(AssertionError):
        ops.quant_fp8(x, 128, dst_pos=pos[:7], fanout=2, rows_out=8)
    with pytest.raises(AssertionError):
        ops.quant_fp8(x, 128, rows_out=3)
    _, _, _, _, ws = ops.topk_gating(torch.zeros(6, 8, device=DEV), 2, 3, return_workspace=True)
    one = torch.ones((), device=DEV)
    ops.topk_gating_bwd(ws, torch.float32, 6, 8, 2, 3, one, torch.ones(12, device=DEV))
    with pytest.raises(AssertionError):
        ops.topk_gating_bwd(ws, torch.float32, 6, 8, 2, 3, one, torch.ones(11, device=DEV))


# ---- routing weights divided by their sum -------------------------------------------------------------------------
@pytest.mark.gpu
@pytest.mark.parametrize("top_k", [1, 2, 3, 4, 5, 6, 7, 8, 9, 12, 15, 16, 17, 24, 31, 32])
@pytest.mark.parametrize("tokens", [1, 37, 3000])          # one block, one block with several ids per lane, chunks
def test_plan_normalises_as_torch_does(tokens, top_k):
    """Bit for bit: the expert-parallel path divides by torch's sum."""
    from dlblas_b200 import _C
    g = torch.Generator().manual_seed(tokens + top_k)
    ids = torch.randint(0, 40, (tokens, top_k), generator=g).to(DEV)
    w = torch.rand(tokens, top_k, generator=g).to(DEV)
    lib, slots = _C.lib(), tokens * top_k
    got, pos = torch.empty_like(w), torch.empty(slots, dtype=torch.int32, device=DEV)
    max_tiles = slots // 128 + 40
    tiles = torch.empty((max_tiles + 1) * 4, dtype=torch.int32, device=DEV)
    ws = torch.empty(max(lib.dlb_sort_by_expert_workspace_size(slots, 40), 1), dtype=torch.uint8, device=DEV)
    _C.check(lib.dlb_moe_plan(_C.ptr(ids), _C.DLB_I64, tokens, top_k, 40, 0, 40, 128, None, _C.ptr(pos), _C.ptr(tiles),
                              max_tiles, _C.ptr(w), _C.ptr(got), _C.ptr(ws), ws.numel(), _C.stream()))
    assert torch.equal(got, w / w.sum(-1, keepdim=True))


@pytest.mark.gpu
def test_layer_normalises_weights_of_any_layout():
    from dlblas_b200.layers.moe.ep_moe import DlblasTritonFusedMoEBlockedF8Impl
    x, logits, *weights = (t.to(DEV) for t in O.make_layer_inputs(50, 256, 256, 16, seed=8))
    w, ids = (t.to(DEV) for t in O.softmax_topk(logits.cpu(), 6, False))
    layer, plain = (DlblasTritonFusedMoEBlockedF8Impl(top_k=6, num_experts=16, renormalize=r, out_dtype=torch.bfloat16)
                    for r in (True, False))
    for given in (w, w.t().contiguous().t(), w.half(), w.half().t().contiguous().t()):
        want = plain.forward(x, given / given.sum(-1, keepdim=True), ids, *weights)
        assert torch.equal(layer.forward(x, given, ids, *weights), want)


# ---- routing scores that are no numbers, or minus infinity --------------------------------------------------------
@pytest.mark.gpu
@pytest.mark.parametrize("experts,groups", [(256, 8), (160, 8), (64, 8), (256, 32), (32, 1), (96, 8)])   # the last: general kernel
@pytest.mark.parametrize("off", [0.02, 0.5, 0.9, 1.0])
def test_grouped_routing_with_experts_switched_off(experts, groups, off):
    """A bias of minus infinity switches an expert off, down to fewer experts and groups than are wanted; so does a NaN."""
    from dlblas_b200 import ops
    g = torch.Generator().manual_seed(int(100 * off) + experts + groups)
    topk_group, top_k = max(groups // 2, 1), 6
    x = torch.randn(200, experts, generator=g)
    for trial in range(4):
        bias = torch.randn(experts, generator=g) * 0.1
        dead = torch.rand(experts, generator=g) < off
        if trial == 1:
            dead[0::experts // 32] = True                     # the first expert of every lane
        bias[dead] = -float("inf")
        want_w, want_ids = O.biased_grouped_topk(x, bias, top_k, False, groups, topk_group)
        w, ids = ops.route_grouped_topk(x.to(DEV), bias.to(DEV), top_k, False, groups, topk_group)
        assert torch.equal(ids.cpu(), want_ids) and torch.equal(w.cpu(), want_w)
        if 2 * int(dead.sum()) <= experts:                    # enough left in any topk_group groups
            nan = bias.masked_fill(dead, float("nan"))
            w, ids = ops.route_grouped_topk(x.to(DEV), nan.to(DEV), top_k, False, groups, topk_group)
            live = ~dead[want_ids.long()]
            assert torch.equal(ids.cpu()[live], want_ids[live]) and torch.equal(w.cpu()[live], want_w[live])


# ---- threads ------------------------------------------------------------------------------------------------------
@pytest.mark.gpu
def test_other_threads_run_while_a_launch_waits():
    """Launches behind half a second of work fill the queue, and the next one waits for the GPU; torch's operators let other
    threads run in the meantime, and so do these."""
    import threading
    import time

    from dlblas_b200 import ops
    x = torch.zeros(4, 128, dtype=torch.bfloat16, device=DEV)
    ops.quant_fp8(x, 128)
    torch.cuda.synchronize()
    gaps, done = [], threading.Event()

    def watch():
        last = time.perf_counter()
        while not done.is_set():
            time.sleep(0.001)
            now = time.perf_counter()
            gaps.append(now - last)
            last = now

    thread = threading.Thread(target=watch)
    thread.start()
    torch.cuda._sleep(1_000_000_000)
    begin = time.perf_counter()
    for _ in range(4000):
        ops.quant_fp8(x, 128)
    queued = time.perf_counter() - begin
    done.set()
    thread.join()
    torch.cuda.synchronize()
    if queued < 0.3:
        pytest.skip("the queue took all launches")
    assert max(gaps) < 0.5 * queued, (max(gaps), queued)


@pytest.mark.gpu
def test_threads_on_their_own_streams():
    """Four threads at once, each with its own sizes and stream: the results of one thread alone."""
    import threading

    from dlblas_b200.kernels.permute import permute, unpermute
    from dlblas_b200.layers.moe.ep_moe import DlblasTritonFusedMoEBlockedF8Impl
    layer = DlblasTritonFusedMoEBlockedF8Impl(top_k=2, num_experts=8, renormalize=True, out_dtype=torch.bfloat16)
    jobs, results = [], {}
    for i, tokens in enumerate((3, 70, 500, 2100)):
        x, logits, *weights = (t.to(DEV) for t in O.make_layer_inputs(tokens, 256, 256, 8, seed=i))
        w, ids = (t.to(DEV) for t in O.softmax_topk(logits.cpu(), 2, False))
        jobs.append((x, w, ids, weights))
    torch.cuda.synchronize()

    def run(i):
        x, w, ids, weights = jobs[i]
        a = x.detach().requires_grad_(True)
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(20):
                a.grad = None
                rows, rmap = permute(a, ids)
                y = unpermute(rows, rmap, w)
                y.backward(x)
                out = layer.forward(x, w, ids, *weights)
            torch.cuda.current_stream().synchronize()
        return out, y.detach(), rmap, a.grad

    alone = [run(i) for i in range(4)]
    threads = [threading.Thread(target=lambda i=i: results.__setitem__(i, run(i))) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for i in range(4):
        assert all(torch.equal(p, q) for p, q in zip(alone[i], results[i])), i


@pytest.mark.gpu
def test_operators_in_a_row_wait_for_one_another():
    """Every kernel is launched while its predecessor runs.  Inputs overwritten by torch right before and right after each
    chain, no synchronisation in between, against the same chain with one after every operator."""
    from dlblas_b200 import ops
    from dlblas_b200.kernels.fp8 import per_token_group_quant_fp8
    from dlblas_b200.kernels.moe import biased_grouped_topk
    from dlblas_b200.kernels.permute import permute, unpermute
    g = torch.Generator(device=DEV).manual_seed(5)
    t, h, e, k, rounds = 300, 512, 64, 4, 24
    xs = torch.randn(rounds, t, h, device=DEV, generator=g, dtype=torch.bfloat16)
    ls = torch.randn(rounds, t, e, device=DEV, generator=g)
    bias = torch.randn(e, device=DEV, generator=g) * 0.01
    w = torch.randn(640, h, device=DEV, generator=g).to(torch.float8_e4m3fn)
    ws = torch.rand(5, h // 128, device=DEV, generator=g) + 0.5
    x, logits = torch.empty_like(xs[0]), torch.empty_like(ls[0])

    def chain(sync):
        wait = torch.cuda.synchronize if sync else (lambda: None)
        weights, ids = biased_grouped_topk(x, logits, bias, k, True, 8, 4)
        wait()
        rows, row_map = permute(x, ids)
        wait()
        back = unpermute(rows, row_map, weights)
        wait()
        q, s = per_token_group_quant_fp8(back, 128)
        wait()
        y = ops.fp8_gemm(q, w, s, ws, torch.bfloat16)
        wait()
        return ids, rows, back, q.view(torch.uint8), y

    def run(sync):
        out = []
        for i in range(rounds):
            x.copy_(xs[i])
            logits.copy_(ls[i])
            out.append(chain(sync))
            x.zero_()
            logits.zero_()
        torch.cuda.synchronize()
        return out

    for got, want in zip(run(False), run(True)):
        for a, b in zip(got, want):
            assert torch.equal(a, b)
