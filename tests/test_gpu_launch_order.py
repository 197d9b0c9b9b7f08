"""Kernels are launched while their predecessor in the stream still runs.  The orders that a stream, an event or a CUDA graph
promises hold all the same: inputs that a slow kernel writes right in front of an operator, or on another stream behind an
event, are the ones it reads.  Every result is compared bit for bit with the same operators run one at a time."""
import pytest
import torch

from oracle import moe_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda"
FP8 = torch.float8_e4m3fn
SLOW = 2_000_000      # cycles of the kernel that holds an input back: about a millisecond


class Chain:
    """A chain of operators over buffers of its own; step(i) is what is written into the inputs before pass i."""

    def __init__(self, tokens=2500, hidden=512, experts=64, top_k=4, rounds=4):
        g = torch.Generator(device=DEV).manual_seed(tokens)
        self.top_k = top_k
        self.xs = torch.randn(rounds, tokens, hidden, device=DEV, generator=g, dtype=torch.bfloat16)
        self.ls = torch.randn(rounds, tokens, experts, device=DEV, generator=g)
        self.bias = torch.randn(experts, device=DEV, generator=g) * 0.01
        self.w = torch.randn(640, hidden, device=DEV, generator=g).to(FP8)
        self.ws = torch.rand(5, hidden // 128, device=DEV, generator=g) + 0.5
        self.b16 = torch.randn(experts, 256, hidden, device=DEV, generator=g, dtype=torch.bfloat16) * 0.1
        w13, w2 = (torch.randn(experts, n, k, device=DEV, generator=g).to(FP8) for n, k in ((512, hidden), (hidden, 256)))
        self.moe_w = (w13, torch.rand(experts, 4, hidden // 128, device=DEV, generator=g) * 0.01 + 0.01,
                      w2, torch.rand(experts, hidden // 128, 2, device=DEV, generator=g) * 0.01 + 0.01)
        self.x, self.logits = torch.zeros_like(self.xs[0]), torch.zeros_like(self.ls[0])
        self.rounds = rounds
        # ragged, one group empty
        self.sizes = torch.full((experts,), tokens // experts, dtype=torch.int64, device=DEV)
        self.sizes[2] += self.sizes[1] + tokens % experts
        self.sizes[1] = 0

    def write(self, i):
        self.x.copy_(self.xs[i])
        self.logits.copy_(self.ls[i])

    def clear(self):
        self.x.zero_()
        self.logits.zero_()

    def first(self, wait=lambda: None):
        """What reads the inputs first."""
        from dlblas_b200.kernels.moe import biased_grouped_topk
        weights, ids = biased_grouped_topk(self.x, self.logits, self.bias, self.top_k, True, 8, 4)
        wait()
        return weights, ids

    def rest(self, weights, ids, wait=lambda: None):
        import dlblas_b200
        from dlblas_b200 import ops
        from dlblas_b200.kernels.fp8 import per_token_group_quant_fp8
        from dlblas_b200.kernels.grouped_gemm.BF16 import k_grouped_gemm, m_grouped_gemm
        from dlblas_b200.kernels.moe_align_block_size import moe_align_block_size
        from dlblas_b200.layers.moe.ep_moe import DlblasTritonFusedMoEBlockedF8Impl
        experts = self.bias.numel()
        q, s = per_token_group_quant_fp8(self.x, 128)
        wait()
        y = ops.fp8_gemm(q, self.w, s, self.ws, torch.bfloat16)
        wait()
        sorted_ids, expert_ids, padded = moe_align_block_size(ids, 64, experts, experts)
        wait()
        layer = DlblasTritonFusedMoEBlockedF8Impl(top_k=self.top_k, num_experts=experts, out_dtype=torch.bfloat16)
        out = layer.forward(self.x, weights, ids, *self.moe_w)
        wait()
        gated = dlblas_b200.topk_gating(self.logits, self.top_k, 1.0, 2, False)
        wait()
        m16 = m_grouped_gemm(out, self.b16, self.sizes, trans_b=True)
        wait()
        k16 = k_grouped_gemm(out, m16, self.sizes)
        wait()
        return [ids, weights, q.view(torch.uint8), s, y, padded, out, m16, k16, *gated]


def _apart(chain):
    """Pass by pass and operator by operator, each waited for."""
    wait, out = torch.cuda.synchronize, []
    for i in range(chain.rounds):
        chain.write(i)
        wait()
        out.append(chain.rest(*chain.first(wait), wait))
    chain.clear()
    wait()
    return out


def _same(got, want):
    for a, b in zip(got, want):
        assert len(a) == len(b)
        for j, (p, q) in enumerate(zip(a, b)):
            equal = torch.equal(p, q)
            assert equal, j


def test_chain_on_one_stream():
    chain = Chain()
    want, got = _apart(chain), []
    for i in range(chain.rounds):
        torch.cuda._sleep(SLOW)
        chain.write(i)
        got.append(chain.rest(*chain.first()))
        chain.clear()
    torch.cuda.synchronize()
    _same(got, want)


def test_chain_in_a_graph():
    """Captured once, replayed with other inputs; a replay starts right behind the writes."""
    chain = Chain()
    want, got = _apart(chain), []
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        result = chain.rest(*chain.first())
    for i in range(chain.rounds):
        torch.cuda._sleep(SLOW)
        chain.write(i)
        graph.replay()
        got.append([t.clone() for t in result])
        chain.clear()
    torch.cuda.synchronize()
    _same(got, want)
    graph.reset()


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("before", ["operator", "torch", "nothing"])
def test_streams_joined_by_an_event(captured, before):
    """The inputs arrive from a second stream, late; the operator behind the event's wait must see them, whatever ran on its
    own stream in front of the wait."""
    from dlblas_b200.kernels.fp8 import per_token_group_quant_fp8
    chain = Chain()
    want, got = _apart(chain), []
    other = torch.randn(4096, 512, device=DEV, dtype=torch.bfloat16)
    main, side = torch.cuda.Stream(), torch.cuda.Stream()
    source = [torch.empty_like(chain.x), torch.empty_like(chain.logits)]
    torch.cuda.synchronize()

    def one():
        here = torch.cuda.current_stream()
        fork, done = torch.cuda.Event(), torch.cuda.Event()
        fork.record(here)
        side.wait_event(fork)
        with torch.cuda.stream(side):
            torch.cuda._sleep(SLOW)
            chain.x.copy_(source[0])
            chain.logits.copy_(source[1])
            # the last thing in front of the event is an operator of the package
            early = per_token_group_quant_fp8(chain.x, 128)      # element 2 and 3 of the chain's results
            done.record(side)
        if before == "operator":
            per_token_group_quant_fp8(other, 128)
        elif before == "torch":
            other.add_(0)
        here.wait_event(done)
        return chain.rest(*chain.first()) + [early[0].view(torch.uint8), early[1]]

    if captured:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=main):
            result = one()
    with torch.cuda.stream(main):
        for i in range(chain.rounds):
            source[0].copy_(chain.xs[i])
            source[1].copy_(chain.ls[i])
            if captured:
                graph.replay()
            else:
                result = one()
            got.append([t.clone() for t in result])
            chain.clear()
    torch.cuda.synchronize()
    n = len(want[0])
    _same([r[:n] for r in got], want)
    _same([r[n:] for r in got], [[w[2], w[3]] for w in want])
    if captured:
        graph.reset()


@pytest.mark.parametrize("captured", [False, True])
def test_exchange_kernels_in_between(captured):
    """The masked-layout step: the exchange's kernels are launched the plain way, between kernels that are not."""
    from dlblas_b200 import ops
    from dlblas_b200.layers.moe.ep_moe import FusedMoELowLatency
    x, logits, *weights = (t.to(DEV) for t in O.make_layer_inputs(64, 512, 256, 16, seed=3))
    g = torch.Generator(device=DEV).manual_seed(3)
    xs = torch.randn(4, *x.shape, device=DEV, generator=g, dtype=torch.bfloat16)
    ls = torch.randn(4, *logits.shape, device=DEV, generator=g)
    layer = FusedMoELowLatency(1, None, 16, 512, 0)
    layer.token_dispatcher.dispatch = layer.token_dispatcher.dispatch      # a replaced step: all of them are called

    def step(wait=lambda: None):
        w, ids = ops.route_softmax_topk(logits, 4, True)
        wait()
        out = layer.forward(x, w, ids, *weights)
        wait()
        q, s = ops.quant_fp8(out, 128)
        wait()
        return [w, ids, out, q.view(torch.uint8), s]

    want, got = [], []
    for i in range(4):
        x.copy_(xs[i])
        logits.copy_(ls[i])
        torch.cuda.synchronize()
        want.append([t.clone() for t in step(torch.cuda.synchronize)])
    if captured:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            result = step()
    for i in range(4):
        torch.cuda._sleep(SLOW)
        x.copy_(xs[i])
        logits.copy_(ls[i])
        if captured:
            graph.replay()
        else:
            result = step()
        got.append([t.clone() for t in result])
        x.zero_()
        logits.zero_()
    torch.cuda.synchronize()
    _same(got, want)
    if captured:
        graph.reset()


def test_default_stream_and_a_blocking_stream():
    """The legacy default stream waits for streams that were created without the non-blocking flag, and they for it, without an
    event.  An operator on the default stream, right behind another one, reads what such a stream wrote in between."""
    import ctypes

    from dlblas_b200.kernels.fp8 import per_token_group_quant_fp8
    handle = ctypes.c_void_p()
    assert int(torch.cuda.cudart().cudaStreamCreate(ctypes.addressof(handle))) == 0
    blocking = torch.cuda.ExternalStream(handle.value)
    x, other = (torch.zeros(2048, 512, device=DEV, dtype=torch.bfloat16) for _ in range(2))
    xs = torch.randn(6, 2048, 512, device=DEV, dtype=torch.bfloat16)
    want = [per_token_group_quant_fp8(t, 128) for t in xs]
    torch.cuda.synchronize()
    got = []
    for t in xs:
        per_token_group_quant_fp8(other, 128)
        with torch.cuda.stream(blocking):
            torch.cuda._sleep(SLOW)
            x.copy_(t)
        got.append(per_token_group_quant_fp8(x, 128))
        with torch.cuda.stream(blocking):
            x.zero_()
    torch.cuda.synchronize()
    _same([[q.view(torch.uint8), s] for q, s in got], [[q.view(torch.uint8), s] for q, s in want])
    del blocking
    assert int(torch.cuda.cudart().cudaStreamDestroy(handle.value)) == 0
