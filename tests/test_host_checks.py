"""Arguments that the host side of the operators refuses before anything is launched: the kernels take their sizes from
these, and C++ has no exception for a division by zero."""
import pytest
import torch

DEV = "cuda"
FP8 = torch.float8_e4m3fn


def test_refused_without_a_device():
    from dlblas_b200._C import host
    from dlblas_b200.kernels.fp8 import per_token_group_quant_fp8
    for x in (torch.zeros(2, 128, 4).transpose(1, 2), torch.zeros(128, 4).t(), torch.zeros(())):
        with pytest.raises(AssertionError):
            per_token_group_quant_fp8(x, 128)
    with pytest.raises(AssertionError):
        host().gating_capacity(16, 0, 1.0, 2)


def test_gating_capacity_takes_and_refuses_what_python_would():
    from dlblas_b200.kernels.topk_gating import _capacity
    assert _capacity(64, 8, 1.25, 2) == 10 and _capacity(64, 8, 0.1, 4.7) == 4 and _capacity(64, 8, -3.0, 2) == 2
    assert _capacity(64, 8, -1e30, 2) == 2
    for factor, error in ((float("inf"), OverflowError), (float("-inf"), OverflowError), (1e39, OverflowError),
                          (1e30, OverflowError), (float("nan"), ValueError)):
        with pytest.raises(error):
            _capacity(64, 8, factor, 2)
    with pytest.raises(ValueError):
        _capacity(64, 8, 1.0, float("nan"))


def test_registry_keeps_no_argument():
    import gc
    import weakref

    from dlblas_b200.op_registry import _QUICK_MAX, OpRegistry
    from dlblas_b200.symbolic_var import SymVar
    from dlblas_b200.symbolic_var import Tensor
    r = OpRegistry()

    def impl(x, n):
        return x

    s = SymVar("s")
    r.register("unit_keep", None, (Tensor((s,), dtype=torch.float32, device="cpu"), torch.SymInt), impl, None, impl)
    x = torch.zeros(3)
    gone = weakref.ref(x)
    assert r.get_op("unit_keep", (x, 2)) is r.get_op("unit_keep", (x, 2))
    del x
    gc.collect()
    assert gone() is None
    for n in range(_QUICK_MAX + 5):
        r.get_op("unit_keep", (torch.zeros(3), n))
    assert len(r.quick) <= _QUICK_MAX


def test_host_module_of_another_torch_is_refused_and_rebuilt(monkeypatch):
    from dlblas_b200 import _C, build
    assert _C.host() is not None and _C.host_is_current()
    monkeypatch.setattr(torch, "__version__", torch.__version__ + "1")
    monkeypatch.setattr(_C, "_host_module", None)
    with pytest.raises(RuntimeError, match="another torch"):
        _C.host()
    started = []

    class Started(Exception):
        pass

    def popen(command, **kwargs):
        started.append(command)
        raise Started

    monkeypatch.setattr(build.subprocess, "Popen", popen)
    with pytest.raises(Started):
        build.build()
    assert started[0][0] == "g++" and any(torch.__version__ in word for word in started[0])


@pytest.mark.gpu
def test_refused_on_the_device(monkeypatch):
    from dlblas_b200 import _C, ops
    from dlblas_b200.kernels.fp8_gemm import fp8_gemm
    from dlblas_b200.kernels.grouped_gemm.BF16 import m_grouped_gemm
    from dlblas_b200.kernels.moe_align_block_size import moe_align_block_size
    from dlblas_b200.layers.moe.kernels.blocked_fp8_fused_moe import moe_expert_forward
    host = _C.host()
    x = torch.zeros(4, 256, dtype=torch.bfloat16, device=DEV)
    w13, s13 = torch.zeros(2, 512, 256, device=DEV).to(FP8), torch.ones(2, 4, 2, device=DEV)
    w2, s2 = torch.zeros(2, 256, 256, device=DEV).to(FP8), torch.ones(2, 2, 2, device=DEV)
    w, ids = torch.ones(4, 2, device=DEV), torch.zeros(4, 2, dtype=torch.int64, device=DEV)

    def layer(w2=w2, s2=s2, w=w, ids=ids):
        return moe_expert_forward(x, None, None, w13, s13, w2, s2, w, ids, 2, torch.bfloat16)

    layer()
    step = host.low_latency_forward
    step(x, w, ids, w13, s13, w2, s2, torch.bfloat16)
    with pytest.raises(AssertionError):
        ops.quant_fp8(x, 0)
    with pytest.raises(AssertionError):
        fp8_gemm(torch.zeros(4, 0, device=DEV).to(FP8), torch.zeros(8, 0, device=DEV).to(FP8),
                 torch.zeros(4, 0, device=DEV), torch.zeros(1, 0, device=DEV))
    with pytest.raises(AssertionError):
        moe_align_block_size(torch.zeros(4, dtype=torch.int32, device=DEV), 0, 4, 4)
    for bad in (w2[:1], w2[:, :128], w2[:, :, :128]):           # smaller than what the first GEMM hands over
        with pytest.raises(AssertionError):
            layer(w2=bad.contiguous())
        with pytest.raises(AssertionError):
            step(x, w, ids, w13, s13, bad.contiguous(), s2, torch.bfloat16)
    with pytest.raises(AssertionError):
        layer(s2=s2[:, :1].contiguous())
    for host_side in ({"w": w.cpu()}, {"ids": ids.cpu()}):
        with pytest.raises(RuntimeError, match="CUDA"):
            layer(**host_side)
    with pytest.raises(AssertionError):                          # the layer has converted the weights by then
        step(x, w.half(), ids, w13, s13, w2, s2, torch.bfloat16)
    b = torch.zeros(1, 64, 64, dtype=torch.bfloat16, device=DEV)
    size = torch.tensor([8], device=DEV)
    a = torch.zeros(8, 64, dtype=torch.bfloat16, device=DEV)
    for text, error in (("0", AssertionError), ("wide", ValueError)):
        monkeypatch.setenv("DLBLAS_GEMM16_TILE_ROWS", text)
        with pytest.raises(error):
            m_grouped_gemm(a, b, size)
