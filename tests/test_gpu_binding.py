"""What the Python entry points refuse, and with which exception."""
import ctypes

import pytest
import torch

from caif_b200 import native as nv

pytestmark = pytest.mark.gpu


def _int8(out_dim, in_dim):
    return nv.Weight(torch.zeros(max(1, out_dim * in_dim), dtype=torch.int8, device="cuda"), nv.I8, in_dim, out_dim,
                     torch.ones(1, device="cuda"))


@pytest.mark.parametrize("call", [
    lambda x, w, l: nv.rmsnorm_fwd(x, x.float()),
    lambda x, w, l: nv.rmsnorm_bwd(x, x, x.float(), x.float()),
    lambda x, w, l: nv.linear_fwd(w, x),
    lambda x, w, l: nv.linear_dx(w, x),
    lambda x, w, l: nv.linear_fwd_residual(w, x, x),
    lambda x, w, l: nv.linear_fwd_multi([w, w], x),
    lambda x, w, l: nv.linear_concat([w, w], x, workspace=x),
    lambda x, w, l: nv.linear_concat([w, w], x, backward=True, workspace=x),
    lambda x, w, l: nv.lora_linear_fwd(w, l, x),
    lambda x, w, l: nv.lora_linear_bwd(w, l, x, x, x),
])
def test_rows_of_no_elements_are_a_division_by_zero(call):
    x = torch.empty(3, 0, dtype=torch.bfloat16, device="cuda")
    w = _int8(0, 0)
    lora = nv.Lora(torch.zeros(8, 0, dtype=torch.bfloat16, device="cuda"),
                   torch.zeros(0, 8, dtype=torch.bfloat16, device="cuda"), 8.0)
    with pytest.raises(ZeroDivisionError):
        call(x, w, lora)


@pytest.mark.parametrize("call", [
    lambda x, i: nv.moe_topk(x, 2),
    lambda x, i: nv.moe_normalize_rows(x),
    lambda x, i: nv.moe_softmax(x),
    lambda x, i: nv.moe_build_dispatch(i, 4),
    lambda x, i: nv.moe_dispatch(x, i[0], i[0], i[0, 0], 8),
    lambda x, i: nv.moe_combine_bwd_grad_expert(x, i[0], x[0], i[0], i[0, 0], 8),
    lambda x, i: nv.moe_combine_bwd_grad_weights(x, x, i[0], i[0], i[0, 0]),
    lambda x, i: nv.moe_router_bwd(x[0], x, i[0]),
    lambda x, i: nv.quantize_int8_per_channel(x),
])
def test_operands_of_another_rank_than_two_are_refused(call):
    x = torch.rand(2, 4, 8, device="cuda")
    idx = torch.zeros(2, 4, 2, dtype=torch.int32, device="cuda")
    with pytest.raises(ValueError):
        call(x, idx)


def test_exceptions_are_the_ones_torch_raises():
    x = torch.rand(2, 4, device="cuda")
    idx = torch.zeros(2, 1, dtype=torch.int32, device="cuda")
    with pytest.raises(torch.OutOfMemoryError):
        nv.moe_combine(x, idx, x[:, :1].contiguous(), idx, idx.view(-1), 10 ** 12)
    with pytest.raises(IndexError):
        nv.rmsnorm_fwd(torch.zeros((), device="cuda"), torch.ones(1, device="cuda"))
    with pytest.raises(IndexError):
        nv.moe_combine(x.view(-1), idx, x, idx, idx.view(-1), 2)


def test_calls_with_their_result_allocate_nothing_under_a_capture():
    """A graph captured without torch's knowledge: what its launches use must still be theirs when it is replayed."""
    x = torch.randn(1025, 256, device="cuda").bfloat16()
    w = _int8(384, 256)
    w.codes.random_(-127, 128)
    dy = torch.randn(1025, 384, device="cuda").bfloat16()
    y, dx = torch.empty(1025, 384, device="cuda"), torch.empty(1025, 256, device="cuda")
    stream = torch.cuda.Stream()
    rt = ctypes.CDLL(None)
    if not hasattr(rt, "cudaStreamBeginCapture"):
        import glob
        import os
        rt = ctypes.CDLL((glob.glob(os.path.join(os.path.dirname(torch.__file__), "..", "nvidia", "cuda_runtime", "lib",
                                                 "libcudart.so*")) or ["libcudart.so"])[0])
    handle, graph, executable = ctypes.c_void_p(stream.cuda_stream), ctypes.c_void_p(), ctypes.c_void_p()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        for _ in range(2):      # (what is set up once is set up now, and the allocator has blocks to give)
            nv.linear_fwd(w, x, torch.float32, nv.BF16, out=y)
            nv.linear_dx(w, dy, torch.float32, nv.BF16, out=dx)
        torch.cuda.synchronize()
        want = y.clone(), dx.clone()
        torch.cuda.synchronize()
        before = torch.cuda.memory_stats()["allocation.all.allocated"]
        assert rt.cudaStreamBeginCapture(handle, 1) == 0
        nv.linear_fwd(w, x, torch.float32, nv.BF16, out=y)
        nv.linear_dx(w, dy, torch.float32, nv.BF16, out=dx)
        assert rt.cudaStreamEndCapture(handle, ctypes.byref(graph)) == 0
        assert torch.cuda.memory_stats()["allocation.all.allocated"] == before
        assert rt.cudaGraphInstantiate(ctypes.byref(executable), graph, ctypes.c_ulonglong(0)) == 0
        y.zero_()
        dx.zero_()
        assert rt.cudaGraphLaunch(executable, handle) == 0
        torch.cuda.synchronize()
        rt.cudaGraphExecDestroy(executable)
        rt.cudaGraphDestroy(graph)
    assert torch.equal(y, want[0]) and torch.equal(dx, want[1])


def test_no_output_type_is_the_default_one():
    w = _int8(128, 64)
    w.codes.random_(-127, 128)
    x = torch.randn(4, 64, device="cuda").bfloat16()
    want = nv.linear_fwd(w, x)
    assert want.dtype == torch.float32
    assert torch.equal(nv.linear_fwd(w, x, None), want)
    out = torch.empty(4, 128, dtype=torch.bfloat16, device="cuda")
    assert nv.linear_fwd(w, x, None, out=out) is out and torch.equal(out, want.bfloat16())
    assert nv.linear_dx(w, want.bfloat16(), out_dtype=None).dtype == torch.float32
    assert nv.linear_fwd_multi([w, w], x, None).dtype == torch.float32
