"""GPU parity of the frozen-linear forward and dX against the CPU oracle.

Tolerances (max |err| / max |want|, the reference tests' measure):
  fp32 compute 1e-4, bf16/fp16 compute 2e-2 -- the bounds the task states.
Where the kernel consumes exactly the operands the reference would (generic
path), the bound asserted is the tighter 1e-4 in every cell.
"""
import os

import numpy as np
import pytest
import torch

import caif_oracle as orc
from caif_b200 import native as nv
from gpu_util import TORCH_DTYPE, act, best_time, kernels_of, make_weight, max_rel_err, to_dev

pytestmark = pytest.mark.gpu

TOL_F32 = 1e-4
TOL_16 = 2e-2

STORAGES = [orc.F32, orc.F16, orc.BF16, orc.I8, orc.I4]
COMPUTES = [orc.F32, orc.F16, orc.BF16]


def _oracle_w(weight, codes, scales, compute):
    return orc.weight_to_compute(codes, scales, weight.storage, weight.in_dim, weight.out_dim, compute,
                                 weight.scheme, weight.group_size)


@pytest.mark.parametrize("storage", STORAGES)
@pytest.mark.parametrize("compute", COMPUTES)
def test_every_cell_forward_and_dx(storage, compute, monkeypatch):
    """The reference's 3x5 (compute, storage) grid, shapes that hit every tail:
    in/out not multiples of the tile, int4 groups straddling rows."""
    monkeypatch.setenv("CAIFQ_FORCE_PATH", "generic")
    rng = np.random.default_rng(100 + storage * 10 + compute)
    in_dim, out_dim, m = 72, 52, 37
    weight, codes, scales = make_weight(rng, out_dim, in_dim, storage)
    x_np, x = act(rng, m, in_dim, compute if compute != orc.F32 else orc.F32)
    dy_np, dy = act(rng, m, out_dim, compute if compute != orc.F32 else orc.F32)
    wc = _oracle_w(weight, codes, scales, compute)
    y = nv.linear_fwd(weight, x, torch.float32, compute)
    dx = nv.linear_dx(weight, dy, torch.float32, compute)
    assert nv.last_path() == "generic"
    assert y.dtype == torch.float32 and tuple(y.shape) == (m, out_dim)
    assert max_rel_err(y.cpu().numpy(), orc.frozen_linear_forward(x_np, wc, compute)) <= TOL_F32
    assert max_rel_err(dx.cpu().numpy(), orc.frozen_linear_backward(dy_np, wc, compute)) <= TOL_F32


def test_config1_int8_fp32(monkeypatch):
    """in=1024, out=1024, M=64, fp32 compute, int8 per-tensor weights N(0,0.02):
    codes and scale bit-exact, Y and dX within 1e-4 of the host-sgemm path."""
    rng = np.random.default_rng(1234)
    w = (rng.standard_normal((1024, 1024)) * 0.02).astype(np.float32)
    q, s = nv.quantize_int8_per_tensor(to_dev(w))
    oq, os_ = orc.quantize_int8_per_tensor(w)
    assert np.array_equal(q.cpu().numpy(), oq) and np.array_equal(s.cpu().numpy().view(np.uint32), os_.view(np.uint32))
    weight = nv.Weight(q, nv.I8, 1024, 1024, s)
    x_np, x = act(rng, 64, 1024, orc.F32)
    dy_np, dy = act(rng, 64, 1024, orc.F32)
    wc = orc.weight_to_compute(oq, os_, orc.I8, 1024, 1024)
    y = nv.linear_fwd(weight, x)
    dx = nv.linear_dx(weight, dy)
    for exact in (True, False):  # fp64-accumulated loop and OpenBLAS sgemm (the reference's host GEMM)
        assert max_rel_err(y.cpu().numpy(), orc.frozen_linear_forward(x_np, wc, exact=exact)) <= TOL_F32
        assert max_rel_err(dx.cpu().numpy(), orc.frozen_linear_backward(dy_np, wc, exact=exact)) <= TOL_F32


@pytest.mark.parametrize("scheme,with_scales", [(orc.PER_CHANNEL, True), (orc.PER_TENSOR, False)])
def test_int8_per_channel_quirk_and_raw_cast(scheme, with_scales, monkeypatch):
    rng = np.random.default_rng(7)
    in_dim, out_dim, m = 96, 64, 20
    weight, codes, scales = make_weight(rng, out_dim, in_dim, orc.I8, scheme=scheme, with_scales=with_scales)
    x_np, x = act(rng, m, in_dim, orc.F32)
    wc = _oracle_w(weight, codes, scales, orc.F32)
    y = nv.linear_fwd(weight, x)
    assert max_rel_err(y.cpu().numpy(), orc.frozen_linear_forward(x_np, wc)) <= TOL_F32
    mat = nv.weight_materialize(weight)
    assert np.array_equal(mat.cpu().numpy(), wc)


def test_three_d_input_and_output_dtypes():
    rng = np.random.default_rng(8)
    weight, codes, scales = make_weight(rng, 48, 64, orc.I4)
    x_np = orc.round_through(rng.standard_normal((2, 5, 64)).astype(np.float32), orc.BF16)
    x = to_dev(x_np, torch.bfloat16)
    wc = _oracle_w(weight, codes, scales, orc.F32)
    want = orc.frozen_linear_forward(x_np, wc).reshape(2, 5, 48)
    y = nv.linear_fwd(weight, x, torch.float32, orc.F32)
    assert tuple(y.shape) == (2, 5, 48)
    assert max_rel_err(y.cpu().numpy(), want) <= TOL_F32
    yb = nv.linear_fwd(weight, x, torch.bfloat16, orc.F32)
    assert np.array_equal(yb.float().cpu().numpy(), orc.round_through(y.cpu().numpy(), orc.BF16))


def test_errors():
    rng = np.random.default_rng(9)
    weight, _, _ = make_weight(rng, 16, 16, orc.I8)
    x = torch.zeros((4, 16), device="cuda")
    bad = nv.Weight(weight.codes, 9, 16, 16)
    with pytest.raises(nv.CaifqError):
        nv.linear_fwd(bad, x)
    no_scales = nv.Weight(weight.codes, nv.I4, 16, 16, None)
    with pytest.raises(nv.CaifqError):
        nv.linear_fwd(no_scales, x)
    # m == 0 is a no-op
    y = nv.linear_fwd(weight, torch.zeros((0, 16), device="cuda"))
    assert y.shape[0] == 0


# --------------------------------------------------------------------- decode
@pytest.mark.parametrize("m", [1, 4, 16])
def test_decode_int4_config2(m):
    """in=4096, out=14336, int4 g128, bf16 activations: forward, weight-streaming kernel."""
    g = torch.Generator(device="cuda").manual_seed(1235)
    out_dim, in_dim = 14336, 4096
    wf = torch.randn(out_dim * in_dim, generator=g, device="cuda") * 0.02
    p, s = nv.quantize_int4(wf, 128)
    weight = nv.Weight(p, nv.I4, in_dim, out_dim, s, group_size=128)
    x = torch.randn(m, in_dim, generator=g, device="cuda").to(torch.bfloat16)
    y = nv.linear_fwd(weight, x, torch.float32, orc.F32)
    assert nv.last_path() == "decode"
    wc = orc.dequantize_int4(p.cpu().numpy(), s.cpu().view(torch.int16).numpy().view(np.uint16), out_dim * in_dim,
                             128).reshape(out_dim, in_dim)
    want = orc.gemm_nt(x.float().cpu().numpy(), wc)
    assert max_rel_err(y.cpu().numpy(), want) <= TOL_F32
    # bf16 compute: the reference rounds scale*code to bf16 first; bound 2e-2
    yb = nv.linear_fwd(weight, x, torch.float32, orc.BF16)
    want_b = orc.gemm_nt(x.float().cpu().numpy(), orc.round_through(wc, orc.BF16))
    assert max_rel_err(yb.cpu().numpy(), want_b) <= TOL_16
    os.environ["CAIFQ_FORCE_PATH"] = "generic"
    try:
        yg = nv.linear_fwd(weight, x, torch.float32, orc.F32)
        assert nv.last_path() == "generic"
    finally:
        del os.environ["CAIFQ_FORCE_PATH"]
    assert max_rel_err(y.cpu().numpy(), yg.cpu().numpy()) <= TOL_F32


@pytest.mark.parametrize("storage,in_dim,out_dim,m,group", [
    (orc.I4, 1024, 264, 3, 128),     # one chunk per warp, partial... out multiple of 8
    (orc.I4, 2048, 1000, 8, 256),    # group of two chunks
    (orc.I4, 8192, 128, 5, 128),     # four chunks per warp
    (orc.I4, 4096, 100, 16, 128),    # out not a multiple of 8 (ragged last unit), two token tiles
    (orc.I4, 384, 64, 9, 128),       # fewer chunks than warps
    (orc.I8, 4096, 512, 2, 0),
    (orc.I8, 1024, 136, 12, 0),
    (orc.I8, 5120, 64, 7, 0),       # five chunks per warp
    (orc.I8, 320, 72, 1, 0),
    (orc.I4, 1024, 40000, 16, 128),  # more items per CTA than partial sums can be parked: several rounds
    (orc.I4, 1024, 40000, 3, 128),
    (orc.I8, 512, 33000, 9, 0),
])
def test_decode_shapes(storage, in_dim, out_dim, m, group):
    rng = np.random.default_rng(in_dim + out_dim + m)
    weight, codes, scales = make_weight(rng, out_dim, in_dim, storage, group=group or 128)
    x_np, x = act(rng, m, in_dim, orc.BF16)
    y = nv.linear_fwd(weight, x, torch.float32, orc.F32)
    assert nv.last_path() == "decode"
    wc = _oracle_w(weight, codes, scales, orc.F32)
    assert max_rel_err(y.cpu().numpy(), orc.frozen_linear_forward(x_np, wc)) <= TOL_F32


@pytest.mark.parametrize("storage,in_dim,out_dim,m,sd", [
    (orc.I4, 14336, 136, 5, orc.BF16),   # several passes over k, the last one partial
    (orc.I4, 14336, 1000, 16, orc.F32),
    (orc.I8, 14336, 72, 1, orc.BF16),
    (orc.I8, 9280, 264, 16, orc.BF16),   # 145 chunks
    (orc.I4, 8320, 9000, 9, orc.F32),    # passes over k and several rounds of parked sums
    (orc.I4, 2048, 24, 8, orc.F16),      # eight-warp form, fewer rows than SMs
])
def test_decode_long_rows_and_the_residual_add(storage, in_dim, out_dim, m, sd):
    rng = np.random.default_rng(in_dim + out_dim + m)
    weight, codes, scales = make_weight(rng, out_dim, in_dim, storage)
    wc = _oracle_w(weight, codes, scales, orc.F32)
    x_np, x = act(rng, m, in_dim, orc.BF16)
    res_np, res = act(rng, m, out_dim, sd)
    want = orc.frozen_linear_forward(x_np, wc)
    y = nv.linear_fwd(weight, x, torch.float32, orc.F32)
    assert nv.last_path() == "decode"
    assert max_rel_err(y.cpu().numpy(), want) <= TOL_F32
    got = nv.linear_fwd_residual(weight, x, res.clone(), orc.F32)
    assert nv.last_path() == "decode"
    # the same bits as the product in the stream's dtype followed by an add there
    sep = nv.linear_fwd(weight, x, TORCH_DTYPE[sd], orc.F32)
    assert torch.equal(got, (sep.float() + res.float()).to(TORCH_DTYPE[sd]))


@pytest.mark.parametrize("storage", [orc.I4, orc.I8])
@pytest.mark.parametrize("in_dim,out_dim,m", [(1024, 1024, 4), (4096, 1000, 9), (14336, 520, 1), (14336, 136, 16), (9216, 72, 5)])
def test_decode_is_as_close_to_64_bits_as_the_fma_kernel(storage, in_dim, out_dim, m, monkeypatch):
    rng = np.random.default_rng(in_dim + out_dim + m)
    weight, codes, scales = make_weight(rng, out_dim, in_dim, storage)
    w = torch.from_numpy(_oracle_w(weight, codes, scales, orc.F32)).double().cuda()
    x = torch.from_numpy(rng.standard_normal((m, in_dim)).astype(np.float32)).cuda().bfloat16()
    want = x.double() @ w.T
    y = nv.linear_fwd(weight, x, torch.float32, orc.F32)
    assert nv.last_path() == "decode"
    monkeypatch.setenv("CAIFQ_FORCE_PATH", "generic")
    fma = nv.linear_fwd(weight, x, torch.float32, orc.F32)
    assert (y.double() - want).norm() <= 1.02 * (fma.double() - want).norm()


@pytest.mark.parametrize("storage", [orc.I4, orc.I8])
@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan"), 3.0e38])
@pytest.mark.parametrize("in_dim,m", [(512, 1), (4096, 3), (14336, 12)])
def test_decode_infinities_and_nans_reach_only_their_token(storage, value, in_dim, m, monkeypatch):
    """An infinity times a weight is an infinity of that sign (NaN for a zero), as in a plain fp32 product; and large values
    overflow only where the product itself does.  Three layers in one launch."""
    rng = np.random.default_rng(in_dim + m)
    ws = [make_weight(rng, o, in_dim, storage)[0] for o in (264, 64, 40)]
    x = torch.from_numpy(rng.standard_normal((m, in_dim)).astype(np.float32)).cuda().bfloat16()
    clean = nv.linear_fwd_multi(ws, x, torch.float32, orc.F32)
    x[m // 2, 77] = value
    x[m // 2, in_dim - 1] = value
    y = nv.linear_fwd_multi(ws, x, torch.float32, orc.F32)
    one = nv.linear_fwd(ws[0], x, torch.float32, orc.F32)
    assert nv.last_path() == "decode"
    monkeypatch.setenv("CAIFQ_FORCE_PATH", "generic")
    want = torch.cat([nv.linear_fwd(w, x, torch.float32, orc.F32) for w in ws], 1)
    others = [t for t in range(m) if t != m // 2]
    assert torch.equal(y[others], clean[others]) and torch.equal(one[others], y[others, :264])
    for got, ref in ((y[m // 2], want[m // 2]), (one[m // 2], want[m // 2, :264])):
        assert torch.equal(torch.isnan(got), torch.isnan(ref))
        live = ~torch.isnan(ref)
        assert torch.equal(torch.isinf(got[live]), torch.isinf(ref[live]))
        if live.any():
            # (two huge terms may cancel: the bound is that of the terms, not of the sum)
            scale = ref[live].abs()[torch.isfinite(ref[live])].max() if torch.isfinite(ref[live]).any() else 0.0
            same = got[live] == ref[live]
            assert (same | ((got[live] - ref[live]).abs() <= 1e-5 * scale)).all()


def test_decode_int8_without_scales_and_bf16_out():
    rng = np.random.default_rng(77)
    weight, codes, scales = make_weight(rng, 256, 2048, orc.I8, with_scales=False)
    x_np, x = act(rng, 4, 2048, orc.BF16)
    y = nv.linear_fwd(weight, x, torch.bfloat16, orc.F32)
    assert nv.last_path() == "decode"
    want = orc.frozen_linear_forward(x_np, _oracle_w(weight, codes, scales, orc.F32))
    assert max_rel_err(y.float().cpu().numpy(), want) <= 1e-2  # bf16 output rounding


def test_decode_forward_gather_into_several_buffers():
    """The fused gather: two shards of a wider layer write their slices, at their column offsets,
    into two result buffers each (on one GPU both 'ranks' are local buffers); every buffer ends up
    holding the full-width result, equal to the plain forward of each shard bit for bit."""
    rng = np.random.default_rng(2024)
    in_dim, shard, m = 1024, 520, 5
    shards = [make_weight(rng, shard, in_dim, orc.I4)[0] for _ in range(2)]
    _, x = act(rng, m, in_dim, orc.BF16)
    bufs = [torch.full((m, 2 * shard), float("nan"), device="cuda") for _ in range(2)]
    ptrs = [b.data_ptr() for b in bufs]
    for r, w in enumerate(shards):
        nv.linear_fwd_gather(w, x, ptrs, 2 * shard, r * shard, orc.F32, orc.F32)
        assert nv.last_path() == "decode"
    torch.cuda.synchronize()
    want = torch.cat([nv.linear_fwd(w, x, torch.float32, orc.F32) for w in shards], dim=1)
    for b in bufs:
        assert torch.equal(b, want)
    # shapes the few-token kernel does not take are refused, not silently run elsewhere
    _, x_many = act(rng, 64, in_dim, orc.BF16)
    big = torch.empty((64, 2 * shard), device="cuda")
    with pytest.raises(nv.CaifqError):
        nv.linear_fwd_gather(shards[0], x_many, [big.data_ptr()], 2 * shard, 0, orc.F32, orc.F32)
    with pytest.raises(nv.CaifqError):   # the slice must fit the row pitch
        nv.linear_fwd_gather(shards[0], x, ptrs, shard, shard, orc.F32, orc.F32)


# ------------------------------------------------------------ tensor-core path
def _umma_case(storage, compute, m, in_dim, out_dim, seed, group=128):
    rng = np.random.default_rng(seed)
    weight, codes, scales = make_weight(rng, out_dim, in_dim, storage, group=group)
    x_np, x = act(rng, m, in_dim, orc.BF16)
    dy_np, dy = act(rng, m, out_dim, orc.BF16)
    wc = _oracle_w(weight, codes, scales, compute)
    return weight, wc, x_np, x, dy_np, dy


@pytest.mark.parametrize("storage,compute,tol", [
    (orc.I8, orc.F32, TOL_F32),     # exact products: holds the fp32 bound
    (orc.I8, orc.BF16, TOL_16),
    (orc.I4, orc.BF16, TOL_16),
    (orc.I4, orc.F32, TOL_F32),     # scale*code as two bf16 terms: holds the fp32 bound
    (orc.BF16, orc.F32, TOL_F32),
])
@pytest.mark.parametrize("m,in_dim,out_dim", [(300, 512, 384), (256, 128, 128), (77, 1408, 2048), (1000, 2048, 1408),
                                             (17, 256, 384)])
def test_umma_forward_and_dx(storage, compute, tol, m, in_dim, out_dim):
    weight, wc, x_np, x, dy_np, dy = _umma_case(storage, compute, m, in_dim, out_dim, 500 + storage + m)
    y = nv.linear_fwd(weight, x, torch.float32, compute)
    assert nv.last_path() == "umma"
    dx = nv.linear_dx(weight, dy, torch.float32, compute)
    assert nv.last_path() == "umma"
    assert nv.lib().caifq_device_status() == 0
    assert max_rel_err(y.cpu().numpy(), orc.frozen_linear_forward(x_np, wc, compute)) <= tol
    assert max_rel_err(dx.cpu().numpy(), orc.frozen_linear_backward(dy_np, wc, compute)) <= tol
    if storage == orc.I4 and compute == orc.BF16:
        # the operand is code * bf16(scale), the reference's is bf16(code * scale): they differ by the bf16
        # rounding of the fp16 scale, a small fraction of the bound
        assert max_rel_err(y.cpu().numpy(), orc.frozen_linear_forward(x_np, wc, compute)) <= 4e-3


def test_umma_int4_group_size_that_is_not_a_power_of_two():
    weight, wc, x_np, x, dy_np, dy = _umma_case(orc.I4, orc.BF16, 64, 384, 256, 4321, group=96)
    y = nv.linear_fwd(weight, x, torch.float32, orc.BF16)
    assert nv.last_path() == "umma"
    dx = nv.linear_dx(weight, dy, torch.float32, orc.BF16)
    assert max_rel_err(y.cpu().numpy(), orc.frozen_linear_forward(x_np, wc, orc.BF16)) <= 4e-3
    assert max_rel_err(dx.cpu().numpy(), orc.frozen_linear_backward(dy_np, wc, orc.BF16)) <= 4e-3


def test_umma_bf16_output_and_accumulate_epilogue():
    weight, wc, x_np, x, dy_np, dy = _umma_case(orc.I8, orc.F32, 200, 256, 256, 42)
    yb = nv.linear_fwd(weight, x, torch.bfloat16, orc.F32)
    assert nv.last_path() == "umma"
    want = orc.round_through(orc.frozen_linear_forward(x_np, wc), orc.BF16)
    assert max_rel_err(yb.float().cpu().numpy(), want) <= 1e-2


def test_umma_config3_shape_matches_generic_and_oracle_rows(monkeypatch):
    """4096 -> 4096 int8 per-tensor, M = 8192 bf16 tokens (the training config): the tensor-core
    path against the generic path on the whole output and against the oracle on 16 rows."""
    g = torch.Generator(device="cuda").manual_seed(1236)
    dim, m = 4096, 8192
    wf = torch.randn(dim * dim, generator=g, device="cuda") * 0.02
    q, s = nv.quantize_int8_per_tensor(wf)
    weight = nv.Weight(q.view(dim, dim), nv.I8, dim, dim, s)
    x = torch.randn(m, dim, generator=g, device="cuda").to(torch.bfloat16)
    dy = torch.randn(m, dim, generator=g, device="cuda").to(torch.bfloat16)
    y = nv.linear_fwd(weight, x, torch.float32, orc.F32)
    assert nv.last_path() == "umma"
    dx = nv.linear_dx(weight, dy, torch.float32, orc.F32)
    assert nv.lib().caifq_device_status() == 0
    monkeypatch.setenv("CAIFQ_FORCE_PATH", "generic")
    yg = nv.linear_fwd(weight, x, torch.float32, orc.F32)
    dxg = nv.linear_dx(weight, dy, torch.float32, orc.F32)
    assert nv.last_path() == "generic"
    assert float((y - yg).abs().max() / yg.abs().max()) <= TOL_F32
    assert float((dx - dxg).abs().max() / dxg.abs().max()) <= TOL_F32
    rows = torch.arange(0, m, m // 16, device="cuda")
    wc = orc.dequantize_int8_per_tensor(q.cpu().numpy().reshape(dim, dim), s.cpu().numpy())
    want = orc.gemm_nt(x[rows].float().cpu().numpy(), wc)
    assert max_rel_err(y[rows].cpu().numpy(), want) <= TOL_F32
    want_dx = orc.gemm_nn(dy[rows].float().cpu().numpy(), wc)
    assert max_rel_err(dx[rows].cpu().numpy(), want_dx) <= TOL_F32


def test_decode_misaligned_activations_fall_back():
    """bf16 activations that do not start on a 16-byte boundary (a row slice of a larger tensor)
    are a legal call: the few-token kernel declines them and another kernel family answers."""
    rng = np.random.default_rng(77)
    weight, codes, scales = make_weight(rng, 136, 1024, orc.I8)
    x_np, x = act(rng, 4, 1024, orc.BF16)
    big = torch.zeros(4 * 1024 + 8, dtype=torch.bfloat16, device="cuda")
    shifted = big[1:1 + 4 * 1024].view(4, 1024)     # starts 2 bytes past an aligned address
    shifted.copy_(x)
    assert shifted.data_ptr() % 16 == 2
    y = nv.linear_fwd(weight, shifted, torch.float32, orc.F32)
    assert nv.last_path() != "decode"
    wc = _oracle_w(weight, codes, scales, orc.F32)
    assert max_rel_err(y.cpu().numpy(), orc.frozen_linear_forward(x_np, wc)) <= TOL_F32


def test_decode_wait_that_runs_out_raises_the_flag_and_returns():
    """The library's self-test of its bounded waits: the next few-token launch announces bytes that
    never arrive, with a short wait limit.  The kernel must return (no hang, no fault), the status
    word must report the few-token kernel (bit 0), and the next call must be healthy again."""
    import time

    rng = np.random.default_rng(78)
    weight, codes, scales = make_weight(rng, 1024, 4096, orc.I4)
    x_np, x = act(rng, 4, 4096, orc.BF16)
    wc = _oracle_w(weight, codes, scales, orc.F32)
    want = orc.frozen_linear_forward(x_np, wc)
    y = nv.linear_fwd(weight, x, torch.float32, orc.F32)
    assert nv.last_path() == "decode"
    assert nv.lib().caifq_device_status() == 0
    nv.lib().caifq_selftest_stall_next_decode()
    t0 = time.time()
    nv.linear_fwd(weight, x, torch.float32, orc.F32)
    torch.cuda.synchronize()
    assert time.time() - t0 < 1.0
    assert nv.lib().caifq_device_status() & 1
    y = nv.linear_fwd(weight, x, torch.float32, orc.F32)
    assert nv.lib().caifq_device_status() == 0
    assert max_rel_err(y.cpu().numpy(), want) <= TOL_F32


def test_umma_wait_that_runs_out_raises_the_flag_and_returns():
    """The tensor-core kernel's give-up path: one activation tile announces bytes that never arrive.  The
    first wait that runs out makes every later wait of the CTA return at once, so the kernel ends within
    about one (short, self-test) limit instead of one limit per remaining wait; its tensor memory is
    released (the next launch can allocate it) and the status word reports bit 1."""
    import time

    weight, wc, x_np, x, dy_np, dy = _umma_case(orc.I8, orc.BF16, 512, 1024, 1024, 4242)
    y = nv.linear_fwd(weight, x, torch.float32, orc.BF16)
    assert nv.last_path() == "umma"
    assert nv.lib().caifq_device_status() == 0
    nv.lib().caifq_selftest_stall_next_umma()
    t0 = time.time()
    nv.linear_fwd(weight, x, torch.float32, orc.BF16)
    torch.cuda.synchronize()
    assert time.time() - t0 < 1.0
    assert nv.lib().caifq_device_status() & 2
    y2 = nv.linear_fwd(weight, x, torch.float32, orc.BF16)
    dx = nv.linear_dx(weight, dy, torch.float32, orc.BF16)
    assert nv.lib().caifq_device_status() == 0
    assert torch.equal(y, y2)
    assert max_rel_err(dx.cpu().numpy(), orc.frozen_linear_backward(dy_np, wc, orc.BF16)) <= TOL_16


@pytest.mark.parametrize("storage,compute,tol", [
    (orc.I8, orc.BF16, TOL_16),
    (orc.I8, orc.F32, TOL_F32),
    (orc.I4, orc.BF16, TOL_16),
    (orc.I4, orc.F32, TOL_F32),
    (orc.BF16, orc.F32, TOL_F32),
])
def test_umma_cta_pairs_equal_single_ctas(storage, compute, tol, monkeypatch):
    """256-wide tiles on CTA pairs (one `cta_group::2` MMA of 256 rows over two SMs, operands staged half
    and half, barriers of the leader CTA signalled across the cluster) accumulate every output element
    over k in the same order as a single CTA's two 128-row MMAs: the results are bit-equal, for the
    forward pass (K-major weights) and dX (MN-major), and sampled rows hold the oracle's bound."""
    m, in_dim, out_dim = 10007, 512, 1024
    weight, wc, x_np, x, dy_np, dy = _umma_case(storage, compute, m, in_dim, out_dim, 9100 + storage)
    monkeypatch.setenv("CAIFQ_UMMA_PAIR", "0")
    y1 = nv.linear_fwd(weight, x, torch.float32, compute)
    dx1 = nv.linear_dx(weight, dy, torch.bfloat16, compute)
    monkeypatch.setenv("CAIFQ_UMMA_PAIR", "1")
    y2 = nv.linear_fwd(weight, x, torch.float32, compute)
    assert nv.last_path() == "umma"
    dx2 = nv.linear_dx(weight, dy, torch.bfloat16, compute)
    assert nv.lib().caifq_device_status() == 0
    assert nv.lib().caifq_umma_pair_capacity() >= 1
    assert torch.equal(y1, y2)
    assert torch.equal(dx1, dx2)
    rows = np.r_[0:8, 5000:5008, m - 8:m]
    assert max_rel_err(y2[rows].cpu().numpy(), orc.frozen_linear_forward(x_np[rows], wc, compute)) <= tol
    want_dx = orc.round_through(orc.frozen_linear_backward(dy_np[rows], wc, compute), orc.BF16)
    assert max_rel_err(dx2[rows].float().cpu().numpy(), want_dx) <= max(tol, 1e-2)   # one bf16 rounding of the output


def test_umma_cta_pair_wait_that_runs_out_returns(monkeypatch):
    """The give-up path with CTA pairs: the leader's wait runs out, both CTAs of every pair leave their
    loops, meet at the cluster barrier, release their tensor memory, and the next launch is correct."""
    import time

    monkeypatch.setenv("CAIFQ_UMMA_PAIR", "1")
    weight, wc, x_np, x, dy_np, dy = _umma_case(orc.I8, orc.BF16, 10007, 512, 1024, 4243)
    y = nv.linear_fwd(weight, x, torch.float32, orc.BF16)
    assert nv.lib().caifq_device_status() == 0
    nv.lib().caifq_selftest_stall_next_umma()
    t0 = time.time()
    nv.linear_fwd(weight, x, torch.float32, orc.BF16)
    torch.cuda.synchronize()
    assert time.time() - t0 < 1.0
    assert nv.lib().caifq_device_status() & 2
    y2 = nv.linear_fwd(weight, x, torch.float32, orc.BF16)
    assert nv.lib().caifq_device_status() == 0
    assert torch.equal(y, y2)


@pytest.mark.parametrize("storage,outs,m", [
    (orc.I4, (4096, 1024, 1024), 1),        # q, k, v of the Llama-shaped block
    (orc.I4, (4096, 1024, 1024), 16),
    (orc.I4, (1416, 1032, 520), 4),         # boundaries that are multiples of 8 but not of 16: items straddle layers
    (orc.I8, (1416, 1032, 520, 264), 9),    # int8: every layer has its own per-tensor scale
    (orc.I4, (14336, 14336), 4),            # gate, up
])
def test_decode_several_layers_that_share_the_input_in_one_launch(storage, outs, m):
    """caifq_linear_fwd_multi: one persistent launch streams the code matrices of all layers; every output
    has the bits the layer's own caifq_linear_fwd call gives, and holds the oracle's bound."""
    in_dim = 4096 if outs[0] >= 4096 else 1024
    rng = np.random.default_rng(7700 + sum(outs) + m)
    ws, wcs = [], []
    for o in outs:
        w, codes, scales = make_weight(rng, o, in_dim, storage)
        ws.append(w)
        wcs.append(_oracle_w(w, codes, scales, orc.F32))
    x_np, x = act(rng, m, in_dim, orc.BF16)
    y = nv.linear_fwd_multi(ws, x, torch.float32, orc.F32)
    assert nv.last_path() == "decode"
    assert nv.lib().caifq_device_status() == 0
    col = 0
    for w, wc in zip(ws, wcs):
        single = nv.linear_fwd(w, x, torch.float32, orc.F32)
        assert nv.last_path() == "decode"
        assert torch.equal(y[:, col:col + w.out_dim], single)
        assert max_rel_err(single.cpu().numpy(), orc.frozen_linear_forward(x_np, wc, orc.F32)) <= TOL_F32
        col += w.out_dim
    # refused, not mis-computed: a layer (not the last) whose row count is not a multiple of 8, and many tokens
    odd = [make_weight(rng, 1028, in_dim, storage)[0], ws[0]]
    with pytest.raises(nv.CaifqError):
        nv.linear_fwd_multi(odd, x, torch.float32, orc.F32)
    with pytest.raises(nv.CaifqError):
        nv.linear_fwd_multi(ws, act(rng, 32, in_dim, orc.BF16)[1], torch.float32, orc.F32)


@pytest.mark.parametrize("storage,compute,sd,m", [
    (orc.I4, orc.BF16, orc.BF16, 300),    # tensor-core path, bf16 residual stream
    (orc.I8, orc.F32, orc.F32, 77),       # tensor-core path, fp32 stream
    (orc.I4, orc.BF16, orc.BF16, 4),      # few tokens: the accumulate epilogue lives on the other kernels
    (orc.F16, orc.F16, orc.F16, 20),      # generic kernel
])
def test_forward_with_the_residual_add_in_the_epilogue(storage, compute, sd, m):
    """caifq_linear_fwd_residual: the block's x = x + sub_out with sub_out the projection's output cast to
    the stream's dtype, computed in the product's epilogue: round(round(y) + residual)."""
    in_dim, out_dim = 512, 384
    rng = np.random.default_rng(8800 + storage + m)
    weight, codes, scales = make_weight(rng, out_dim, in_dim, storage)
    wc = _oracle_w(weight, codes, scales, compute)
    x_np, x = act(rng, m, in_dim, sd)
    res_np, res = act(rng, m, out_dim, sd)
    got = nv.linear_fwd_residual(weight, x, res.clone(), compute)
    y = orc.round_through(orc.frozen_linear_forward(x_np, wc, compute), sd)
    want = orc.round_through(y + res_np, sd)
    tol = TOL_F32 if compute == orc.F32 else TOL_16
    assert max_rel_err(got.float().cpu().numpy(), want) <= tol
    # the same bits as the separate product followed by an add in the stream's dtype
    sep = nv.linear_fwd(weight, x, TORCH_DTYPE[sd], compute)
    if nv.last_path() != "decode":     # (the few-token kernel sums in another order than the kernel that accumulates)
        assert torch.equal(got, (sep.float() + res.float()).to(TORCH_DTYPE[sd]))


@pytest.mark.parametrize("storage", [orc.I4, orc.I8, orc.BF16])
def test_layers_sharing_their_input_as_one_product_over_concatenated_weights(storage):
    """caifq_linear_fwd_concat / caifq_linear_dx_concat on the attention shapes of the Llama-like config scaled
    down (q of 1024, k and v of 256 features over 512 inputs, 4099 tokens): the columns of every layer hold what
    the oracle gives for that layer alone (weights as bf16 compute sees them), dX the sum over the layers, and
    both agree with the per-layer calls."""
    rng = np.random.default_rng(700 + storage)
    in_dim, outs, m = 512, (1024, 256, 256), 4099
    layers = [make_weight(rng, o, in_dim, storage, std=0.05) for o in outs]
    ws = [l[0] for l in layers]
    wc = [orc.weight_to_compute(l[1], l[2], storage, in_dim, o, orc.BF16, l[0].scheme, l[0].group_size)
          for l, o in zip(layers, outs)]
    x_np, x = act(rng, m, in_dim, orc.BF16)
    dy_np, dy = act(rng, m, sum(outs), orc.BF16)
    y = nv.linear_concat(ws, x, out_dtype=torch.float32)
    assert nv.last_path() == "umma"
    dx = nv.linear_concat(ws, dy, backward=True, out_dtype=torch.float32)
    assert nv.lib().caifq_device_status() == 0
    rows = np.r_[0:8, 2000:2008, m - 8:m]
    col = 0
    want_dx = np.zeros((rows.size, in_dim), np.float64)
    per_layer_dx = torch.zeros(m, in_dim, device="cuda")
    for w, c, o in zip(ws, wc, outs):
        want = orc.frozen_linear_forward(x_np[rows], c, orc.BF16)
        assert max_rel_err(y[rows, col:col + o].cpu().numpy(), want) <= TOL_16
        alone = nv.linear_fwd(w, x, torch.float32, orc.BF16)
        assert max_rel_err(y[:, col:col + o].cpu().numpy(), alone.cpu().numpy()) <= TOL_16
        want_dx += orc.frozen_linear_backward(dy_np[rows, col:col + o], c, orc.BF16)
        per_layer_dx += nv.linear_dx(w, dy[:, col:col + o].contiguous(), torch.float32, orc.BF16)
        col += o
    assert max_rel_err(dx[rows].cpu().numpy(), want_dx) <= TOL_16
    assert max_rel_err(dx.cpu().numpy(), per_layer_dx.cpu().numpy()) <= TOL_16
    # refusals: fp32 compute has no bf16 operand; a short workspace
    arr = nv._weight_array(ws)
    y2 = torch.empty(m, sum(outs), device="cuda")
    scratch = torch.empty(1024, dtype=torch.uint8, device="cuda")
    rc = nv.lib().caifq_linear_fwd_concat(arr, 3, nv._ptr(x), nv.BF16, m, nv._ptr(y2), nv.F32, nv.BF16, nv._ptr(scratch),
                                          1024, nv._stream())
    assert rc == 1 and b"workspace" in nv.lib().caifq_last_error()
    big = torch.empty(nv.lib().caifq_linear_concat_workspace_bytes(arr, 3), dtype=torch.uint8, device="cuda")
    rc = nv.lib().caifq_linear_fwd_concat(arr, 3, nv._ptr(x), nv.BF16, m, nv._ptr(y2), nv.F32, nv.F32, nv._ptr(big),
                                          big.numel(), nv._stream())
    assert rc == 1 and b"BF16" in nv.lib().caifq_last_error()


@pytest.mark.parametrize("m,in_dim,out_dim,sd", [
    (1, 2048, 64, orc.F32), (16, 2048, 20, orc.F32), (17, 96, 8, orc.BF16), (64, 1056, 96, orc.F16), (9, 1056, 4096, orc.F16),
    (40, 32, 33, orc.F32),     # fewer k-steps than warps, a ragged last column tile
])
def test_few_rows_on_a_bf16_weight(m, in_dim, out_dim, sd):
    rng = np.random.default_rng(m + in_dim + out_dim)
    weight, codes, _ = make_weight(rng, out_dim, in_dim, orc.BF16)
    x_np, x = act(rng, m, in_dim, orc.BF16)
    res_np, res = act(rng, m, out_dim, sd)
    want = orc.frozen_linear_forward(x_np, _oracle_w(weight, codes, None, orc.F32))
    y = nv.linear_fwd(weight, x, torch.float32, orc.F32)
    assert nv.last_path() == "decode"
    assert max_rel_err(y.cpu().numpy(), want) <= TOL_F32
    got = nv.linear_fwd_residual(weight, x, res.clone(), orc.F32)
    sep = nv.linear_fwd(weight, x, TORCH_DTYPE[sd], orc.F32)
    assert torch.equal(got, (sep.float() + res.float()).to(TORCH_DTYPE[sd]))


@pytest.mark.parametrize("compute", [orc.F32, orc.BF16])
@pytest.mark.parametrize("m,in_dim,out_dim", [
    (65, 2048, 64), (300, 512, 96), (700, 256, 160), (17, 14336, 8),
    (2500, 4096, 33),      # more rows than a wave of CTAs, a ragged last column tile
    (16, 14336, 4096), (257, 8192, 4104),
])
def test_bf16_weight_outside_the_tensor_core_tiles_keeps_fp32_precision(m, in_dim, out_dim, compute, monkeypatch):
    """Products of bf16 values are exact in fp32 and the sums are fp32's: no further from 64 bits than the fp32-FMA kernel."""
    g = torch.Generator(device="cuda").manual_seed(m + in_dim + out_dim)
    w = (torch.randn(out_dim, in_dim, generator=g, device="cuda") / in_dim ** 0.5).bfloat16()
    x = torch.randn(m, in_dim, generator=g, device="cuda").bfloat16()
    weight = nv.Weight(w, nv.BF16, in_dim, out_dim)
    want = x.double() @ w.double().T
    y = nv.linear_fwd(weight, x, torch.float32, compute)
    assert nv.last_path() == "decode"
    monkeypatch.setenv("CAIFQ_FORCE_PATH", "generic")
    fma = nv.linear_fwd(weight, x, torch.float32, compute)
    assert nv.last_path() == "generic"
    assert (y.double() - want).norm() <= 1.02 * (fma.double() - want).norm()


def test_layers_over_ragged_widths_are_refused_as_one_product():
    """The concatenated product needs whole 128-column tiles: 96 + 64 output features are not."""
    ws = [make_weight(np.random.default_rng(o), o, 256, orc.I8)[0] for o in (96, 64)]
    with pytest.raises(nv.CaifqError, match="tensor-core path"):
        nv.linear_concat(ws, torch.zeros(64, 256, dtype=torch.bfloat16, device="cuda"))


@pytest.mark.parametrize("offset", [0, 8])
def test_layers_as_one_product_take_what_one_scale_inside_the_values_can_hold(offset):
    """Codes that start on 16 bytes or on 8: the same values, and the same refusals."""
    codes = torch.randint(-127, 128, (offset + 128 * 256,), dtype=torch.int8, device="cuda")[offset:]
    scales = torch.rand(128, device="cuda") * 0.01 + 0.01
    x = torch.randn(64, 256, device="cuda").bfloat16()
    good = nv.Weight(codes, nv.I8, 256, 128, scales[:1].contiguous())
    want = x.double() @ (codes.view(128, 256).float() * scales[0]).bfloat16().double().T
    y = nv.linear_concat([good, good], x, out_dtype=torch.float32)
    assert (y.double() - torch.cat([want, want], 1)).norm() <= 1e-5 * (2 ** 0.5) * want.norm()
    for bad in (nv.Weight(codes, nv.I8, 256, 128), nv.Weight(codes, nv.I8, 256, 128, scales, scheme=nv.PER_CHANNEL)):
        with pytest.raises(nv.CaifqError, match="per-tensor scale"):
            nv.linear_concat([bad, bad], x)


@pytest.mark.parametrize("storage,group", [(orc.I8, 128), (orc.I4, 128), (orc.I4, 64)])
@pytest.mark.parametrize("m,in_dim,out_dim", [(1, 1024, 128), (64, 1024, 1024), (65, 128, 64), (130, 64, 192), (1000, 384, 2048)])
def test_fp32_activations_on_the_tensor_core(storage, group, m, in_dim, out_dim):
    """Three bf16 terms per activation: tile edges in m, one block of k, every split of k over a cluster.  Held to an
    fp32 GEMM's own error, far below the layer's bound."""
    if storage == orc.I4 and in_dim % group:
        pytest.skip("groups straddle rows: the generic kernel's")
    rng = np.random.default_rng(m + in_dim + out_dim + group)
    weight, codes, scales = make_weight(rng, out_dim, in_dim, storage, group=group)
    wc = _oracle_w(weight, codes, scales, orc.F32)
    x_np, x = act(rng, m, in_dim, orc.F32)
    dy_np, dy = act(rng, m, out_dim, orc.F32)
    y = nv.linear_fwd(weight, x)
    assert nv.last_path() == "umma"
    want = x_np.astype(np.float64) @ wc.astype(np.float64).T
    assert np.linalg.norm(y.cpu().numpy() - want) <= 1e-6 * np.linalg.norm(want)
    dx = nv.linear_dx(weight, dy)
    assert nv.last_path() == "umma"
    want = dy_np.astype(np.float64) @ wc.astype(np.float64)
    assert np.linalg.norm(dx.cpu().numpy() - want) <= 1e-6 * np.linalg.norm(want)
    res_np, res = act(rng, m, out_dim, orc.F32)
    assert torch.equal(nv.linear_fwd_residual(weight, x, res.clone()), y + res)


@pytest.mark.parametrize("storage,group", [(orc.I8, 128), (orc.I4, 128), (orc.I4, 64)])
@pytest.mark.parametrize("m,in_dim,out_dim", [(1, 64, 64), (3, 192, 320), (16, 1152, 64), (16, 128, 1088), (17, 64, 128),
                                              (2, 4096, 640)])
def test_fp32_activations_of_few_rows(storage, group, m, in_dim, out_dim):
    """The 16-row tile takes 128 of k at a time: k that ends half way through them (or never gets there), two scale groups
    in one of them, k over clusters; 17 rows are the other tile's.  Bound: as above, an fp32 GEMM's own error."""
    if storage == orc.I4 and in_dim % group:
        pytest.skip("groups straddle rows: the generic kernel's")
    rng = np.random.default_rng(7 * m + in_dim + out_dim + group)
    weight, codes, scales = make_weight(rng, out_dim, in_dim, storage, group=group)
    wc = _oracle_w(weight, codes, scales, orc.F32).astype(np.float64)
    x_np, x = act(rng, m, in_dim, orc.F32)
    dy_np, dy = act(rng, m, out_dim, orc.F32)
    for got, want in ((nv.linear_fwd(weight, x), x_np.astype(np.float64) @ wc.T),
                      (nv.linear_dx(weight, dy), dy_np.astype(np.float64) @ wc)):
        assert nv.last_path() == "umma"
        assert np.linalg.norm(got.cpu().numpy() - want) <= 1e-6 * np.linalg.norm(want)


@pytest.mark.parametrize("bits", [0x7FC00000, 0x7F800001, 0xFF80FFFF, 0x7F800000, 0xFF800000])
def test_fp32_activations_that_are_not_finite(bits, monkeypatch):
    """A NaN of any payload stays one; an infinity gives what the fp32-FMA kernel gives; other rows keep their bits."""
    rng = np.random.default_rng(99)
    weight, codes, scales = make_weight(rng, 192, 128, orc.I8)
    for f, width in ((nv.linear_fwd, 128), (nv.linear_dx, 192)):
        x = torch.randn(5, width, device="cuda")
        clean = f(weight, x)
        x.view(torch.int32)[2, 9] = bits - (1 << 32) if bits >= 1 << 31 else bits
        y = f(weight, x)
        assert nv.last_path() == "umma"
        monkeypatch.setenv("CAIFQ_FORCE_PATH", "generic")
        want = f(weight, x)
        monkeypatch.delenv("CAIFQ_FORCE_PATH")
        rest = [0, 1, 3, 4]
        assert torch.equal(y[rest], clean[rest])
        assert torch.equal(torch.isnan(y[2]), torch.isnan(want[2]))
        live = ~torch.isnan(want[2])
        assert torch.equal(y[2][live], want[2][live])


@pytest.mark.parametrize("storage,compute,group", [(orc.I8, orc.BF16, 128), (orc.I4, orc.BF16, 32), (orc.I4, orc.F32, 128)])
@pytest.mark.parametrize("m,in_dim,out_dim", [
    (17, 128, 128),        # one stage of k
    (17, 64, 192512),      # half a stage of k, more tiles a CTA than there are barriers for them
    (33, 320, 128),        # an odd 64 k at the end, a box of tokens with one row
    (64, 384, 19072),      # more tiles than SMs: both accumulator sets, tiles of one unit
    (128, 2048, 256),      # k over clusters of eight
    (129, 1408, 640),      # clusters of four; one accumulator set, or two tiles of tokens
    (257, 1152, 6272), (512, 4096, 128), (768, 256, 384),
])
def test_tens_to_hundreds_of_tokens(storage, compute, group, m, in_dim, out_dim):
    if in_dim % group:
        pytest.skip("groups straddle rows: the generic kernel's")
    weight, wc, x_np, x, dy_np, dy = _umma_case(storage, compute, m, in_dim, out_dim, m + in_dim, group)
    y = nv.linear_fwd(weight, x, torch.float32, compute)
    assert nv.last_path() == "umma"
    want = x_np.astype(np.float64) @ wc.astype(np.float64).T
    assert np.abs(y.cpu().numpy() - want).max() <= (TOL_F32 if compute == orc.F32 else 5e-3) * np.abs(want).max()
    for sd in (orc.BF16, orc.F32):
        res_np, res = act(np.random.default_rng(m), m, out_dim, sd)
        got = nv.linear_fwd_residual(weight, x, res.clone(), compute)
        sep = nv.linear_fwd(weight, x, TORCH_DTYPE[sd], compute)
        assert torch.equal(got, (sep.float() + res.float()).to(TORCH_DTYPE[sd]))
    assert nv.lib().caifq_device_status() == 0


@pytest.mark.parametrize("m,out_dim", [(64, 1024), (512, 14336)])
def test_streaming_wait_that_runs_out_raises_the_flag_and_returns(m, out_dim):
    import time

    weight, wc, x_np, x, dy_np, dy = _umma_case(orc.I4, orc.BF16, m, 1024, out_dim, 4243)
    y = nv.linear_fwd(weight, x, torch.float32, orc.BF16)
    assert nv.lib().caifq_device_status() == 0
    nv.lib().caifq_selftest_stall_next_umma()
    t0 = time.time()
    nv.linear_fwd(weight, x, torch.float32, orc.BF16)
    torch.cuda.synchronize()
    assert time.time() - t0 < 1.0
    assert nv.lib().caifq_device_status() & 2
    y2 = nv.linear_fwd(weight, x, torch.float32, orc.BF16)
    assert nv.lib().caifq_device_status() == 0
    assert torch.equal(y, y2)


@pytest.mark.parametrize("storage,m,out_dim", [(orc.I4, 64, 1024), (orc.I8, 96, 14336), (orc.I4, 300, 19072)])
def test_streaming_launch_behind_a_long_kernel_waits_for_it(storage, m, out_dim):
    """A launch that is placed beside the end of a long one (here one CTA's, a few hundred ms) must not count that one's
    time as its own waiting."""
    weight, wc, x_np, x, dy_np, dy = _umma_case(storage, orc.BF16, m, 256, out_dim, 4321)
    want = nv.linear_fwd(weight, x, torch.float32, orc.BF16)
    assert nv.lib().caifq_device_status() == 0
    rng = np.random.default_rng(3)
    big, _, _ = make_weight(rng, 2048, 4096, orc.I8)
    rows = torch.ones(131072, 4096, dtype=torch.bfloat16, device="cuda")
    y_big = torch.empty(131072, 2048, dtype=torch.bfloat16, device="cuda")
    y = torch.empty_like(want)
    start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    nv.lib().caifq_set_cta_limit(1)
    try:
        start.record()
        # (the plain entry point: the weight is converted in the kernel, which takes a single CTA)
        assert nv.lib().caifq_linear_fwd(big.ref(), nv._ptr(rows), nv.BF16, rows.shape[0], nv._ptr(y_big), nv.BF16, nv.BF16,
                                         nv._stream()) == 0
    finally:
        nv.lib().caifq_set_cta_limit(0)
    assert nv.lib().caifq_linear_fwd(weight.ref(), nv._ptr(x), nv.BF16, m, nv._ptr(y), nv.F32, nv.BF16, nv._stream()) == 0
    end.record()
    assert nv.lib().caifq_device_status() == 0
    assert start.elapsed_time(end) > 150.0
    assert torch.equal(y, want)


@pytest.mark.parametrize("width", ["64", "96", "128", "160", "192", "224", "256", None])
@pytest.mark.parametrize("m,in_dim,out_dim", [(300, 320, 384), (2305, 128, 1152)])   # partial tiles both ways; 10 row tiles
def test_umma_bf16_tile_widths(width, m, in_dim, out_dim, monkeypatch):
    if width is not None:
        monkeypatch.setenv("CAIFQ_UMMA_BN", width)
    weight, wc, x_np, x, dy_np, dy = _umma_case(orc.BF16, orc.F32, m, in_dim, out_dim, m + out_dim)
    y = nv.linear_fwd(weight, x, torch.float32, orc.F32)
    assert nv.last_path() == "umma"
    assert max_rel_err(y.cpu().numpy(), x_np.astype(np.float64) @ wc.astype(np.float64).T) <= TOL_F32
    out = torch.empty(m * out_dim + 8, dtype=torch.bfloat16, device="cuda")[8:].view(m, out_dim)   # 16-byte aligned only
    nv.linear_fwd(weight, x, torch.bfloat16, orc.F32, out=out)
    assert torch.equal(out, y.to(torch.bfloat16))
    in_dx = (in_dim + 127) // 128 * 128      # dX has in_dim columns: whole 128-column tiles
    weight, wc, x_np, x, dy_np, dy = _umma_case(orc.BF16, orc.F32, m, in_dx, out_dim, m + out_dim)
    dx = nv.linear_dx(weight, dy, torch.float32, orc.F32)
    assert nv.last_path() == "umma"
    assert max_rel_err(dx.cpu().numpy(), dy_np.astype(np.float64) @ wc.astype(np.float64)) <= TOL_F32
    assert nv.lib().caifq_device_status() == 0


@pytest.mark.parametrize("storage,compute,group", [(orc.I8, orc.F32, 128), (orc.I8, orc.BF16, 128), (orc.I4, orc.BF16, 32),
                                                   (orc.I4, orc.BF16, 96)])
@pytest.mark.parametrize("m,in_dim,out_dim", [(128, 384, 640), (769, 1152, 384), (1025, 768, 128)])
def test_many_tokens_through_an_expanded_weight(storage, compute, group, m, in_dim, out_dim):
    """The binding hands linear_fwd / linear_dx a scratch for the weight as bf16; without one (the plain C calls) the same
    values come from the in-kernel conversion.  int4: code times scale rounded once, so the bound is a bf16 GEMM's own."""
    weight, wc, x_np, x, dy_np, dy = _umma_case(storage, compute, m, in_dim, out_dim, m + out_dim, group)
    need = nv.lib().caifq_linear_workspace_bytes
    assert need(weight.ref(), 1, nv.BF16, m, compute) == in_dim * out_dim * 2
    assert (need(weight.ref(), 0, nv.BF16, m, compute) > 0) == (m > 768)
    assert need(weight.ref(), 1, nv.F32, m, compute) == 0 and need(weight.ref(), 1, nv.BF16, 127, compute) == 0
    tol = TOL_F32 if compute == orc.F32 else 4e-3
    y = nv.linear_fwd(weight, x, torch.float32, compute)
    dx = nv.linear_dx(weight, dy, torch.float32, compute)
    assert nv.last_path() == "umma"
    assert max_rel_err(y.cpu().numpy(), x_np.astype(np.float64) @ wc.astype(np.float64).T) <= tol
    assert max_rel_err(dx.cpu().numpy(), dy_np.astype(np.float64) @ wc.astype(np.float64)) <= tol
    plain = torch.empty_like(dx)
    rc = nv.lib().caifq_linear_dx(weight.ref(), dy.data_ptr(), nv.BF16, m, plain.data_ptr(), nv.F32, compute, nv._stream())
    assert rc == 0 and max_rel_err(plain.cpu().numpy(), dx.cpu().numpy()) <= 2 * tol


@pytest.mark.parametrize("limit", [1, 3])
def test_products_under_a_limit_of_few_ctas(limit):
    """One CTA leaves no pair, three leave one: the same numbers from the expanded products, plain and with an adapter, and
    from experts."""
    weight, wc, x_np, x, dy_np, dy = _umma_case(orc.I8, orc.BF16, 1025, 256, 384, 11)
    dense = nv.Weight(torch.randn(384, 256, device="cuda").bfloat16(), nv.BF16, 256, 384)
    lora = nv.Lora(torch.randn(16, 256, device="cuda").bfloat16() / 16, torch.randn(384, 16, device="cuda").bfloat16() / 16, 32.0)
    rng = np.random.default_rng(12)
    gate, up, down = ([make_weight(rng, o, i, orc.I4)[0] for _ in range(2)] for o, i in ((384, 256), (384, 256), (256, 384)))
    offsets = [0, 700, 1025]
    need = nv.grouped_expert_expanded_bytes(gate, up, down, nv.BF16, nv.BF16)
    expanded = torch.empty(need, dtype=torch.uint8, device="cuda")

    def products():
        y = nv.linear_fwd(weight, x, torch.bfloat16, orc.BF16)
        dx = nv.linear_dx(weight, dy, torch.bfloat16, orc.BF16)
        few = nv.linear_fwd(weight, x[:64], torch.bfloat16, orc.BF16)
        d = nv.linear_fwd(dense, x, torch.bfloat16, orc.BF16)
        ly, h = nv.lora_linear_fwd(weight, lora, x, orc.F32, expanded=True)
        ldx, _, _ = nv.lora_linear_bwd(weight, lora, dy, x, h, orc.F32, expanded=True)
        nv.grouped_expert_expand(gate, up, down, expanded, nv.BF16, nv.BF16)
        out, g, u = nv.grouped_expert_fwd(gate, up, down, offsets, x, nv.BF16, expanded)
        edx = nv.grouped_expert_bwd(gate, up, down, offsets, x, g, u, nv.BF16, expanded)
        out2, g2, u2 = nv.grouped_expert_fwd(gate, up, down, offsets, x, nv.BF16)
        edx2 = nv.grouped_expert_bwd(gate, up, down, offsets, x, g2, u2, nv.BF16)
        return [y, dx, few, d, ly, h, ldx, out, g, u, edx, out2, edx2]

    want = products()
    nv.lib().caifq_set_cta_limit(limit)
    try:
        got = products()
        assert nv.lib().caifq_device_status() == 0
    finally:
        nv.lib().caifq_set_cta_limit(0)
    for a, b in zip(got, want):
        assert max_rel_err(a.float().cpu().numpy(), b.float().cpu().numpy()) <= 1e-2


def test_a_wide_layer_on_one_cta():
    """More tiles than a CTA can keep records of go to the kernel that needs none."""
    out_dim, in_dim, m = 128 * 4800, 64, 17
    codes = torch.randint(-127, 128, (out_dim, in_dim), dtype=torch.int8, device="cuda")
    weight = nv.Weight(codes, nv.I8, in_dim, out_dim, torch.full((1,), 0.01, device="cuda"))
    x = torch.randn(m, in_dim, device="cuda").bfloat16()
    want = nv.linear_fwd(weight, x, torch.bfloat16, orc.BF16)
    nv.lib().caifq_set_cta_limit(1)
    try:
        got = nv.linear_fwd(weight, x, torch.bfloat16, orc.BF16)
        assert nv.lib().caifq_device_status() == 0
    finally:
        nv.lib().caifq_set_cta_limit(0)
    assert torch.equal(got, want)


@pytest.mark.parametrize("storage", [orc.I8, orc.I4])
def test_wide_outputs_of_few_hundred_rows_convert_in_the_kernel(storage):
    """One wave of tiles converts in place; more rows expand.  With an adapter the workspace is that of the largest call."""
    rng = np.random.default_rng(8)
    compute = orc.BF16
    weight, codes, scales = make_weight(rng, 256, 14336, storage)         # dX has 14336 columns
    turned, tcodes, tscales = make_weight(rng, 14336, 256, storage)       # so has this forward product
    dense = torch.from_numpy(_oracle_w(weight, codes, scales, compute)).double().cuda()
    tdense = torch.from_numpy(_oracle_w(turned, tcodes, tscales, compute)).double().cuda()
    need = nv.lib().caifq_linear_workspace_bytes
    for m in (128, 256):
        assert need(weight.ref(), 1, nv.BF16, m, compute) == 0
    assert need(weight.ref(), 1, nv.BF16, 1024, compute) > 0
    assert need(turned.ref(), 1, nv.BF16, 128, compute) > 0               # (256 columns)
    lora = nv.Lora(torch.randn(16, 256, device="cuda").bfloat16() / 16, torch.randn(14336, 16, device="cuda").bfloat16() / 64, 16.0)
    small = nv.lora_fwd_workspace_bytes(turned, lora, 128, compute, True)
    assert small <= nv.lora_fwd_workspace_bytes(turned, lora, 256, compute, True) <= nv.lora_fwd_workspace_bytes(
        turned, lora, 1024, compute, True)
    for m in (128, 256, 257, 1024):
        dy = torch.randn(m, 256, device="cuda").bfloat16()
        want = dy.double() @ dense
        dx = nv.linear_dx(weight, dy, torch.float32, compute)
        assert (dx.double() - want).norm() <= 4e-3 * want.norm()
        want = dy.double() @ tdense.T + (dy.double() @ lora.a.double().T) @ lora.b.double().T
        y, _ = nv.lora_linear_fwd(turned, lora, dy, compute, expanded=True)
        assert (y.double() - want).norm() <= 1e-2 * want.norm()


def _early_reader(name, weight):
    """A product by one of the kernels that read codes and scales ahead of the previous kernel's end."""
    g = torch.Generator(device="cuda").manual_seed(29)
    m = {"decode": 4, "stream": 64, "fp32_rows": 8, "fp32": 64, "experts": 8, "experts_stream": 96}[name]
    x = torch.randn(m, weight.in_dim, generator=g, device="cuda")
    if name.startswith("fp32"):
        return lambda: nv.linear_fwd(weight, x)
    x = x.bfloat16()
    if not name.startswith("experts"):
        return lambda: nv.linear_fwd(weight, x, torch.float32, nv.BF16)
    ws = [weight] * 4
    offsets = [m // 4 * e for e in range(5)]
    return lambda: nv.grouped_expert_fwd(ws, ws, ws, offsets, x, nv.BF16)[1]


@pytest.mark.parametrize("reader", ["decode", "stream", "fp32_rows", "fp32", "experts", "experts_stream"])
@pytest.mark.parametrize("writer", ["cast_scales", "cast_scale", "cast_codes", "int4", "int8"])
def test_products_see_what_was_just_written(reader, writer):
    """The library's own writers of codes and scales let the next kernel in at once, and the products read codes and scales
    before their wait: what was written just ahead on the stream has to be what is multiplied, bit for bit.  The weight lies
    at the end of a large buffer, so that its writer is under way for long after its successor could have started."""
    lib, stream = nv.lib(), torch.cuda.current_stream().cuda_stream
    dim, pad = 1024, 1 << 26
    n = dim * dim
    g = torch.Generator(device="cuda").manual_seed(31)
    source = 40.0 * torch.randn(pad + n, generator=g, device="cuda").clamp_(-3.0, 3.0)
    if writer in ("cast_scales", "int4"):
        codes = torch.randint(0, 256, ((pad + n) // 2,), dtype=torch.uint8, generator=g, device="cuda")
        scales = torch.rand(pad + n // 128, generator=g, device="cuda").half()
        at = pad if writer == "cast_scales" else pad // 128
        weight = nv.Weight(codes[pad // 2:], nv.I4, dim, dim, scales[at:at + n // 128], group_size=128)
    else:
        codes = torch.randint(-127, 128, (pad + n,), dtype=torch.int8, generator=g, device="cuda")
        scales = torch.rand(pad + 1, generator=g, device="cuda")
        at = pad if writer == "cast_scale" else 0
        weight = nv.Weight(codes[pad:], nv.I8, dim, dim, None if writer == "cast_codes" else scales[at:at + 1])
    half = source.half()

    def write():
        if writer == "cast_scales":
            return lib.caifq_cast(source.data_ptr(), nv.F32, scales.data_ptr(), nv.F16, scales.numel(), stream)
        if writer == "cast_scale":
            return lib.caifq_cast(half.data_ptr(), nv.F16, scales.data_ptr(), nv.F32, scales.numel(), stream)
        if writer == "cast_codes":
            return lib.caifq_cast(source.data_ptr(), nv.F32, codes.data_ptr(), nv.I8, codes.numel(), stream)
        if writer == "int4":
            return lib.caifq_quantize_int4_per_group(source.data_ptr(), codes.data_ptr(), scales.data_ptr(), pad + n, 128, stream)
        return lib.caifq_quantize_int8_per_tensor(source.data_ptr(), codes.data_ptr(), scales.data_ptr(), pad + n, stream)

    product = _early_reader(reader, weight)
    before = product()
    filler = torch.empty(1 << 28, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    for _ in range(4):
        filler.zero_()      # (the host is ahead of the device from here on)
    assert write() == 0
    got = product()
    torch.cuda.synchronize()
    want = product()
    assert torch.equal(got, want)
    assert not torch.equal(before, want)


@pytest.mark.parametrize("m", [1, 16, 17, 33, 48, 65])
@pytest.mark.parametrize("out_dim", [1176, 3144, 3176, 3544, 3552, 3553, 3560, 4712, 4737])
def test_bf16_weight_either_side_of_a_resident_wave(m, out_dim):
    """147, 443 to 445 and 589 CTAs of 8 columns (two chains' loads at a time while three CTAs an SM take them all), and 32
    columns a CTA beyond, fewer registers from two CTAs an SM to three with three tiles of rows (3144 and 3176: 297 and 300).  Bound: products are exact, an fp32 sum of chains of 128 is within 1e-6 of the norm."""
    in_dim = 544       # 17 steps of 32: warps of two and of three
    g = torch.Generator(device="cuda").manual_seed(out_dim + m)
    w = torch.randn(out_dim, in_dim, generator=g, device="cuda").bfloat16()
    x = torch.randn(m, in_dim, generator=g, device="cuda").bfloat16()
    want = x.double() @ w.double().T
    weight = nv.Weight(w, nv.BF16, in_dim, out_dim)
    got = nv.linear_fwd(weight, x)
    assert (got.double() - want).norm() <= 1e-6 * want.norm()
    res = torch.randn(m, out_dim, generator=g, device="cuda")
    assert torch.equal(nv.linear_fwd_residual(weight, x, res.clone()), got + res)


def test_a_wider_bf16_weight_takes_no_second_wave():
    """14336 -> 4096, one row, is 15 % more bytes than 14336 -> 3552.  (With two chains' loads a time its 512 CTAs were two
    waves: 49 us against 25; 32 us with one.)"""
    x = torch.randn(1, 14336, device="cuda").bfloat16()
    t = {}
    for out_dim in (3552, 4096):
        weight = nv.Weight(torch.randn(out_dim, 14336, device="cuda").bfloat16(), nv.BF16, 14336, out_dim)
        t[out_dim] = best_time(lambda: nv.linear_fwd(weight, x))
    assert t[4096] < 1.6 * t[3552], t


@pytest.mark.parametrize("storage", [orc.I4, orc.I8])
@pytest.mark.parametrize("limit,how", [(1, "call"), (37, "call"), (132, "call"), (90, "CAIFQ_DECODE_CTAS"),
                                       (90, "CAIFQ_UMMA_CTAS")])
def test_experts_of_few_rows_keep_to_a_limit_of_ctas(storage, limit, how, monkeypatch):
    """A host's collective finds the SMs that the limit leaves it: no launch of the experts' products has more CTAs.  (Without
    a limit the few-token kernel has two an SM; the streaming kernel, which rounds an int4 weight to bf16, keeps to one.)"""
    rng = np.random.default_rng(59)
    counts = [1, 5, 0, 8] * 8
    gate, up, down = ([make_weight(rng, o, i, storage)[0] for _ in counts] for o, i in ((384, 512), (384, 512), (512, 384)))
    offsets = np.concatenate([[0], np.cumsum(counts)]).astype(np.int32).tolist()
    x = torch.randn(offsets[-1], 512, device="cuda").bfloat16()
    sms = torch.cuda.get_device_properties(0).multi_processor_count

    def run():
        return nv.grouped_expert_fwd(gate, up, down, offsets, x, nv.BF16)

    def products():
        return [(name.split("linear_")[1].split("_kernel")[0], ctas) for name, ctas in kernels_of(run) if "linear_" in name]

    want = run()
    assert products() == [("decode", 2 * sms), ("decode", 2 * sms)]
    if how == "call":
        nv.lib().caifq_set_cta_limit(limit)
    else:
        monkeypatch.setenv(how, str(limit))
    try:
        got = run()
        ran = products()
        most = sms if how == "CAIFQ_DECODE_CTAS" else limit     # (the other kernel's variable)
        assert len(ran) == 2 and all(name == "stream" and ctas <= most for name, ctas in ran)
        assert nv.lib().caifq_device_status() == 0
    finally:
        nv.lib().caifq_set_cta_limit(0)
    for a, b in zip(got, want):
        assert (a.float() - b.float()).norm() <= 1e-2 * b.float().norm()
