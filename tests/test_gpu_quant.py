"""GPU parity: quantize / dequantize / cast kernels are bit-exact against the
CPU oracle and against the reference's own kernels (oracle/_ref)."""
import numpy as np
import pytest
import torch

import caif_oracle as orc
import refkernels as ref
from caif_b200 import native as nv
from gpu_util import best_time, dev, to_dev

pytestmark = pytest.mark.gpu


def _bits(t):
    return t.detach().cpu().contiguous().view(torch.int32).numpy() if t.dtype == torch.float32 else t.cpu().numpy()


def _f16bits(t):
    return t.detach().cpu().contiguous().view(torch.int16).numpy().view(np.uint16)


INT8_CASES = {
    "c1_1024x1024": lambda g: (torch.randn(1024, 1024, generator=g) * 0.02),
    "odd_length": lambda g: torch.randn(100003, generator=g),
    "unaligned_view": lambda g: torch.randn(4099, generator=g)[3:],
    "zeros": lambda g: torch.zeros(777),
    "ties": lambda g: torch.arange(-127, 128).float() * 0.5,
    "one": lambda g: torch.tensor([0.3]),
    "with_inf_nan": lambda g: torch.tensor([1.0, float("nan"), -2.0, 0.5]),
}


@pytest.mark.parametrize("name", sorted(INT8_CASES))
def test_int8_per_tensor_bit_exact(name):
    g = torch.Generator().manual_seed(11)
    x = INT8_CASES[name](g).float()
    xd = x.to(dev())
    if name == "unaligned_view":
        xd = torch.randn(4099, generator=g).to(dev())[3:]
        x = xd.cpu()
    else:
        xd = xd.contiguous()
    q, s = nv.quantize_int8_per_tensor(xd)
    dq = nv.dequantize_int8_per_tensor(q, s)
    oq, os_ = orc.quantize_int8_per_tensor(x.numpy())
    assert np.array_equal(q.cpu().numpy(), oq)
    assert np.array_equal(_bits(s), os_.view(np.int32))
    assert np.array_equal(_bits(dq), orc.dequantize_int8_per_tensor(oq, os_).view(np.int32))
    if ref.available():
        rq, rs = ref.quantize_int8_per_tensor(xd.contiguous())
        assert torch.equal(rq, q) and torch.equal(rs.view(torch.int32), s.view(torch.int32))
        assert torch.equal(ref.dequantize_int8_per_tensor(rq, rs).view(torch.int32), dq.view(torch.int32))


def test_int8_empty_is_a_no_op():
    x = torch.empty(0, device=dev())
    q, s = nv.quantize_int8_per_tensor(x)
    assert q.numel() == 0


@pytest.mark.parametrize("shape", [(1024, 1024), (48, 80), (1, 7), (513, 3)])
def test_int8_per_channel_bit_exact(shape):
    g = torch.Generator().manual_seed(12)
    x = (torch.randn(*shape, generator=g) * 0.02).float()
    if shape[1] > 3:
        x[:, 3] = 0.0
    xd = x.to(dev()).contiguous()
    q, s = nv.quantize_int8_per_channel(xd)
    dq = nv.dequantize_int8_per_channel(q, s)
    oq, os_ = orc.quantize_int8_per_channel(x.numpy())
    assert np.array_equal(q.cpu().numpy(), oq)
    assert np.array_equal(_bits(s), os_.view(np.int32))
    assert np.array_equal(_bits(dq), orc.dequantize_int8_per_channel(oq, os_).view(np.int32))
    if ref.available():
        rq, rs = ref.quantize_int8_per_channel(xd)
        assert torch.equal(rq, q) and torch.equal(rs.view(torch.int32), s.view(torch.int32))


INT4_CASES = [
    ((14336 // 8, 4096), 128),   # an eighth of the decode config's weight
    ((16, 8), 128),              # the reference tests' shape: one group straddles all rows
    ((37, 24), 128),
    ((131,), 128),               # ragged tail, lone last nibble
    ((32, 96), 64),
    ((2048, 1408), 128),         # expert projection
    ((5, 30), 6),                # small even group
    ((1,), 128),
]


@pytest.mark.parametrize("shape,group", INT4_CASES)
def test_int4_bit_exact(shape, group):
    g = torch.Generator().manual_seed(13)
    x = (torch.randn(*shape, generator=g) * 0.02).float().reshape(-1)
    if x.numel() >= 512:
        x[128:256] = 0.0
    xd = x.to(dev()).contiguous()
    p, s = nv.quantize_int4(xd, group)
    dq = nv.dequantize_int4(p, s, x.numel(), group)
    op, os_ = orc.quantize_int4(x.numpy(), group)
    assert np.array_equal(p.cpu().numpy(), op)
    assert np.array_equal(_f16bits(s), os_)
    assert np.array_equal(_bits(dq), orc.dequantize_int4(op, os_, x.numel(), group).view(np.int32))
    if ref.available():
        rp, rs = ref.quantize_int4(xd, group)
        assert torch.equal(rp, p) and torch.equal(rs.view(torch.int16), s.view(torch.int16))
        assert torch.equal(ref.dequantize_int4(rp, rs, x.numel(), group).view(torch.int32), dq.view(torch.int32))


def test_int4_full_size_round_trip_properties():
    """Decode config weight (14336 x 4096): error bound of the reference's test
    (tests/test_quantize_ops.cpp:296) and idempotence of quantize(dequantize(.))."""
    g = torch.Generator(device="cuda").manual_seed(14)
    x = torch.randn(14336 * 4096, generator=g, device=dev()) * 0.02
    p, s = nv.quantize_int4(x, 128)
    dq = nv.dequantize_int4(p, s, x.numel(), 128)
    gmax = x.view(-1, 128).abs().amax(dim=1, keepdim=True)
    assert bool(((x.view(-1, 128) - dq.view(-1, 128)).abs() <= gmax / 7.0 * 0.5 + gmax * 1e-3 + 1e-7).all())
    p2, s2 = nv.quantize_int4(dq, 128)
    dq2 = nv.dequantize_int4(p2, s2, x.numel(), 128)
    assert float((dq2 - dq).abs().max()) <= float(gmax.max()) * 2e-3


@pytest.mark.parametrize("src,dst", [(torch.float32, torch.bfloat16), (torch.float32, torch.float16),
                                     (torch.bfloat16, torch.float32), (torch.float16, torch.float32),
                                     (torch.float16, torch.bfloat16), (torch.float32, torch.int8),
                                     (torch.int8, torch.float32)])
def test_cast_matches_oracle(src, dst):
    g = torch.Generator().manual_seed(15)
    x = torch.randn(10007, generator=g) * 50.0
    xs = x.to(src) if src != torch.int8 else x.clamp(-127, 127).round().to(torch.int8)
    got = nv.cast(xs.to(dev()).contiguous(), dst).cpu()
    base = xs.float().numpy()
    if dst == torch.int8:
        assert np.array_equal(got.numpy(), orc.cast_f32_to_int8(base))
    elif dst == torch.float32:
        assert np.array_equal(got.numpy(), base)
    else:
        code = orc.BF16 if dst == torch.bfloat16 else orc.F16
        assert np.array_equal(got.float().numpy(), orc.round_through(base, code))


def test_oracle_matches_reference_kernels_on_routing():
    if not ref.available():
        pytest.skip("reference kernels not built")
    g = torch.Generator().manual_seed(16)
    probs = torch.softmax(torch.randn(512, 68, generator=g), dim=-1).to(torch.bfloat16).float()
    pd = probs.to(dev()).contiguous()
    ridx, rval = ref.topk(pd, 6)
    rnorm = ref.normalize_rows(rval)
    oidx, oval = orc.topk(probs.numpy(), 6)
    assert np.array_equal(ridx.cpu().numpy(), oidx)
    assert np.array_equal(_bits(rval), oval.view(np.int32))
    assert np.array_equal(_bits(rnorm), orc.normalize_rows(oval).view(np.int32))
    wide = torch.rand(7, 1000, generator=g).to(dev())
    assert np.array_equal(_bits(ref.normalize_rows(wide)), orc.normalize_rows(wide.cpu().numpy()).view(np.int32))


@pytest.mark.parametrize("group,n", [(32, 8192 * 3 + 40), (64, 4096 * 5), (64, 100), (128, 8192 * 2 + 131), (256, 8192 + 257)])
def test_int4_eight_elements_a_thread_bit_exact(group, n):
    """Edges of a block's 8192 elements, a shorter last group, a buffer shorter than one group."""
    g = torch.Generator().manual_seed(15)
    x = torch.randn(n, generator=g) * 0.02
    x[:min(n, group)] = 0.0
    p, s = nv.quantize_int4(x.to(dev()), group)
    op, os_ = orc.quantize_int4(x.numpy(), group)
    assert np.array_equal(p.cpu().numpy(), op)
    assert np.array_equal(_f16bits(s), os_)


@pytest.mark.parametrize("shape", [(1000, 516), (4097, 130), (64, 128), (65, 131), (3, 4096)])
def test_int8_slices_of_rows_bit_exact(shape):
    """Per channel: several row slices, aligned and unaligned rows, a partial block of columns; per tensor: the same
    elements, with and without a remainder of four."""
    g = torch.Generator().manual_seed(16)
    x = torch.randn(*shape, generator=g) * 0.02
    q, s = nv.quantize_int8_per_channel(x.to(dev()))
    oq, os_ = orc.quantize_int8_per_channel(x.numpy())
    assert np.array_equal(q.cpu().numpy(), oq)
    assert np.array_equal(_bits(s), os_.view(np.int32))
    q, s = nv.quantize_int8_per_tensor(x.to(dev()))
    oq, os_ = orc.quantize_int8_per_tensor(x.numpy())
    assert np.array_equal(q.cpu().numpy(), oq)
    assert np.array_equal(_bits(s), os_.view(np.int32))


@pytest.mark.parametrize("n", [1, 3, 4, 5, 8192, 8193, 40961])
@pytest.mark.parametrize("offset", [0, 1])
def test_int8_block_maxima_lie_where_the_codes_will(n, offset):
    """Fewer codes than a block's maximum has bytes, one block and several, codes that start on any byte; and a value and a
    weight quantized again into the same codes."""
    g = torch.Generator().manual_seed(18)
    codes = torch.zeros(n + offset + 4, dtype=torch.int8, device=dev())
    scale = torch.zeros(1, device=dev())
    for std in (0.02, 3.0):
        x = torch.randn(n, generator=g) * std
        xd = x.to(dev())
        rc = nv.lib().caifq_quantize_int8_per_tensor(xd.data_ptr(), codes.data_ptr() + offset, scale.data_ptr(), n,
                                                     torch.cuda.current_stream().cuda_stream)
        assert rc == 0
        oq, os_ = orc.quantize_int8_per_tensor(x.numpy())
        assert np.array_equal(codes[offset:offset + n].cpu().numpy(), oq)
        assert np.array_equal(_bits(scale), os_.view(np.int32))
        assert not codes[:offset].any() and not codes[offset + n:].any()


@pytest.mark.parametrize("rows,cols", [(1, 1), (7, 30), (9, 4096), (2049, 36), (1025, 31), (300, 9600), (65, 19000)])
def test_int8_per_channel_clusters_bit_exact(rows, cols):
    """Eight row slices a column block of 16 (512 threads), 32, 64 and 128; slices without rows; infinities and NaNs."""
    g = torch.Generator().manual_seed(19)
    x = torch.randn(rows, cols, generator=g) * 0.02
    x[0, 0] = float("inf")
    x[rows - 1, cols // 2] = float("nan")
    q, s = nv.quantize_int8_per_channel(x.to(dev()))
    oq, os_ = orc.quantize_int8_per_channel(x.numpy())
    assert np.array_equal(_bits(s), os_.view(np.int32))
    live = np.isfinite(x.numpy() / os_[None, :])   # (what a NaN or an infinity is cast to is not defined on the CPU)
    assert np.array_equal(q.cpu().numpy()[live], oq[live])


@pytest.mark.parametrize("n", [1, 255, 257, 606207, 606209, 3 * 606208, 3 * 606208 + 1, 4 * 606208 - 1, 4 * 606208, 4 * 606208 + 1,
                               7 * 606208 + 300])
@pytest.mark.parametrize("src,dst", [(torch.float32, torch.bfloat16), (torch.float16, torch.float32),
                                     (torch.bfloat16, torch.bfloat16)])
def test_cast_trips_of_four(n, src, dst):
    """A grid of 2368 blocks takes 606208 elements at a time, four times a trip: whole trips, trips that are cut, none; a
    source that starts on any element; the same buffer as source and result."""
    g = torch.Generator(device="cuda").manual_seed(n)
    base = torch.randn(n + 1, generator=g, device="cuda").to(src)
    for x in (base[:n], base[1:]):
        assert torch.equal(nv.cast(x, dst), x.to(dst))
    if src == dst:
        want = base[:n].clone()
        rc = nv.lib().caifq_cast(base.data_ptr(), nv.dtype_code(src), base.data_ptr(), nv.dtype_code(dst), n,
                                 torch.cuda.current_stream().cuda_stream)
        assert rc == 0 and torch.equal(base[:n], want)


def test_cast_to_a_byte_moves_fewer_bytes_than_to_a_word():
    """500 MB against 800.  (With a bound for each element of a trip 109 us against 128; 80 without.)"""
    x = torch.randn(100_000_000, device="cuda")
    byte = best_time(lambda: nv.cast(x, torch.int8), calls=5)
    word = best_time(lambda: nv.cast(x, torch.float32), calls=5)
    assert byte < 0.74 * word, (byte, word)


@pytest.mark.parametrize("rows,cols", [(4096, 33), (4097, 33), (2049, 257), (10241, 1152), (16384, 132), (16385, 132), (16385, 1),
                                       (65536, 31), (40000, 300)])
def test_int8_per_channel_of_tall_tensors_bit_exact(rows, cols):
    """Either side of the lines between clusters of eight row slices and slices that fill the device: rows that 16-byte loads can
    and cannot read, a last slice that is cut; infinities and NaNs."""
    g = torch.Generator().manual_seed(23)
    x = torch.randn(rows, cols, generator=g) * 0.02
    x[rows - 1, 0] = float("-inf")
    x[rows // 2, cols // 2] = float("nan")
    x[:, cols - 1] = 0.0
    q, s = nv.quantize_int8_per_channel(x.to(dev()))
    oq, os_ = orc.quantize_int8_per_channel(x.numpy())
    assert np.array_equal(_bits(s), os_.view(np.int32))
    with np.errstate(invalid="ignore"):
        live = np.isfinite(x.numpy() / os_[None, :])   # (what a NaN or an infinity is cast to is not defined on the CPU)
    assert np.array_equal(q.cpu().numpy()[live], oq[live])


def test_int8_per_channel_of_a_tall_tensor_uses_the_whole_device():
    """262144 x 31, against one scale for all of it.  (As two clusters of eight CTAs 160 us, 12 times as long; 52 us with the
    rows over all SMs.)"""
    x = torch.randn(262144, 31, device="cuda")
    channel = best_time(lambda: nv.quantize_int8_per_channel(x))
    tensor = best_time(lambda: nv.quantize_int8_per_tensor(x))
    assert channel < 7.0 * tensor, (channel, tensor)


def test_a_launch_that_was_refused_leaves_no_error_behind():
    """A launch into a capture that something else has broken fails on the host; the next call is none the worse."""
    import ctypes

    rt = ctypes.CDLL("libcudart.so.12")
    lib = nv.lib()
    x = torch.randn(4096, device="cuda")
    y = torch.empty(4096, dtype=torch.bfloat16, device="cuda")
    packed = torch.empty(2048, dtype=torch.uint8, device="cuda")
    scales = torch.empty(32, dtype=torch.float16, device="cuda")
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    raw = ctypes.c_void_p(stream.cuda_stream)
    assert rt.cudaStreamBeginCapture(raw, 0) == 0                       # the mode that forbids allocations meanwhile
    p = ctypes.c_void_p()
    assert rt.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(256)) != 0    # and with one the capture is void
    rc = lib.caifq_cast(x.data_ptr(), nv.F32, y.data_ptr(), nv.BF16, x.numel(), stream.cuda_stream)
    graph = ctypes.c_void_p()
    rt.cudaStreamEndCapture(raw, ctypes.byref(graph))
    rt.cudaGetLastError()
    assert rc != 0
    here = torch.cuda.current_stream().cuda_stream
    assert lib.caifq_quantize_int4_per_group(x.data_ptr(), packed.data_ptr(), scales.data_ptr(), x.numel(), 128, here) == 0
    assert lib.caifq_cast(x.data_ptr(), nv.F32, y.data_ptr(), nv.BF16, x.numel(), here) == 0
    assert torch.equal(y, x.bfloat16())
