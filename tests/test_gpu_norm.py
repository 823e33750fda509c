"""RMSNorm in front of the frozen projections (caif_b200/csrc/norm.cu) against the reference's own kernels
(src/caif_cuda_kernels_normalization.cu, compiled unmodified into oracle/_ref) and the oracle: y, the cached rms
and dx bit for bit, grad_gamma to rounding (the reference adds it with atomics in no fixed order)."""
import numpy as np
import pytest
import torch

import caif_oracle as orc
import refkernels as ref
from caif_b200 import native as nv

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,dim", [(333, 4096), (1, 4096), (1100, 14336), (50, 700), (7, 33), (3, 8192)])
def test_rmsnorm_bit_exact_with_the_reference_kernels(dtype, rows, dim):
    if dtype == torch.float32 and dim * 8 > 96 * 1024:
        pytest.skip("two fp32 rows of this width exceed the backward's row buffers")
    code = orc.F32 if dtype == torch.float32 else orc.BF16
    g = torch.Generator(device="cuda").manual_seed(rows * 7 + dim)
    x = (torch.randn(rows, dim, generator=g, device="cuda") * 1.5).to(dtype)
    dy = torch.randn(rows, dim, generator=g, device="cuda").to(dtype)
    gamma = 1.0 + 0.1 * torch.randn(dim, generator=g, device="cuda")
    eps = 1e-5
    y, rms = nv.rmsnorm_fwd(x, gamma, eps)
    f = lambda t: t.float().cpu().numpy()
    o_y, o_rms = orc.rmsnorm_forward(f(x), f(gamma), eps, code)
    assert np.array_equal(f(rms), o_rms)
    assert np.array_equal(f(y), o_y)
    if dim > 8192:      # the backward keeps a thread's share of grad_gamma in registers: rows up to 8192 wide
        if ref.available():
            r_y, r_rms = ref.rmsnorm_fwd(x, gamma, eps)
            assert torch.equal(r_rms, rms) and torch.equal(r_y, y)
        with pytest.raises(nv.CaifqError, match="too long"):
            nv.rmsnorm_bwd(dy, x, gamma, rms)
        return
    dx, gg = nv.rmsnorm_bwd(dy, x, gamma, rms)
    o_dx, o_gg = orc.rmsnorm_backward(f(dy), f(x), f(gamma), o_rms, code)
    assert np.array_equal(f(dx), o_dx)
    assert np.max(np.abs(f(gg) - o_gg)) <= 1e-4 * max(1.0, float(np.max(np.abs(o_gg))))
    if ref.available():
        r_y, r_rms = ref.rmsnorm_fwd(x, gamma, eps)
        assert torch.equal(r_rms, rms) and torch.equal(r_y, y)
        r_dx, r_gg = ref.rmsnorm_bwd(dy, x, gamma, rms, eps)
        assert torch.equal(r_dx, dx)
        assert torch.allclose(r_gg, gg, rtol=1e-4, atol=1e-4 * float(gg.abs().max()))
    # in place, and accumulation onto an existing grad_gamma
    x2 = x.clone()
    nv._check(nv.lib().caifq_rmsnorm_fwd(nv._ptr(x2), nv._ptr(gamma), nv._ptr(x2), None, eps, nv.dtype_code(x2), rows,
                                         dim, nv._stream()), "in place")
    assert torch.equal(x2, y)
    _, gg2 = nv.rmsnorm_bwd(dy, x, gamma, rms, grad_gamma=gg.clone())
    assert torch.allclose(gg2, 2 * gg, rtol=1e-5, atol=1e-5 * float(gg.abs().max()))


def test_rmsnorm_edge_cases():
    gamma = torch.ones(16, device="cuda")
    y, rms = nv.rmsnorm_fwd(torch.zeros(0, 16, device="cuda"), gamma)
    assert y.shape == (0, 16) and rms.numel() == 0
    z, rms = nv.rmsnorm_fwd(torch.zeros(2, 16, device="cuda"), gamma, 1e-6)
    assert torch.equal(z, torch.zeros(2, 16, device="cuda")) and torch.all(rms == np.float32(1e-6) ** 0.5)
    with pytest.raises(nv.CaifqError, match="row buffer"):
        nv.rmsnorm_fwd(torch.zeros(1, 30000, device="cuda"), torch.ones(30000, device="cuda"))


@pytest.mark.parametrize("dtype,rows,dim", [
    (torch.bfloat16, 1, 2048), (torch.bfloat16, 5, 4096), (torch.bfloat16, 1185, 4096), (torch.bfloat16, 1190, 6144),
    (torch.bfloat16, 1201, 1416), (torch.bfloat16, 7, 16384), (torch.float32, 600, 4096), (torch.float32, 3, 6144),
    (torch.float16, 1184, 2056), (torch.bfloat16, 300, 264),
])
def test_rmsnorm_rows_in_registers_match_the_element_kernels(dtype, rows, dim):
    """Edges of the register forms (rows per CTA, stripes of 256 columns, the last one partial) against the kernels
    with one thread per column, which rows that do not start on 16 bytes take: the same bits."""
    g = torch.Generator(device="cuda").manual_seed(rows + dim)
    x = torch.randn(rows, dim, generator=g, device="cuda").to(dtype)
    dy = torch.randn(rows, dim, generator=g, device="cuda").to(dtype)
    gamma = torch.randn(dim, generator=g, device="cuda")

    def shifted(t):
        flat = torch.empty(t.numel() + 1, dtype=t.dtype, device="cuda")
        flat[1:] = t.reshape(-1)
        return flat[1:].view(rows, dim)

    y, rms = nv.rmsnorm_fwd(x, gamma)
    if dim * x.element_size() <= 96 * 1024:
        y2, rms2 = nv.rmsnorm_fwd(shifted(x), gamma)
        assert torch.equal(y, y2) and torch.equal(rms, rms2)
    want = x.float() / torch.sqrt(x.float().square().mean(-1, keepdim=True) + 1e-5) * gamma
    assert float((y.float() - want).abs().max()) <= (1e-5 if dtype == torch.float32 else 5e-2) * float(want.abs().max())
    if dim <= 8192:
        dx, dg = nv.rmsnorm_bwd(dy, x, gamma, rms)
        dx2, dg2 = nv.rmsnorm_bwd(shifted(dy), shifted(x), gamma, rms)
        assert torch.equal(dx, dx2)
        assert float((dg - dg2).abs().max()) <= 1e-4 * float(dg2.abs().max())


@pytest.mark.parametrize("dim", [6016, 6017, 6143, 6144, 6145])
def test_rmsnorm_backward_of_rows_that_just_fill_the_shared_memory(dim):
    """Two fp32 rows of 6144 are 48 KB, what a launch has without asking, beside the kernel's own few words: against the
    oracle, bit for bit."""
    rows, eps = 5, 1e-5
    g = torch.Generator(device="cuda").manual_seed(dim)
    x, dy = (torch.randn(rows, dim, generator=g, device="cuda") for _ in range(2))
    gamma = 1.0 + 0.1 * torch.randn(dim, generator=g, device="cuda")
    f = lambda t: t.cpu().numpy()
    _, rms = nv.rmsnorm_fwd(x, gamma, eps)
    dx, gg = nv.rmsnorm_bwd(dy, x, gamma, rms)
    o_dx, o_gg = orc.rmsnorm_backward(f(dy), f(x), f(gamma), f(rms), orc.F32)
    assert np.array_equal(f(dx), o_dx)
    assert np.max(np.abs(f(gg) - o_gg)) <= 1e-4 * max(1.0, float(np.max(np.abs(o_gg))))
