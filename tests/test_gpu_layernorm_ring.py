"""Layer-norm backward at the edges of its ring of rows, against fp64."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu

EPS = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -10, torch.float32: 2e-6}


# one row, fewer rows than warps, one row per warp of the largest grid, a ring that wraps with a remainder; the narrowest and
# widest rows of each type
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("rows", [1, 7, 1184, 4737, 6000])
def test_layer_norm_backward_ring(dtype, rows):
    from torchmpi_b200.ops.layernorm import LayerNorm, check_status, supported
    unit = 128 if dtype == torch.float32 else 256
    for C in (unit, 3 * unit, 4 * unit, 8 * unit):
        torch.manual_seed(C)
        m = LayerNorm(C, device="cuda", dtype=dtype)
        with torch.no_grad():
            m.weight.copy_(1 + 0.1 * torch.randn(C))
        x = ((torch.randn(rows, C, device="cuda") * 1.5).to(dtype) + 0.25).requires_grad_(True)
        assert supported(x, m.weight, m.bias)
        dy = torch.randn(rows, C, device="cuda").to(dtype)
        m(x).backward(dy)
        check_status()
        xr, w, b = x.detach().double().requires_grad_(True), m.weight.detach().double().requires_grad_(True), m.bias.detach().double().requires_grad_(True)
        F.layer_norm(xr, (C,), w, b, m.eps).backward(dy.double())
        eps = EPS[dtype]
        assert (x.grad.double() - xr.grad).abs().max() <= eps * xr.grad.abs().max() + 1e-5
        for got, ref in ((m.weight.grad, w.grad), (m.bias.grad, b.grad)):       # fp32 sums over the rows, one rounding
            assert (got.double() - ref).abs().max() <= eps * ref.abs().max() + 2e-6 * rows
