"""Batch-norm passes at the edges of their unrolled loops and residual gradients that travel as a mask, against fp64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _cl(*shape, dtype):
    n, c, h, w = shape
    return torch.randn(n, h, w, c, device="cuda").to(dtype).permute(0, 3, 1, 2)


# vectors of 16 bytes per tensor: one, a few blocks with a remainder, just above one and above four per thread of the largest grid
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("N,C,H,W", [(1, 8, 1, 2), (3, 64, 7, 5), (1, 64, 101, 97), (2, 512, 53, 61)])
@pytest.mark.parametrize("relu,res", [(True, True), (True, False), (False, True), (False, False)])
def test_bn_passes_at_loop_edges(dtype, N, C, H, W, relu, res):
    from torchmpi_b200.ops.bn_relu import FusedBatchNormReLU
    torch.manual_seed(3)
    x = (_cl(N, C, H, W, dtype=dtype) + 0.25).requires_grad_(True)
    r = _cl(N, C, H, W, dtype=dtype).requires_grad_(True) if res else None
    m = FusedBatchNormReLU(C, relu=relu).cuda()
    with torch.no_grad():
        m.weight.copy_(torch.rand(C) + 0.5)
        m.bias.copy_(torch.randn(C) * 0.1)
    y = m(x, r)
    dy = _cl(N, C, H, W, dtype=dtype)
    y.backward(dy)
    xr, rr = x.detach().double().requires_grad_(True), r.detach().double().requires_grad_(True) if res else None
    g, b = m.weight.detach().double().requires_grad_(True), m.bias.detach().double().requires_grad_(True)
    z = torch.nn.functional.batch_norm(xr, None, None, g, b, True, 0.1, m.eps)
    z = z + rr if res else z
    yr = torch.relu(z) if relu else z
    yr.backward(dy.double())
    # fp32 arithmetic on values of order one (x times scale: 1e-6 each), one rounding to dtype
    eps = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -10, torch.float32: 1e-5}[dtype]
    assert torch.allclose(y.double(), yr, rtol=eps, atol=3e-5)
    sure = z.detach().abs() > 1e-4 if relu else torch.ones_like(z, dtype=torch.bool)     # the mask may differ where z is about 0
    scale = xr.grad.abs().max().item()
    assert ((x.grad.double() - xr.grad).abs() * sure).max() <= eps * scale + 3e-5 * (1 + scale)
    if res:
        assert torch.equal((r.grad.double() * sure), (rr.grad * sure))
    M = N * H * W
    for got, ref in ((m.weight.grad, g.grad), (m.bias.grad, b.grad)):
        assert (got.double() - ref).abs().max() <= 2e-6 * M + 1e-4      # fp32 sums of M terms of order one, and the few unsure ones
