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


# rows that end inside a 32-row slice, column tiles of one to four slices and several column tiles
@pytest.mark.parametrize("N,H,W,Cin,Cout", [(1, 3, 5, 64, 64), (2, 13, 11, 192, 64), (3, 28, 28, 512, 128), (5, 7, 7, 576, 64), (8, 40, 41, 256, 64)])
def test_masked_second_gradient(N, H, W, Cin, Cout):
    """The input gradient plus a second one under mask bits equals the sum with the masked tensor, bit for bit."""
    from torchmpi_b200.ops import conv
    from torchmpi_b200.parallel.flat_buckets import MaskedGrad
    torch.manual_seed(5)
    dy, add = _cl(N, Cout, H, W, dtype=torch.bfloat16), _cl(N, Cin, H, W, dtype=torch.bfloat16)
    w = (_cl(Cout, Cin, 1, 1, dtype=torch.float32) * Cin ** -0.5).to(torch.bfloat16)
    bits = torch.randint(0, 256, (N * H * W * Cin // 8,), device="cuda", dtype=torch.uint8)
    rows = add.permute(0, 2, 3, 1)
    rows[0, 0, 0] = float("nan")                                  # a masked NaN is not added either
    keep = (bits[:, None].int() >> torch.arange(8, device="cuda") & 1).view(N, H, W, Cin).permute(0, 3, 1, 2).bool()
    masked = add.masked_fill(~keep, 0.0).contiguous(memory_format=torch.channels_last)
    assert torch.equal(MaskedGrad(add, bits).tensor().nan_to_num(7.0), masked.nan_to_num(7.0))
    product = conv.conv_dgrad(dy, w, (N, Cin, H, W), 1, 0)
    expect = (product + masked).nan_to_num(7.0)
    assert torch.equal(conv.conv_dgrad(dy, w, (N, Cin, H, W), 1, 0, add=add, add_bits=bits).nan_to_num(7.0), expect)
    assert torch.equal(conv.conv_dgrad(dy, w, (N, Cin, H, W), 1, 0, add=masked).nan_to_num(7.0), expect)
    ref = torch.einsum("nohw,oc->nchw", dy.double(), w.double()[:, :, 0, 0])
    assert (product.double() - ref).abs().max() <= 2.0 ** -8 * ref.abs().max()


@pytest.mark.parametrize("conv1_frozen,own_library", [(False, False), (True, False), (False, True)])
def test_residual_gradient_reaches_the_block_input(conv1_frozen, own_library):
    """The residual's share of the input gradient, whoever adds it: the first convolution's kernel, or autograd where that
    convolution runs in the library."""
    from torchmpi_b200.models.resnet import Bottleneck
    torch.manual_seed(2)
    planes = 32 if own_library else 64                     # 32 channels: not a multiple of 64, so a library convolution
    m = Bottleneck(planes * 4, planes, 1, None, fused_bn=True).cuda()
    for c in (m.conv1, m.conv2, m.conv3):
        c.to(torch.bfloat16)
    m = m.to(memory_format=torch.channels_last)
    with torch.no_grad():
        m.bn3.weight.zero_()                                  # the branch passes nothing back: dx is the residual's gradient alone
        m.bn3.bias.zero_()
    m.conv1.weight.requires_grad_(not conv1_frozen)
    x = _cl(3, planes * 4, 9, 9, dtype=torch.bfloat16).requires_grad_(True)
    y = m(x)
    dy = torch.randn_like(y)
    y.backward(dy)
    assert torch.equal(x.grad, torch.where(x > 0, dy, torch.zeros_like(dy)))
