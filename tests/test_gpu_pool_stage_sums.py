"""The pooling stage's kept inputs and window indices, element by element, against PyTorch on the same rounded values."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


# even and odd heights and widths, one window, several strips; values that tie and windows that are closed throughout
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("N,C,H,W", [(1, 8, 1, 1), (2, 8, 2, 3), (1, 16, 7, 6), (3, 64, 61, 9), (2, 24 * 8, 30, 31)])
def test_pool_stage_keeps_inputs_and_positions(dtype, N, C, H, W):
    from torchmpi_b200.ops.bn_relu import FusedBatchNormReLUMaxPool, supported
    torch.manual_seed(H)
    C = C if 256 % (C * {2: 1, 4: 2}[torch.empty((), dtype=dtype).element_size()] // 8) == 0 else 64
    x = torch.randint(-6, 3, (N, H, W, C), device="cuda").to(dtype).permute(0, 3, 1, 2).requires_grad_(True)
    m = FusedBatchNormReLUMaxPool(C).cuda().eval()              # mean 0, variance 1: all but the identity, exact up to eps
    assert supported(x)
    y = m(x)
    _, xmax, idx = y.grad_fn.saved_tensors[:3]
    z = torch.relu(x.detach().float().contiguous())
    ref, flat = F.max_pool2d(z, 3, 2, 1, return_indices=True)
    oh = torch.arange(y.shape[2], device="cuda")[:, None]
    ow = torch.arange(y.shape[3], device="cuda")[None]
    code = (flat // W - (2 * oh - 1)) * 3 + flat % W - (2 * ow - 1)
    code[ref == 0] = 255
    assert torch.equal(idx.permute(0, 3, 1, 2).long(), code)
    kept = x.detach().float().flatten(2).gather(2, flat.flatten(2)).view_as(ref)
    assert torch.equal(xmax.float()[ref > 0], kept[ref > 0]) and (xmax.float()[ref == 0] <= 0).all()
    dy = torch.randn_like(y)
    y.backward(dy)
    # sums of N * OH * OW terms of order one in fp32, xhat within 5e-6 of x (eps); whole small values: exact products
    open_ = (ref > 0).double() * dy.double()
    assert (m.bias.grad.double() - open_.sum((0, 2, 3))).abs().max() <= 2e-6 * ref.numel() / C + 1e-5
    assert (m.weight.grad.double() - (open_ * kept.double() * (1 + m.eps) ** -0.5).sum((0, 2, 3))).abs().max() <= 1e-5 * ref.numel() / C + 1e-4
