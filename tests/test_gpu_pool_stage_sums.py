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


# packs of four and eight channels, both element sizes; odd sizes, several strips
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("N,C,H,W", [(1, 8, 1, 1), (2, 64, 30, 31), (1, 2048, 5, 4)])
def test_pool_stage_entries_without_kept_inputs(dtype, N, C, H, W):
    """The C entries that take no kept inputs sum over all of x; they give what the ones with kept inputs give."""
    from torchmpi_b200._lib import check, dtype_code, lib, stream_ptr
    if 256 % (C // (16 // dtype.itemsize)):
        pytest.skip("channels the kernel does not take")
    torch.manual_seed(C + H)
    x = (torch.randn(N, H, W, C, device="cuda") + 0.25).to(dtype)
    gamma, beta = torch.rand(C, device="cuda") + 0.5, torch.randn(C, device="cuda") * 0.1
    out = (N, (H - 1) // 2 + 1, (W - 1) // 2 + 1, C)
    dy = torch.randn(out, device="cuda").to(dtype)
    got = []
    for keep in (False, True):
        y, idx, xmax = torch.empty_like(dy), torch.empty(out, dtype=torch.uint8, device="cuda"), torch.empty_like(dy)
        mean, invstd, dgamma, dbeta = (torch.empty(C, device="cuda") for _ in range(4))
        dx, scratch = torch.empty_like(x), torch.empty(lib.tmpi_bn_scratch_bytes(C), dtype=torch.uint8, device="cuda")
        kept = [xmax.data_ptr()] if keep else []
        fwd, bwd = ((lib.tmpi_bn_relu_pool_fwd_keep, lib.tmpi_bn_relu_pool_bwd_kept) if keep else
                    (lib.tmpi_bn_relu_pool_fwd, lib.tmpi_bn_relu_pool_bwd))
        check(fwd(x.data_ptr(), y.data_ptr(), idx.data_ptr(), *kept, gamma.data_ptr(), beta.data_ptr(), None, None, mean.data_ptr(),
                  invstd.data_ptr(), N, H, W, C, 1e-5, 0.1, 1, dtype_code(dtype), scratch.data_ptr(), stream_ptr()))
        check(bwd(x.data_ptr(), *kept, dy.data_ptr(), idx.data_ptr(), dx.data_ptr(), gamma.data_ptr(), beta.data_ptr(), mean.data_ptr(),
                  invstd.data_ptr(), dgamma.data_ptr(), dbeta.data_ptr(), N, H, W, C, dtype_code(dtype), scratch.data_ptr(), stream_ptr()))
        got.append((y, idx, dx, dgamma, dbeta))
    (y0, idx0, dx0, dg0, db0), (y1, idx1, dx1, dg1, db1) = got
    assert torch.equal(y0, y1) and torch.equal(idx0, idx1)
    # the same terms of order one in another order, in fp32; dx is rounded to its type after that
    terms = N * out[1] * out[2]
    assert (dg0 - dg1).abs().max() <= 2e-6 * terms + 1e-5 and (db0 - db1).abs().max() <= 2e-6 * terms + 1e-5
    eps = {torch.bfloat16: 2.0 ** -7, torch.float16: 2.0 ** -9, torch.float32: 1e-5}[dtype]
    assert (dx0.float() - dx1.float()).abs().max() <= eps * dx1.float().abs().max() + 1e-6


def test_pool_stage_keeps_nothing_without_gradients():
    """Inference allocates the output and its index, not the inputs that only a backward reads; neither setting of the backward's
    tunable has to be the one that held during forward."""
    from torchmpi_b200 import config
    from torchmpi_b200.ops.bn_relu import FusedBatchNormReLUMaxPool
    m = FusedBatchNormReLUMaxPool(64).cuda()
    x = torch.randn(16, 112, 112, 64, device="cuda").to(torch.bfloat16).permute(0, 3, 1, 2)
    for mode in (torch.no_grad, torch.inference_mode):
        with mode():
            m(x)
            torch.cuda.synchronize()
            before = torch.cuda.memory_allocated()
            torch.cuda.reset_peak_memory_stats()
            y = m(x)
            out = y.numel()
            assert torch.cuda.max_memory_allocated() - before <= 3 * out + (2 << 20)       # y, the index and what the allocator leaves unsplit
    grads = []
    for fwd, bwd in ((1, 1), (0, 1), (1, 0)):
        try:
            config.set("bn_pool_fused_bwd", fwd)
            xs = x.detach().requires_grad_(True)
            m.zero_grad(set_to_none=True)
            y = m(xs)
            config.set("bn_pool_fused_bwd", bwd)
            y.backward(torch.ones_like(y))
        finally:
            config.set("bn_pool_fused_bwd", 1)
        grads.append((xs.grad, m.weight.grad, m.bias.grad))
    for dx, dg, db in grads[1:]:
        # sums of 50176 terms of order one in fp32, in another order; bf16 gradients of positions under several windows
        assert (dg - grads[0][1]).abs().max() < 0.1 and (db - grads[0][2]).abs().max() < 0.1
        assert (dx.float() - grads[0][0].float()).norm() <= 1e-2 * grads[0][0].float().norm()
