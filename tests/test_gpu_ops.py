"""Single-GPU hot ops against plain PyTorch fp32 references of the same op."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_native_library_is_loaded():
    from torchmpi_b200 import _lib
    assert _lib.lib.tmpi_has_cuda() == 1
    for sym in ("tmpi_sgd_momentum", "tmpi_xent_fwd_bwd", "tmpi_bn_relu_fwd", "tmpi_cuda_allreduce_sgd"):
        assert _lib.has_symbol(sym)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("nesterov", [False, True])
def test_sgd_momentum_matches_torch(dtype, nesterov):
    from torchmpi_b200.ops import elementwise
    torch.manual_seed(0)
    n = 8 * 12345
    w0 = torch.randn(n, device="cuda")
    w = w0.to(dtype).clone()
    master = w.float().clone() if dtype != torch.float32 else None
    mom = torch.zeros(n, device="cuda")
    ref = torch.nn.Parameter(w.float().clone())
    opt = torch.optim.SGD([ref], lr=0.05, momentum=0.9, weight_decay=1e-4, nesterov=nesterov)
    for step in range(4):
        g = torch.randn(n, device="cuda").to(dtype)
        ref.grad = g.float() * 0.5
        opt.step()
        gbuf = g.clone()
        elementwise.sgd_momentum_(w, gbuf, lr=0.05, momentum=0.9, weight_decay=1e-4, nesterov=nesterov,
                                  grad_scale=0.5, master=master, momentum_buf=mom, first_step=(step == 0),
                                  zero_grad=True)
        got = master if master is not None else w
        assert torch.allclose(got, ref.detach(), atol=2e-6, rtol=1e-5)
        assert torch.count_nonzero(gbuf) == 0
        if master is not None:
            assert torch.equal(w, master.to(dtype))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_xent_forward_and_gradient(dtype):
    from torchmpi_b200.ops import xent
    torch.manual_seed(1)
    for rows, cols in ((256, 1000), (7, 10), (33, 50257)):
        logits = (torch.randn(rows, cols, device="cuda") * 3).to(dtype).requires_grad_(True)
        labels = torch.randint(0, cols, (rows,), device="cuda")
        loss = xent.cross_entropy(logits, labels)
        loss.backward()
        ref_in = logits.detach().float().requires_grad_(True)
        ref = torch.nn.functional.cross_entropy(ref_in, labels)
        ref.backward()
        assert torch.allclose(loss.float(), ref, atol=1e-4, rtol=1e-5), (rows, cols, loss.item(), ref.item())
        tol = 1e-6 if dtype == torch.float32 else 2e-3 / rows + 1e-5
        assert torch.allclose(logits.grad.float(), ref_in.grad, atol=tol, rtol=2e-2)
        # same input, same bits
        loss2 = xent.cross_entropy(logits.detach(), labels)
        assert torch.equal(loss.detach(), loss2)


def test_absmean_var_and_check():
    from torchmpi_b200.ops import stats
    torch.manual_seed(2)
    for dtype in (torch.float32, torch.bfloat16, torch.float64):
        for n in (1, 1000, 3_000_001):
            x = torch.randn(n, device="cuda").to(dtype)
            m, v = stats.absmean_var(x)
            a = x.double().abs()
            # fp64 accumulation of fp32 partial sums over at most 32 elements (fp64 inputs: fp64 throughout)
            tol_m, tol_v = (1e-9, 1e-7) if dtype == torch.float64 else (5e-7, 2e-6)
            assert abs(m - a.mean().item()) <= tol_m * max(1.0, abs(m))
            if n > 1:
                assert abs(v - a.var().item()) <= tol_v * max(1.0, v)
            assert stats.absmean_var(x) == (m, v)      # deterministic


def test_easgd_and_downpour_kernels():
    from torchmpi_b200.ops import elementwise
    torch.manual_seed(3)
    for dtype, n in ((torch.float32, 100003), (torch.bfloat16, 8 * 4096), (torch.float32, 4096)):
        x = torch.randn(n, device="cuda").to(dtype)
        c = torch.randn(n, device="cuda").to(dtype)
        d = torch.empty_like(x)
        x0 = x.float().clone()
        elementwise.easgd_elastic(x, c, d, 0.3)
        diff = c.float() - x0
        tol = 1e-6 if dtype == torch.float32 else 2e-2
        assert torch.allclose(x.float(), x0 + 0.3 * diff, atol=tol, rtol=tol)
        assert torch.allclose(d.float(), -0.3 * diff, atol=tol, rtol=tol)
        acc = torch.randn(n, device="cuda").to(dtype)
        g = torch.randn(n, device="cuda").to(dtype)
        a0 = acc.float().clone()
        elementwise.downpour_accum(acc, g, scale=2.0)
        assert torch.allclose(acc.float(), a0 + 2.0 * g.float(), atol=tol, rtol=tol)
        elementwise.downpour_accum(acc, g, zero_first=True)
        assert torch.allclose(acc.float(), g.float(), atol=tol, rtol=tol)


@pytest.mark.parametrize("C,hw,relu,res", [(64, 56, True, False), (256, 14, True, True), (2048, 7, False, False),
                                           (16, 9, True, True)])
def test_fused_bn_relu_matches_torch(C, hw, relu, res):
    from torchmpi_b200.ops.bn_relu import FusedBatchNormReLU, supported
    torch.manual_seed(4)
    N = 16
    x = (torch.randn(N, C, hw, hw, device="cuda") * 2 + 0.5).to(torch.bfloat16).contiguous(memory_format=torch.channels_last)
    r = torch.randn(N, C, hw, hw, device="cuda").to(torch.bfloat16).contiguous(memory_format=torch.channels_last) if res else None
    assert supported(x)
    m = FusedBatchNormReLU(C, relu=relu).cuda()
    with torch.no_grad():
        m.weight.uniform_(0.5, 1.5)
        m.bias.uniform_(-0.5, 0.5)
    ref = torch.nn.BatchNorm2d(C).cuda()
    ref.load_state_dict({k: v for k, v in m.state_dict().items()})
    xa = x.clone().requires_grad_(True)
    ra = r.clone().requires_grad_(True) if res else None
    y = m(xa, ra)
    xb = x.float().clone().requires_grad_(True)
    rb = r.float().clone().requires_grad_(True) if res else None
    z = ref(xb) + (rb if res else 0)
    yr = torch.relu(z) if relu else z
    assert torch.allclose(y.float(), yr, atol=3e-2, rtol=2e-2)
    assert torch.allclose(m.running_mean, ref.running_mean, atol=1e-3, rtol=1e-3)
    assert torch.allclose(m.running_var, ref.running_var, atol=1e-3, rtol=1e-3)
    dy = torch.randn_like(y)
    # use the same ReLU mask in both: derive the reference gradient from the fused output's mask
    y.backward(dy)
    mask = (y > 0).float() if relu else torch.ones_like(yr)
    z.backward(dy.float() * mask)
    scale = xb.grad.abs().max().item()
    assert torch.allclose(xa.grad.float(), xb.grad, atol=3e-2 * scale + 1e-3, rtol=5e-2)
    assert torch.allclose(m.weight.grad, ref.weight.grad, atol=2e-2 * ref.weight.grad.abs().max().item(), rtol=2e-2)
    assert torch.allclose(m.bias.grad, ref.bias.grad, atol=2e-2 * ref.bias.grad.abs().max().item(), rtol=2e-2)
    if res:
        assert torch.allclose(ra.grad.float(), (dy.float() * mask), atol=1e-2, rtol=1e-2)
    # eval mode uses the running statistics
    m.eval(), ref.eval()
    ye = m(x, r)
    ze = ref(x.float()) + (r.float() if res else 0)
    assert torch.allclose(ye.float(), torch.relu(ze) if relu else ze, atol=3e-2, rtol=2e-2)


@pytest.mark.parametrize("shape,k,s,p", [((8, 64, 112, 112), 3, 2, 1), ((3, 16, 17, 23), 3, 2, 1), ((2, 8, 9, 9), 2, 2, 0)])
def test_maxpool_nhwc_matches_torch(shape, k, s, p):
    from torchmpi_b200.ops.pool import MaxPool2d, supported
    torch.manual_seed(5)
    x = torch.relu(torch.randn(*shape, device="cuda")).to(torch.bfloat16).contiguous(memory_format=torch.channels_last)
    assert supported(x)
    xa = x.clone().requires_grad_(True)
    y = MaxPool2d(k, s, p)(xa)
    xb = x.clone().requires_grad_(True)
    yr = torch.nn.functional.max_pool2d(xb, k, s, p)
    assert torch.equal(y, yr)
    dy = torch.randn_like(y)
    y.backward(dy)
    yr.backward(dy)
    # many ties (zeros after ReLU): the first maximum of a window must receive the gradient
    assert torch.allclose(xa.grad.float(), xb.grad.float(), atol=2e-2, rtol=2e-2)


def test_stem_conv_matches_conv2d():
    """im2col + tcgen05 GEMM stem against an fp32 conv2d of the same bf16 operands, forward and dW."""
    from torchmpi_b200.ops import stem_conv, gemm
    torch.manual_seed(5)
    for N, H, W in ((4, 224, 224), (3, 64, 96), (2, 40, 56)):
        conv = stem_conv.StemConv7x7(64).cuda().to(torch.bfloat16).to(memory_format=torch.channels_last)
        x = torch.randn(N, 3, H, W, device="cuda").to(torch.bfloat16).contiguous(memory_format=torch.channels_last)
        assert stem_conv.supported(x, conv.weight)
        y = conv(x)
        assert y.is_contiguous(memory_format=torch.channels_last)
        dy = torch.randn_like(y)
        y.backward(dy)
        wr = conv.weight.detach().float().requires_grad_(True)
        yr = torch.nn.functional.conv2d(x.float(), wr, None, 2, 3)
        yr.backward(dy.float())
        assert y.shape == yr.shape
        assert torch.allclose(y.float(), yr, rtol=2e-2, atol=5e-2), (N, H, W, (y.float() - yr).abs().max().item())
        rel = (conv.weight.grad.float() - wr.grad).norm() / wr.grad.norm()
        assert rel < 1e-2, (N, H, W, rel.item())
        gemm.check_status()


@pytest.mark.parametrize("fused_bwd", [0, 1])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_bn_relu_maxpool_stage_matches_separate_ops(dtype, fused_bwd):
    """Batch-norm + ReLU + max-pool in one stage against the three PyTorch ops in fp32 on the same input."""
    from torchmpi_b200 import config
    from torchmpi_b200.ops.bn_relu import FusedBatchNormReLUMaxPool
    config.set("bn_pool_fused_bwd", fused_bwd)
    torch.manual_seed(7)
    for N, C, H, W in ((4, 64, 112, 112), (2, 16, 33, 47), (3, 32, 16, 16)):
        x = torch.randn(N, C, H, W, device="cuda").to(dtype).contiguous(memory_format=torch.channels_last).requires_grad_(True)
        m = FusedBatchNormReLUMaxPool(C).cuda()
        with torch.no_grad():
            m.weight.copy_(torch.randn(C).abs() + 0.5)
            m.weight[::3] *= -1                      # negative scales reverse the order inside a window
            m.bias.copy_(torch.randn(C) * 0.3)
        y = m(x)
        dy = torch.randn_like(y)
        y.backward(dy)
        xr = x.detach().float().requires_grad_(True)
        ref_bn = torch.nn.BatchNorm2d(C).cuda()
        with torch.no_grad():
            ref_bn.weight.copy_(m.weight)
            ref_bn.bias.copy_(m.bias)
        z = torch.relu(ref_bn(xr))
        if dtype == torch.bfloat16:
            z = z + (z.to(dtype).float() - z).detach()      # the stage pools the bf16-rounded activation
        yr = torch.nn.functional.max_pool2d(z, 3, 2, 1)
        yr.backward(dy.float())
        tol = 2e-2 if dtype == torch.bfloat16 else 1e-4
        assert y.shape == yr.shape
        assert torch.allclose(y.float(), yr, rtol=tol, atol=tol), (N, C, H, W)
        assert torch.allclose(m.running_mean, ref_bn.running_mean, atol=1e-4)
        assert torch.allclose(m.running_var, ref_bn.running_var, atol=1e-3, rtol=1e-3)
        rel = (x.grad.float() - xr.grad).norm() / xr.grad.norm()
        assert rel < (2e-2 if dtype == torch.bfloat16 else 1e-4), (N, C, H, W, rel.item())
        assert torch.allclose(m.weight.grad, ref_bn.weight.grad, rtol=2e-2, atol=2e-2 * ref_bn.weight.grad.abs().max().item())
        assert torch.allclose(m.bias.grad, ref_bn.bias.grad, rtol=2e-2, atol=2e-2 * ref_bn.bias.grad.abs().max().item())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_layernorm_matches_torch(dtype):
    """One-pass layer norm (forward, dx, dgamma, dbeta) against fp32 PyTorch on the same operands."""
    from torchmpi_b200.ops.layernorm import LayerNorm, supported
    torch.manual_seed(9)
    for rows, C in ((8192, 1024), (777, 256), (33, 2048 if dtype == torch.bfloat16 else 1024), (4096, 768)):
        ln = LayerNorm(C).cuda().to(dtype)
        with torch.no_grad():
            ln.weight.copy_(torch.randn(C) * 0.5 + 1.0)
            ln.bias.copy_(torch.randn(C) * 0.2)
        x = (torch.randn(rows, C, device="cuda") * 2 + 0.5).to(dtype).requires_grad_(True)
        assert supported(x, ln.weight, ln.bias), (rows, C)
        y = ln(x)
        dy = torch.randn_like(y)
        y.backward(dy)
        xr = x.detach().float().requires_grad_(True)
        wr, br = ln.weight.detach().float().requires_grad_(True), ln.bias.detach().float().requires_grad_(True)
        yr = torch.nn.functional.layer_norm(xr, (C,), wr, br, ln.eps)
        yr.backward(dy.float())
        tol = 3e-2 if dtype == torch.bfloat16 else 1e-4
        assert torch.allclose(y.float(), yr, rtol=tol, atol=tol), (rows, C)
        for g, gr in ((x.grad, xr.grad), (ln.weight.grad, wr.grad), (ln.bias.grad, br.grad)):
            rel = (g.float() - gr).norm() / gr.norm()
            assert rel < (2e-2 if dtype == torch.bfloat16 else 1e-5), (rows, C, rel.item())


@pytest.mark.parametrize("N,H,W,cl", [(1, 8, 8, True), (2, 17, 24, False), (3, 64, 256, True), (1, 224, 224, True), (150, 16, 40, False)])
def test_stem_conv_implicit_gemm(N, H, W, cl):
    """Forward and weight gradient of the implicit-GEMM stem against an fp32 convolution: the narrowest and widest rows, odd
    heights, chunks cut by the image's end, more chunks than CTAs, both weight layouts."""
    import torch.nn.functional as F
    from torchmpi_b200.ops import stem_conv, gemm
    torch.manual_seed(N + H + W)
    conv = stem_conv.StemConv7x7(64).cuda().to(torch.bfloat16)
    if cl:
        conv = conv.to(memory_format=torch.channels_last)
    x = torch.randn(N, 3, H, W, device="cuda").to(torch.bfloat16).contiguous(memory_format=torch.channels_last)
    assert stem_conv.supported(x, conv.weight) and stem_conv.direct(x, conv.weight)
    y = conv(x)
    dy = torch.randn_like(y)
    y.backward(dy)
    gemm.check_status()
    w = conv.weight.detach().float().requires_grad_(True)
    ref = F.conv2d(x.float(), w, None, 2, 3)
    ref.backward(dy.float())
    assert y.shape == ref.shape and y.is_contiguous(memory_format=torch.channels_last)
    rel = lambda a, b: ((a.float() - b).norm() / b.norm()).item()
    # one bf16 rounding of an fp32 sum: 2^-9 at most, 2^-9 / sqrt(3) in the mean
    assert rel(y, ref.detach()) < 4e-3, rel(y, ref.detach())
    assert rel(conv.weight.grad, w.grad) < 4e-3, rel(conv.weight.grad, w.grad)


@pytest.mark.parametrize("W", [8, 40, 256])
def test_stem_conv_non_finite_pixels(W):
    """A non-finite pixel reaches the windows that contain it and no other."""
    import torch.nn.functional as F
    from torchmpi_b200.ops import stem_conv, gemm
    torch.manual_seed(W)
    H = 21
    conv = stem_conv.StemConv7x7(64).cuda().to(torch.bfloat16)
    x = torch.randn(3, 3, H, W).to(torch.bfloat16)
    x[0, 0, 0, 0], x[0, 1, 9, W - 2], x[0, 2, 20, 4], x[1, 1, 5, 2], x[1, 0, 12, 5] = (float(v) for v in ("inf", "-inf", "nan", "nan", "inf"))
    xc = x.cuda().contiguous(memory_format=torch.channels_last)
    assert stem_conv.direct(xc, conv.weight)
    with torch.no_grad():
        y = conv(xc).float().cpu()
    gemm.check_status()
    w = conv.weight.detach().double().cpu().reshape(64, 147)
    ref = (w @ F.unfold(x.double(), 7, padding=3, stride=2)).reshape(y.shape)
    assert torch.equal(y.isnan(), ref.isnan()) and torch.equal(y.isinf(), ref.isinf())
    assert torch.equal(y[ref.isinf()].double(), ref[ref.isinf()])
    ok = ref.isfinite()
    # 2^-9 for the rounding to bf16, 147 fp32 additions to sums below 4 (seven standard deviations)
    assert ((y.double() - ref)[ok].abs() <= 2 ** -8 * ref[ok].abs() + 147 * 4 * 2 ** -23).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("N,C,H,W", [(1, 8, 1, 1), (2, 64, 2, 3), (5, 128, 29, 30), (3, 16, 64, 5)])
def test_bn_pool_stage_edges_and_ties(dtype, N, C, H, W):
    """The pooling stage at single rows and columns, odd sizes and several strips, on values with many ties: the first
    maximum of a window takes the gradient, a window that the ReLU closed passes none."""
    from torchmpi_b200 import config
    from torchmpi_b200.ops.bn_relu import FusedBatchNormReLUMaxPool
    torch.manual_seed(N * H + W)
    x = torch.randint(-2, 3, (N, C, H, W), device="cuda").to(dtype).contiguous(memory_format=torch.channels_last)
    m = FusedBatchNormReLUMaxPool(C).cuda().eval()                 # fixed statistics: (x - 0) / 1 exactly, ties stay ties
    with torch.no_grad():
        m.running_var.fill_(1.0 - m.eps)
        m.weight[::2] *= -1
    xg = x.clone().requires_grad_(True)
    y = m(xg)
    z = torch.relu(x.float() * m.weight.detach()[None, :, None, None]).to(dtype).float().requires_grad_(True)
    ref = torch.nn.functional.max_pool2d(z, 3, 2, 1)
    assert torch.allclose(y.float(), ref, rtol=1e-3, atol=1e-3)
    # backward uses batch statistics in its formula; with both parameter sums removed it is the routed gradient, which the
    # two-stage path (pool, then batch-norm) computes separately
    dy = torch.randn_like(y)
    got = {}
    for fused in (1, 0):
        config.set("bn_pool_fused_bwd", fused)
        try:
            xg.grad = m.weight.grad = m.bias.grad = None
            m(xg).backward(dy)
            got[fused] = (xg.grad.float().clone(), m.weight.grad.clone(), m.bias.grad.clone())
        finally:
            config.set("bn_pool_fused_bwd", 1)
    ref.backward(dy.float())
    # the bias gradient is the sum of the routed gradient over the positions that the ReLU lets through
    routed = (z.grad * (z > 0)).sum((0, 2, 3))
    scale = dy.float().abs().sum((0, 2, 3)).max().item() + 1e-6
    assert (got[1][2] - routed).abs().max().item() <= 1e-5 * scale
    tol = {torch.float32: 1e-5, torch.float16: 2e-3, torch.bfloat16: 1.6e-2}[dtype]      # two-stage rounds the routed gradient to dtype
    for a, b in zip(got[1], got[0]):
        assert (a - b).abs().max().item() <= tol * max(1.0, b.abs().max().item()) * 2, (dtype, (a - b).abs().max().item())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows,cols,pitch", [(1, 1, 0), (7, 33, 0), (336, 10, 0), (900, 128, 0), (300, 1000, 1008), (5, 1024, 0),
                                             (3, 1025, 0), (700, 5003, 5008), (2, 60001, 0)])
def test_cross_entropy_row_lengths(rows, cols, pitch, dtype):
    """A warp per row, a block per row in shared memory (misaligned rows, a pitch) and the fallback for rows that do not fit
    there: loss and gradient against fp64, padding columns left out."""
    from torchmpi_b200.ops import xent
    torch.manual_seed(rows + cols)
    buf = torch.randn(rows, pitch or cols, device="cuda").mul_(3.0).to(dtype)
    x = buf[:, :cols].detach().requires_grad_(True)
    labels = torch.randint(0, cols, (rows,), device="cuda")
    loss = xent.cross_entropy(x, labels)
    loss.backward()
    ref_x = x.detach().double().requires_grad_(True)
    ref = torch.nn.functional.cross_entropy(ref_x, labels)
    ref.backward()
    assert loss.shape == ref.shape
    assert abs(loss.item() - ref.item()) <= 2e-6 * max(1.0, abs(ref.item()))
    # exponentials from the special-function unit (2 ulp), fp16 between the passes of long 16-bit rows, one final rounding
    unit = {torch.float32: 2e-6, torch.float16: 2 ** -9, torch.bfloat16: 2 ** -7.5}[dtype]
    err = (x.grad.double() - ref_x.grad).abs()
    # fp16 subnormals of the result; exponentials below 2^-14 kept as fp16 subnormals, and the label's p - 1, which cancels
    floor = (2 ** -24 if dtype == torch.float16 else 0.0) + 1e-6 / rows
    assert bool((err <= unit * ref_x.grad.abs() + floor).all()), (err / (ref_x.grad.abs() + 1e-30)).max().item()
    with pytest.raises(RuntimeError):
        loss.backward()                                    # the stored gradient has been handed out


def test_cross_entropy_infinities_and_bad_labels():
    from torchmpi_b200.ops import xent
    for cols in (40, 3000):
        x = torch.randn(6, cols, device="cuda")
        x[0, 1:] = float("-inf")                           # one class left
        x[1, ::2] = float("-inf")
        x[2, 3] = float("nan")
        x[3] = torch.finfo(torch.float32).min              # a mask of the type's lowest value: uniform
        xg = x.clone().requires_grad_(True)
        labels = torch.zeros(6, dtype=torch.int64, device="cuda")
        labels[1] = 1
        bad = labels.clone()
        bad[4], bad[5] = -1, cols                          # no class: nothing is taken off the gradient
        loss = xent.cross_entropy(xg, bad)
        loss.backward()
        ref = x.clone().requires_grad_(True)
        torch.nn.functional.cross_entropy(ref, labels).backward()
        ref.grad[4:, 0] += 1.0 / 6
        assert torch.isnan(loss)
        for r in (0, 1, 3, 4, 5):
            assert torch.allclose(xg.grad[r], ref.grad[r], rtol=1e-5, atol=1e-8), (cols, r)
        assert torch.isnan(xg.grad[2]).all()


@pytest.mark.parametrize("n", [8, 4096, 511 * 8, 1_000_008])
def test_elementwise_updates_at_block_edges(n):
    """One pack per thread (SGD) and two (EASGD, Downpour): tensors of one pack, whole blocks, a cut last block."""
    from torchmpi_b200.ops import elementwise as ew
    torch.manual_seed(n)
    for dtype in (torch.bfloat16, torch.float32):
        local, center = torch.randn(n, device="cuda").to(dtype), torch.randn(n, device="cuda").to(dtype)
        l0, delta = local.clone(), torch.full_like(local, 7.0)
        ew.easgd_elastic(local, center, delta, 0.25)
        d = center.float() - l0.float()
        assert torch.equal(local, (l0.float() + 0.25 * d).to(dtype)) and torch.equal(delta, (-0.25 * d).to(dtype))
        acc = l0.clone()
        ew.downpour_accum(acc, center, scale=0.5)
        assert torch.equal(acc, (l0.float() + 0.5 * center.float()).to(dtype))
        w, m = l0.clone(), torch.zeros(n, device="cuda")
        master = l0.float() if dtype != torch.float32 else None
        ew.sgd_momentum_(w, center, lr=0.5, momentum=0.5, master=master, momentum_buf=m, first_step=True, zero_grad=False)
        assert torch.equal(m, center.float()) and torch.equal(w, (l0.float() - 0.5 * center.float()).to(dtype))


def test_native_autograd_functions_save_through_hooks():
    """The C++ functions keep their inputs as saved tensors: pack / unpack hooks see them, and the gradients are the same."""
    from torchmpi_b200.ops import attention, gemm, layernorm
    torch.manual_seed(0)
    lin = gemm.Linear(128, 384, gelu=True).cuda().to(torch.bfloat16)
    ln = layernorm.LayerNorm(256).cuda().to(torch.bfloat16)
    cases = [(lambda t: lin(t), torch.randn(64, 128)), (lambda t: ln(t), torch.randn(40, 256)),
             (lambda t: attention.causal_attention(t, 2), torch.randn(1, 128, 384))]
    for fn, x in cases:
        x = x.cuda().to(torch.bfloat16)
        a, b = x.clone().requires_grad_(True), x.clone().requires_grad_(True)
        fn(a).float().square().sum().backward()
        seen = []
        with torch.autograd.graph.saved_tensors_hooks(lambda t: (seen.append(t.shape), t.cpu())[1], lambda t: t.cuda()):
            fn(b).float().square().sum().backward()
        assert seen
        assert ((a.grad.float() - b.grad.float()).norm() / a.grad.float().norm()).item() < 1e-3


@pytest.mark.parametrize("dtype,C,H,W", [(torch.bfloat16, 64, 9, 219), (torch.bfloat16, 64, 8, 224), (torch.bfloat16, 64, 7, 256),
                                         (torch.float32, 64, 9, 120), (torch.float32, 64, 6, 130), (torch.float16, 256, 5, 96)])
@pytest.mark.parametrize("fused_bwd", [1, 0])
def test_bn_pool_stage_long_rows(dtype, C, H, W, fused_bwd):
    """Rows that would not fit in an SM's shared memory: forward and both backward routes against separate ops."""
    from torchmpi_b200 import config
    from torchmpi_b200.ops.bn_relu import FusedBatchNormReLUMaxPool
    torch.manual_seed(W)
    x = torch.randn(2, C, H, W, device="cuda").to(dtype).contiguous(memory_format=torch.channels_last).requires_grad_(True)
    m = FusedBatchNormReLUMaxPool(C).cuda()
    before = config.get("bn_pool_fused_bwd")
    config.set("bn_pool_fused_bwd", fused_bwd)
    try:
        y = m(x)
        dy = torch.randn_like(y)
        y.backward(dy)
    finally:
        config.set("bn_pool_fused_bwd", before)
    xr = x.detach().float().requires_grad_(True)
    bn = torch.nn.BatchNorm2d(C).cuda()
    z = torch.relu(bn(xr))
    z = z + (z.to(dtype).float() - z).detach()              # the stage pools the rounded activation
    yr = torch.nn.functional.max_pool2d(z, 3, 2, 1)
    yr.backward(dy.float())
    # one rounding of the result (2^-8 for bf16, 2^-11 for fp16), and a window whose two largest values round alike now and then
    # sends its gradient to the other one
    tol = {torch.bfloat16: 2e-2, torch.float16: 4e-3, torch.float32: 1e-4}[dtype]
    assert torch.allclose(y.float(), yr, rtol=tol, atol=tol)
    rel = lambda a, b: ((a.float() - b).norm() / b.norm()).item()
    assert rel(x.grad, xr.grad) < tol and rel(m.weight.grad, bn.weight.grad) < tol and rel(m.bias.grad, bn.bias.grad) < tol


def test_cross_entropy_on_two_streams_at_once():
    """Losses of equal row counts that run at the same time on two streams keep their own arrival counters and row losses."""
    from torchmpi_b200 import _native
    from torchmpi_b200.ops import xent
    torch.manual_seed(3)
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    for rows, cols in ((8192, 1000), (600, 20000), (96, 10)):
        x = [torch.randn(rows, cols, device="cuda") for _ in streams]
        labels = [torch.randint(0, cols, (rows,), device="cuda") for _ in streams]
        want = [xent.cross_entropy(a, b) for a, b in zip(x, labels)]
        torch.cuda.synchronize()
        got = [[], []]
        for _ in range(20):
            for k, s in enumerate(streams):
                with torch.cuda.stream(s):
                    got[k].append(xent.cross_entropy(x[k], labels[k]))
        torch.cuda.synchronize()
        for k in (0, 1):
            assert all(torch.equal(v, want[k]) for v in got[k]), (rows, cols, k)
    buffers = set()
    for s in streams:
        with torch.cuda.stream(s):
            buffers.add(_native.ext().cross_entropy_scratch(x[0], 96).data_ptr())
    assert len(buffers) == 2


def test_cross_entropy_first_called_under_capture():
    """A captured loss clears its own counter: right on every replay, and eager calls around it are right before the first."""
    from torchmpi_b200.ops import xent
    torch.manual_seed(4)
    x = torch.randn(77, 300, device="cuda")
    labels = torch.randint(0, 300, (77,), device="cuda")
    want = xent.cross_entropy(x, labels)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        captured = xent.cross_entropy(x, labels)
    with torch.cuda.stream(side):
        eager = xent.cross_entropy(x, labels)
    torch.cuda.synchronize()
    assert torch.equal(eager, want)
    for _ in range(3):
        captured.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(captured, want)
    torch.cuda.synchronize()
    assert torch.equal(xent.cross_entropy(x, labels), want)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("cols", [40, 3000, 60001])
def test_cross_entropy_rows_at_the_lowest_value(cols, dtype):
    """A row filled with the type's lowest finite value is uniform, and so are two such logits beside -inf: the largest logit
    times log2(e) overflows there and must not be formed."""
    from torchmpi_b200.ops import xent
    lowest = torch.finfo(dtype).min
    x = torch.full((3, cols), lowest, device="cuda", dtype=dtype)
    x[1, 2:] = float("-inf")
    x[2] = -lowest                                         # the largest value
    labels = torch.tensor([1, 0, cols - 1], device="cuda")
    x.requires_grad_(True)
    loss = xent.cross_entropy(x, labels)
    loss.backward()
    # logsumexp - x[label]: log(n) is lost beside 3e38 in 32 bits, and the loss is that of a uniform row without the cancellation
    p = torch.zeros(3, cols, dtype=torch.double, device="cuda")
    p[0], p[1, :2], p[2] = 1.0 / cols, 0.5, 1.0 / cols
    p[torch.arange(3), labels] -= 1.0
    unit = {torch.float32: 2e-6, torch.float16: 2 ** -9, torch.bfloat16: 2 ** -7.5}[dtype]
    floor = (2 ** -24 if dtype == torch.float16 else 0.0) + 1e-6 / 3
    assert bool(((x.grad.double() - p / 3).abs() <= unit * p.abs() / 3 + floor).all())
    assert torch.isfinite(loss)


@pytest.mark.parametrize("H,W", [(21, 8), (24, 40), (22, 40), (21, 104), (50, 200), (23, 256), (5, 24), (2, 16)])
def test_stem_weight_gradient_non_finite_pixels(H, W):
    """A non-finite pixel reaches the taps that multiply it by an output gradient and no other: output widths that are not a
    multiple of 16 and odd output heights, where the products run over padding."""
    import torch.nn.functional as F
    from torchmpi_b200.ops import stem_conv, gemm
    torch.manual_seed(H * W)
    conv = stem_conv.StemConv7x7(64).cuda().to(torch.bfloat16)
    clean = torch.randn(4, 3, H, W).to(torch.bfloat16)
    nan, inf = float("nan"), float("inf")
    spots = [(0, 1, H - 1, W - 1, inf), (1, 0, H - 1, W // 2, nan), (2, 2, H // 2, W - 2, -inf), (3, 1, H - 2, W - 3, nan), (0, 2, 0, 0, inf)]
    dy = None
    for n, c, ih, iw, v in spots:
        x = clean.clone()
        x[n, c, ih, iw] = v
        xc = x.cuda().contiguous(memory_format=torch.channels_last)
        assert stem_conv.direct(xc, conv.weight)
        conv.weight.grad = None
        y = conv(xc)
        dy = torch.randn_like(y) if dy is None else dy
        y.backward(dy)
        gemm.check_status()
        got = conv.weight.grad.double().cpu()
        col = F.unfold(x.double(), 7, padding=3, stride=2)                     # [N, 147, OH * OW]
        ref = torch.einsum("nop,nkp->ok", dy.double().cpu().flatten(2), col).reshape(64, 3, 7, 7)
        assert torch.equal(got.isnan(), ref.isnan()) and torch.equal(got.isinf(), ref.isinf()), (n, c, ih, iw, v)
        ok = ref.isfinite()
        assert ok.any() or min(H, W) <= 8
        # one rounding to bf16 (2^-9 at most) and fp32 sums
        assert ((got - ref)[ok].norm() <= 4e-3 * ref[ok].norm()), (n, c, ih, iw, v)


def test_stem_weight_gradient_in_a_graph_beside_an_eager_one():
    """A captured weight gradient, replayed while eager ones run on the stream it was captured on: each has its own partial
    sums."""
    from torchmpi_b200.ops.stem_conv import _StemDirectFn
    torch.manual_seed(8)
    w = torch.randn(64, 3, 7, 7, device="cuda").to(torch.bfloat16)
    x = [torch.randn(64, 3, 64, 64, device="cuda").to(torch.bfloat16).contiguous(memory_format=torch.channels_last) for _ in range(2)]
    dy = [torch.randn(64, 64, 32, 32, device="cuda").to(torch.bfloat16).contiguous(memory_format=torch.channels_last) for _ in range(2)]

    def grad(k):
        leaf = w.detach().requires_grad_(True)             # of the stream that this runs on
        return torch.autograd.grad(_StemDirectFn.apply(x[k], leaf), leaf, dy[k])[0]

    want = [grad(0), grad(1)]
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        captured = grad(0)
    for _ in range(10):
        graph.replay()
        with torch.cuda.stream(side):
            eager = grad(1)
        torch.cuda.synchronize()
        assert torch.equal(captured, want[0]) and torch.equal(eager, want[1])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
def test_operands_between_16_byte_boundaries(dtype):
    """Views that start one element into a buffer, as inputs, parameters and incoming gradients: the bits of aligned operands."""
    from torchmpi_b200.ops import gemm, layernorm
    torch.manual_seed(6)

    def shifted(t):
        v = torch.empty(t.numel() + 1, device="cuda", dtype=t.dtype)[1:].view(t.shape)
        return v.copy_(t)

    x, dy = torch.randn(37, 512, device="cuda").to(dtype), torch.randn(37, 512, device="cuda").to(dtype)
    g, b = torch.randn(512, device="cuda").to(dtype), torch.randn(512, device="cuda").to(dtype)
    out = []
    for place in (torch.clone, shifted):
        ln = layernorm.LayerNorm(512, device="cuda", dtype=dtype)
        ln.weight, ln.bias = torch.nn.Parameter(place(g)), torch.nn.Parameter(place(b))
        leaf = place(x).requires_grad_(True)
        y = ln(leaf)
        y.backward(place(dy))
        out.append([y.detach(), leaf.grad, ln.weight.grad, ln.bias.grad])
    assert all(torch.equal(a, c) for a, c in zip(*out))
    rows, n = 64, 1024
    dy, z = torch.randn(rows, n, device="cuda").to(dtype), torch.randn(rows, n, device="cuda").to(dtype)
    (dz, db), (dz2, db2) = gemm.bias_grad(dy, z), gemm.bias_grad(shifted(dy), shifted(z))
    unit = {torch.float32: 1e-5, torch.float16: 2 ** -9, torch.bfloat16: 2 ** -6}[dtype]       # PyTorch's passes round once more
    assert torch.allclose(dz, dz2, rtol=unit, atol=unit) and torch.allclose(db, db2, rtol=unit, atol=unit * rows ** 0.5)
    if dtype == torch.bfloat16:
        w, bias, xl = (torch.randn(*s, device="cuda").to(dtype) for s in ((n, 256), (n,), (rows, 256)))
        for gelu in (False, True):
            out = []
            for place in (torch.clone, shifted):
                leaves = [t.clone().requires_grad_(True) for t in (xl, w, bias)]
                y = gemm.linear(*leaves, gelu=gelu)
                out.append(torch.autograd.grad(y, leaves, place(dy)))
            assert all(torch.equal(a, c) for a, c in zip(*out))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("cols", [10, 1000, 5003, 60001])
def test_cross_entropy_labels_outside_the_row(cols, dtype):
    """A label that names no class counts as the largest logit in the loss and takes nothing off the gradient, in the kernel of
    short rows, of rows in shared memory and of rows that are read three times."""
    from torchmpi_b200.ops import xent
    torch.manual_seed(cols)
    x = torch.randn(6, cols, device="cuda").mul_(2.0).to(dtype).requires_grad_(True)
    labels = torch.tensor([-100, cols, cols - 1, -1, 2 ** 31 - 1, 0], device="cuda")
    loss = xent.cross_entropy(x, labels)
    loss.backward()
    xd = x.detach().double()
    inside = (labels >= 0) & (labels < cols)
    picked = torch.where(inside, xd.gather(1, labels.clamp(0, cols - 1)[:, None])[:, 0], xd.max(1).values)
    want = (torch.logsumexp(xd, 1) - picked).mean()
    assert abs(loss.item() - want.item()) <= 2e-6 * max(1.0, abs(want.item()))
    p = torch.softmax(xd, 1)
    p[inside, labels[inside]] -= 1.0
    p /= 6
    # exponentials from the special-function unit, fp16 between the passes of long 16-bit rows, one final rounding
    unit = {torch.float32: 2e-6, torch.float16: 2 ** -9, torch.bfloat16: 2 ** -7.5}[dtype]
    floor = (2 ** -24 if dtype == torch.float16 else 0.0) + 1e-6 / 6
    assert bool(((x.grad.double() - p).abs() <= unit * p.abs() + floor).all())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows,cols", [(1, 1), (3, 10), (336, 10), (17, 5003), (5, 60001)])
def test_cross_entropy_gradient_scaled_by_the_incoming_one(rows, cols, dtype):
    """The bits of a multiplication by the incoming gradient in the logits' type; packs and remainders."""
    from torchmpi_b200.ops import xent
    torch.manual_seed(cols)
    x = torch.randn(rows, cols, device="cuda").to(dtype)
    labels = torch.randint(0, cols, (rows,), device="cuda")
    grads = []
    for unit in (True, False):
        leaf = x.clone().requires_grad_(True)
        loss = xent.cross_entropy(leaf, labels, unit)
        (loss if unit else loss * 0.3).backward()
        grads.append(leaf.grad)
    assert torch.equal(grads[1], grads[0] * torch.tensor(0.3, device="cuda").to(dtype))
    for bad in (float("inf"), float("nan")):
        leaf = x.clone().requires_grad_(True)
        (xent.cross_entropy(leaf, labels) * bad).backward()
        assert torch.equal(leaf.grad.isnan(), (grads[0] * bad).isnan())
