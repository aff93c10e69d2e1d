"""The tcgen05 bf16 GEMM against a plain PyTorch fp32 matmul of the same operands."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _ref(a, b, bias=None, gelu=False):
    y = a.float() @ b.float().t()
    if bias is not None:
        y = y + bias.float()
    return torch.nn.functional.gelu(y) if gelu else y


@pytest.mark.parametrize("M,N,K", [(128, 256, 64), (128, 256, 512), (256, 512, 128), (1024, 1024, 1024),
                                   (100, 72, 40), (129, 257, 72), (4096, 2048, 4096), (37, 1000, 2048)])
def test_gemm_matches_fp32_reference(M, N, K):
    from torchmpi_b200.ops import gemm
    torch.manual_seed(M * 7 + N * 3 + K)
    a = torch.randn(M, K, device="cuda").to(torch.bfloat16)
    b = torch.randn(N, K, device="cuda").to(torch.bfloat16)
    y = gemm.matmul_nt(a, b)
    torch.cuda.synchronize()
    gemm.check_status()
    ref = _ref(a, b)
    err = (y.float() - ref).abs().max().item()
    assert err <= 0.02 * (K ** 0.5) + 0.05, (M, N, K, err)
    # bf16 rounding of an fp32-accumulated result: relative error of one bf16 ulp
    assert torch.allclose(y.float(), ref, rtol=1e-2, atol=0.02 * (K ** 0.5))


@pytest.mark.parametrize("M,N,K", [(256, 256, 64), (256, 512, 448), (300, 520, 136), (1024, 1024, 1024),
                                   (4096, 2048, 4096), (2304, 1280, 512)])
def test_gemm_cta_pair_and_single_cta_paths(M, N, K):
    """The 256 x 256 CTA-pair kernel (cta_group::2) and the 128 x 256 single-CTA kernel give the same
    product; both are checked against fp32, with a bias + GELU epilogue as well."""
    from torchmpi_b200 import config
    from torchmpi_b200.ops import gemm
    torch.manual_seed(M + N + K)
    a = torch.randn(M, K, device="cuda").to(torch.bfloat16)
    b = torch.randn(N, K, device="cuda").to(torch.bfloat16) * 0.2
    bias = torch.randn(N, device="cuda").to(torch.bfloat16)
    out = {}
    try:
        for pair in (1, 0):
            config.set("gemm_pair", pair)
            out[pair] = (gemm.matmul_nt(a, b), gemm.matmul_nt(a, b, bias, gelu=True))
            torch.cuda.synchronize()
            gemm.check_status()
    finally:
        config.set("gemm_pair", 1)
    ref, ref_g = _ref(a, b), _ref(a, b, bias, True)
    for pair in (1, 0):
        assert torch.allclose(out[pair][0].float(), ref, rtol=1e-2, atol=0.02 * (K ** 0.5)), pair
        assert torch.allclose(out[pair][1].float(), ref_g, rtol=2e-2, atol=0.02 * (K ** 0.5)), pair
    # same operands, same fp32 accumulation order along K: the two kernels agree bit for bit
    assert torch.equal(out[0][0], out[1][0])


@pytest.mark.parametrize("M,N,K", [(256, 256, 64), (512, 384, 200), (1024, 2048, 1024), (2048, 4096, 8192)])
def test_gemm_reads_second_operand_as_k_by_n(M, N, K):
    """``matmul_nn(a, b)`` with ``b [K, N]`` (MN-major shared-memory descriptor) equals the K-major
    kernel on a transposed copy bit for bit, and the fp32 product within rounding."""
    from torchmpi_b200.ops import gemm
    torch.manual_seed(M + 3 * N + 5 * K)
    a = torch.randn(M, K, device="cuda").to(torch.bfloat16)
    b = (torch.randn(K, N, device="cuda") * 0.2).to(torch.bfloat16)
    y = gemm.matmul_nn(a, b)
    y_t = gemm.matmul_nt(a, b.t().contiguous())
    torch.cuda.synchronize()
    gemm.check_status()
    ref = a.float() @ b.float()
    assert torch.allclose(y.float(), ref, rtol=1e-2, atol=0.02 * (K ** 0.5))
    assert torch.equal(y, y_t)


@pytest.mark.parametrize("M,N,K", [(256, 256, 64), (384, 512, 200), (1024, 2048, 1000), (4096, 1024, 8192)])
def test_gemm_transposed_first_operand(M, N, K):
    """``matmul_tn(a, b) = a.T @ b`` with ``a [K, M]`` and ``b [K, N]`` as stored (the weight-gradient layout):
    same bits as the K-major kernel on transposed copies, and the fp32 product within rounding."""
    from torchmpi_b200.ops import gemm
    torch.manual_seed(2 * M + 3 * N + K)
    a = torch.randn(K, M, device="cuda").to(torch.bfloat16)
    b = (torch.randn(K, N, device="cuda") * 0.2).to(torch.bfloat16)
    y = gemm.matmul_tn(a, b)
    y_t = gemm.matmul_nt(a.t().contiguous(), b.t().contiguous())
    torch.cuda.synchronize()
    gemm.check_status()
    ref = a.float().t() @ b.float()
    assert torch.allclose(y.float(), ref, rtol=1e-2, atol=0.02 * (K ** 0.5))
    assert torch.equal(y, y_t)


def test_gemm_epilogues_and_identity():
    from torchmpi_b200.ops import gemm
    torch.manual_seed(0)
    M, N, K = 384, 768, 256
    a = torch.randn(M, K, device="cuda").to(torch.bfloat16)
    b = torch.randn(N, K, device="cuda").to(torch.bfloat16) * 0.1
    bias = torch.randn(N, device="cuda").to(torch.bfloat16)
    for use_bias in (False, True):
        for gelu in (False, True):
            y = gemm.matmul_nt(a, b, bias if use_bias else None, gelu=gelu)
            ref = _ref(a, b, bias if use_bias else None, gelu)
            assert torch.allclose(y.float(), ref, rtol=2e-2, atol=5e-2), (use_bias, gelu)
    # identity weight: the product must reproduce the input exactly (checks tile placement and swizzle)
    eye = torch.eye(256, device="cuda").to(torch.bfloat16)
    x = torch.randn(512, 256, device="cuda").to(torch.bfloat16)
    assert torch.equal(gemm.matmul_nt(x, eye), x)
    gemm.check_status()


def test_linear_autograd_matches_torch():
    from torchmpi_b200.ops import gemm
    torch.manual_seed(1)
    x = torch.randn(4, 64, 512, device="cuda").to(torch.bfloat16).requires_grad_(True)
    lin = gemm.Linear(512, 1024, gelu=True).cuda().to(torch.bfloat16)
    y = lin(x)
    dy = torch.randn_like(y)
    y.backward(dy)
    xr = x.detach().float().requires_grad_(True)
    wr = lin.weight.detach().float().requires_grad_(True)
    br = lin.bias.detach().float().requires_grad_(True)
    yr = torch.nn.functional.gelu(torch.nn.functional.linear(xr, wr, br))
    yr.backward(dy.float())
    assert torch.allclose(y.float(), yr, rtol=2e-2, atol=5e-2)
    assert torch.allclose(x.grad.float(), xr.grad, rtol=3e-2, atol=0.5)
    assert torch.allclose(lin.weight.grad.float(), wr.grad, rtol=3e-2, atol=0.5)
    assert torch.allclose(lin.bias.grad.float(), br.grad, rtol=3e-2, atol=0.5)
    gemm.check_status()


def test_fused_gemms_single_rank():
    """With one rank the fused kernels degenerate to copy-engine + GEMM and GEMM + local slot sum:
    checks the flag hand-off between the copy CTAs and the TMA producers, and the slot epilogue."""
    import torchmpi_b200 as mpi
    from torchmpi_b200.parallel.tensor_parallel import TPGroup
    from torchmpi_b200.ops import gemm
    mpi.start(with_cuda=True)
    try:
        torch.manual_seed(3)
        rows, D, F = 512, 512, 1024
        tp = TPGroup(rows, D)
        full_buf, full_off = tp.new_full_buffer()
        x = torch.randn(rows, D, device="cuda").to(torch.bfloat16)
        w1 = (torch.randn(F, D, device="cuda") / D ** 0.5).to(torch.bfloat16)
        b1 = torch.randn(F, device="cuda").to(torch.bfloat16)
        w2 = (torch.randn(D, F, device="cuda") / F ** 0.5).to(torch.bfloat16)
        for rep in range(3):                 # flags and counters are epoch based: repeated calls must work
            z = tp.ag_gemm(x, full_off, full_buf, w1, b1)
            assert torch.equal(full_buf[:rows * D].view(rows, D), x)
            ref = x.float() @ w1.float().t() + b1.float()
            assert torch.allclose(z.float(), ref, rtol=2e-2, atol=5e-2), rep
            y = tp.gemm_rs(z, w2)
            ref2 = z.float() @ w2.float().t()
            assert torch.allclose(y.float(), ref2, rtol=2e-2, atol=5e-2), rep
        # the weight handed over as [K, N] (what backward does) gives the same bits as its transpose
        z_kn = tp.ag_gemm(x, full_off, full_buf, w1.t().contiguous(), None, w_is_kn=True)
        assert torch.equal(z_kn, tp.ag_gemm(x, full_off, full_buf, w1, None))
        y_kn = tp.gemm_rs(z, w2.t().contiguous(), w_is_kn=True)
        assert torch.equal(y_kn, tp.gemm_rs(z, w2))
        torch.cuda.synchronize()
        tp.check()
    finally:
        mpi.stop()


def test_wide_head_and_pitched_cross_entropy():
    """LM head with a vocabulary that is not a multiple of 8: logits live in a pitched buffer, the loss kernel
    takes the pitch, and forward / dX / dW all run on the CTA-pair kernel.  Against fp32 PyTorch."""
    from torchmpi_b200.ops import gemm, xent
    torch.manual_seed(11)
    for T, d, V in ((256, 256, 50257), (512, 384, 1003)):
        x = (torch.randn(T, d, device="cuda") * 0.5).to(torch.bfloat16).requires_grad_(True)
        w = (torch.randn(V, d, device="cuda") * 0.05).to(torch.bfloat16).requires_grad_(True)
        y = torch.randint(0, V, (T,), device="cuda")
        logits = gemm.wide_head(x, w)
        assert logits.shape == (T, V) and logits.stride(0) % 8 == 0
        loss = xent.cross_entropy(logits, y)
        loss.backward()
        xr, wr = x.detach().float().requires_grad_(True), w.detach().float().requires_grad_(True)
        lr = torch.nn.functional.linear(xr, wr)
        ref = torch.nn.functional.cross_entropy(lr, y)
        ref.backward()
        assert torch.allclose(logits.float(), lr, rtol=2e-2, atol=2e-2), (T, d, V)
        assert abs(loss.item() - ref.item()) < 2e-2 * max(1.0, abs(ref.item())), (loss.item(), ref.item())
        for g, gr in ((x.grad, xr.grad), (w.grad, wr.grad)):
            rel = (g.float() - gr).norm() / gr.norm()
            assert rel < 3e-2, (T, d, V, rel.item())
        gemm.check_status()


def test_bias_grad_with_and_without_gelu():
    """Column sum fused with the GELU backward against PyTorch in fp32."""
    from torchmpi_b200.ops import gemm
    torch.manual_seed(13)
    for rows, C in ((8192, 1024), (777, 4096), (33, 3072)):
        dy = torch.randn(rows, C, device="cuda").to(torch.bfloat16)
        z = (torch.randn(rows, C, device="cuda") * 1.5).to(torch.bfloat16)
        dz, db = gemm.bias_grad(dy, z)
        ref = torch.ops.aten.gelu_backward(dy.float(), z.float())
        assert torch.allclose(dz.float(), ref, rtol=2e-2, atol=2e-2)
        assert torch.allclose(db.float(), dz.float().sum(0), rtol=1e-2, atol=0.05 * rows ** 0.5)
        same, db2 = gemm.bias_grad(dy)
        assert same is dy
        assert torch.allclose(db2.float(), dy.float().sum(0), rtol=1e-2, atol=0.05 * rows ** 0.5)


def test_gelu_forward_kernel():
    """The erf-form GELU through the rational approximation against PyTorch in fp32."""
    from torchmpi_b200.ops import gemm
    torch.manual_seed(17)
    for shape, dt in (((8192, 4096), torch.bfloat16), ((333, 1000), torch.float32), ((64, 40), torch.float16)):
        z = (torch.randn(*shape, device="cuda") * 2.5).to(dt)
        y = gemm.gelu(z)
        ref = torch.nn.functional.gelu(z.float())
        tol = 1e-5 if dt == torch.float32 else 2e-2
        assert torch.allclose(y.float(), ref, rtol=tol, atol=tol), (shape, dt)
    edge = torch.tensor([-30.0, -8.0, -0.0, 0.0, 8.0, 30.0, float("inf")], device="cuda").repeat(4)[:24].contiguous()
    assert torch.allclose(gemm.gelu(edge), torch.nn.functional.gelu(edge), atol=1e-5)


@pytest.mark.parametrize("M,N,K,bias", [(256, 256, 64, True), (300, 520, 136, True), (384, 264, 72, False), (3072, 1000, 200, True),
                                        (8200, 4104, 136, True), (4104, 3000, 72, False), (2056, 2056, 136, True), (3592, 1032, 200, False)])
def test_gelu_epilogue_equals_product_then_gelu(M, N, K, bias):
    """One kernel that writes z and gelu(z): the same bits as the product followed by the elementwise pass (GELU of the
    rounded z), ragged edges.  On 74 clusters the first three shapes have a few tiles of 128 columns and the fourth 72 of 192, one
    per cluster; the others several per cluster (accumulators and staging tiles used again): up to eight of 256 columns, three
    of 256, two of 192, two of 128."""
    from torchmpi_b200.ops import gemm
    torch.manual_seed(M + N)
    a = torch.randn(M, K, device="cuda").to(torch.bfloat16)
    b = (torch.randn(N, K, device="cuda") * K ** -0.5).to(torch.bfloat16)
    c = torch.randn(N, device="cuda").to(torch.bfloat16) if bias else None
    z, y = gemm.matmul_nt_gelu(a, b, c)
    torch.cuda.synchronize()
    gemm.check_status()
    assert torch.equal(z, gemm.matmul_nt(a, b, c))
    assert torch.equal(y, gemm.gelu(z))
    ref = a.float() @ b.float().t() + (c.float() if bias else 0.0)
    assert ((z.float() - ref).norm() / ref.norm()).item() < 4e-3          # one bf16 rounding: 2^-9 at most


@pytest.mark.parametrize("M,N,K", [(3072, 1024, 200), (3072, 1000, 72), (8192, 384, 136), (2056, 2056, 136), (3592, 1032, 200)])
def test_pair_gemm_narrow_tiles(M, N, K):
    """Shapes whose tiles are 192 columns wide (they fill the SMs better than 256), the last one 128, all operand layouts, a
    bias; the last two with more tiles than clusters."""
    from torchmpi_b200.ops import gemm
    torch.manual_seed(M + N + K)
    a = torch.randn(M, K, device="cuda").to(torch.bfloat16)
    b = torch.randn(N, K, device="cuda").to(torch.bfloat16)
    c = torch.randn(N, device="cuda").to(torch.bfloat16)
    ref = a.float() @ b.float().t()
    rel = lambda got, want: ((got.float() - want).norm() / want.norm()).item()
    assert rel(gemm.matmul_nt(a, b, c), ref + c.float()) < 4e-3
    assert rel(gemm.matmul_nn(a, b.t().contiguous()), ref) < 4e-3
    assert rel(gemm.matmul_tn(a.t().contiguous(), b.t().contiguous()), ref) < 4e-3
    odd = torch.randn(N + 1, device="cuda").to(torch.bfloat16)[1:]         # a bias that 16-byte loads cannot read
    assert rel(gemm.matmul_nt(a, b, odd), ref + odd.float()) < 4e-3
    gemm.check_status()


@pytest.mark.parametrize("gelu", [False, True])
@pytest.mark.parametrize("rows,n", [(8, 16), (264, 512)])
@pytest.mark.parametrize("bias,frozen", [(False, ""), (False, "x"), (True, "w"), (True, "b"), (True, "xw")])
def test_linear_without_bias_and_with_frozen_inputs(gelu, rows, n, bias, frozen):
    """Every combination of a missing bias and inputs that want no gradient, with small operands and on the CTA-pair kernel."""
    from torchmpi_b200.ops import gemm
    torch.manual_seed(rows)
    k = 256
    t = {"x": torch.randn(2, rows, k), "w": torch.randn(n, k) / 16, "b": torch.randn(n)}
    t = {a: v.cuda().to(torch.bfloat16).requires_grad_(a not in frozen) for a, v in t.items()}
    r = {a: v.detach().float().requires_grad_(a not in frozen) for a, v in t.items()}
    y = gemm.linear(t["x"], t["w"], t["b"] if bias else None, gelu=gelu)
    z = torch.nn.functional.linear(r["x"], r["w"], r["b"] if bias else None)
    ref = torch.nn.functional.gelu(z) if gelu else z
    dy = torch.randn_like(y)
    y.backward(dy)
    ref.backward(dy.float())
    gemm.check_status()
    # one rounding to bf16 (2^-9) of the result, and with GELU of z before it and of dz in front of the products
    assert (y.float() - ref).norm() <= 2 ** -7 * ref.norm()
    for a in "xwb":
        if a in frozen or (a == "b" and not bias):
            assert t[a].grad is None
        else:
            assert (t[a].grad.float() - r[a].grad).norm() <= 2 ** -7 * r[a].grad.norm(), a


def test_refused_operands_of_linear_and_cross_entropy():
    """Operands that do not fit each other, an empty batch and types that no kernel takes raise before anything is launched."""
    from torchmpi_b200._lib import TorchMPIError
    from torchmpi_b200.ops import gemm, xent
    x = torch.zeros(16, 64, device="cuda", dtype=torch.bfloat16)
    for w in (torch.zeros(32, 128, device="cuda"), torch.zeros(32, 56, device="cuda"), torch.zeros(32, 64), torch.zeros(32, device="cuda")):
        for gelu in (False, True):
            with pytest.raises(ValueError):
                gemm.linear(x, w.to(torch.bfloat16), None, gelu=gelu)
    with pytest.raises(ZeroDivisionError):
        xent.cross_entropy(torch.zeros(0, 10, device="cuda"), torch.zeros(0, device="cuda", dtype=torch.int64))
    for dtype in (torch.float64, torch.int32, torch.int64):
        with pytest.raises(TorchMPIError):
            xent.cross_entropy(torch.zeros(4, 10, device="cuda", dtype=dtype), torch.zeros(4, device="cuda", dtype=torch.int64))
    with pytest.raises(TypeError):
        xent.cross_entropy(torch.zeros(4, 10, device="cuda", dtype=torch.complex64), torch.zeros(4, device="cuda", dtype=torch.int64))


def test_first_cuda_call_of_a_thread_encodes_a_tensor_map():
    """A thread without a current context (the autograd thread of a process whose backward begins here) may call a kernel
    that takes tensor maps before anything else has made the context current."""
    import threading
    from torchmpi_b200.ops import attention, conv, gemm, stem_conv
    from torchmpi_b200._lib import lib, check, stream_ptr
    a = torch.randn(256, 256, device="cuda").to(torch.bfloat16)
    want, out = gemm.matmul_nt(a, a), torch.empty(256, 256, device="cuda", dtype=torch.bfloat16)
    small, out_small = gemm.matmul_nt(a[:128], a), torch.empty(128, 256, device="cuda", dtype=torch.bfloat16)
    x = torch.randn(2, 64, 8, 8, device="cuda").to(torch.bfloat16).contiguous(memory_format=torch.channels_last)
    w = torch.randn(64, 64, 1, 1, device="cuda").to(torch.bfloat16).contiguous(memory_format=torch.channels_last)
    y = torch.nn.functional.conv2d(x, w)
    stem = stem_conv.StemConv7x7(64).cuda().to(torch.bfloat16)
    img = torch.randn(1, 3, 16, 16, device="cuda").to(torch.bfloat16).contiguous(memory_format=torch.channels_last)
    z = stem(img).detach()
    qkv = torch.randn(1, 128, 192, device="cuda").to(torch.bfloat16)
    o, _ = attention.attention_forward(qkv, 1)
    torch.cuda.synchronize()
    calls = {"pair": lambda: gemm.matmul_nt(a, a, out=out), "single": lambda: gemm.matmul_nt(a[:128], a, out=out_small),
             "conv": lambda: got.update(conv=conv.conv2d(x, w)), "stem": lambda: got.update(stem=stem(img).detach()),
             "attention": lambda: got.update(attention=attention.attention_forward(qkv, 1)[0])}
    got, errors = {}, {}

    def run(name, fn):
        try:
            with torch.no_grad():
                fn()
        except Exception as e:
            errors[name] = repr(e)
    for name, fn in calls.items():
        t = threading.Thread(target=run, args=(name, fn))
        t.start()
        t.join()
    assert not errors, errors
    torch.cuda.synchronize()
    assert torch.equal(out, want) and torch.equal(out_small, small) and torch.equal(got["stem"], z) and torch.equal(got["attention"], o)
    assert ((got["conv"].float() - y.float()).norm() / y.float().norm()).item() < 1e-2
