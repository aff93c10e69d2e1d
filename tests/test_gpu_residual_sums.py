"""Residual sums inside the projection's epilogue and the layer norm's backward, against fp64 and against the separate sums."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def _rand(*shape, dtype=torch.bfloat16, scale=1.0):
    return (torch.randn(*shape, device="cuda") * scale).to(dtype)


# one pack, remainders of a 64-column slice and of a tile in both directions, several rounds of tiles
@pytest.mark.parametrize("rows,inp,out", [(8, 8, 8), (136, 64, 72), (256, 128, 320), (1000, 520, 1000), (8192, 256, 1024), (8200, 64, 3072)])
@pytest.mark.parametrize("bias", [True, False])
def test_linear_add(rows, inp, out, bias):
    from torchmpi_b200.ops import gemm
    torch.manual_seed(rows)
    x, w, r = _rand(rows, inp).requires_grad_(True), _rand(out, inp, scale=inp ** -0.5).requires_grad_(True), _rand(rows, out).requires_grad_(True)
    b = _rand(out).requires_grad_(True) if bias else None
    y = gemm.linear_add(x, w, b, r)
    dy = _rand(rows, out)
    y.backward(dy)
    gemm.check_status()
    ref = x.detach().double() @ w.detach().double().t() + (b.detach().double() if bias else 0) + r.detach().double()
    # one rounding to bf16 (8 significant bits), and the fp32 sums: inp / 16 roundings of partial sums of about sqrt(inp) * inp^-0.5
    assert bool(((y.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + (inp / 16 + 4) * 2.0 ** -23 * 16).all())
    assert torch.equal(r.grad, dy)
    xl, wl = x.detach().clone().requires_grad_(True), w.detach().clone().requires_grad_(True)
    bl = b.detach().clone().requires_grad_(True) if bias else None
    gemm.linear(xl, wl, bl).backward(dy)
    assert torch.equal(x.grad, xl.grad) and torch.equal(w.grad, wl.grad) and (not bias or torch.equal(b.grad, bl.grad))


@pytest.mark.parametrize("dtype,widths", [(torch.bfloat16, (256, 768, 1024, 1280, 1536, 2048)), (torch.float16, (512,)), (torch.float32, (128, 512, 640, 768, 1024))])
@pytest.mark.parametrize("rows", [1, 9, 2500])
def test_layer_norm_adds_the_other_gradient(dtype, widths, rows):
    from torchmpi_b200.ops import layernorm
    for width in widths:
        torch.manual_seed(width)
        x, w, b = _rand(rows, width, dtype=dtype).requires_grad_(True), _rand(width, dtype=dtype).requires_grad_(True), _rand(width, dtype=dtype).requires_grad_(True)
        y, same = layernorm.layer_norm_fork(x, w, b, 1e-5)
        assert torch.equal(same, x)
        dy, dr = _rand(rows, width, dtype=dtype), _rand(rows, width, dtype=dtype)
        got = torch.autograd.grad((y, same), (x, w, b), (dy, dr))
        layernorm.check_status()
        xd, wd, bd = (t.detach().double().requires_grad_(True) for t in (x, w, b))
        ref = torch.autograd.grad((F.layer_norm(xd, (width,), wd, bd, 1e-5), xd * 1.0), (xd, wd, bd), (dy.double(), dr.double()))
        unit = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11, torch.float32: 2.0 ** -20}[dtype]
        for g, r in zip(got, ref):       # one rounding, and fp32 arithmetic on values around one (sums over the rows for w and b)
            assert bool(((g.double() - r).abs() <= unit * r.abs() + 2.0 ** -19 * (rows ** 0.5 + 4)).all()), width


def test_layer_norm_fork_with_one_branch():
    from torchmpi_b200.ops import layernorm
    x, w, b = _rand(64, 512).requires_grad_(True), _rand(512).requires_grad_(True), _rand(512).requires_grad_(True)
    dy = _rand(64, 512)
    (alone,) = torch.autograd.grad(layernorm.layer_norm_fork(x, w, b, 1e-5)[1], x, dy)
    assert torch.equal(alone, dy)
    got = torch.autograd.grad(layernorm.layer_norm_fork(x, w, b, 1e-5)[0], (x, w, b), dy)
    from torchmpi_b200 import _native
    want = torch.autograd.grad(_native.ext().layer_norm(x, w, b, 1e-5), (x, w, b), dy)
    assert all(torch.equal(a, c) for a, c in zip(got, want))


@pytest.mark.parametrize("batch,seq,heads", [(1, 128, 4), (3, 256, 8)])
def test_block_with_and_without_hooks(batch, seq, heads):
    """A hooked projection sees its own output, so the block forms the sums outside; both forms agree to the rounding of the sums."""
    from torchmpi_b200.models.gpt2 import Block, GPT2Config
    torch.manual_seed(1)
    width = heads * 64
    m = Block(GPT2Config(n_head=heads, n_embd=width, tc_linear=True)).cuda().to(torch.bfloat16)
    x, dy = _rand(batch, seq, width), _rand(batch, seq, width)
    seen, out = [], []
    for hooked in (False, True):
        h = m.proj.register_forward_hook(lambda mod, args, y: seen.append(y.detach())) if hooked else None
        m.zero_grad(set_to_none=True)
        leaf = x.clone().requires_grad_(True)
        y = m(leaf)
        y.backward(dy)
        out.append([y.detach(), leaf.grad] + [p.grad for p in m.parameters()])
        if h is not None:
            h.remove()
    assert len(seen) == 1 and float((seen[0].float() - x.float()).norm() / x.float().norm()) > 0.5       # not the sum
    for a, c in zip(*out):
        assert float((a.float() - c.float()).norm() / c.float().norm()) < 2e-2


@pytest.mark.parametrize("rows,width", [(256, 256), (1024, 1024)])
def test_residual_and_bias_of_the_kernel_in_front(rows, width):
    """The product starts before the layer norm that writes its residual (and a row of which is its bias) has ended."""
    from torchmpi_b200 import _native
    from torchmpi_b200.ops import gemm
    torch.manual_seed(rows)
    x, w, one, zero = _rand(rows, width), _rand(width, width, scale=width ** -0.5), _rand(width), _rand(width)
    outs = []
    for sync in (torch.cuda.synchronize, lambda: None):
        out = []
        for k in range(8):                                                   # each norm's output lies where the one before lay
            t = x + k
            sync()
            r = _native.ext().layer_norm(t * (k + 1.0), one, zero, 1e-5 * (k + 1))
            sync()
            out.append(gemm.linear_add(x, w, r[k], r * 1.0 if k % 2 else r))
            sync()
            del r
        outs.append(out)
    assert all(torch.equal(a, b) for a, b in zip(*outs))
