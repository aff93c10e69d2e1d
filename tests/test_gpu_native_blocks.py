"""The C++ functions of convolution and batch norm against the Python ones that blocks in flat buckets take: the same bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _block(first, planes=64):
    from torchmpi_b200.models import to_bf16_mixed
    from torchmpi_b200.models.resnet import Bottleneck, _bn
    inp, stride, down = planes * 4, 1, None
    torch.manual_seed(2)
    with torch.device("cuda"):
        if first:
            inp, stride = planes * 2, 2
            down = torch.nn.Sequential(torch.nn.Conv2d(inp, planes * 4, 1, stride=stride, bias=False), _bn(planes * 4, True, relu=False))
        m = Bottleneck(inp, planes, stride, down, fused_bn=True)
        for p in m.parameters():
            if p.dim() == 1:
                torch.nn.init.uniform_(p, 0.5, 1.5)
    return inp, to_bf16_mixed(m).to(memory_format=torch.channels_last)


@pytest.mark.parametrize("mode", ["train", "eval", "frozen input", "hooked", "no fork"])
@pytest.mark.parametrize("first", [False, True])
def test_bottleneck_takes_either_path(first, mode):
    from torchmpi_b200 import _native, config
    from torchmpi_b200.ops import bn_relu, conv

    def launched():                              # by the C++ functions, by the Python ones
        return [_native.launches(_native.CONV), _native.launches(_native.BATCHNORM)], [conv._launches, bn_relu._launches]
    inp, m = _block(first)
    m.train(mode != "eval")
    x = torch.randn(3, 12, 10, inp, device="cuda").to(torch.bfloat16).permute(0, 3, 1, 2)
    out, state = [], {k: v.clone() for k, v in m.state_dict().items()}
    config.set("grad_fork", 0 if mode == "no fork" else 1)
    try:
        for native in (True, False):
            m.load_state_dict(state)
            m.zero_grad(set_to_none=True)
            if not native:
                for p in m.parameters():
                    p._tmpi_grad_sink = lambda *a, **k: None                 # a gradient buffer that is not there yet: returned to autograd
            hook = m.bn3.register_forward_hook(lambda mod, args, y: None) if mode == "hooked" else None
            leaf = x.clone().requires_grad_(mode != "frozen input")
            before = launched()
            y = m(leaf)
            dy = torch.randn(y.shape, device="cuda", generator=torch.Generator("cuda").manual_seed(1)).to(y.dtype).contiguous(memory_format=torch.channels_last)
            y.backward(dy)
            cpp, py = ([n - o for n, o in zip(a, b)] for a, b in zip(launched(), before))
            assert all(cpp) and (mode == "hooked" or not any(py)) if native else all(py) and not any(cpp)      # (the hooked layer is Python's)
            conv.check_status()
            if hook is not None:
                hook.remove()
            out.append([y.detach(), leaf.grad] + [p.grad for p in m.parameters()] + [b.clone() for b in m.buffers()])
        with torch.no_grad():
            assert m(x).grad_fn is None
    finally:
        config.set("grad_fork", 1)
    for a, b in zip(*out):
        assert (a is None) == (b is None)
        if a is None:
            continue
        if mode == "hooked":                     # the hooked layer's statistics come from a pass of their own on one side
            assert (a.float() - b.float()).norm() <= 2e-2 * b.float().norm() + 1e-6
        else:
            assert torch.equal(a, b)


def _odd(t):
    """The values of a channels-last tensor, in a buffer in which they start two bytes behind a 16-byte boundary."""
    rows = t.permute(0, 2, 3, 1)
    buf = torch.empty(t.numel() + 8, device=t.device, dtype=t.dtype)[1:1 + t.numel()].view(rows.shape).copy_(rows).permute(0, 3, 1, 2)
    assert buf.data_ptr() % 16 == t.element_size() and buf.is_contiguous(memory_format=torch.channels_last)
    return buf


@pytest.mark.parametrize("layer", ["block", "block in flat buckets", "pool", "stem"])
def test_inputs_and_gradients_at_odd_addresses(layer):
    """Views into larger buffers are read through a copy: the kernels' loads need 16-byte boundaries."""
    from torchmpi_b200.models import to_bf16_mixed
    from torchmpi_b200.ops.bn_relu import FusedBatchNormReLUMaxPool
    from torchmpi_b200.ops.pool import MaxPool2d
    from torchmpi_b200.ops.stem_conv import StemConv7x7
    torch.manual_seed(3)
    if layer == "pool":
        m, shape = MaxPool2d(3, 2, 1), (2, 64, 12, 10)
    elif layer == "stem":
        m, shape = to_bf16_mixed(torch.nn.Sequential(StemConv7x7(64), FusedBatchNormReLUMaxPool(64)).cuda()).to(memory_format=torch.channels_last), (2, 3, 32, 64)
    else:
        inp, m = _block(False)
        shape = (3, inp, 12, 10)
        if layer == "block in flat buckets":
            for p in m.parameters():
                p._tmpi_grad_sink = lambda *a, **k: None
    x = torch.randn(shape, device="cuda").to(torch.bfloat16).contiguous(memory_format=torch.channels_last)
    state, out = {k: v.clone() for k, v in m.state_dict().items()}, []
    for place in (lambda t: t, _odd):
        m.load_state_dict(state)
        leaf = place(x).detach().requires_grad_(layer != "stem")
        y = m(leaf)
        dy = torch.randn(y.shape, device="cuda", generator=torch.Generator("cuda").manual_seed(1)).to(y.dtype).contiguous(memory_format=torch.channels_last)
        out.append([y] + list(torch.autograd.grad(y, ([leaf] if layer != "stem" else []) + list(m.parameters()), place(dy))))
    assert all(torch.equal(a, b) for a, b in zip(*out))


def test_masked_gradient_without_a_kernel_that_takes_it():
    """A residual's gradient that is parked as the incoming gradient and mask bits, and whose last consumer is another residual, or a
    strided convolution, which leave the mask to tensor operations."""
    from torchmpi_b200 import _native
    from torchmpi_b200.ops.bn_relu import FusedBatchNormReLU
    torch.manual_seed(4)
    new = lambda *s: torch.randn(*s, device="cuda").to(torch.bfloat16).to(memory_format=torch.channels_last)
    first, second = FusedBatchNormReLU(64).cuda(), FusedBatchNormReLU(64).cuda()
    w = new(64, 64, 1, 1).requires_grad_(True)
    a, b, r, dy, dz = (new(2, 64, 6, 6) for _ in range(5))
    for strided in (False, True):
        grads = []
        for fork in (_native.ext().Fork(2), None):
            leaf = r.clone().requires_grad_(True)
            # of the two consumers the one that ran last in forward is first in backward
            z = _native.ext().conv2d(leaf, w, 2, 0, fork) if strided else second(b, leaf, res_fork=fork)
            y = first(a, leaf, res_fork=fork)
            grads.append(torch.autograd.grad((z, y), leaf, (dz[:, :, ::2, ::2].contiguous(memory_format=torch.channels_last) if strided else dz, dy))[0].float())
        # one rounding of the sum to bf16, where autograd's own sum rounds the same terms
        assert bool(((grads[0] - grads[1]).abs() <= 2.0 ** -7 * grads[1].abs() + 1e-6).all()), strided


def test_block_on_a_side_stream_and_in_a_graph():
    """The functions' scratch is of the stream and the call."""
    inp, m = _block(False)
    x = torch.randn(2, 8, 8, inp, device="cuda").to(torch.bfloat16).permute(0, 3, 1, 2)

    def grads():
        leaf = x.clone().requires_grad_(True)
        y = m(leaf)
        return torch.autograd.grad(y, [leaf] + list(m.parameters()), torch.ones_like(y))
    want = grads()
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        got = grads()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            captured = grads()
    graph.replay()
    torch.cuda.synchronize()
    for a, b, c in zip(want, got, captured):
        assert torch.equal(a, b) and torch.equal(a, c)


def _layers():
    """(module, input, whether its gradient is wanted)"""
    from torchmpi_b200.models import to_bf16_mixed
    from torchmpi_b200.ops import attention, gemm, layernorm
    from torchmpi_b200.ops.bn_relu import FusedBatchNormReLUMaxPool
    from torchmpi_b200.ops.stem_conv import StemConv7x7
    bf16 = {"device": "cuda", "dtype": torch.bfloat16}

    class Head(torch.nn.Module):
        def __init__(self):
            super().__init__()
            self.weight = torch.nn.Parameter(torch.randn(1003, 256, **bf16))

        def forward(self, x):
            return gemm.wide_head(x, self.weight)

    class Attention(torch.nn.Module):
        def forward(self, x):
            return attention.causal_attention(x, 2)
    image = torch.randn(2, 32, 64, 3, **bf16).permute(0, 3, 1, 2)
    stem = to_bf16_mixed(torch.nn.Sequential(StemConv7x7(64), FusedBatchNormReLUMaxPool(64)).cuda()).to(memory_format=torch.channels_last)
    with torch.device("cuda"):
        up, wide, down = (gemm.Linear(128, n, gelu=g, dtype=torch.bfloat16) for n, g in ((384, True), (1024, True), (384, False)))
    x = torch.randn(256, 128, **bf16)
    sinks = _block(False)[1]
    for p in sinks.parameters():
        p._tmpi_grad_sink = lambda *a, **k: None
    yield from ((up, x, True), (up, x, False), (wide, x, True), (down, x, True), (Head(), torch.randn(256, 256, **bf16), True),
                (layernorm.LayerNorm(256, **bf16), torch.randn(40, 256, **bf16), True), (Attention(), torch.randn(2, 128, 384, **bf16), True), (stem, image, False))
    for first in (False, True):
        inp, m = _block(first)
        yield m, torch.randn(3, 12, 10, inp, **bf16).permute(0, 3, 1, 2), True
    yield sinks, torch.randn(3, 12, 10, 256, **bf16).permute(0, 3, 1, 2), True


def test_saved_tensors_in_another_layout():
    """Hooks on saved tensors may hand back the same values in another order in memory (save_on_cpu with pinned memory does)."""
    torch.manual_seed(5)
    for at, (m, x, grad) in enumerate(_layers()):
        out, state = [], {k: v.clone() for k, v in m.state_dict().items()}
        for relayout in (lambda t: t, lambda t: t.clone(memory_format=torch.contiguous_format), lambda t: t.transpose(0, 1).contiguous().transpose(0, 1) if t.dim() > 1 else t):
            m.load_state_dict(state)
            m.zero_grad(set_to_none=True)
            leaf = x.clone().requires_grad_(grad)
            with torch.autograd.graph.saved_tensors_hooks(lambda t: t, relayout):
                y = m(leaf)
            y.backward(torch.randn(y.shape, device="cuda", generator=torch.Generator("cuda").manual_seed(1)).to(y.dtype))
            out.append([leaf.grad] + [p.grad for p in m.parameters()])
        for other in out[1:]:
            for a, b in zip(out[0], other):
                # the sums of attention's dQ have no fixed order, and the library's 3 x 3 convolutions go by the layout: some roundings to bf16
                # (2^-8) differ; values in the wrong places differ by more than their norm
                same = a is None and b is None or (torch.equal(a, b) if at < 6 or at == 7 else (a.float() - b.float()).norm() <= 2e-2 * a.float().norm())
                assert same, (at, m)
    # a bias alone
    m, x, _ = next(_layers())
    m.weight.requires_grad_(False)
    out = []
    for relayout in (lambda t: t, lambda t: t.t().contiguous().t() if t.dim() > 1 else t):
        m.bias.grad = None
        with torch.autograd.graph.saved_tensors_hooks(lambda t: t, relayout):
            y = m(x)
        y.backward(torch.ones_like(y))
        out.append(m.bias.grad)
    assert torch.equal(*out)
