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
    from torchmpi_b200 import config
    from torchmpi_b200.ops import bn_relu, conv
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
                m.conv1.weight._tmpi_grad_sink = lambda *a, **k: None        # a gradient buffer that is not there yet: returned to autograd
                for b in (m.bn1, m.bn2, m.bn3):
                    b.weight._tmpi_grad_sink = lambda *a, **k: None
            hook = m.bn3.register_forward_hook(lambda mod, args, y: None) if mode == "hooked" else None
            leaf = x.clone().requires_grad_(mode != "frozen input")
            before = conv.launch_count, bn_relu.launch_count
            y = m(leaf)
            dy = torch.randn(y.shape, device="cuda", generator=torch.Generator("cuda").manual_seed(1)).to(y.dtype).contiguous(memory_format=torch.channels_last)
            y.backward(dy)
            assert conv.launch_count > before[0] and bn_relu.launch_count > before[1]
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
