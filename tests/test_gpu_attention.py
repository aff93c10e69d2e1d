"""The tcgen05 causal attention forward against fp32 softmax(Q K^T / sqrt(d)) V, its log-sum-exp, and the gradient
of the autograd op against PyTorch's own attention in fp32."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _ref(qkv, H):
    B, T, C3 = qkv.shape
    C = C3 // 3
    q, k, v = (t.view(B, T, H, 64).transpose(1, 2).float() for t in qkv.split(C, dim=2))
    s = q @ k.transpose(-1, -2) / math.sqrt(64)
    mask = torch.ones(T, T, dtype=torch.bool, device=qkv.device).tril()
    s = s.masked_fill(~mask, float("-inf"))
    lse = torch.logsumexp(s, dim=-1)
    out = torch.softmax(s, dim=-1) @ v
    return out.transpose(1, 2).reshape(B, T, C), lse


@pytest.mark.parametrize("B,T,H", [(1, 128, 1), (2, 256, 3), (2, 1024, 4), (1, 512, 16), (1, 2048, 2)])
def test_attention_forward_matches_fp32(B, T, H):
    from torchmpi_b200.ops import attention
    from torchmpi_b200._lib import lib
    torch.manual_seed(B * 1000 + T + H)
    qkv = (torch.randn(B, T, 3 * H * 64, device="cuda") * 1.5).to(torch.bfloat16)
    assert attention.supported(qkv, H)
    out, lse = attention.attention_forward(qkv, H)
    torch.cuda.synchronize()
    attention.check_status()
    ref, ref_lse = _ref(qkv, H)
    assert torch.allclose(lse, ref_lse, atol=2e-3, rtol=1e-4), (lse - ref_lse).abs().max().item()
    err = (out.float() - ref).abs().max().item()
    assert err < 2e-2, err                         # bf16 probabilities and bf16 output of values of order 1
    rel = ((out.float() - ref).norm() / ref.norm()).item()
    assert rel < 6e-3, rel
    # same input, same bits
    out2, _ = attention.attention_forward(qkv, H)
    assert torch.equal(out, out2)
    assert lib.tmpi_attention_ctas_per_sm() >= 1


def test_attention_autograd_and_fallback():
    from torchmpi_b200.ops import attention
    torch.manual_seed(5)
    B, T, H = 2, 256, 4
    qkv = torch.randn(B, T, 3 * H * 64, device="cuda").to(torch.bfloat16).requires_grad_(True)
    before = attention.launch_count
    out = attention.causal_attention(qkv, H)
    assert attention.launch_count == before + 1
    g = torch.randn_like(out)
    out.backward(g)
    assert attention.last_backward == "own"
    attention.check_status()
    leaf = qkv.detach().float().requires_grad_(True)
    ref, _ = _ref(leaf, H)
    ref.backward(g.float())
    rel = ((qkv.grad.float() - leaf.grad).norm() / leaf.grad.norm()).item()
    assert rel < 2e-2, (rel, attention.last_backward)
    # every backward route gives the same gradient
    first = attention.last_backward
    for route in ("cudnn", "flash", "none"):
        attention._BACKWARDS = (route,)
        try:
            q2 = qkv.detach().clone().requires_grad_(True)
            attention.causal_attention(q2, H).backward(g)
            assert attention.last_backward == ("recompute" if route == "none" else route) or attention.last_backward == "recompute"
            rel = ((q2.grad.float() - leaf.grad).norm() / leaf.grad.norm()).item()
            assert rel < 2e-2, (rel, route)
        finally:
            attention._BACKWARDS = ("own", "cudnn", "flash")
    assert first == "own"
    # shapes the kernel does not take go to PyTorch's attention
    odd = torch.randn(1, 100, 3 * 2 * 64, device="cuda").to(torch.bfloat16)
    assert not attention.supported(odd, 2)
    o = attention.causal_attention(odd, 2)
    r, _ = _ref(odd, 2)
    assert ((o.float() - r).norm() / r.norm()).item() < 1e-2


def test_gpt2_block_uses_own_attention():
    from torchmpi_b200.models import gpt2
    from torchmpi_b200.ops import attention
    torch.manual_seed(0)
    m = gpt2.gpt2_tiny(n_head=2, n_embd=128, block_size=256, tc_linear=True).cuda().to(torch.bfloat16)
    ref = gpt2.gpt2_tiny(n_head=2, n_embd=128, block_size=256, tc_linear=False).cuda().to(torch.bfloat16)
    ref.load_state_dict(m.state_dict())
    idx = torch.randint(0, 512, (2, 256), device="cuda")
    before = attention.launch_count
    y = m(idx)
    assert attention.launch_count == before + len(m.blocks)
    yr = ref(idx)
    rel = ((y.float() - yr.float()).norm() / yr.float().norm()).item()
    assert rel < 3e-2, rel


def test_attention_phase_trace_is_ordered():
    """The tuning aid: CTA 0 stamps the phases of every key block in order, and switching it off stops the writes."""
    from torchmpi_b200.ops import attention
    from torchmpi_b200._lib import lib
    T, H = 512, 2
    qkv = torch.randn(1, T, 3 * H * 64, device="cuda").to(torch.bfloat16)
    buf = torch.zeros((T // 128) * 16, dtype=torch.int64, device="cuda")
    lib.tmpi_attention_set_trace(buf.data_ptr())
    try:
        attention.attention_forward(qkv, H)
        torch.cuda.synchronize()
    finally:
        lib.tmpi_attention_set_trace(None)
    t = buf.cpu().view(T // 128, 16)
    for j in range(T // 128):                      # CTA 0 handles the last query block: T / 128 key blocks
        has_s, max_known, p_written, has_o, updated = (int(t[j, e]) for e in (1, 2, 3, 5, 6))
        assert 0 < has_s <= max_known <= p_written <= has_o <= updated, (j, t[j].tolist())
    buf.zero_()
    attention.attention_forward(qkv, H)
    torch.cuda.synchronize()
    assert int(buf.abs().sum()) == 0


@pytest.mark.parametrize("B,T,H", [(1, 128, 1), (2, 384, 2), (1, 1024, 3), (1, 2048, 2)])
def test_attention_backward_matches_fp32(B, T, H):
    """dQ, dK, dV of the tcgen05 backward kernel against fp32 autograd of softmax(Q K^T / sqrt(d)) V."""
    from torchmpi_b200.ops import attention
    torch.manual_seed(B + T + H)
    qkv = torch.randn(B, T, 3 * H * 64, device="cuda").to(torch.bfloat16)
    out, lse = attention.attention_forward(qkv, H)
    dout = torch.randn_like(out)
    dqkv = attention.attention_backward(qkv, out, lse, dout, H)
    torch.cuda.synchronize()
    attention.check_status()
    leaf = qkv.detach().float().requires_grad_(True)
    ref, _ = _ref(leaf, H)
    ref.backward(dout.float())
    C = H * 64
    for name, sl in (("dq", slice(0, C)), ("dk", slice(C, 2 * C)), ("dv", slice(2 * C, 3 * C))):
        got, want = dqkv[:, :, sl].float(), leaf.grad[:, :, sl]
        rel = ((got - want).norm() / want.norm()).item()
        assert rel < 1.5e-2, (name, rel)
    # dK and dV are bit-reproducible; dQ is summed in arrival order
    dqkv2 = attention.attention_backward(qkv, out, lse, dout, H)
    assert torch.equal(dqkv[:, :, C:], dqkv2[:, :, C:])
    assert torch.allclose(dqkv[:, :, :C].float(), dqkv2[:, :, :C].float(), atol=1e-2, rtol=1e-2)


@pytest.mark.parametrize("B,T,H", [(5, 384, 24), (40, 128, 16), (1, 640, 1)])
def test_attention_several_items_per_team_and_growing_maxima(B, T, H):
    """More (block, head) items than persistent teams (rings and accumulators reused across items), and keys that grow
    along the sequence, so that the running maximum of most rows moves in every block and O is rescaled."""
    from torchmpi_b200.ops import attention
    torch.manual_seed(B * T + H)
    C = H * 64
    qkv = torch.randn(B, T, 3 * C, device="cuda")
    qkv[:, :, C:2 * C] *= torch.linspace(0.2, 2.5, T, device="cuda")[None, :, None]
    qkv = qkv.to(torch.bfloat16)
    leaf = qkv.detach().float().requires_grad_(True)
    ref, ref_lse = _ref(leaf, H)
    out, lse = attention.attention_forward(qkv, H)
    dout = torch.randn_like(out)
    dqkv = attention.attention_backward(qkv, out, lse, dout, H)
    torch.cuda.synchronize()
    attention.check_status()
    ref.backward(dout.float())
    assert torch.allclose(lse, ref_lse, atol=2e-3, rtol=1e-4), (lse - ref_lse).abs().max().item()
    rel = lambda a, b: ((a.float() - b).norm() / b.norm()).item()
    # bf16 P and outputs: 2^-9 relative rounding each; the gradients go through two more roundings (dS, the result)
    assert rel(out, ref.detach()) < 6e-3, rel(out, ref.detach())
    for name, sl in (("dq", slice(0, C)), ("dk", slice(C, 2 * C)), ("dv", slice(2 * C, 3 * C))):
        assert rel(dqkv[:, :, sl], leaf.grad[:, :, sl]) < 1.5e-2, (name, rel(dqkv[:, :, sl], leaf.grad[:, :, sl]))


@pytest.mark.parametrize("t0", [1, 6, 39, 70, 135, 200])
def test_attention_later_tokens_leave_earlier_rows_alone(t0):
    """Values of 1e38 behind the mask change no bit of the rows in front of them, and visible values of zero give zero:
    a masked key has a probability of exactly 0."""
    from torchmpi_b200.ops import attention
    torch.manual_seed(t0)
    B, T, H = 2, 256, 3
    C = H * 64
    qkv = torch.randn(B, T, 3 * C, device="cuda").to(torch.bfloat16)
    out, lse = attention.attention_forward(qkv, H)
    big = qkv.clone()
    big[:, t0:, 2 * C:] = 1e38
    out2, lse2 = attention.attention_forward(big, H)
    big[:, :t0, 2 * C:] = 0.0
    out3, _ = attention.attention_forward(big, H)
    torch.cuda.synchronize()
    attention.check_status()
    assert torch.equal(out2[:, :t0], out[:, :t0]) and torch.equal(lse2, lse)
    assert torch.count_nonzero(out3[:, :t0]) == 0


@pytest.mark.parametrize("key", [0, 5, 6, 7, 38, 63, 100, 134, 191])
def test_attention_non_finite_scores(key):
    """A score that is NaN or overflows to infinity makes its row NaN wherever its key lies; rows before the key and the
    other head keep their bits."""
    from torchmpi_b200.ops import attention
    torch.manual_seed(key)
    T, H, row = 256, 2, 250
    C = H * 64
    qkv = torch.randn(1, T, 3 * C, device="cuda").to(torch.bfloat16)
    out, lse = attention.attention_forward(qkv, H)
    bad = qkv.clone()
    bad[0, key, C + 3] = float("nan")
    out_nan, lse_nan = attention.attention_forward(bad, H)
    huge = qkv.clone()
    huge[0, row, :64] = 1e30
    huge[0, key, C:C + 64] = 1e30
    out_inf, lse_inf = attention.attention_forward(huge, H)
    torch.cuda.synchronize()
    attention.check_status()
    for o, l in ((out_nan, lse_nan), (out_inf, lse_inf)):
        assert torch.equal(o[:, :key], out[:, :key]) and torch.equal(o[:, :, 64:], out[:, :, 64:])
        assert torch.equal(l[:, 0, :key], lse[:, 0, :key]) and torch.equal(l[:, 1], lse[:, 1])
    assert out_nan[0, key:, :64].isnan().all() and lse_nan[0, 0, key:].isnan().all()
    assert out_inf[0, row, :64].isnan().all() and lse_inf[0, 0, row].isnan()


def test_last_backward_names_a_backward_that_ran():
    from torchmpi_b200.ops import attention
    qkv = torch.randn(1, 128, 3 * 64, device="cuda").to(torch.bfloat16).requires_grad_(True)
    attention._BACKWARDS = ("none",)
    try:
        attention.causal_attention(qkv, 1).sum().backward()
    finally:
        attention._BACKWARDS = ("own", "cudnn", "flash")
    assert attention.last_backward == "recompute"
    out = attention.causal_attention(qkv, 1)
    assert attention.last_backward == "recompute"          # a forward names nothing
    out.sum().backward()
    assert attention.last_backward == "own"
    out, lse = attention.attention_forward(qkv.detach(), 1)
    assert attention.last_backward == "own"
