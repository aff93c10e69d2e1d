"""Causal attention whose items are shared by the two teams of a CTA, against fp64."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _rand(*shape):
    return torch.randn(*shape, device="cuda").to(torch.bfloat16)


def _attention64(qkv, heads):
    B, T, C3 = qkv.shape
    q, k, v = (t.reshape(B, T, heads, 64).transpose(1, 2) for t in qkv.split(C3 // 3, dim=2))
    s = (q @ k.transpose(-1, -2)) * 0.125
    s = s.masked_fill(torch.ones(T, T, dtype=torch.bool, device=qkv.device).triu(1), -math.inf)
    return (torch.softmax(s, -1) @ v).transpose(1, 2).reshape(B, T, C3 // 3)


# one to sixteen key blocks per item; fewer items than CTAs, one to two and more rounds of items shared by two teams
@pytest.mark.parametrize("B,T,H", [(1, 128, 1), (1, 256, 3), (1, 384, 1), (1, 640, 2), (1, 1920, 4), (1, 2048, 16), (3, 1024, 12), (2, 2048, 11)])
def test_attention_items_shared_by_teams(B, T, H):
    from torchmpi_b200.ops import attention
    torch.manual_seed(T + H)
    qkv = _rand(B, T, 3 * H * 64)
    qkv[0, T // 3, : H * 64] *= 8.0                        # one query whose weights lie far apart
    qkv.requires_grad_(True)
    y = attention.causal_attention(qkv, H)
    dy = _rand(B, T, H * 64)
    y.backward(dy)
    x = qkv.detach().double().requires_grad_(True)
    ref = _attention64(x, H)
    ref.backward(dy.double())
    shared, _ = _forward(qkv.detach(), H, True)            # whichever form the rule takes at this size
    # probabilities in bf16: 2^-9 of sums of order one each way; the gradient's products twice
    assert ((shared.double() - ref).norm() / ref.norm()) < 5e-3
    assert (shared.double() - ref).abs().max() < 3e-2
    assert ((y.double() - ref).norm() / ref.norm()) < 5e-3
    assert (y.double() - ref).abs().max() < 3e-2
    assert ((qkv.grad.double() - x.grad).norm() / x.grad.norm()) < 1e-2


@pytest.mark.parametrize("T", [256, 1024])
def test_attention_shared_items_non_finite(T):
    """A key that scores -inf weighs nothing wherever the split lies; NaN and +inf reach the rows that see them, and no others."""
    from torchmpi_b200._lib import lib
    from torchmpi_b200.ops import attention
    torch.manual_seed(1)
    for value, at in ((-math.inf, T - 3), (math.nan, T // 2 + 5), (math.inf, 70)):
        qkv = _rand(1, T, 192)
        qkv[:, :, 0] = 1.0                                  # first query coordinate: the key's decides the score
        qkv[0, at, 64] = value
        with torch.no_grad():
            y = attention.causal_attention(qkv, 1)
        assert lib.tmpi_attention_fwd_shares(1, T, 1) and torch.equal(y.nan_to_num(9.0), _forward(qkv, 1, True)[0].nan_to_num(9.0))
        assert torch.isfinite(y[0, :at]).all()
        if value == -math.inf:
            ref = _attention64(torch.cat([qkv[..., :64], qkv[..., 64:128].nan_to_num(neginf=-1e30), qkv[..., 128:]], -1).double(), 1)
            assert torch.isfinite(y).all() and (y.double() - ref)[0].abs().max() < 3e-2
        else:
            assert torch.isnan(y[0, at:]).all()


def _forward(qkv, heads, shared, scale=0.125):
    """(out, lse) of one form of the kernel: a team per item, or items shared by the two teams of a CTA."""
    from torchmpi_b200._lib import check, lib, stream_ptr
    B, T, C3 = qkv.shape
    C = C3 // 3
    out = torch.empty((B, T, C), dtype=qkv.dtype, device=qkv.device)
    lse = torch.empty((B, heads, T), dtype=torch.float32, device=qkv.device)
    base = qkv.data_ptr()
    check(lib.tmpi_attention_fwd_form(base, base + 2 * C, base + 4 * C, C3, out.data_ptr(), C, lse.data_ptr(), B, T, heads, scale,
                                      int(shared), stream_ptr()))
    return out, lse


# keys of whole blocks that score -inf: the middle one, where the second team of the last items starts; the first; the one on the
# last diagonal, all but its last key; several, so that a team has none or only some of its keys left
@pytest.mark.parametrize("shared", [False, True])
@pytest.mark.parametrize("T,keys,scale", [(1024, (512, 640), 0.125), (1024, (0, 128), 0.125), (1024, (896, 1023), 0.125),
                                          (1024, (512, 1023), 0.125), (1024, (128, 900), 0.125), (1024, (0, 600), 0.125),
                                          (1024, (0, 600), 0.69), (384, (256, 383), 0.125), (256, (128, 255), 0.125), (640, (384, 512), 0.125)])
def test_attention_blocks_of_minus_infinity(shared, T, keys, scale):
    from torchmpi_b200.ops import attention
    torch.manual_seed(T + keys[0])
    qkv = _rand(2, T, 192)
    qkv[:, :, 0] = 1.0                                      # first query coordinate: the key's decides the score
    qkv[:, keys[0]:keys[1], 64] = -math.inf
    y, lse = _forward(qkv, 1, shared, scale)
    attention.check_status()
    finite = torch.cat([qkv[..., :64], qkv[..., 64:128].nan_to_num(neginf=-1e30), qkv[..., 128:]], -1).double()
    s = (finite[..., :64] @ finite[..., 64:128].transpose(1, 2)) * scale
    s = s.masked_fill(torch.ones(T, T, dtype=torch.bool, device="cuda").triu(1), -math.inf)
    s = s.masked_fill(s < -1e20, -math.inf)
    ref = torch.softmax(s, -1) @ finite[..., 128:]          # NaN where every key of a row scores -inf
    sees = torch.arange(T, device="cuda") >= (keys[1] if keys[0] == 0 else 0)
    assert torch.isnan(y[:, ~sees]).all() and torch.isfinite(y[:, sees]).all()
    # probabilities and output in bf16 of values of order one
    assert (y.double() - ref)[:, sees].abs().max() < 3e-2
    assert (lse[:, 0].double() - torch.logsumexp(s, -1))[:, sees].abs().max() < 2e-3
