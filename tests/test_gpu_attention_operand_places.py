"""Q, K and V as column blocks of one matrix in either order, and as matrices of their own: the same bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,T,H", [(1, 128, 1), (2, 384, 3)])
def test_packed_and_separate_operands(B, T, H):
    from torchmpi_b200._lib import check, lib, stream_ptr
    torch.manual_seed(T)
    C = H * 64
    parts = [torch.randn(B * T, C, device="cuda").to(torch.bfloat16) for _ in range(3)]
    dout = torch.randn(B * T, C, device="cuda").to(torch.bfloat16)

    def run(place, ld):
        """place: one buffer and the columns of q, k, v in it, or None for three buffers."""
        if place is None:
            q, k, v = (p.clone() for p in parts)
            grads = [torch.full_like(p, float("nan")) for p in parts]
        else:
            buf, gbuf = (torch.full((B * T, ld), float("nan"), device="cuda", dtype=torch.bfloat16) for _ in range(2))
            q, k, v = (buf[:, c:c + C].copy_(p) for c, p in zip(place, parts))
            grads = [gbuf[:, c:c + C] for c in place]
        out, lse = torch.empty(B * T, C, device="cuda", dtype=torch.bfloat16), torch.empty(B, H, T, device="cuda")
        check(lib.tmpi_attention_fwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), ld, out.data_ptr(), C, lse.data_ptr(), B, T, H, 0.125, stream_ptr()))
        delta, acc = torch.empty_like(lse), torch.empty(B * T, C, device="cuda")
        check(lib.tmpi_attention_bwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), ld, out.data_ptr(), C, dout.data_ptr(), C, lse.data_ptr(), delta.data_ptr(),
                                     acc.data_ptr(), *(g.data_ptr() for g in grads), ld, B, T, H, 0.125, stream_ptr()))
        return [out, lse] + [g.clone() for g in grads]

    want = run(None, C)
    for place, ld in (((0, C, 2 * C), 3 * C), ((2 * C, C, 0), 3 * C), ((C, 0, 2 * C), 3 * C), ((8, C + 16, 2 * C + 24), 3 * C + 40)):
        got = run(place, ld)
        for i, (a, b) in enumerate(zip(got, want)):
            if i == 2:                    # dQ is summed in an order that is not fixed
                assert float((a.float() - b.float()).norm()) <= 2.0 ** -8 * float(b.float().norm())
            else:
                assert torch.equal(a, b), (place, i)
    assert lib.tmpi_attention_status() == 0 and lib.tmpi_attention_bwd_status() == 0
