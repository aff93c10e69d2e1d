"""Linear layers of few rows or columns, and weight gradients split over their rows, against fp64."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def _rand(*shape, scale=1.0):
    return (torch.randn(*shape, device="cuda") * scale).to(torch.bfloat16)


# fewer rows or columns than a tile of the pair kernel, one pack, remainders of tiles; the last three split the weight gradient
@pytest.mark.parametrize("rows,inp,out", [(8, 8, 8), (8, 128, 384), (24, 2048, 1000), (200, 256, 128), (256, 1024, 1536), (1000, 136, 768),
                                          (4096, 128, 104), (8192, 128, 512), (8200, 1024, 1000)])
@pytest.mark.parametrize("gelu", [False, True])
def test_linear_of_few_rows_or_columns(rows, inp, out, gelu):
    from torchmpi_b200.ops import gemm
    torch.manual_seed(rows + out)
    x = _rand(rows, inp).requires_grad_(True)
    w = _rand(out, inp, scale=inp ** -0.5).requires_grad_(True)
    b = _rand(out, scale=0.1).requires_grad_(True)
    y = gemm.linear(x, w, b, gelu)
    dy = _rand(rows, out)
    y.backward(dy)
    xr, wr, br = (t.detach().double().requires_grad_(True) for t in (x, w, b))
    z = F.linear(xr, wr, br)
    z = z + (z.to(torch.bfloat16).double() - z).detach()     # the pre-activation is kept in bf16
    yr = F.gelu(z) if gelu else z
    yr.backward(dy.double())
    for got, ref in ((y, yr), (x.grad, xr.grad), (w.grad, wr.grad), (b.grad, br.grad)):
        # dz is rounded to bf16 before the products and the sum; each result once more
        assert ((got.double() - ref).norm() / ref.norm()) < 6e-3
        assert (got.double() - ref).abs().max() <= 2.0 ** -6 * ref.abs().max()
