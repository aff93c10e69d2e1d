"""Entries whose kernels use 16-byte loads and stores refuse tensors that do not start on a 16-byte boundary, before anything is launched."""
import pytest
import torch

from torchmpi_b200._lib import TorchMPIError, check, has_symbol, lib

# only where no kernel could run: an entry that failed to refuse would launch one on addresses that are made up
pytestmark = pytest.mark.skipif(torch.cuda.is_available() or not has_symbol("tmpi_bn_relu_fwd"), reason="needs the CUDA library and no GPU")
A = 1 << 20


def _bf16():
    from torchmpi_b200._lib import dtype_code
    return dtype_code(torch.bfloat16)


# name, its tensors, and the call with those at the addresses p
CALLS = {
    "bn forward": (("x", "residual", "y"), lambda p, t: lib.tmpi_bn_relu_fwd(p[0], p[1], p[2], A, A, None, None, A, A, 64, 64, 1e-5, 0.1, 1, 1, t, A, A, None)),
    "bn backward": (("x", "y", "dy", "dx", "dresidual"), lambda p, t: lib.tmpi_bn_relu_bwd_acc(p[0], p[1], p[2], p[3], p[4], A, A, A, A, A, A, 64, 64, 1, t, A, A, None, None, None)),
    "bn pool forward": (("x", "y", "idx", "xmax"), lambda p, t: lib.tmpi_bn_relu_pool_fwd_keep(p[0], p[1], p[2], p[3], A, A, None, None, A, A, 1, 8, 8, 64, 1e-5, 0.1, 1, t, A, None)),
    "bn pool backward": (("x", "xmax", "dy", "idx", "dx"), lambda p, t: lib.tmpi_bn_relu_pool_bwd_kept(p[0], p[1], p[2], p[3], p[4], A, A, A, A, A, A, 1, 8, 8, 64, t, A, None)),
    "max pool": (("x", "y", "idx"), lambda p, t: lib.tmpi_maxpool_fwd(p[0], p[1], p[2], 1, 8, 8, 64, 4, 4, 3, 2, 1, t, None)),
    "max pool backward": (("dy", "idx", "dx"), lambda p, t: lib.tmpi_maxpool_bwd(p[0], p[1], p[2], 1, 8, 8, 64, 4, 4, 3, 2, 1, t, None)),
    "layer norm": (("x", "gamma", "beta", "y"), lambda p, t: lib.tmpi_layernorm_fwd(p[0], p[1], p[2], p[3], A, A, 8, 256, 1e-5, t, None)),
    "layer norm backward": (("x", "dy", "add", "gamma", "dx"), lambda p, t: lib.tmpi_layernorm_bwd_add(p[0], p[1], p[2], p[3], A, A, p[4], A, A, 8, 256, t, A, None)),
    "bias gradient": (("dy", "z", "dz"), lambda p, t: lib.tmpi_bias_grad(p[0], p[1], p[2], A, 8, 1024, t, A, None)),
    "GELU backward": (("dy", "z", "dz"), lambda p, t: lib.tmpi_gelu_bwd(p[0], p[1], p[2], 1024, t, None)),
    "stem patches": (("x", "col"), lambda p, t: lib.tmpi_stem_im2col(p[0], p[1], 1, 32, 32, t, None)),
}


@pytest.mark.parametrize("name", CALLS)
def test_odd_addresses_are_refused(name):
    tensors, call = CALLS[name]
    for odd in range(len(tensors)):
        with pytest.raises(TorchMPIError, match="-byte aligned"):
            check(call([A + (2 if k == odd else 0) for k in range(len(tensors))], _bf16()))
