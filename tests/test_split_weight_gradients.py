"""Which weight gradients of linear layers run on the kernels that split their rows over the SMs."""
import pytest

from torchmpi_b200._lib import has_symbol, lib

pytestmark = pytest.mark.skipif(not has_symbol("tmpi_gemm_tn_prefers_splitk"), reason="built without the CUDA kernels")


# rows x outputs x inputs: both ways measured on 148 SMs, the faster one
@pytest.mark.parametrize("K,M,N,split", [(8192, 1024, 1024, True), (8192, 512, 512, True), (4096, 104, 128, True), (16384, 1536, 768, True),
                                         (8192, 1536, 1536, False), (1024, 1024, 1024, False), (256, 128, 128, False),
                                         # more tiles than half the SMs: nothing to split
                                         (8192, 3072, 2048, False), (8192, 4096, 4096, False), (16384, 4096, 2048, False), (8192, 50264, 1024, False),
                                         (1 << 20, 4096, 4096, False)])
def test_split_where_it_is_faster(K, M, N, split):
    assert bool(lib.tmpi_gemm_tn_prefers_splitk(M, N, K)) == split


def test_no_split_without_slices():
    """A product that the plan leaves in one slice never takes the partial tiles' way."""
    for M in range(128, 8193, 128):
        for N in (256, 1024, 2048, 4096, 8192):
            if -(-M // 128) * -(-N // 256) > 74:
                assert not lib.tmpi_gemm_tn_prefers_splitk(M, N, 1 << 16), (M, N)
