"""Which weight gradients of linear layers are cut into slices of their rows (csrc/kernels/linear_bwd.cu), as the plan of a call shows by
its arrival counters and its workspace of fp32 partial tiles."""
import ctypes
import time

import pytest

from torchmpi_b200._lib import check, has_symbol, lib

pytestmark = pytest.mark.skipif(not has_symbol("tmpi_linear_bwd_plan"), reason="built without the CUDA kernels")
DW = 2


def _plan(rows, inp, out, want=DW):
    size, n = ctypes.c_size_t(0), ctypes.c_int(0)
    check(lib.tmpi_linear_bwd_plan(rows, inp, out, want, 0, ctypes.byref(size), ctypes.byref(n)))
    assert (size.value > 0) == (n.value > 0)
    return size.value, n.value


# rows x outputs x inputs on 148 SMs: few tiles and many rows are sliced, an output that fills the chip or few rows are not
@pytest.mark.parametrize("rows,out,inp,sliced", [(8192, 1024, 1024, True), (8192, 512, 512, True), (4096, 104, 128, True), (16384, 1536, 768, True),
                                                 (1024, 1024, 1024, False), (256, 128, 128, False), (512, 4096, 1024, False), (8192, 4096, 4096, False),
                                                 # two rounds and a half of whole tiles: slices fill the last one
                                                 (1 << 20, 4096, 3072, True)])
def test_sliced_where_the_tiles_leave_clusters_idle(rows, out, inp, sliced):
    assert (_plan(rows, inp, out)[1] > 0) == sliced


def test_slices_have_eight_k_blocks():
    """Fewer than sixteen K blocks of 64 rows are never cut in two."""
    for out in range(8, 4097, 136):
        for inp in (8, 256, 1000, 4096):
            assert _plan(15 * 64, inp, out)[1] == 0, (out, inp)


def test_workspace_is_bounded():
    """At most eight units of 256 x 256 floats for each of 74 clusters and product."""
    for rows in (64, 1000, 8192, 65536, 1 << 20):
        for out in (8, 512, 1000, 4096, 50264):
            for inp in (64, 768, 1024, 4096):
                for want in (1, 2, 3, 7):
                    assert _plan(rows, inp, out, want)[0] <= 2 * 8 * 74 * 256 * 256 * 4 + 2 * 32 * 256 * 4 * -(-out // 256), (rows, out, inp, want)


@pytest.mark.parametrize("rows,width", [(2048, 512), (8192, 1024), (128, 512)])
def test_plans_of_a_model_are_kept(rows, width):
    """The plans of a block's four layers, asked for in turn, are found again rather than made anew, which takes twice as long or longer."""
    layers = [(rows, width, 3 * width), (rows, width, width), (rows, width, 4 * width), (rows, 4 * width, width)]
    size, n = ctypes.c_size_t(0), ctypes.c_int(0)

    def took(sizes):
        best = float("inf")
        for _ in range(20):
            start = time.perf_counter()
            for s in sizes * 50:
                lib.tmpi_linear_bwd_plan(*s, 7, 0, ctypes.byref(size), ctypes.byref(n))
            best = min(best, (time.perf_counter() - start) / len(sizes))
        return best
    for _ in range(10):                                      # a busy machine: once is enough
        alone, turns = sum(took([s]) for s in layers) / 4, took(layers)
        if turns < 1.3 * alone:
            return
    assert turns < 1.3 * alone, (alone, turns)
