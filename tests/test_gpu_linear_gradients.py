"""The one launch of a linear layer's gradients against fp64, in every form of its work list."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def _form(bx, sx, bw, sw, sb):
    return bx // 64 | sx << 4 | bw // 64 << 8 | sw << 12 | sb << 16


def _rand(*shape):
    """Rows that are not whole 16-byte units sit in a pitched buffer, whose padding is NaN."""
    t = torch.full(shape[:-1] + ((shape[-1] + 7) // 8 * 8,), float("nan"), device="cuda", dtype=torch.bfloat16)
    t[:, :shape[-1]] = torch.randn(*shape, device="cuda")
    return t[:, :shape[-1]]


def _run(dy, x, w, want, form):
    from torchmpi_b200._lib import check, lib, stream_ptr
    rows, out = dy.shape
    inp = x.shape[1]
    size, n = ctypes.c_size_t(0), ctypes.c_int(0)
    check(lib.tmpi_linear_bwd_plan(rows, inp, out, want, form, ctypes.byref(size), ctypes.byref(n)))
    ws = torch.full((max(16, size.value),), 255, device="cuda", dtype=torch.uint8)             # NaN wherever it is read before it is written
    counters = torch.zeros(max(1, n.value), device="cuda", dtype=torch.int32)
    res = [torch.full(s, float("nan"), device="cuda", dtype=torch.bfloat16) for s in ((rows, inp), (out, inp), (out,))]
    for _ in range(2):                                                                          # the second on the counters of the first
        check(lib.tmpi_linear_bwd(dy.data_ptr(), dy.stride(0), x.data_ptr(), w.data_ptr(), *(t.data_ptr() if want >> k & 1 else None for k, t in enumerate(res)),
                                  rows, inp, out, form, ws.data_ptr(), size.value, counters.data_ptr(), n.value, stream_ptr()))
        assert not counters.any()
    return res


# one pack, a row more and a row less than a tile, remainders in every dimension, several rounds of units, long K
@pytest.mark.parametrize("rows,inp,out", [(1, 8, 8), (255, 264, 72), (257, 136, 520), (1000, 768, 1000), (2056, 200, 8), (72, 2056, 264), (4096, 1024, 1536), (520, 256, 1003)])
@pytest.mark.parametrize("form", [0, _form(256, 1, 256, 1, 1), _form(192, 2, 128, 3, 2), _form(128, 3, 192, 8, 4), _form(256, 5, 256, 15, 15), 1 << 20 | _form(128, 2, 192, 3, 4)])
def test_forms_of_the_work_list(rows, inp, out, form):
    from torchmpi_b200.ops import gemm
    torch.manual_seed(rows)
    dy, x, w = (_rand(*s) for s in ((rows, out), (rows, inp), (out, inp)))
    d = dy.double()
    refs = (d @ w.double(), d.t() @ x.double(), d.sum(0))
    # absolute sums of the products: an fp32 sum of K terms is off by K / 16 roundings of a partial sum at most (an MMA adds 16
    # terms), each 2^-23 of it; a result is rounded to bf16 (8 significant bits) once, by half a unit in the last place: up to 2^-8 of it
    sums = (d.abs() @ w.double().abs(), d.abs().t() @ x.double().abs(), d.abs().sum(0))
    steps = (out / 16 + 16, rows / 16 + 16, rows / 16 + 16)
    for want in (7, 1, 2, 3, 5, 6):
        got = _run(dy, x, w, want, form)
        gemm.check_status()
        for k in range(3):
            if want >> k & 1:
                assert bool(((got[k].double() - refs[k]).abs() <= 2.0 ** -8 * refs[k].abs() + steps[k] * 2.0 ** -23 * sums[k]).all()), (want, k)
            else:
                assert bool(got[k].isnan().all())
        assert all(torch.equal(a, b) for k, (a, b) in enumerate(zip(got, _run(dy, x, w, want, form))) if want >> k & 1)      # order of sums fixed


def test_refused_sizes_and_scratch():
    from torchmpi_b200._lib import TorchMPIError, check, lib
    size, n = ctypes.c_size_t(0), ctypes.c_int(0)
    t = torch.zeros(8192, 8, device="cuda", dtype=torch.bfloat16)
    for rows, inp, out, want, form in ((0, 8, 8, 7, 0), (8, 12, 8, 7, 0), (8, 8, 8, 4, 0), (8, 8, 8, 8, 0), (8, 8, 8, 7, 1)):
        with pytest.raises(TorchMPIError):
            check(lib.tmpi_linear_bwd_plan(rows, inp, out, want, form, ctypes.byref(size), ctypes.byref(n)))
    form = _form(128, 1, 128, 4, 1)
    check(lib.tmpi_linear_bwd_plan(8192, 8, 8, 2, form, ctypes.byref(size), ctypes.byref(n)))
    ws, counters, dw = torch.empty(size.value, device="cuda", dtype=torch.uint8), torch.zeros(n.value, device="cuda", dtype=torch.int32), torch.empty_like(t[:8])
    for got in ((size.value - 4, n.value), (size.value, n.value - 1)):
        with pytest.raises(TorchMPIError):
            check(lib.tmpi_linear_bwd(t.data_ptr(), 0, t.data_ptr(), None, None, dw.data_ptr(), None, 8192, 8, 8, form, ws.data_ptr(), got[0],
                                      counters.data_ptr(), got[1], None))


def test_gradients_on_several_streams_and_in_a_graph():
    """Sliced tiles: each stream and each captured call has arrival counters of its own."""
    from torchmpi_b200.ops import gemm
    torch.manual_seed(0)
    x, w, dy = (torch.randn(*s, device="cuda").to(torch.bfloat16) for s in ((8192, 512), (512, 512), (8192, 512)))
    leaves = [t.clone().requires_grad_(True) for t in (x, w, torch.zeros(512, device="cuda", dtype=torch.bfloat16))]

    def grads():
        return torch.autograd.grad(gemm.linear(*leaves), leaves, dy)
    want = grads()
    streams = [torch.cuda.Stream() for _ in range(3)]
    torch.cuda.synchronize()
    got = []
    for _ in range(4):
        for s in streams:
            with torch.cuda.stream(s):
                got.append(grads())
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for g in got for a, b in zip(g, want))
    with torch.cuda.stream(streams[0]):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=streams[0]):
            captured = grads()
    for _ in range(3):
        graph.replay()
        eager = grads()
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for g in (captured, eager) for a, b in zip(g, want))


def test_counters_after_waits_that_ran_out():
    """A kernel that gave up may leave its counters half way: none that was in use before or during a report is handed out after it."""
    from torchmpi_b200 import _native
    from torchmpi_b200._lib import TorchMPIError, check, lib
    from torchmpi_b200.ops import gemm
    like = torch.empty(1, device="cuda", dtype=torch.bfloat16)
    take = _native.ext().arrival_counters
    gemm.check_status()
    first = take(like, 64)
    assert take(like, 64).data_ptr() == first.data_ptr()                      # kept for the stream
    held = [first]                                                            # alive, so that no new one lies where an old one was
    try:
        for again in (False, True):                                           # the second report while the first is unread
            check(lib.tmpi_gemm_report(1024))
            for _ in range(2):
                fresh = take(like, 64)
                assert not fresh.any() and all(fresh.data_ptr() != t.data_ptr() for t in held)
                fresh.fill_(1)                                                # as the next kernel that gives up
                held.append(fresh)
            if again:
                check(lib.tmpi_gemm_report(1025))
    finally:
        with pytest.raises(TorchMPIError, match="1024"):
            gemm.check_status()
    fresh = take(like, 64)
    assert not fresh.any() and all(fresh.data_ptr() != t.data_ptr() for t in held)
    assert take(like, 64).data_ptr() == fresh.data_ptr()
    gemm.check_status()


def _absorbing(rows, cols):
    """Two large values that cancel, and small ones between them that a sum in one chain loses one by one."""
    t = torch.full((rows, cols), 2.0 ** -14, device="cuda")
    t[0], t[-1] = 2.0 ** 15, -2.0 ** 15
    return t


def _cancelling(rows, cols):
    t = torch.randn(rows, cols, device="cuda") + 1.0
    t[-64:] -= t.sum(0) / 64
    return t


@pytest.mark.parametrize("values", [_absorbing, _cancelling])
@pytest.mark.parametrize("form", [0, 1 << 21 | _form(256, 1, 256, 1, 5)])                  # 21 slices of the sums
@pytest.mark.parametrize("rows,out", [(512, 1024), (640, 20480), (2048, 520), (8192, 1024), (8192, 4096), (24576, 1000)])
def test_bias_gradient_is_a_sum_of_short_chains(rows, out, form, values):
    """Column sums that cancel show the error of the fp32 sum, and not the rounding of the result."""
    torch.manual_seed(rows)
    dy = values(rows, out).to(torch.bfloat16)
    x, w = (torch.randn(*s, device="cuda").to(torch.bfloat16) for s in ((rows, 64), (out, 64)))
    db = _run(dy, x, w, 7, form)[2].double()
    ref, total = dy.double().sum(0), dy.double().abs().sum(0)
    # a value passes the batches of 256 rows of its thread, at most 24 of a slice, four levels inside its batch, four over the threads, and
    # the slices in fours, of which there are eight at most: so many roundings by half a unit, each of at most the sum of the absolute values
    bound = (min(rows / 256, 24) + 4 + 4 + 2 + 8) * 2.0 ** -24 * total
    assert bool(((db - ref).abs() <= 2.0 ** -9 * ref.abs() + bound).all())
