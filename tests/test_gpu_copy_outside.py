"""The copy of the cells outside a loop box: every rank, rows at the edges of a warp and of the 1024 elements a warp
copies, strided innermost axes, boxes at the array's faces -- and long rows, which must not be left to a warp each."""
import ctypes
import itertools

import pytest

import __graft_entry__ as ge

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rt():
    ge.build()
    _, g = ge.package()
    g.init()
    return g.runtime()


def copy(rt, src, dst, lo, hi):
    import torch
    r = src.dim()
    A = ctypes.c_long * r
    return rt.dvmhgb_copy_outside_box(r, ctypes.c_void_p(src.data_ptr()), ctypes.c_void_p(dst.data_ptr()), A(*src.stride()),
                                      A(*src.shape), A(*lo), A(*hi),
                                      ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))


CASES = [((1, 31), (0, 0), (0, 30)), ((9000,), (17,), (4100,)), ((40,), (5,), (8,)), ((2500,), (1024,), (1055,))]
CASES += [((5, m), (1, lo), (3, m - 2)) for m, lo in itertools.product((33, 64, 1025, 2080), (1, 31))]
CASES += [((4, 6, m), (1, 2, lo), (2, 4, lo + 2)) for m, lo in itertools.product((3 + 31, 1056, 3100), (0, 30))]


@pytest.mark.parametrize("step", [1, 3])
@pytest.mark.parametrize("n,lo,hi", CASES)
def test_cells(rt, n, lo, hi, step):
    import torch
    src = torch.rand(*n, step, dtype=torch.float64, device="cuda")[..., 0]
    dst = torch.full((*n, step), 7.0, dtype=torch.float64, device="cuda")
    want = dst.clone()
    want[..., 0] = src
    want[..., 0][tuple(slice(a, b + 1) for a, b in zip(lo, hi))] = 7.0
    assert copy(rt, src, dst[..., 0], lo, hi) == 0
    assert torch.equal(dst, want)


@pytest.mark.parametrize("n,lo,hi", [((4000000,), (10,), (20,)), ((3, 1500000), (1, 1), (1, 1499998))])
def test_long_rows_are_shared_out(rt, n, lo, hi):
    import torch
    src, dst = torch.rand(*n, dtype=torch.float64, device="cuda"), torch.zeros(*n, dtype=torch.float64, device="cuda")
    best = [float("inf")] * 2
    for _ in range(5):
        for q, call in enumerate((lambda: copy(rt, src, dst, lo, hi), lambda: dst.copy_(src))):
            e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            torch.cuda.synchronize()
            e0.record()
            call()
            e1.record()
            torch.cuda.synchronize()
            best[q] = min(best[q], e0.elapsed_time(e1))
    assert best[0] < 6 * best[1] + 0.02  # a warp a row: over 1000 times
