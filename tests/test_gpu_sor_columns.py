"""The SOR sweep by columns of hyperplane tiles (variant 5) against the box tiles (variant 1: every sum on the FP64 unit)
and the items of the tiles handed out one by one (variant 4), bit for bit: boxes at the edges of the 16 x 8 tiles and of
the 8 hyperplanes, one cell thick, starting past the first 64-wide chunk, with more columns than the GPU holds at once;
fields that the FP32 limbs hold, move to, or leave to the FP64 unit, and two sweeps in a row."""
import ctypes

import pytest

import __graft_entry__ as ge
from tests.test_gpu_jacobi_ranges import field

pytestmark = pytest.mark.gpu
BOXES = [((18, 10, 18), (1, 1, 1), (16, 8, 16)), ((19, 11, 75), (1, 1, 1), (17, 9, 73)),
         ((17, 9, 139), (0, 0, 65), (15, 7, 130)), ((40, 41, 9), (3, 2, 4), (39, 40, 4)),
         ((9, 60, 66), (4, 1, 1), (4, 58, 64)), ((50, 9, 70), (1, 5, 63), (48, 5, 64))]
KINDS = ["unit", "degrees", "huge", "subnormal", "growing", "hot wall", "mixed", "spots", "signed", "zero"]


def data(kind, n, seed):
    import torch
    if kind in ("unit", "signed"):
        a = torch.rand(*n, generator=torch.Generator().manual_seed(seed), dtype=torch.float64)
        return a - 0.5 if kind == "signed" else a
    if kind == "zero":
        a = torch.zeros(*n, dtype=torch.float64)
        a[:, 0] = 0.75
        return a
    return field(kind, tuple(max(q, 8) for q in n), seed)[:n[0], :n[1], :n[2]].contiguous()


def sweeps(L, a, lo, hi, variant, count=2):
    import torch
    L3 = ctypes.c_long * 3
    n, d = a.shape, a.cuda()
    st, ext, clo, chi = L3(n[1] * n[2], n[2], 1), L3(*n), L3(*lo), L3(*hi)
    vp = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    w = torch.tensor([1.2], dtype=torch.float64, device="cuda")
    items = torch.full((L.dvmhgb_sor3d_items(clo, chi, variant),), float("nan"), dtype=torch.float64, device="cuda")
    scratch = torch.zeros(L.dvmhgb_sor3d_scratch_bytes(clo, chi, variant) // 4 + 1, dtype=torch.int32, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    sp = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    for _ in range(count):
        assert L.dvmhgb_sor3d_sweep(vp(d), st, ext, clo, chi, vp(w), vp(items), vp(scratch), vp(status), variant,
                                    sp) == 0
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    return d.cpu(), items.cpu()


def same(x, y):
    import torch
    return bool(((x.view(torch.int64) == y.view(torch.int64)) | (x.isnan() & y.isnan())).all())


@pytest.fixture(scope="module")
def rt():
    ge.build()
    _, g = ge.package()
    g.init()
    L = g.runtime()
    L.dvmhgb_sor3d_items.restype = L.dvmhgb_sor3d_scratch_bytes.restype = ctypes.c_long
    return L


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("box", range(len(BOXES)))
def test_fields_and_edges(rt, box, kind):
    n, lo, hi = BOXES[box]
    a = data(kind, n, box)
    array, items = sweeps(rt, a, lo, hi, 5)
    assert same(array, sweeps(rt, a, lo, hi, 1)[0])
    assert same(items, sweeps(rt, a, lo, hi, 4)[1])


@pytest.mark.parametrize("n", [(300, 260, 12), (24, 700, 40)])
def test_more_columns_than_the_gpu_holds(rt, n):
    lo, hi = (1, 1, 1), tuple(q - 2 for q in n)
    a = data("unit", n, 7)
    array, items = sweeps(rt, a, lo, hi, 5)
    assert same(array, sweeps(rt, a, lo, hi, 1)[0])
    assert same(items, sweeps(rt, a, lo, hi, 4)[1])
