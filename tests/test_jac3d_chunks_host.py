"""The chunks of planes that the cross-step Jacobi-3D pass takes (no GPU: dvmhgb_jac3d_stnupd_items is the CTA count of
its grid): the cheapest by the cost that all counts of chunks are compared with here, and found without going through
them one by one -- a box of many planes and few rows would wait for the host."""
import ctypes
import time

import pytest

L3 = ctypes.c_long * 3
SHAPES = {0: (1, 4), 1: (1, 3), 2: (2, 2), 3: (1, 3), 4: (2, 2)}  # rows per thread, CTAs per SM
SMS = 152  # without a GPU


@pytest.fixture(scope="module")
def rt():
    import __graft_entry__ as ge
    import torch
    if torch.cuda.is_available():
        pytest.skip("sizes for the SM count of a machine without a GPU")
    ge.build()
    _, g = ge.package()
    r = g.runtime()
    r.dvmhgb_jac3d_stnupd_items.restype = ctypes.c_long
    return r


def ceil(a, b):
    return -(-a // b)


@pytest.mark.parametrize("variant", sorted(SHAPES))
@pytest.mark.parametrize("n", [(3, 3, 3), (67, 67, 67), (258, 255, 255), (512, 512, 512), (3000, 12, 40), (9, 1500, 700)])
def test_cheapest_chunks(rt, n, variant):
    jt, ctas = SHAPES[variant]
    ni, tiles, resident = n[0] - 2, ceil((n[2] - 2) // 2 + 1, 32) * ceil(n[1] - 2, 8 * jt), SMS * ctas
    cost = lambda length: ceil(tiles * ceil(ni, length), resident) * (length + 4)  # noqa: E731
    lengths = {ceil(ni, want) for want in range(1, ni + 1)}
    least = min(cost(q) for q in lengths)
    items = rt.dvmhgb_jac3d_stnupd_items(L3(1, 1, 1), L3(*[q - 2 for q in n]), variant)
    assert items in {tiles * ceil(ni, q) for q in lengths if cost(q) == least}


def test_many_planes_do_not_cost_host_time(rt):
    lo, hi = L3(1, 1, 1), L3(59998, 8, 32)
    t = time.perf_counter()
    for _ in range(200):
        rt.dvmhgb_jac3d_stnupd_items(lo, hi, 4)
    assert (time.perf_counter() - t) / 200 < 20e-6  # 1 us; 130 when every count was looked at


@pytest.mark.parametrize("rows,variant", [(1, 3), (8, 3), (9, 4), (16, 4), (17, 3), (65, 3), (72, 3), (73, 4), (81, 4), (510, 4)])
def test_few_rows_take_one_a_thread(rt, rows, variant):
    assert rt.dvmhgb_jac3d_stnupd_default(L3(1, 3, 1), L3(500, 2 + rows, 70)) == variant
