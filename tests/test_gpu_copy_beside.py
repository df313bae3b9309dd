"""The Jacobi passes whose copy of the cells outside the loop box runs beside them: a chain of steps queued at once gives
what the same steps give one at a time, bit for bit, where the copy is the longer part (a small box in a large array) and
where it is the shorter."""
import ctypes

import pytest

import __graft_entry__ as ge
from tests.util import kernel_macros

pytestmark = pytest.mark.gpu
K = kernel_macros()
STEPS = 12


@pytest.fixture(scope="module")
def rt():
    ge.build()
    _, g = ge.package()
    g.init()
    L = g.runtime()
    L.dvmhgb_jac3d_stnupd_items.restype = L.dvmhgb_jac2d_fused_items.restype = ctypes.c_long
    return L


def vp(t):
    return ctypes.c_void_p(t.data_ptr())


@pytest.mark.parametrize("n,lo,hi", [((200, 180, 192), (90, 80, 100), (95, 84, 103)), ((66, 65, 130), (1, 1, 1), (64, 63, 128)),
                                     ((40, 300, 64), (20, 1, 1), (20, 298, 62))])
def test_cross_step_pass(rt, n, lo, hi):
    import torch
    L3 = ctypes.c_long * 3
    st, ext, clo, chi = L3(n[1] * n[2], n[2], 1), L3(*n), L3(*lo), L3(*hi)
    a0 = torch.rand(*n, generator=torch.Generator().manual_seed(3), dtype=torch.float64).cuda()
    items = torch.zeros(rt.dvmhgb_jac3d_stnupd_items(clo, chi, 5), dtype=torch.float64, device="cuda")
    sp = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)

    def run(wait):
        a, alt, b = a0.clone(), torch.zeros_like(a0), torch.zeros_like(a0)
        seen = []
        for _ in range(STEPS):
            assert rt.dvmhgb_jac3d_stnupd(vp(a), vp(alt), vp(b), st, ext, clo, chi, vp(items), 5, sp) == 0
            if wait:
                torch.cuda.synchronize()
            seen.append(items.max())
            a, alt = alt, a
        torch.cuda.synchronize()
        return a, b, torch.stack(seen)

    assert all(torch.equal(x, y) for x, y in zip(run(False), run(True)))


@pytest.mark.parametrize("n,lo,hi", [((3000, 2048), (1400, 900), (1404, 940)), ((130, 192), (1, 1), (128, 190)),
                                     ((900, 640), (6, 1), (893, 638))])
def test_update_with_stencil_2d(rt, n, lo, hi):
    import torch
    L2 = ctypes.c_long * 2
    st, ext, clo, chi = L2(n[1], 1), L2(*n), L2(*lo), L2(*hi)
    b0 = torch.rand(*n, generator=torch.Generator().manual_seed(4), dtype=torch.float64).cuda()
    items = torch.zeros(rt.dvmhgb_jac2d_fused_items(clo, chi), dtype=torch.float64, device="cuda")
    sp = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)

    def run(wait):
        a, b, c = b0.flip(0).contiguous(), b0.clone(), torch.zeros_like(b0)
        seen = []
        for _ in range(STEPS):
            assert rt.dvmhgb_jac2d_fused(vp(a), vp(b), vp(c), st, ext, clo, chi, vp(items), K["DVMHGB_JAC2D_FUSED_LIMBS"],
                                         sp) == 0
            if wait:
                torch.cuda.synchronize()
            seen.append(items.max())
            b, c = c, b
        torch.cuda.synchronize()
        return a, b, torch.stack(seen)

    assert all(torch.equal(x, y) for x, y in zip(run(False), run(True)))
