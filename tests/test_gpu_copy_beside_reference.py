"""The Jacobi passes with the copy of the cells outside the loop box beside them, a chain of steps queued at once against
the same steps in torch, bit for bit: the variants that programs get (test_gpu_copy_beside.py compares a chain with its own
steps one at a time).  Second buffers begin with a value that no step makes, so a cell that nobody writes differs."""
import ctypes

import pytest

import __graft_entry__ as ge
from tests.util import J3_STNUPD, kernel_macros

pytestmark = pytest.mark.gpu
K = kernel_macros()
STEPS, NOBODY = 6, -77.0


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


def random(n, seed):
    import torch
    return torch.rand(*n, generator=torch.Generator(device="cuda").manual_seed(seed), dtype=torch.float64, device="cuda")


def neighbours(a, lo, hi, order):
    """The sum of the box's neighbours, (axis, offset) by (axis, offset)."""
    s = None
    for axis, off in order:
        part = a[tuple(slice(lo[d] + (off if d == axis else 0), hi[d] + 1 + (off if d == axis else 0))
                       for d in range(a.dim()))]
        s = part.clone() if s is None else s + part
    return s


BOXES3 = [((200, 180, 192), (90, 80, 100), (95, 84, 103)), ((66, 65, 130), (1, 1, 1), (64, 63, 128)),
          ((40, 300, 64), (20, 1, 1), (20, 298, 62)), ((30, 50, 202), (3, 5, 7), (25, 38, 190))]
BOXES2 = [((3000, 2048), (1400, 900), (1404, 940)), ((130, 192), (1, 1), (128, 190)), ((900, 640), (6, 1), (893, 638)),
          ((70, 300), (3, 65), (60, 250))]


@pytest.mark.parametrize("n,lo,hi", BOXES3)
@pytest.mark.parametrize("variant", range(J3_STNUPD))
def test_cross_step_pass(rt, variant, n, lo, hi):
    import torch
    L3 = ctypes.c_long * 3
    st, ext, clo, chi = L3(n[1] * n[2], n[2], 1), L3(*n), L3(*lo), L3(*hi)
    a, alt, b = random(n, 3), torch.full(n, NOBODY, dtype=torch.float64, device="cuda"), random(n, 5)
    box = tuple(slice(p, q + 1) for p, q in zip(lo, hi))
    wa, wb, weps = a.clone(), b.clone(), []
    six = torch.tensor(6.0, dtype=torch.float64, device="cuda")  # (by a number torch multiplies with its reciprocal)
    for _ in range(STEPS):
        new = neighbours(wa, lo, hi, [(0, -1), (1, -1), (2, -1), (2, 1), (1, 1), (0, 1)]) / six
        weps.append((new - wa[box]).abs().max())
        wb[box] = new
        wa[box] = new
    items = torch.zeros(rt.dvmhgb_jac3d_stnupd_items(clo, chi, variant), dtype=torch.float64, device="cuda")
    sp, eps = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream), []
    torch.cuda.synchronize()
    for _ in range(STEPS):
        assert rt.dvmhgb_jac3d_stnupd(vp(a), vp(alt), vp(b), st, ext, clo, chi, vp(items), variant, sp) == 0
        eps.append(items.max())
        a, alt = alt, a
    assert torch.equal(a, wa) and torch.equal(b, wb) and torch.equal(torch.stack(eps), torch.stack(weps))


@pytest.mark.parametrize("n,lo,hi", BOXES2)
def test_update_with_stencil_2d(rt, n, lo, hi):
    import torch
    L2 = ctypes.c_long * 2
    st, ext, clo, chi = L2(n[1], 1), L2(*n), L2(*lo), L2(*hi)
    a, b, c = random(n, 3), random(n, 4), torch.full(n, NOBODY, dtype=torch.float64, device="cuda")
    box = tuple(slice(p, q + 1) for p, q in zip(lo, hi))
    wa, wb, weps = a.clone(), b.clone(), []
    for _ in range(STEPS):
        weps.append((wb[box] - wa[box]).abs().max())
        wa[box] = wb[box]
        wb[box] = neighbours(wa, lo, hi, [(0, -1), (1, -1), (1, 1), (0, 1)]) / 4.0
    items = torch.zeros(rt.dvmhgb_jac2d_fused_items(clo, chi), dtype=torch.float64, device="cuda")
    sp, eps = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream), []
    torch.cuda.synchronize()
    for _ in range(STEPS):
        assert rt.dvmhgb_jac2d_fused(vp(a), vp(b), vp(c), st, ext, clo, chi, vp(items), K["DVMHGB_JAC2D_FUSED_LIMBS"],
                                     sp) == 0
        eps.append(items.max())
        b, c = c, b
    assert torch.equal(a, wa) and torch.equal(b, wb) and torch.equal(torch.stack(eps), torch.stack(weps))
