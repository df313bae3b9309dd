"""The Jacobi 2-D limb kernels (stencil, and update with stencil) against float64 on the CPU, bit for bit: boxes that
touch the array's edges (a neighbour outside the array counts as 0), start past the first 64-wide chunk, are one cell
wide or high, and fields that the limbs hold, move to, or leave to the FP64 unit.  Every older variant gives the same."""
import ctypes

import pytest

import __graft_entry__ as ge
from tests.test_gpu_jacobi_ranges import field
from tests.util import kernel_macros

pytestmark = pytest.mark.gpu
K = kernel_macros()
BOXES = [((40, 131), (1, 1), (38, 129)), ((9, 64), (0, 0), (8, 63)), ((33, 200), (5, 70), (27, 190)),
         ((12, 66), (1, 1), (10, 64)), ((7, 129), (3, 64), (3, 64)), ((70, 193), (1, 0), (68, 192))]


def reference(a, lo, hi):
    import torch
    p = torch.nn.functional.pad(a, (1, 1, 1, 1))  # 0 outside the array
    i, j = slice(lo[0] + 1, hi[0] + 2), slice(lo[1] + 1, hi[1] + 2)
    s = lambda q, d: slice(q.start + d, q.stop + d)  # noqa: E731
    return (((p[s(i, -1), j] + p[i, s(j, -1)]) + p[i, s(j, 1)]) + p[s(i, 1), j]) / 4.0


@pytest.mark.parametrize("kind", ["unit", "degrees", "huge", "subnormal", "growing", "hot wall", "mixed", "spots"])
@pytest.mark.parametrize("box", range(len(BOXES)))
def test_stencil_and_pair(box, kind):
    import torch
    ge.build()
    _, g = ge.package()
    g.init()
    L = g.runtime()
    L.dvmhgb_jac2d_fused_items.restype = ctypes.c_long
    n, lo, hi = BOXES[box]

    def data(seed):
        if kind == "unit":
            return torch.rand(*n, generator=torch.Generator().manual_seed(seed), dtype=torch.float64)
        return field(kind, (max(n[0], 8), max(n[1], 8), 8), seed)[:n[0], :n[1], 3].contiguous()

    a, b = data(box), data(box + 50)
    w = (n[1] + 1) // 2 * 2
    L2 = ctypes.c_long * 2
    st, ext, clo, chi = L2(w, 1), L2(*n), L2(*lo), L2(*hi)
    vp = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    sp = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)

    def dev(t, fill=0.0):
        d = torch.full((n[0], w), fill, dtype=torch.float64, device="cuda")
        if t is not None:
            d[:, :n[1]] = t.cuda()
        return d

    def same(x, y):
        x, y = x.cpu(), y.cpu()
        return bool(((x.view(torch.int64) == y.view(torch.int64)) | (x.isnan() & y.isnan())).all())

    i, j = slice(lo[0], hi[0] + 1), slice(lo[1], hi[1] + 1)
    for v in range(K["DVMHGB_JAC2D_STENCIL_LIMBS"] + 1):
        out = dev(None, 7.0)
        assert L.dvmhgb_jac2d_stencil(vp(dev(a)), vp(out), st, ext, clo, chi, v, sp) == 0
        torch.cuda.synchronize()
        want = torch.full((n[0], w), 7.0, dtype=torch.float64)
        want[i, j] = reference(a, lo, hi)
        assert same(out, want), (kind, box, v)
    new = a.clone()
    new[i, j] = b[i, j]
    wantB = b.clone()
    wantB[i, j] = reference(new, lo, hi)
    d = (b[i, j] - a[i, j]).abs()
    d = d[~d.isnan()]
    for v in range(K["DVMHGB_JAC2D_FUSED_LIMBS"] + 1):
        da, db, out = dev(a), dev(b), dev(None, 7.0)
        items = torch.full((L.dvmhgb_jac2d_fused_items(clo, chi),), float("nan"), dtype=torch.float64, device="cuda")
        assert L.dvmhgb_jac2d_fused(vp(da), vp(db), vp(out), st, ext, clo, chi, vp(items), v, sp) == 0
        torch.cuda.synchronize()
        assert same(da[:, :n[1]], new) and same(db[:, :n[1]], b), (kind, box, v)
        assert same(out[:, :n[1]].contiguous(), wantB), (kind, box, v)
        assert bool((out[:, n[1]:] == 7.0).all()), (kind, box, v)
        assert not bool(items.isnan().any()), (kind, box, v)
        assert items.max().item() == (d.max().item() if d.numel() else 0.0), (kind, box, v)
