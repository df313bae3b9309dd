"""The Jacobi-3D limb kernels on fields where planes that their range holds and planes that none holds (negative values)
take turns, over chunks of many planes: the change between the limbs and the plain planes and back, bit for bit.  And on
fields that no range holds at all, where they may not be slower than kernels that sum on the FP64 unit alone."""
import ctypes

import pytest

import __graft_entry__ as ge
from tests.util import J3_STENCILS, J3_STNUPD

pytestmark = pytest.mark.gpu
L3 = ctypes.c_long * 3


@pytest.fixture(scope="module")
def rt():
    ge.build()
    _, g = ge.package()
    g.init()
    L = g.runtime()
    L.dvmhgb_jac3d_stnupd_items.restype = L.dvmhgb_jac3d_update_items.restype = ctypes.c_long
    return L


def vp(t):
    return ctypes.c_void_p(t.data_ptr())


def bands(n, kind):
    """[0.25, 1) with negative values in runs of 1 .. 40 planes: everywhere in them, or in one cell in 5000."""
    import torch
    gen = torch.Generator(device="cuda").manual_seed(11)
    a = 0.25 + 0.75 * torch.rand(*n, generator=gen, dtype=torch.float64, device="cuda")
    runs, i = torch.Generator().manual_seed(12), 0
    if kind == "whole":
        while i < n[0]:
            i += int(torch.randint(1, 40, (1,), generator=runs))
            m = int(torch.randint(1, 40, (1,), generator=runs))
            a[i:i + m] -= 0.6
            i += m
    else:
        a = torch.where(torch.rand(*n, generator=gen, dtype=torch.float64, device="cuda") < 1 / 5000, -a, a)
    return a


@pytest.mark.parametrize("kind", ["whole", "single"])
@pytest.mark.parametrize("n", [(190, 250, 700), (230, 330, 390)])
def test_bands(rt, kind, n):
    import torch
    a = bands(n, kind)
    st, ext, lo, hi = L3(n[1] * n[2], n[2], 1), L3(*n), L3(1, 1, 1), L3(*[q - 2 for q in n])
    inner = (slice(1, -1),) * 3
    s = a[:-2, 1:-1, 1:-1] + a[1:-1, :-2, 1:-1]
    for x in (a[1:-1, 1:-1, :-2], a[1:-1, 1:-1, 2:], a[1:-1, 2:, 1:-1], a[2:, 1:-1, 1:-1]):
        s += x
    new = a.clone()
    new[inner] = s / torch.full((1,), 6.0, dtype=torch.float64, device="cuda")  # (a scalar would be a product by 1 / 6)
    eps = (new - a).abs().max().item()
    sp = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    b, alt = torch.empty_like(a), torch.empty_like(a)
    for v in range(22, J3_STENCILS):
        b.copy_(a)
        assert rt.dvmhgb_jac3d_stencil(vp(a), vp(b), st, ext, lo, hi, v, sp) == 0
        assert torch.equal(b, new), v
    for v in range(J3_STNUPD):
        b.copy_(a)
        alt.fill_(9.0)
        items = torch.full((rt.dvmhgb_jac3d_stnupd_items(lo, hi, v),), -1.0, dtype=torch.float64, device="cuda")
        assert rt.dvmhgb_jac3d_stnupd(vp(a), vp(alt), vp(b), st, ext, lo, hi, vp(items), v, sp) == 0
        assert torch.equal(b, new) and torch.equal(alt, new) and items.max().item() == eps, v


def fastest(call, runs=7):
    import torch
    best = float("inf")
    for _ in range(runs + 1):
        e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        torch.cuda.synchronize()
        torch.cuda._sleep(300000)
        e0.record()
        for _ in range(3):
            assert call() == 0
        e1.record()
        torch.cuda.synchronize()
        best = min(best, e0.elapsed_time(e1))
    return best


@pytest.mark.parametrize("n", [(255, 255, 256), (2000, 4, 2000)])
def test_signed_fields_are_not_slower(rt, n):
    """The stencil alone, variant 25, against all additions on the FP64 unit (13); the cross-step pass against that and
    an update loop.  Measured at 255^3: 178 against 204 us, 270 against 300."""
    import torch
    a = torch.rand(*n, generator=torch.Generator(device="cuda").manual_seed(1), dtype=torch.float64, device="cuda") * 2 - 1
    b, alt = torch.zeros_like(a), torch.zeros_like(a)
    st, ext, lo, hi = L3(n[1] * n[2], n[2], 1), L3(*n), L3(1, 1, 1), L3(*[q - 2 for q in n])
    items = torch.zeros(max(rt.dvmhgb_jac3d_stnupd_items(lo, hi, 4), rt.dvmhgb_jac3d_update_items(lo, hi)),
                        dtype=torch.float64, device="cuda")
    sp = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    fp64 = fastest(lambda: rt.dvmhgb_jac3d_stencil(vp(a), vp(b), st, ext, lo, hi, 13, sp))
    assert fastest(lambda: rt.dvmhgb_jac3d_stencil(vp(a), vp(b), st, ext, lo, hi, 25, sp)) < 1.05 * fp64
    update = fastest(lambda: rt.dvmhgb_jac3d_update(vp(a), vp(b), st, lo, hi, vp(items), 2, sp))
    a.copy_(torch.rand_like(a) * 2 - 1)
    cross = fastest(lambda: rt.dvmhgb_jac3d_stnupd(vp(a), vp(alt), vp(b), st, ext, lo, hi, vp(items), 4, sp))
    assert cross < 1.05 * (fp64 + update)


@pytest.mark.parametrize("n", [(2000, 4, 2000), (60000, 10, 34), (600, 26, 600), (256, 255, 256)])
def test_the_default_shape_is_a_fast_one(rt, n):
    import torch
    a = 0.5 + 0.25 * torch.rand(*n, generator=torch.Generator(device="cuda").manual_seed(1), dtype=torch.float64, device="cuda")
    b, alt = torch.zeros_like(a), torch.zeros_like(a)
    st, ext, lo, hi = L3(n[1] * n[2], n[2], 1), L3(*n), L3(1, 1, 1), L3(*[q - 2 for q in n])
    sp = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)

    def time(v):
        items = torch.zeros(rt.dvmhgb_jac3d_stnupd_items(lo, hi, v), dtype=torch.float64, device="cuda")
        return fastest(lambda: rt.dvmhgb_jac3d_stnupd(vp(a), vp(alt), vp(b), st, ext, lo, hi, vp(items), v, sp))

    assert time(rt.dvmhgb_jac3d_stnupd_default(lo, hi)) < 1.15 * min(time(v) for v in (0, 1, 2, 3, 4))
