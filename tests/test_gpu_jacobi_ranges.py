"""The Jacobi-3D stencil and cross-step kernels on fields outside [0, 1): the limb kernels move their range to the
values they meet, and compute on the FP64 unit what does not fit.  Bit-exact against float64 on the CPU."""
import ctypes

import pytest

import __graft_entry__ as ge
from tests.util import J3_STENCILS, J3_STNUPD

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def g():
    ge.build()
    _, g = ge.package()
    g.init()
    return g


def field(kind, n, seed):
    import torch
    gen = torch.Generator().manual_seed(seed)
    a = torch.rand(*n, generator=gen, dtype=torch.float64)
    i = torch.arange(n[0], dtype=torch.float64)[:, None, None]
    if kind == "degrees":
        return a * 100.0
    if kind == "huge":
        return a * 2.0 ** 990
    if kind == "tiny":  # the smallest normal numbers' neighbourhood: sums and quotients stay normal
        return (a + 0.5) * 2.0 ** -1000
    if kind == "subnormal":
        return a * 2.0 ** -1030
    if kind == "growing":  # a binade more every three planes: the range moves along
        return a * 2.0 ** (i / 3).floor()
    if kind == "hot wall":  # zeros everywhere but on one face
        a = torch.zeros(*n, dtype=torch.float64)
        a[0] = 1.0
        return a
    if kind == "mixed":  # no range holds these
        return a * 10.0 ** (torch.rand(*n, generator=gen, dtype=torch.float64) * 24 - 12).round()
    if kind == "spots":  # single values far from the rest, one negative, one infinite
        a[3, 4, 5], a[n[0] // 2, 7, 2], a[2, n[1] - 2, n[2] - 2] = 1e40, -0.25, 1e-30
        a[n[0] - 3, 3, 3] = float("inf")
        return a
    if kind == "equal":  # every difference the same
        return torch.full(n, 0.3, dtype=torch.float64)
    raise ValueError(kind)


KINDS = ["degrees", "huge", "tiny", "subnormal", "growing", "hot wall", "mixed", "spots", "equal"]


def reference(a):
    s = a[:-2, 1:-1, 1:-1] + a[1:-1, :-2, 1:-1]
    for x in (a[1:-1, 1:-1, :-2], a[1:-1, 1:-1, 2:], a[1:-1, 2:, 1:-1], a[2:, 1:-1, 1:-1]):
        s = s + x
    return s / 6.0


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n", [(13, 21, 70), (40, 12, 133)])
def test_stencil_and_cross_step(g, kind, n):
    import torch
    L = g.runtime()
    L.dvmhgb_jac3d_stnupd_items.restype = ctypes.c_long
    ld = (n[2] + 1) // 2 * 2
    A3 = ctypes.c_long * 3
    st, ext, lo, hi = A3(n[1] * ld, ld, 1), A3(*n), A3(1, 1, 1), A3(n[0] - 2, n[1] - 2, n[2] - 2)
    a = field(kind, n, KINDS.index(kind))
    inner = (slice(1, -1),) * 3
    new = reference(a)
    eps = (new - a[inner]).abs()
    eps = eps[~eps.isnan()].max()
    dev = torch.zeros(n[0], n[1], ld, dtype=torch.float64, device="cuda")
    dev[:, :, :n[2]] = a.cuda()
    vp = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    bits = lambda t: t.cpu().contiguous().view(torch.int64)  # noqa: E731
    stream = torch.cuda.current_stream().cuda_stream
    for v in range(22, J3_STENCILS):
        b = torch.full_like(dev, 7.0)
        assert L.dvmhgb_jac3d_stencil(vp(dev), vp(b), st, ext, lo, hi, v, ctypes.c_void_p(stream)) == 0
        b = b.cpu()
        assert torch.equal(bits(b[1:-1, 1:-1, 1:n[2] - 1]), bits(new)), (kind, v)
        b[1:-1, 1:-1, 1:n[2] - 1] = 7.0
        assert bool((b == 7.0).all()), (kind, v)  # nothing outside the box
    for v in range(J3_STNUPD):
        b, alt = torch.full_like(dev, 7.0), torch.full_like(dev, 9.0)
        items = torch.full((L.dvmhgb_jac3d_stnupd_items(lo, hi, v),), -1.0, dtype=torch.float64, device="cuda")
        assert L.dvmhgb_jac3d_stnupd(vp(dev), vp(alt), vp(b), st, ext, lo, hi, vp(items), v,
                                     ctypes.c_void_p(stream)) == 0
        want = a.clone()
        want[inner] = new
        assert torch.equal(bits(alt[:, :, :n[2]]), bits(want)), (kind, v)  # outside the box: A's values
        assert torch.equal(bits(b[1:-1, 1:-1, 1:n[2] - 1]), bits(new)), (kind, v)
        assert bool((alt.cpu()[:, :, n[2]:] == 9.0).all()), (kind, v)  # no write past the rows' ends
        assert items.max().item() == eps.item(), (kind, v)


@pytest.mark.parametrize("kind", KINDS)
def test_update(g, kind):
    """The update loop's |B - A|, whose fixed point follows the values too."""
    import torch
    L = g.runtime()
    L.dvmhgb_jac3d_update_items.restype = ctypes.c_long
    n = (9, 14, 131)
    ld = 132
    A3 = ctypes.c_long * 3
    st, lo, hi = A3(n[1] * ld, ld, 1), A3(1, 1, 1), A3(n[0] - 2, n[1] - 2, n[2] - 2)
    a, b = field(kind, n, 3), field(kind, n, 4)
    da, db = (torch.zeros(n[0], n[1], ld, dtype=torch.float64, device="cuda") for _ in range(2))
    da[:, :, :n[2]], db[:, :, :n[2]] = a.cuda(), b.cuda()
    items = torch.full((L.dvmhgb_jac3d_update_items(lo, hi),), -1.0, dtype=torch.float64, device="cuda")
    vp = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert L.dvmhgb_jac3d_update(vp(da), vp(db), st, lo, hi, vp(items), 2, stream) == 0
    inner = (slice(1, -1),) * 3
    d = (b[inner] - a[inner]).abs()
    assert items.max().item() == d[~d.isnan()].max().item()
    a[inner] = b[inner]
    assert torch.equal(da[:, :, :n[2]].cpu(), a)
