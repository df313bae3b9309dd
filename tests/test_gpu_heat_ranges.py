"""The heat kernel's strips on fields that its limbs hold, move to, or leave to the FP64 unit, at strip lengths around
the batches of 8 rows and at widths around the 64-wide chunks.  Every item -- the SUM tree and the MINLOC of each row of
a chunk -- and every cell is compared with numpy, bit for bit."""
import ctypes

import numpy as np
import pytest

import __graft_entry__ as ge
from tests.test_gpu_heat_kernel import HeatDesc

pytestmark = pytest.mark.gpu

KINDS = ["unit", "degrees", "negative", "zeros", "subnormal", "growing", "far apart", "special"]


def field(kind, n, m):
    rng = np.random.default_rng(KINDS.index(kind) * 100 + n)
    a = rng.random((n, m))
    if kind == "degrees":
        a *= 100.0
    if kind == "negative":
        a -= 0.5
    if kind == "zeros":
        a[:, : m // 2] = 0.0
        a[n // 2, 2] = -0.0
    if kind == "subnormal":
        a *= 2.0 ** -1040
    if kind == "growing":
        a *= 2.0 ** np.floor(np.arange(n) / 2)[:, None]
    if kind == "far apart":
        a *= 10.0 ** np.round(rng.random((n, m)) * 20 - 10)
    if kind == "special":
        a[n // 2, m // 2], a[1, 1], a[n - 2, m - 2] = np.inf, np.nan, -np.inf
    return a


def tree(v):
    v = v.copy()
    while len(v) > 1:
        v = v[0::2] + v[1::2]
    return v[0]


def reference(a, lo, hi, c):
    """dst over the box, and per (row, chunk) the SUM, the minimum and its place."""
    i, j = np.arange(lo[0], hi[0] + 1), np.arange(lo[1], hi[1] + 1)
    g = lambda di, dj: a[np.ix_(i + di, j + dj)]  # noqa: E731
    with np.errstate(all="ignore"):
        new = g(0, 0) + c * ((((g(-1, 0) + g(1, 0)) + g(0, -1)) + g(0, 1)) - 4.0 * g(0, 0))
        items = []
        for r in range(len(i)):
            for ch in range(lo[1] // 64, hi[1] // 64 + 1):
                s = np.full(64, -0.0)
                best, at = np.inf, None
                for q in range(64):
                    col = 64 * ch + q
                    if lo[1] <= col <= hi[1]:
                        v = new[r, col - lo[1]]
                        s[q] = v
                        if v < best:
                            best, at = v, col
                items.append((tree(s), best, at))
    return new, items


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n,m,lo1", [(4, 3, 1), (12, 66, 1), (21, 67, 3), (30, 131, 1), (11, 200, 65)])
def test_strips(kind, n, m, lo1):
    import torch
    ge.build()
    _, g = ge.package()
    g.init()
    L = g.runtime()
    c = 0.2
    coef = torch.tensor([c], dtype=torch.float64, device="cuda")
    a = field(kind, n, m)
    lo, hi = (1, lo1), (n - 2, m - 2)
    new, items = reference(a, lo, hi, c)
    w = m + (m & 1) + 2
    S = torch.full((n, w), 1e30, dtype=torch.float64, device="cuda")  # the rows' padding is not the loop's business
    S[:, :m] = torch.from_numpy(a).cuda()
    sp = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    vp = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    for sr in (0, 1, 7, 8, 9, 17, 64):  # 0: the single loop's own choice
        D = torch.full_like(S, 7.0)
        d = HeatDesc()
        assert L.dvmhgb_heat_desc_fill(ctypes.byref(d), vp(S), vp(D), ctypes.c_long(w), (ctypes.c_long * 2)(*lo),
                                       (ctypes.c_long * 2)(*hi), vp(coef)) == 0
        si = torch.full((d.units + 1,), 7.0, dtype=torch.float64, device="cuda")
        mi = torch.full_like(si, 7.0)
        li = torch.full((2 * d.units + 1,), 7, dtype=torch.int32, device="cuda")
        d.sumItems, d.minItems, d.locItems = si.data_ptr(), mi.data_ptr(), li.data_ptr()
        if sr == 0:
            assert L.dvmhgb_heat(ctypes.byref(d), sp) == 0
        else:
            assert L.dvmhgb_heat_desc_rows(ctypes.byref(d), ctypes.c_long(sr)) == 0
            dev = torch.empty(ctypes.sizeof(d), dtype=torch.uint8, device="cuda")
            dev.copy_(torch.frombuffer(bytearray(d), dtype=torch.uint8))
            assert L.dvmhgb_heat_many(vp(dev), 1, ctypes.c_long(d.strips), sp) == 0
        got = D.cpu().numpy()
        where = (kind, n, m, sr)
        box = got[lo[0]:hi[0] + 1, lo[1]:hi[1] + 1]
        assert ((box.view(np.int64) == new.view(np.int64)) | (np.isnan(box) & np.isnan(new))).all(), where
        got[lo[0]:hi[0] + 1, lo[1]:hi[1] + 1] = 7.0
        assert (got == 7.0).all(), where
        si, mi, li = si.cpu().numpy(), mi.cpu().numpy(), li.cpu().numpy()
        assert si[-1] == 7.0 and mi[-1] == 7.0 and li[-1] == 7, where
        for q, (s, best, at) in enumerate(items):
            assert si[q] == s or (np.isnan(si[q]) and np.isnan(s)), (where, q)
            assert mi[q] == best, (where, q)
            if at is not None:
                row = lo[0] + q // (hi[1] // 64 - lo[1] // 64 + 1)
                assert (li[2 * q], li[2 * q + 1]) == (row, at), (where, q)
