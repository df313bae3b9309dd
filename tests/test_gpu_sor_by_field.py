"""The SOR sweep whose kernel the field chooses (columns of hyperplane tiles or tiles one by one), and the choice by the
box's shape: bit for bit the box tiles' cells and residual items (variant 2: items of 8 positions too, no hyperplane
tiles), and no slower than the better of the two kernels where the columns alone were."""
import ctypes

import pytest

import __graft_entry__ as ge
from tests.test_gpu_sor_columns import BOXES, data, same
from tests.util import kernel_macros

pytestmark = pytest.mark.gpu
BY_FIELD = kernel_macros()["DVMHGB_SOR3D_VARIANTS"]
L3 = ctypes.c_long * 3


@pytest.fixture(scope="module")
def rt():
    ge.build()
    _, g = ge.package()
    g.init()
    L = g.runtime()
    for f in ("items", "scratch_bytes", "by_field_scratch_bytes"):
        getattr(L, "dvmhgb_sor3d_" + f).restype = ctypes.c_long
    return L


def vp(t):
    return ctypes.c_void_p(t.data_ptr())


class Sweep:
    """A box of an array and a variant's buffers: call() runs one sweep in place."""

    def __init__(self, L, a, lo, hi, variant, fill=7.0):
        import torch
        n, self.a = a.shape, a.cuda() if not a.is_cuda else a.clone()
        self.w = torch.tensor([1.2], dtype=torch.float64, device="cuda")
        st, ext, lo, hi = L3(n[1] * n[2], n[2], 1), L3(*n), L3(*lo), L3(*hi)
        field = variant == BY_FIELD
        self.items = torch.full((L.dvmhgb_sor3d_items(lo, hi, 5 if field else variant),), fill, dtype=torch.float64,
                                device="cuda")
        size = L.dvmhgb_sor3d_by_field_scratch_bytes(lo, hi) if field else L.dvmhgb_sor3d_scratch_bytes(lo, hi, variant)
        self.scratch = torch.full((size + 64,), 0x5A, dtype=torch.uint8, device="cuda")
        self.size = size
        self.status = torch.zeros(1, dtype=torch.int32, device="cuda")
        sp = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        head = (vp(self.a), st, ext, lo, hi, vp(self.w), vp(self.items), vp(self.scratch), vp(self.status))
        self.call = (lambda: L.dvmhgb_sor3d_sweep_by_field(*head, sp)) if field else (
            lambda: L.dvmhgb_sor3d_sweep(*head, variant, sp))

    def run(self, count):
        import torch
        for _ in range(count):
            assert self.call() == 0
        torch.cuda.synchronize()
        assert int(self.status.item()) == 0
        assert bool((self.scratch[self.size:] == 0x5A).all())  # nothing beyond the scratch asked for
        return self.a.cpu(), self.items.cpu()


# fields that the limbs hold (columns), that they do not (tiles), and both in one
@pytest.mark.parametrize("kind", ["unit", "signed", "mixed", "spots", "zero", "growing"])
@pytest.mark.parametrize("box", range(len(BOXES)))
@pytest.mark.parametrize("variant", [BY_FIELD, 5, 4])
def test_cells_and_items(rt, box, kind, variant):
    n, lo, hi = BOXES[box]
    a = data(kind, n, box)
    cells, items = Sweep(rt, a, lo, hi, variant, 7.0).run(2)
    want, want_items = Sweep(rt, a, lo, hi, 2, -3.0).run(2)  # (an item that one of them leaves out differs)
    assert same(cells, want)
    assert same(items, want_items)


@pytest.mark.parametrize("kind", ["unit", "signed"])
def test_more_columns_than_the_gpu_holds(rt, kind):
    n = (300, 260, 12)
    lo, hi = (1, 1, 1), tuple(q - 2 for q in n)
    a = data(kind, n, 7)
    cells, items = Sweep(rt, a, lo, hi, BY_FIELD, 7.0).run(2)
    want, want_items = Sweep(rt, a, lo, hi, 2, -3.0).run(2)
    assert same(cells, want) and same(items, want_items)


@pytest.mark.parametrize("n,signed", [((384, 384, 384), True), ((40, 500, 400), False), ((240, 240, 240), True)])
def test_default_is_not_slower_than_the_tiles(rt, n, signed):
    import torch
    lo, hi = (1, 1, 1), tuple(q - 2 for q in n)
    a = torch.rand(*n, generator=torch.Generator(device="cuda").manual_seed(1), dtype=torch.float64, device="cuda")
    if signed:
        a = 2 * a - 1
    times = {}
    for variant in (4, rt.dvmhgb_sor3d_default_variant(L3(*lo), L3(*hi))):
        s, best = Sweep(rt, a, lo, hi, variant), 1e9
        for _ in range(8):
            b, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            b.record()
            assert s.call() == 0
            e.record()
            torch.cuda.synchronize()
            best = min(best, b.elapsed_time(e))
        times[variant] = best
    assert all(t < 1.025 * times[4] for t in times.values()), times
