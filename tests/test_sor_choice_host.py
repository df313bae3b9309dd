"""dvmhgb_sor3d_default_variant: which of the two hyperplane sweeps a box takes, on the 152 SMs of a GB300."""
import ctypes

import pytest

import __graft_entry__ as ge
from tests.util import kernel_macros

K = kernel_macros()
L3 = ctypes.c_long * 3


@pytest.fixture(scope="module")
def rt():
    ge.build()
    _, g = ge.package()
    L = g.runtime()
    L.dvmhgb_sor3d_scratch_bytes.restype = L.dvmhgb_sor3d_by_field_scratch_bytes.restype = ctypes.c_long
    return L


@pytest.mark.parametrize("n,want", [((3, 3, 3), 4), ((12, 12, 12), 5), ((34, 34, 34), 5), ((97, 97, 97), 5),
                                    ((190, 190, 190), 5), ((200, 200, 200), 6), ((384, 384, 384), 6),
                                    ((40, 500, 400), 4), ((500, 40, 400), 5), ((60, 60, 2000), 4), ((100, 100, 1000), 5),
                                    ((18, 200, 300), 4), ((400, 400, 40), 6), ((100, 2000, 40), 4), ((4000, 20, 20), 5)])
def test_by_shape(rt, n, want):
    import torch
    if torch.cuda.is_available():
        pytest.skip("another number of SMs")
    assert K["DVMHGB_SOR3D_VARIANTS"] == 6
    lo, hi = L3(1, 1, 1), L3(*[q - 2 for q in n])
    assert rt.dvmhgb_sor3d_default_variant(lo, hi) == want


@pytest.mark.parametrize("box", [((1, 1, 1), (1, 1, 1)), ((1, 1, 1), (382, 382, 382)), ((3, 2, 100), (40, 39, 101))])
def test_scratch_holds_either_sweep(rt, box):
    lo, hi = L3(*box[0]), L3(*box[1])
    ti = [(hi[d] - lo[d] + t) // t for d, t in ((0, 16), (1, 8))]
    assert rt.dvmhgb_sor3d_by_field_scratch_bytes(lo, hi) >= max(rt.dvmhgb_sor3d_scratch_bytes(lo, hi, 4),
                                                                 256 + 4 * ti[0] * ti[1])


def test_empty_box(rt):
    assert rt.dvmhgb_sor3d_by_field_scratch_bytes(L3(5, 1, 1), L3(4, 10, 10)) == -1
