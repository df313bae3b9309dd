"""Reduction results that a fold also writes to pinned host memory: what get_actual returns is the device copy's value
where folds wrote all of the variable, some of it, or where a kernel wrote the device copy itself, in every mode and on
replayed graphs."""
import ctypes
import importlib.util
import os

import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def cases():
    import __graft_entry__ as ge
    ge.build()
    spec = importlib.util.spec_from_file_location("perf_cases", os.path.join(HERE, "..", "perf", "cases.py"))
    m = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(m)
    return m


def plates(cases, mode, scale=1.0):
    """A program whose steps run in the given mode."""
    p = cases.prepare({"kind": "heat", "count": 3, "lo": 16, "hi": 64, "steps": 1, "scale": scale, "mode": mode}, 5)
    step = p.step

    def in_mode():
        p.set_mode(p.mode)
        return step()

    p.step = in_mode
    return p


@pytest.mark.parametrize("mode", ["plain", "async", "batched"])
def test_whole_and_partial_results(cases, mode):
    """Three plates share arrays of sums, minima and places: steps over all of them, over the outer two (the middle
    entries are the program's own), and over all again."""
    p, ref = plates(cases, mode), plates(cases, "plain")
    both = p.loops
    for step in range(6):
        want = ref.step()
        some = step % 3 == 1
        p.loops = tuple([q for k, q in enumerate(way) if not (some and k == 1)] for way in both)
        got = p.step()
        for k in range(3):
            if some and k == 1:
                assert (got[0][1], got[1][1]) == (0, 1e300) and (got[2][1] == -1).all()
            elif k != 1 or step == 0:  # the middle plate has skipped a step from then on
                assert got[0][k] == want[0][k] and got[1][k] == want[1][k] and (got[2][k] == want[2][k]).all()
    p.set_mode(ctypes.c_int(cases.gb.MODES["batched"]))


@pytest.mark.parametrize("mode", ["plain", "async", "batched"])
def test_device_copy_written_by_a_kernel(cases, mode):
    """A program that asks for the device address may write there: its value is what get_actual returns, then and after
    the next steps."""
    import torch
    p, ref = plates(cases, mode), plates(cases, "plain")
    address = cases._abi("dvmh_get_device_addr_C", ctypes.c_void_p, ctypes.c_long, ctypes.c_void_p)
    fetch, p.get_actual = p.get_actual, lambda v: None  # a step that does not read its results
    p.step()
    ref.step()
    d = address(1, p.sums.ctypes.data)
    raw = type("Sums", (), {"__cuda_array_interface__": {"shape": (3,), "typestr": "<f8", "data": (d, False),
                                                         "version": 2}})()
    p.flush()
    with torch.cuda.stream(p.stream):
        torch.as_tensor(raw, device="cuda")[1] = 42.0
    for v in p.results:
        fetch(v)
    assert p.sums[1] == 42.0
    p.get_actual = fetch
    for _ in range(3):
        got, want = p.step(), ref.step()
        assert all((g == w).all() for g, w in zip(got, want))
    p.set_mode(ctypes.c_int(cases.gb.MODES["batched"]))
