"""The limb kernels' shapes (rows per thread, plane slots, CTAs per SM) of the cross-step Jacobi-3D variants: no two alike,
or the tuner times one kernel under two numbers, and the handlers' table for the tuner's model says the same ones."""
import os
import re

from tests.util import J3_STNUPD

PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dvm-snapshot-r6603-fork_gb300")


def test_shapes():
    text = open(os.path.join(PKG, "csrc", "kernels", "jacobi.cu")).read()
    lines = " ".join(re.findall(r"#define DVMHGB_LIMB_S\w+\(C\) (.*)", text))
    shapes = [tuple(map(int, m)) for m in re.findall(r"C\((\d+), (\d+), (\d+), (\d+)\)", lines)]
    assert [s[0] for s in shapes] == list(range(J3_STNUPD))
    assert len({s[1:] for s in shapes}) == J3_STNUPD
    text = open(os.path.join(PKG, "workloads", "jac3d_cuda.cu")).read()
    table = re.search(r"c\[6\]\[3\] = \{(.*)\};", text).group(1)
    assert [tuple(map(int, m)) for m in re.findall(r"\{(\d+), (\d+), (\d+)\}", table)] == [s[1:] for s in shapes]
