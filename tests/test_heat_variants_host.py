"""The names of the heat step's strip geometries as a C program uses them: a constant default, rows and CTAs of a variant."""
import os
import subprocess

CODE = r"""
#include <stdio.h>
#include "dvmh_gb_kernels.h"
static const int usual = DVMHGB_HEAT_DEFAULT;
int main(void) {
    for (int v = 0; v < DVMHGB_HEAT_VARIANTS; v++)
        if (DVMHGB_HEAT_ROWS(v) < 1 || DVMHGB_HEAT_CTAS(v) < 1 || DVMHGB_HEAT_CTAS(v) > 8) return 1;
    printf("%ld %d\n", (long)DVMHGB_HEAT_ROWS(usual), (int)DVMHGB_HEAT_CTAS(usual));
    return usual >= 0 && usual < DVMHGB_HEAT_VARIANTS ? 0 : 1;
}
"""


def test_c_program(tmp_path):
    src, exe = tmp_path / "v.c", str(tmp_path / "v")
    src.write_text(CODE)
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "include")
    subprocess.check_call(["gcc", "-std=c99", "-I" + include, str(src), "-o", exe])
    rows, ctas = subprocess.check_output([exe], text=True).split()
    assert (int(rows), int(ctas)) == (32, 2)  # what takes the fewest rounds for many uneven plates
