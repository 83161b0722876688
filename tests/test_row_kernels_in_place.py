"""The row passes transform frame sums in place (input and output are one buffer),
so none of them may promise the compiler that the two do not overlap: under that
promise the input may be read through the non-coherent path."""

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "pyturb_gb300" / "csrc"
ROW_PASSES = ["k_rows", "k_rows_reg", "k_rows_gt", "k_rows_blu"]


@pytest.mark.parametrize("kernel", ROW_PASSES)
def test_row_pass_makes_no_aliasing_promise(kernel):
    found = [m for p in CSRC.glob("*.cu*")
             for m in re.findall(r"__global__[^;{}]*?\b%s\(([^{}]*?)\)\s*\{" % kernel, p.read_text())]
    assert len(found) == 1
    args = {a.split()[-1].lstrip("*"): a for a in found[0].split(",")}
    assert "__restrict__" not in args["in"] and "__restrict__" not in args["work"]
