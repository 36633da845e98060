"""Launch shapes of the compiled marches, read from the tables in the sources: no GPU needed."""
import glob
import os
import re

from conftest import ROOT

CSRC = os.path.join(ROOT, "cushg_b200", "csrc")


def rows():
    """(macro, threads) of every variant of the fused and adjoint marches."""
    for f in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        text = re.sub(r"//[^\n]*", "", open(f).read())
        for macro, args in re.findall(r"\b(SHG_VARIANT|SHG_SPLIT_VARIANT|SHG_ADJ)\((float|double[^()]*|float[^()]*)\)", text):
            a = [x.strip() for x in args.split(",")]
            yield f"{os.path.basename(f)}: {macro}({args})", int(a[5 if macro == "SHG_ADJ" else 4])


def test_every_split_has_whole_warps():
    """The power sums and the adjoint's reductions work warp by warp: a thread count that ends in a
    part of a warp has two warps on one row, one of them with lanes missing."""
    found = list(rows())
    assert len(found) > 40
    assert [name for name, threads in found if threads % 32] == []
