"""What holds for the kernels' sources."""
import glob
import os

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rustymath_b200", "csrc")


@pytest.mark.parametrize("name", ["getrf.cu", "getrf_block.cu", "mixed.cu", "potrf.cu", "short_pivot.cuh",
                                  "batched_kernels.cuh"])
def test_reciprocals_are_correctly_rounded(name):
    """rustymath multiplies a pivot's column by the pivot's correctly rounded reciprocal. The kernels take it
    from CUDA's intrinsics and operators, not from the hardware's approximation."""
    (path,) = glob.glob(os.path.join(CSRC, name))
    assert "rcp.approx" not in open(path).read()


def test_a_change_to_any_source_or_header_rebuilds_the_library():
    from rustymath_b200 import build
    assert set(glob.glob(os.path.join(CSRC, "*"))) <= set(build.sources() + build.headers())
