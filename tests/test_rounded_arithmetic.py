"""The kernels' divisions and roots are the rounded ones: no approximate
intrinsic and no approximate instruction in the sources, and no compiler flag
that would put them there."""
import glob
import os
import re

PACKAGE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "vlasiator_b200")
APPROXIMATE = r"\.approx|__fdividef|__frsqrt|__(exp|exp10|log|log2|log10|pow|sin|cos|tan)f\b"


def test_no_approximate_arithmetic():
    found = []
    for path in sorted(glob.glob(os.path.join(PACKAGE, "csrc", "*.cu*"))):
        with open(path) as f:
            for n, line in enumerate(f, 1):
                if re.search(APPROXIMATE, line.split("//")[0]):
                    found.append((os.path.basename(path), n, line.strip()))
    assert not found, found


def test_no_approximate_build():
    from vlasiator_b200.build import FLAGS
    assert not [f for f in FLAGS if re.search(r"fast_math|prec-div=false|prec-sqrt=false|ftz=true", f)]
