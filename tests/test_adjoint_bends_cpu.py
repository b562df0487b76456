"""The adjoint of exact bends outside the range of its short form (csrc/adjoint.cuh): steps of negative
length and angles beyond a quarter turn, against central finite differences of the same element's forward
map (the method and tolerance of test_adjoint_cpu.py)."""
import pytest

import test_adjoint_cpu
from test_adjoint_cpu import abi, ha  # noqa: F401 (fixture)

# (l, g, ref_tilt); the angle is g l
BENDS = {
    "negative": (-0.3, 2.0, 0.0),
    "negative_both": (-1.0, -0.3, 0.0),
    "negative_tilted": (-0.3, 2.0, 0.2),
    "angle_1.49": (1.49, 1.0, 0.0),
    "angle_1.51": (1.51, 1.0, 0.0),
    "angle_2": (1.0, 2.0, 0.0),
    "angle_-3": (1.5, -2.0, 0.3),
    "angle_4.5": (2.25, 2.0, 0.0),
    "angle_-7.8": (3.772, -2.067, 0.0),
}


@pytest.mark.parametrize("name", sorted(BENDS))
def test_vjp_matches_finite_differences(ha, name):  # noqa: F811
    l, g, ref_tilt = BENDS[name]
    ele = abi.default_element(abi.SBEND, l=l, g=g, ref_tilt=ref_tilt, fringe_type=abi.FRINGE_NONE)
    test_adjoint_cpu.test_element_vjp_matches_finite_differences(ha, name, ele)
