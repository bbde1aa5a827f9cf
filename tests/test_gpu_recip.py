"""rcp64 and rsqrt64 over every exponent they are claimed for.

Bounds: a seed of relative error e <= 2^-19 and one step whose remainder is e^3
(2^-57) leave the rounding of the last operation, half a unit in the last place,
and for the root that of x y in the residual, halved by the step: another half.
With room for the remainder: 0.6 and 1.1 units.  The signed mean of a million
roundings to nearest is zero to 3e-4 units; a one-signed remainder would show as
a drift of whatever sums them (0.003 allowed)."""
import pytest

import _device_check

pytestmark = pytest.mark.gpu


def test_error_of_the_fp64_reciprocals(native_lib, tmp_path):
    got = {}
    for line in _device_check.run("recip_check", tmp_path).splitlines():
        name, worst, mean, count = line.split()
        got[name] = (float(worst), float(mean), int(count))
    assert got["rcp"][2] > 10 ** 6
    assert got["rcp"][0] <= 0.6 and abs(got["rcp"][1]) <= 0.003, got
    assert got["rsqrt"][0] <= 1.1 and abs(got["rsqrt"][1]) <= 0.003, got
