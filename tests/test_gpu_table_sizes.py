"""Kernel tables of every size in the mixed mode: an odd number of intervals
leaves the packed FP32 table aligned for its 16-byte loads, and the derivatives
agree with the FP64 oracle on the same table (2e-5 of the largest)."""
import pytest

from spheral_gb300 import problems

from _parity import compare_fields

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("points", [990, 994, 998, 1000])
@pytest.mark.parametrize("make", ["sph", "asph", "crksph"])
def test_table_sizes(native_lib, oracle_mod, make, points):
    from spheral_gb300.engine import Engine
    p = {"sph": lambda: problems.random_box(n_side=12, seed=2), "asph": lambda: problems.stretched_box(16, 13, 10),
         "crksph": lambda: problems.crksph_box(n_side=12)}[make]()
    p.config.update(num_table_points=points, kernel="wendland_c4" if make == "sph" else "bspline")
    if make == "sph":
        p.nodelists[0].update(nPerh=3.02)
        p.H *= 0.5   # the kernel's extent is 1
    eng, orc = Engine.from_problem(p, precision="fp32"), oracle_mod.Oracle(p)
    for e in (eng, orc):
        e.initialize()
        e.evaluate_derivatives()
    bad = compare_fields(eng, orc, ["DvDt", "DepsDt", "DvDx", "massZerothMoment"], 2e-5)
    assert not bad, bad
