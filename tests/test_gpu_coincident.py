"""eps2 = 0 in the artificial viscosity: nodes at the same place (and a node on
a wall with its own image) take no viscosity from each other, their mu being
0/0, in every form of the pair sweep."""
import numpy as np
import pytest

from spheral_gb300 import problems

from _parity import compare_fields

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("fp32", 2e-5)])
@pytest.mark.parametrize("side,limited", [(9, False), (9, True), (20, False), (30, True), (54, False)])
def test_coincident_nodes_without_eps2(native_lib, oracle_mod, side, limited, precision, tol):
    from spheral_gb300.engine import Engine
    if side > 50 and precision == "fp64":
        pytest.skip("the FP64 sweep has one form of the quotient")
    p = problems.random_box(n_side=side, seed=side, nPerh=1.25)
    p.config.update(eps2=0.0)
    if limited:
        p.config.update(viscosity="limited_monaghan_gingold", Cl=2.0, Cq=2.0)
    for a, b in ((0, 1), (p.n // 2, p.n // 2 + 1)):
        p.pos[b] = p.pos[a]
        p.vel[b] = p.vel[a] + np.array([0.1, 0.2, 0.3])   # v_ij . 0 is -0 from one side
    eng, orc = Engine.from_problem(p, precision=precision), oracle_mod.Oracle(p)
    for e in (eng, orc):
        e.initialize()
        e.evaluate_derivatives()
    bad = compare_fields(eng, orc, ["DvDt", "DepsDt", "DvDx", "maxViscousPressure", "effViscousPressure"], tol)
    assert not bad, bad
    assert np.all(np.isfinite(eng.field("DvDt")))
