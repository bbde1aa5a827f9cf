"""The mixed pair sweep's two forms are equally accurate: the reduced one of
small runs is no further from the FP64 oracle (root mean square over the nodes,
within the 15 % that two samples of the same roundings may differ by) than the
one large runs and domains of a decomposed run take."""
import numpy as np
import pytest

from spheral_gb300 import problems

pytestmark = pytest.mark.gpu

FIELDS = ["DvDt", "DepsDt", "DvDx", "gradRho", "M", "maxViscousPressure", "DHDt", "Hideal", "massZerothMoment"]


@pytest.mark.parametrize("limited", [False, True], ids=["mg", "limited"])
@pytest.mark.parametrize("make", [lambda: problems.kelvin_helmholtz(n1=20, seed=20),
                                  lambda: problems.kelvin_helmholtz(n1=41, seed=41),
                                  lambda: problems.random_box(n_side=30, seed=30)], ids=["kh20", "kh41", "box30"])
def test_reduced_form_is_as_accurate(native_lib, oracle_mod, make, limited):
    from spheral_gb300.engine import Engine
    p = make()
    if limited:
        p.config.update(viscosity="limited_monaghan_gingold", Cl=2.0, Cq=2.0)
    orc = oracle_mod.Oracle(p)
    orc.initialize()
    orc.evaluate_derivatives()
    err = []
    for domain in (False, True):
        eng = Engine.from_problem(p, precision="fp32")
        if domain:
            eng.set_domain(0, lambda point, dt: dt)
        eng.initialize()
        eng.evaluate_derivatives()
        err.append({f: np.sqrt(np.mean((eng.field(f) - orc.field(f)) ** 2)) for f in FIELDS})
    worse = {f: err[0][f] / err[1][f] for f in FIELDS if err[0][f] > 1.15 * err[1][f]}
    assert not worse, worse
