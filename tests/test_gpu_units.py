"""The mixed sweeps in the units of a star (CGS: 3e28 g and 3e9 cm per node,
velocities of 100 km/s): the sums of a node stay inside FP32 in every form of
the pair sweep, so the derivatives, their moment matrix M and the viscous
pressures agree with the FP64 oracle as they do in units of order one (2e-5 of
the largest, FP32 rounding of pair terms that cancel)."""
import numpy as np
import pytest

from spheral_gb300 import problems

from _parity import compare_fields

pytestmark = pytest.mark.gpu

FIELDS = ["massDensitySum", "normalization", "DvDt", "DepsDt", "DvDx", "internalDvDx", "gradRho", "M",
          "maxViscousPressure", "effViscousPressure", "DHDt", "massZerothMoment", "omegaGradh"]


def _star(p, nodes_across):
    """p, a unit box of unit density and sound speed, as a box of 7e10 cm
    across at 6 g/cm^3 and 3e7 cm/s."""
    length = 1.75e9 * nodes_across
    density, speed = 6.0, 3.0e7
    p.pos *= length
    p.vel *= speed
    p.mass *= density * length ** 3
    p.rho *= density
    p.eps *= speed ** 2
    p.H /= length
    for b in p.boundaries:
        b["lo"] *= length
        b["hi"] *= length
    for d in p.nodelists:
        d.update(hmin=d["hmin"] * length, hmax=d["hmax"] * length)
    return p


def _compare(oracle_mod, p, fields):
    from spheral_gb300.engine import Engine
    eng, orc = Engine.from_problem(p, precision="fp32"), oracle_mod.Oracle(p)
    for e in (eng, orc):
        e.initialize()
        e.evaluate_derivatives()
    bad = compare_fields(eng, orc, fields, 2e-5)
    assert not bad, bad


# 16, 8, 4 and 2 lanes per node and the one-lane form of large runs; walls
@pytest.mark.parametrize("side,limited", [(12, False), (20, True), (40, False), (46, True), (54, False), (54, True)])
def test_isotropic_forms_in_stellar_units(native_lib, oracle_mod, side, limited):
    p = problems.random_box(n_side=side, seed=side, nPerh=1.25, boundaries="reflecting" if side == 20 else "periodic")
    if limited:
        p.config.update(viscosity="limited_monaghan_gingold", Cl=2.0, Cq=2.0)
    _compare(oracle_mod, _star(p, side), FIELDS)


@pytest.mark.parametrize("options", [dict(xsph=True), dict(compatible_energy=False)], ids=["xsph", "no_compat"])
def test_general_forms_in_stellar_units(native_lib, oracle_mod, options):
    p = problems.random_box(n_side=24, seed=3, nPerh=1.25)
    p.config.update(options)
    _compare(oracle_mod, _star(p, 24), FIELDS)


def test_tensor_form_in_stellar_units(native_lib, oracle_mod):
    p = problems.stretched_box(24, 20, 16, seed=4)
    _compare(oracle_mod, _star(p, 20), ["massDensitySum", "normalization", "DvDt", "DepsDt", "DvDx", "gradRho", "M",
                                        "maxViscousPressure", "effViscousPressure"])
