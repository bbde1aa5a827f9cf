"""The sweeps change form with the node count: lanes per node, the mixed pair
loop's arithmetic (from 150,000 nodes), four warps or one per search item, the
tiles of the node sort.  On both sides of every line the neighbour sets equal
the FP64 oracle's exactly, and the fields stay within the bounds of the
precision mode: FP64 1e-12 normwise (summation order and the 2-ulp reciprocals
of ~130 terms), mixed 2e-5 for derivatives (FP32 rounding of pair terms that
cancel; ten times that at 33 nodes, where the corrected gradients of nodes with
a handful of neighbours amplify it by their moment matrix's condition) and 2e-6
for the density and grad-h sums (compensated)."""
import numpy as np
import pytest

from spheral_gb300 import problems

from _parity import compare_fields

pytestmark = pytest.mark.gpu

FP64 = ["massDensitySum", "normalization", "DvDt", "DepsDt", "DvDx", "gradRho", "M", "maxViscousPressure",
        "effViscousPressure", "DHDt", "Hideal", "massZerothMoment", "omegaGradh"]
FP32 = ["massDensitySum", "DvDt", "DepsDt", "DvDx", "gradRho", "M", "maxViscousPressure", "DHDt", "Hideal",
        "massZerothMoment"]


def _box(n, seed, boundaries="open", **config):
    """n nodes of a jittered lattice in the unit cube (a random subset of the
    next larger cube), about 60 neighbours each."""
    side = int(np.ceil(n ** (1.0 / 3.0) - 1e-9))
    p = problems.random_box(n_side=side, seed=seed, nPerh=1.25, boundaries=boundaries)
    keep = np.sort(np.random.default_rng(seed).permutation(p.n)[:n])
    for k in ("pos", "vel", "mass", "rho", "eps", "H", "nodelist"):
        setattr(p, k, np.ascontiguousarray(getattr(p, k)[keep]))
    p.config.update(config)
    return p


def _keys(i, j, n):
    return np.unique(np.asarray(i, np.int64) * n + np.asarray(j, np.int64))


def _pair(oracle_mod, p, precision, sets=True):
    from spheral_gb300.engine import Engine
    eng, orc = Engine.from_problem(p, precision=precision), oracle_mod.Oracle(p)
    eng.initialize()
    orc.initialize()
    if not sets:   # the derivatives see every neighbour; comparing 10^7 keys takes longer than they do
        assert eng.neighbor_entries() > 0
        return eng, orc
    i, j, _ = eng.pairs()
    a, b, _ = orc.pairs()
    assert np.array_equal(_keys(i, j, p.n), np.union1d(_keys(a, b, p.n), _keys(b, a, p.n)))
    return eng, orc


@pytest.mark.parametrize("n", [1, 2, 33, 2047, 2048, 2049, 5999, 6000, 19999, 20001])
@pytest.mark.parametrize("limited", [False, True], ids=["mg", "limited"])
def test_mixed_forms(native_lib, oracle_mod, n, limited):
    cfg = dict(viscosity="limited_monaghan_gingold", Cl=2.0, Cq=2.0) if limited else {}
    eng, orc = _pair(oracle_mod, _box(n, 31 + n, **cfg), "fp32")
    eng.evaluate_derivatives()
    orc.evaluate_derivatives()
    bad = compare_fields(eng, orc, FP32 if n > 2 else ["DvDt"], 2e-5 if n > 33 else 2e-4)
    assert not bad, bad
    bad = compare_fields(eng, orc, ["omegaGradh"], 2e-6)
    assert not bad, bad
    dt, ref = eng.dt()[0], orc.hydro_dt()
    assert abs(dt - ref) <= (1e-5 if n > 33 else 2e-4) * ref
    eng.sum_density()
    orc.sum_density()
    bad = compare_fields(eng, orc, ["massDensity"], 2e-6)
    assert not bad, bad


@pytest.mark.parametrize("n", [79999, 80000, 149999, 150000])
def test_mixed_forms_large(native_lib, oracle_mod, n):
    p = _box(n, 7, boundaries="reflecting" if n == 149999 else "open")
    eng, orc = _pair(oracle_mod, p, "fp32")
    eng.evaluate_derivatives()
    orc.evaluate_derivatives()
    bad = compare_fields(eng, orc, FP32, 2e-5)
    assert not bad, bad
    a, b = eng.step(), orc.step()
    assert abs(a - b) <= 1e-5 * b
    bad = compare_fields(eng, orc, ["massDensity", "specificThermalEnergy", "H"], 5e-5)
    assert not bad, bad


@pytest.mark.parametrize("n", [1, 2, 33, 7999, 8000, 19999, 20000, 59999, 60000])
def test_fp64_forms(native_lib, oracle_mod, n):
    limited = n in (33, 7999, 20000)
    cfg = dict(viscosity="limited_monaghan_gingold", Cl=2.0, Cq=2.0, xsph=True) if limited else {}
    p = _box(n, 3 + n, boundaries="reflecting" if n == 8000 else "open", **cfg)
    eng, orc = _pair(oracle_mod, p, "fp64")
    eng.evaluate_derivatives()
    orc.evaluate_derivatives()
    bad = compare_fields(eng, orc, FP64 if n > 2 else ["DvDt", "omegaGradh"], 1e-12)
    assert not bad, bad
    dt, ref = eng.dt()[0], orc.hydro_dt()
    assert abs(dt - ref) <= 1e-12 * ref
    a, b = eng.step(), orc.step()
    assert abs(a - b) <= 1e-12 * b
    bad = compare_fields(eng, orc, ["position", "velocity", "massDensity", "specificThermalEnergy", "H"], 1e-11)
    assert not bad, bad


@pytest.mark.parametrize("shape", [(96, 4, 4), (4, 4, 96), (5, 40, 5)])
def test_elongated_grids(native_lib, oracle_mod, shape):
    """Grids whose axes have different bit counts (the cell key keeps the extra
    bits of the longer axes above the interleaved ones)."""
    nx, ny, nz = shape
    rng = np.random.default_rng(nx)
    p = problems.random_box(n_side=12, seed=1, boundaries="open")
    pos = problems._lattice(nx, ny, nz, (0.0, 0.0, 0.0), (float(nx), float(ny), float(nz)))
    n = len(pos)
    pos = pos + rng.normal(0.0, 0.1, pos.shape)
    q = problems.Problem("bar", pos, rng.normal(0.0, 0.1, pos.shape), np.ones(n), np.ones(n), np.full(n, 1.5),
                         np.full(n, 0.6), None, [dict(p.nodelists[0], hmax=10.0)], [], dict(p.config))
    eng, orc = _pair(oracle_mod, q, "fp64")
    eng.evaluate_derivatives()
    orc.evaluate_derivatives()
    bad = compare_fields(eng, orc, ["DvDt", "DepsDt", "DvDx"], 1e-12)
    assert not bad, bad


ASPH_SHAPES = [(30, 20, 19), (30, 20, 21), (45, 32, 27), (45, 32, 28), (60, 48, 34), (60, 48, 35)]


@pytest.mark.parametrize("shape,boundaries", [(s, "periodic") for s in ASPH_SHAPES] +
                         [(s, "reflecting") for s in ASPH_SHAPES[1::2]])
def test_asph_forms(native_lib, oracle_mod, shape, boundaries):
    """Tensor H on both sides of 12,000, 40,000 and 100,000 nodes; the bound is
    the one of the mixed ASPH derivatives.  With walls only the boxes that have
    no node on one: 1e-9 from a wall, 2e-9 from its own image, the FP32 second
    moment's |r|^-5 overflows and Hideal falls back to the isotropic one."""
    p = problems.stretched_box(*shape, seed=sum(shape), boundaries=boundaries)
    eng, orc = _pair(oracle_mod, p, "fp32", p.n < 20000)
    eng.evaluate_derivatives()
    orc.evaluate_derivatives()
    bad = compare_fields(eng, orc, ["DvDt", "DepsDt", "DvDx", "massDensitySum", "DHDt", "Hideal", "massZerothMoment",
                                    "maxViscousPressure"], 2e-5)
    assert not bad, bad


@pytest.mark.parametrize("side", [24, 25, 27, 28, 34, 35, 46, 47, 53, 54])
def test_crk_forms(native_lib, oracle_mod, side):
    """CRKSPH on both sides of 15,000, 20,000, 40,000, 100,000 and 150,000 nodes
    with the standard Q, the limited Q at the odd sides; the bounds are twice
    those of the mixed CRKSPH evaluation, the vote's the same."""
    q = dict(viscosity="limited_monaghan_gingold") if side % 2 else dict(viscosity="monaghan_gingold", Cl=1.0, Cq=1.0)
    p = problems.crksph_box(n_side=side, seed=side, boundaries="reflecting" if side in (25, 46) else "periodic")
    p.config.update(xsph=False, **q)
    eng, orc = _pair(oracle_mod, p, "fp32", p.n < 20000)
    eng.sum_density()
    orc.sum_density()
    eng.evaluate_derivatives()
    orc.rk_corrections()
    orc.evaluate_derivatives()
    bad = compare_fields(eng, orc, ["massDensity", "DvDt", "DepsDt", "DvDx", "Hideal", "massZerothMoment",
                                    "rkCorrections"], 2e-5)
    assert not bad, bad
    dt, ref = eng.dt()[0], orc.hydro_dt()
    assert abs(dt - ref) <= 1e-6 * ref
    if side < 40 or side == 54:   # the vote on the density sweep
        a, b = eng.step(), orc.step()
        assert abs(a - b) <= 1e-5 * b


@pytest.mark.parametrize("n", [2, 3, 7, 8, 9, 31, 33, 127, 1025])
@pytest.mark.parametrize("softening", [1e-15, 0.01, 30.0])
def test_gravity_forms(native_lib, oracle_mod, n, softening):
    """Eight nodes per warp (FP64) and 32 (mixed); softenings whose separation
    limit, 1e-5 of them, excludes no node, none but the node itself, and many.
    The bounds are the FP64 and mixed walks' of the gravity parity tests."""
    from spheral_gb300.engine import Engine
    p = problems.evrard(n=n, seed=n, softening=softening)
    p.pos[n // 2] = p.pos[0] + 1e-5   # close to and, at 30, inside the limit
    orc = oracle_mod.Oracle(p)
    orc.initialize()
    orc.evaluate_derivatives()
    orc.gravity()
    for precision, tol in (("fp64", 1e-12), ("fp32", 2e-6)):
        eng = Engine.from_problem(p, precision=precision)
        eng.initialize()
        eng.evaluate_derivatives()
        bad = compare_fields(eng, orc, ["DvDtGravity", "potential"], tol)
        assert not bad, (precision, bad)
