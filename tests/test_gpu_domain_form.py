"""The mixed pair sweep has one form for large runs and another for small ones.
In a decomposed run every domain takes the first, whatever its own node count,
so that the two sides of a pair across a cut come from the same arithmetic.

A box just above the line and the same box without the nodes of a small ball
(just below it) have the same cells and the same lists away from the ball: the
derivatives there are bitwise the same when both are domains, and differ by
rounding when the smaller box is a run of its own."""
import numpy as np
import pytest

from spheral_gb300 import problems

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("limited", [False, True], ids=["mg", "limited"])
def test_form_of_a_domain_does_not_depend_on_its_size(native_lib, limited):
    from spheral_gb300.engine import Engine
    p = problems.random_box(n_side=54, seed=6, nPerh=1.25, boundaries="open")
    if limited:
        p.config.update(viscosity="limited_monaghan_gingold", Cl=2.0, Cq=2.0)
    p.config.update(gradh_correction=False)   # the grad-h sweep's own forms do not touch the pair
    h = 1.25 / 54
    p.H[:, [0, 3, 5]] = 1.0 / h               # the same cells with and without the ball
    r = np.linalg.norm(p.pos - 0.5, axis=1)
    keep = np.argsort(-r, kind="stable")[:149000]
    keep = np.sort(keep)
    far = r > np.sort(r)[p.n - 149000] + 5.0 * h     # whose neighbours' neighbours are all kept
    q = p.copy()
    for name in ("pos", "vel", "mass", "rho", "eps", "H", "nodelist"):
        setattr(q, name, np.ascontiguousarray(getattr(p, name)[keep]))
    assert q.n < 150000 <= p.n and far[keep].sum() > 1000

    def derivs(prob, domain):
        eng = Engine.from_problem(prob, precision="fp32")
        if domain:
            eng.set_domain(0, lambda point, dt: dt)
        eng.initialize()
        eng.evaluate_derivatives()
        return [eng.field(f).copy() for f in ("DvDt", "DepsDt", "DvDx")]

    large, small, alone = derivs(p, True), derivs(q, True), derivs(q, False)
    for a, b in zip(large, small):
        assert np.array_equal(a[far], b[far[keep]])
    assert not np.array_equal(large[0][far], alone[0][far[keep]])
