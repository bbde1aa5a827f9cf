"""Neighbour sets for tensor H with large axis ratios at an angle to the axes.

The search culls candidates by a lower bound of |H r|^2 per chunk of nodes; it
has to hold for every H.  On sheared smoothing tensors (ratios of 3 to 10, the
hminratio limit, turned by 10 to 40 degrees about one axis and about all three)
the sets equal the FP64 oracle's exactly in both precision modes: with periodic
images and with walls, with four warps per work item (the small boxes) and with
one (the box of 79,507 nodes)."""
import numpy as np
import pytest

from spheral_gb300 import problems

pytestmark = pytest.mark.gpu


def _rotation(angles):
    R = np.eye(3)
    for a, t in enumerate(angles):
        c, s = np.cos(t), np.sin(t)
        Q = np.eye(3)
        b, d = [k for k in range(3) if k != a]
        Q[b, b], Q[b, d], Q[d, b], Q[d, d] = c, -s, s, c
        R = Q @ R
    return R


def sheared_box(side, ratio, angles, boundaries, seed):
    """A jittered cubic lattice whose H has principal values in the proportion
    1 : sqrt(ratio) : ratio, turned by ``angles`` (radians about x, y, z) and by
    up to 0.03 more per node; about 45 neighbours."""
    p = problems.stretched_box(side, side, side, seed=seed, nPerh=1.1, tilt=0.03, boundaries=boundaries)
    H = np.zeros((p.n, 3, 3))
    for k, (a, b) in enumerate(((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2))):
        H[:, a, b] = H[:, b, a] = p.H[:, k]
    half = np.diag([ratio ** -0.25, 1.0, ratio ** 0.25])
    R = _rotation(angles)
    H = np.einsum("ai,nij,bj->nab", R @ half, H, R @ half)
    p.H = np.ascontiguousarray(np.stack([H[:, 0, 0], H[:, 0, 1], H[:, 0, 2], H[:, 1, 1], H[:, 1, 2], H[:, 2, 2]],
                                        axis=1))
    return p


def _sets_equal(native, oracle_mod, p, precision):
    from spheral_gb300.engine import Engine
    eng, orc = Engine.from_problem(p, precision=precision), oracle_mod.Oracle(p)
    eng.connectivity()
    orc.connectivity()
    i, j, _ = eng.pairs()
    a, b, _ = orc.pairs()
    keys = lambda x, y: np.unique(np.asarray(x, np.int64) * p.n + np.asarray(y, np.int64))
    want = np.union1d(keys(a, b), keys(b, a))
    got = keys(i, j)
    assert np.array_equal(got, want), (len(np.setdiff1d(want, got)), "lost of", len(want))


ANGLES = {"z10": (0, 0, 10), "z20": (0, 0, 20), "x30": (30, 0, 0), "y40": (0, 40, 0), "all": (25, -35, 15)}


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("boundaries", ["periodic", "reflecting"])
@pytest.mark.parametrize("ratio", [3.0, 5.0, 10.0])
@pytest.mark.parametrize("angles", list(ANGLES))
def test_sheared_sets(native_lib, oracle_mod, angles, ratio, boundaries, precision):
    # the periodic axes are at least three supports wide
    p = sheared_box(26 if ratio > 5.0 else 20, ratio, np.radians(ANGLES[angles]), boundaries, seed=int(ratio) + len(angles))
    _sets_equal(native_lib, oracle_mod, p, precision)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("angles,ratio,boundaries", [("z20", 3.0, "reflecting"), ("x30", 10.0, "periodic"),
                                                     ("all", 5.0, "reflecting")])
def test_sheared_sets_one_warp(native_lib, oracle_mod, angles, ratio, boundaries, precision):
    p = sheared_box(43, ratio, np.radians(ANGLES[angles]), boundaries, seed=9)
    _sets_equal(native_lib, oracle_mod, p, precision)
