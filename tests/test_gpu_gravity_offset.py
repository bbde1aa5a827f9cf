"""The octree walk far from the origin: the set of accepted cells is the one of
the reference's expressions wherever the system lies.

512 nodes of equal mass on multiples of 2^-19 in a box of 2^-8 at 2^24 + 3/4
from the origin (away from the FP32 numbers there, so that the low halves of
double-float coordinates are large): every sum m x is exact in FP64, so a centre of mass is one rounded
quotient whatever the order of summation.  (The reference adds nodes to a
centre one by one and rounds each time, so its own centres depend on the
insertion order here; the walk below takes the quotient.)  Accelerations and
potentials agree with a plain octree walk in numpy to the walks' own rounding,
1e-12 and 2e-6, unless a cell is accepted by one and opened by the other."""
import numpy as np
import pytest

from spheral_gb300 import problems

from _parity import rel_err

pytestmark = pytest.mark.gpu

LEVELS = 20


def _octree_walk(pos, mass, G, soft2, opening):
    """TreeGravity.cc:362-480, 819-932 with the far cells and leaves of every
    node summed in FP64."""
    n = len(mass)
    lo = pos.min(axis=0)
    length = (pos.max(axis=0) - lo).max()
    coord = np.minimum(((pos - lo) / length * 2.0 ** LEVELS).astype(np.int64), 2 ** LEVELS - 1)
    acc, phi = np.zeros((n, 3)), np.zeros(n)

    def add(nodes, m, d, r2):
        unit = np.where(r2[:, None] > 0.0, d / np.sqrt(np.where(r2 > 0.0, r2, 1.0))[:, None], [1.0, 0.0, 0.0])
        acc[nodes] += (m / (r2 + soft2))[..., None] * unit
        phi[nodes] -= m / np.sqrt(r2 + soft2)

    def visit(members, level, nodes):
        leaf = len(members) == 1 or level == LEVELS
        if level > 0:
            M = mass[members].sum()
            xcm = (mass[members, None] * pos[members]).sum(axis=0) / M if len(members) > 1 else pos[members[0]]
            size = length * 2.0 ** -level
            centre = lo + ((coord[members[0]] >> (LEVELS - level)) + 0.5) * size
            d = xcm - pos[nodes]
            r2 = (d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]) + d[:, 2] * d[:, 2]
            e = xcm - centre
            limit = (length * length / 4.0 ** level) / (opening * opening) + ((e[0] * e[0] + e[1] * e[1]) + e[2] * e[2])
            far = r2 > limit
            add(nodes[far], M, d[far], r2[far])
            nodes = nodes[~far]
        if len(nodes) == 0:
            return
        if leaf:
            for j in members:
                d = pos[j] - pos[nodes]
                r2 = (d * d).sum(axis=1)
                use = r2 / soft2 > 1.0e-10
                add(nodes[use], mass[j], d[use], r2[use])
            return
        child = (coord[members] >> (LEVELS - 1 - level)) & 1
        octant = child[:, 0] + 2 * child[:, 1] + 4 * child[:, 2]
        for o in range(8):
            part = members[octant == o]
            if len(part):
                visit(part, level + 1, nodes)

    visit(np.arange(n), 0, np.arange(n))
    return G * acc, G * phi


@pytest.mark.parametrize("seed", range(6))
@pytest.mark.parametrize("offset", [0.0, 2.0 ** 24 + 0.75], ids=["origin", "far"])
def test_walk_far_from_the_origin(native_lib, offset, seed):
    from spheral_gb300.engine import Engine
    n, side = 512, 2.0 ** -8
    p = problems.evrard(n=n, seed=seed, softening=side / 64)
    rng = np.random.default_rng(seed)
    p.pos[:] = offset + rng.integers(0, 2 ** 11, (n, 3)) * 2.0 ** -19
    p.mass[:] = 2.0 ** -9
    p.vel[:] = 0.0
    p.H[:, [0, 3, 5]] = 8.0 / (1.51 * side)
    acc, phi = _octree_walk(p.pos, p.mass, p.config["G"], p.config["softening"] ** 2, p.config["opening"])
    for precision, tol in (("fp64", 1e-12), ("fp32", 2e-6)):
        eng = Engine.from_problem(p, precision=precision)
        eng.initialize()
        eng.evaluate_derivatives()
        for name, want in (("DvDtGravity", acc), ("potential", phi)):
            err = rel_err(eng.field(name), want)
            assert err <= tol, (precision, name, err)
