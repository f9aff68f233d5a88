"""Advection (gale_b200/csrc/gg_advect.cu; needs a B200) on both sides of the swarm size from
which the velocities are packed per node: the same points, alone and repeated past it, move
to the same bits, and those agree with the oracle."""
import numpy as np
import pytest

from gale_b200 import workloads
from gale_b200.stokes import Mesh, StokesProblem

pytestmark = pytest.mark.gpu

PACK = 1 << 20  # points × dim


@pytest.mark.parametrize("n,order", [((13, 7), 1), ((13, 7), 2), ((5, 9, 4), 1), ((5, 9, 4), 2)], ids=str)
def test_packed_and_component_velocities(oracle_mod, n, order):
    dim = len(n)
    rng = np.random.default_rng(order + dim)
    mesh = Mesh(dim, n)
    u = rng.standard_normal(int(np.prod(np.add(n, 1))) * dim)
    x = workloads.random_points(mesh, 40, rng)

    def advect(points):
        G = StokesProblem(mesh)
        G.set_points(points)
        G.locate()
        return G.advect(0.05, u, order=order)  # some predictor and corrector positions leave the mesh
    small = advect(x)
    assert not np.array_equal(small, x)
    for total in ((PACK - 1) // dim, -(-PACK // dim), PACK):
        reps = -(-total // len(x))
        big = advect(np.concatenate([x] * reps)[:total])
        assert np.array_equal(big, np.concatenate([small] * reps)[:total])
    O = oracle_mod.OracleProblem(mesh)
    O.set_points(x, np.zeros(len(x), dtype=np.int32))
    if order == 2:
        xo = O.advect(0.05, u)
        assert np.max(np.abs(small - xo)) <= 1e-12  # one step of O(1) velocities in double
