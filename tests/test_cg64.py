"""The one-launch FP64 Jacobi CG (gale_b200/csrc/gg_cg64.cu) at the sizes where its work
split changes (needs a B200): against the CPU oracle's Uzawa solve, which takes the same
steps (same outer count), and against itself (same bits)."""
import numpy as np
import pytest

from gale_b200 import workloads
from gale_b200.stokes import (BodyForce, MaterialViscosity, Mesh, RheologyMaterial, StokesProblem, UzawaSolver,
                              free_slip)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(2, 2), (1, 1), (3, 2), (33, 5), (100, 3), (5, 90), (31, 17), (64, 33), (64, 64), (65, 63), (75, 70), (2, 2, 2), (5, 3, 2), (33, 4, 3),
                               (12, 11, 9)],
                         ids=lambda n: "x".join(map(str, n)))
def test_cg64_against_oracle(oracle_mod, n):
    """Partial tiles, single rows, one vector block, strips of one to several row pairs in a
    cluster of 1 to 16 CTAs, and a grid of CTAs."""
    dim = len(n)
    rng = np.random.default_rng(sum(n))
    mesh = Mesh(dim, n)
    x = workloads.random_points(mesh, 9, rng)
    mat = (np.sum((x - 0.55) ** 2, 1) < 0.1).astype(np.int32)
    mats = [RheologyMaterial([MaterialViscosity(1.0)], density=1.0),
            RheologyMaterial([MaterialViscosity(30.0)], density=1.3)]

    def load(prob):
        prob.set_velocity_bc(free_slip(dim))
        prob.set_materials(mats)
        prob.set_body_force(BodyForce(gravity=1.0))
        prob.set_points(x, mat)
        return prob
    prm = UzawaSolver(tolerance=1e-8)
    G = load(StokesProblem(mesh))
    G.locate()
    G.build_operator("fp64")
    u, p, st = G.solve(prm)
    u2, p2, st2 = G.solve(prm)
    assert np.array_equal(u, u2) and np.array_equal(p, p2)
    assert st["inner_iterations"] == st2["inner_iterations"]
    O = load(oracle_mod.OracleProblem(mesh))
    O.assemble()
    uo, po, so = O.uzawa(prm)
    # the same steps on operators that agree to 1e-12: rounding, amplified by the Krylov
    # recurrences, stays an order below the solver's own tolerance
    assert np.linalg.norm(u - uo) <= 1e-7 * np.linalg.norm(uo)
    pc, poc = p - p.mean(), po - po.mean()
    assert np.linalg.norm(pc - poc) <= 1e-6 * np.linalg.norm(poc)
    assert abs(st["outer_iterations"] - so["outer_iterations"]) <= 1
