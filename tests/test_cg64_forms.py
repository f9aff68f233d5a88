"""The forms of the plain FP64 CG (gale_b200/csrc/gg_cg64.cu; needs a B200): the captured class
launches, the cooperative grid and the cluster give the same bits and the same counts, and so
do solves that share the GPU."""
import time

import numpy as np
import pytest

from gale_b200 import abi, workloads
from gale_b200.stokes import (BodyForce, MaterialViscosity, Mesh, RheologyMaterial, StokesProblem, UzawaSolver,
                              free_slip)

pytestmark = pytest.mark.gpu


def problem(n, seed):
    dim = len(n)
    rng = np.random.default_rng(seed)
    mesh = Mesh(dim, n)
    x = workloads.random_points(mesh, 9, rng)
    G = StokesProblem(mesh)
    G.set_velocity_bc(free_slip(dim))
    G.set_materials([RheologyMaterial([MaterialViscosity(1.0)], density=1.0),
                     RheologyMaterial([MaterialViscosity(30.0)], density=1.3)])
    G.set_body_force(BodyForce(gravity=1.0))
    G.set_points(x, (np.sum((x - 0.55) ** 2, 1) < 0.1).astype(np.int32))
    return G


# a strip of one cluster; a grid; more than 592 blocks of 256 vector entries, so that a CTA takes
# a second tile and a thread a second entry; the same in 3D
@pytest.mark.parametrize("n", [(40, 37), (100, 90), (290, 270), (12, 11, 9), (41, 38, 36)], ids=lambda n: "x".join(map(str, n)))
def test_forms_give_the_same_bits(n):
    G = problem(n, sum(n))
    G.locate()
    G.build_operator("fp64")
    prm = UzawaSolver(tolerance=1e-2)
    out = []
    for form in (0, 1, 2):
        assert G.lib.gg_select_cg64(G.h, form) == abi.GG_OK
        out.append(G.solve(prm))
    # the launches did run: three are counted per iteration, one per inner solve in the other forms
    its = out[0][2]["inner_iterations"]
    assert out[1][2]["kernel_launches"] >= 3 * its
    assert out[0][2]["kernel_launches"] < its and out[2][2]["kernel_launches"] < its
    for u, p, st in out[1:]:
        assert np.array_equal(u, out[0][0]) and np.array_equal(p, out[0][1])
        for k in ("outer_iterations", "inner_iterations", "rel_residual"):
            assert st[k] == out[0][2][k]
    assert G.lib.gg_select_cg64(G.h, 3) == abi.GG_ERR_INVALID


# shares of the SMs (6 × 9.7 k and 8 × 20 k dofs), and the launches beside others (8 × 117 k dofs)
@pytest.mark.parametrize("n,count", [((75, 63), 6), ((19, 17, 17), 8), ((34, 32, 32), 8)], ids=str)
def test_solves_that_share_the_gpu(n, count):
    prm = UzawaSolver(tolerance=1e-2)
    probs = [problem(n, k % 3) for k in range(count)]
    alone = []
    for G in probs[:3]:
        G.locate()
        G.build_operator("fp64")
        alone.append(G.solve(prm))
    for k, (u, p, st) in enumerate(StokesProblem.solve_batch(probs, prm, workers=count)):
        assert np.array_equal(u, alone[k % 3][0]) and np.array_equal(p, alone[k % 3][1])
        assert st["inner_iterations"] == alone[k % 3][2]["inner_iterations"]


def test_shared_solves_do_not_take_turns():
    """8 of 192² on 8 threads, each solve wide enough for the whole GPU: 5 times one alone on a
    B200, 8 times when they took turns."""
    prm = UzawaSolver(tolerance=1e-4)
    probs = [problem((192, 192), k) for k in range(8)]
    for G in probs:
        G.locate()
        G.build_operator("fp64")

    def best(f):
        t = []
        for _ in range(3):
            t0 = time.perf_counter()
            f()
            t.append(time.perf_counter() - t0)
        return min(t)
    one = np.mean([best(lambda: G.solve(prm)) for G in probs])
    for _ in range(4):  # a busy host delays single calls
        together = best(lambda: StokesProblem.solve_batch(probs, prm, workers=8))
        if together < 6.5 * one:
            break
    assert together < 6.5 * one
