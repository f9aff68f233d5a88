"""The batched CTA solver (gale_b200/csrc/gg_cta.cu): one launch solves every problem of a
batch, one CTA per problem (needs a B200).

- every problem reaches the Uzawa tolerance, and its velocity and pressure are as close to
  the oracle's converged solution as the FP64 oracle's own solve at the same tolerance
  (within 1.5× plus 1e-6), on uneven sizes;
- the element applies sum over parity classes and the reductions run in a fixed order, so
  solving the same batch twice gives the same bits;
- the batch reports one kernel launch per problem (the shared launch).
"""
from dataclasses import replace

import numpy as np
import pytest

from gale_b200 import workloads
from gale_b200.stokes import Mesh, StokesProblem, UzawaSolver

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


def test_cta_batch_against_oracle_and_reproducible(oracle_mod):
    ws = workloads.batch_sinkers(count=8, sizes=(16, 24, 32, 48))
    prm = UzawaSolver(tolerance=1e-6, precision="mixed", inner="mg")
    probs = [w.apply(StokesProblem(w.mesh)) for w in ws]
    first = StokesProblem.solve_batch(probs, prm, workers=4)
    second = StokesProblem.solve_batch(probs, prm, workers=4)
    for (u1, p1, s1), (u2, p2, s2) in zip(first, second):
        assert np.array_equal(u1, u2) and np.array_equal(p1, p2)
        assert s1["kernel_launches"] == 1
    for w, (u, p, st) in zip(ws, first):
        assert st["rel_residual"] <= 1e-6
        O = w.apply(oracle_mod.OracleProblem(w.mesh))
        O.assemble()
        ut, pt, _ = O.uzawa(UzawaSolver(tolerance=1e-11, innerRtolFactor=0.01, maxIterations=5000,
                                        innerMaxIterations=200000))
        uo, po, _ = O.uzawa(UzawaSolver(tolerance=1e-6))
        pc, ptc, poc = p - p.mean(), pt - pt.mean(), po - po.mean()
        assert rel(u, ut) <= 1.5 * rel(uo, ut) + 1e-6, (w.mesh.elements[0], rel(u, ut), rel(uo, ut))
        assert rel(pc, ptc) <= 1.5 * rel(poc, ptc) + 1e-6, (w.mesh.elements[0], rel(pc, ptc), rel(poc, ptc))


def test_cta_batch_of_an_odd_count():
    """Three problems in one launch (the statistics sit behind an odd number of 4-byte words
    unless the device block is laid out for it) give the bits they give in a batch of four."""
    ws = workloads.batch_sinkers(count=4, sizes=(16, 20), seed=11)

    def solve(part):
        return StokesProblem.solve_batch([w.apply(StokesProblem(w.mesh)) for w in part],
                                         UzawaSolver(tolerance=1e-5, precision="mixed", inner="mg"))
    three, four = solve(ws[:3]), solve(ws)
    for (ua, pa, sa), (ub, pb, sb) in zip(three, four):
        assert np.array_equal(ua, ub) and np.array_equal(pa, pb)
        assert sa["outer_iterations"] == sb["outer_iterations"] > 0


@pytest.mark.parametrize("nx,ny", [(16, 32), (22, 24), (64, 8), (34, 30), (40, 26)])
def test_cta_batch_of_ragged_2d_meshes(oracle_mod, nx, ny):
    """Element counts around the block size and twice it (512, 528, 1020 and 1040 elements on
    512 threads), uneven axes and odd coarse levels: as close to the converged solution as
    the FP64 oracle at the same tolerance."""
    mesh = Mesh(2, (nx, ny), (0.0, 0.0), (1.0, 1.0))
    x = workloads.random_points(mesh, 12, np.random.default_rng(17))
    inside = (x[:, 0] - 0.5) ** 2 + (x[:, 1] - 0.6) ** 2 < 0.04
    w = replace(workloads.sinker_2d(n=4), mesh=mesh, coords=x, material=inside.astype(np.int32))
    (u, p, _), = StokesProblem.solve_batch([w.apply(StokesProblem(mesh))],
                                           UzawaSolver(tolerance=1e-6, precision="mixed", inner="mg"))
    O = w.apply(oracle_mod.OracleProblem(mesh))
    O.assemble()
    ut, pt, _ = O.uzawa(UzawaSolver(tolerance=1e-11, innerRtolFactor=0.01, maxIterations=5000,
                                    innerMaxIterations=200000))
    uo, po, _ = O.uzawa(UzawaSolver(tolerance=1e-6))
    pc, ptc, poc = p - p.mean(), pt - pt.mean(), po - po.mean()
    assert rel(u, ut) <= 1.5 * rel(uo, ut) + 1e-6
    assert rel(pc, ptc) <= 1.5 * rel(poc, ptc) + 1e-6


@pytest.mark.parametrize("n", [(8, 8), (9, 7), (4, 3), (27, 19), (31, 33), (5, 4, 3), (9, 7, 5)],
                         ids=lambda n: "x".join(map(str, n)))
def test_cta_batch_of_meshes_that_do_not_coarsen(oracle_mod, n):
    """One multigrid level: an odd axis, or few enough dofs.  As close to the converged
    solution as the FP64 oracle at the same tolerance."""
    dim = len(n)
    mesh = Mesh(dim, n)
    w = workloads.sinker_2d(n=4) if dim == 2 else workloads.creep_3d(n=4)
    x = workloads.random_points(mesh, 12, np.random.default_rng(17))
    inside = np.sum((x - 0.55) ** 2, 1) < 0.06
    w = replace(w, mesh=mesh, coords=x, material=inside.astype(np.int32) if dim == 2 else np.zeros(len(x), np.int32),
                temperature=None if dim == 2 else np.random.default_rng(3).random(int(np.prod(np.add(n, 1)))))
    probs = [w.apply(StokesProblem(mesh)) for _ in range(2)]
    (u, p, st), (u2, p2, _) = StokesProblem.solve_batch(probs, UzawaSolver(tolerance=1e-6, precision="mixed", inner="mg"))
    assert st["rel_residual"] <= 1e-6 and np.array_equal(u, u2) and np.array_equal(p, p2)
    O = w.apply(oracle_mod.OracleProblem(mesh))
    O.assemble()
    ut, pt, _ = O.uzawa(UzawaSolver(tolerance=1e-11, innerRtolFactor=0.01, maxIterations=5000,
                                    innerMaxIterations=200000))
    uo, po, _ = O.uzawa(UzawaSolver(tolerance=1e-6))
    pc, ptc, poc = p - p.mean(), pt - pt.mean(), po - po.mean()
    assert rel(u, ut) <= 1.5 * rel(uo, ut) + 1e-6
    assert rel(pc, ptc) <= 1.5 * rel(poc, ptc) + 1e-6
