"""2D levels smoothed by patches of 16 × 16 nodes (gale_b200/csrc/gg_fused.cu; needs a B200)
against the graph-captured V-cycle, one kernel per step: partial patches, single rows of
patches, every smoothing degree (halos of 2 to 5 rings), and a fine level with more patches
than one phase takes."""
import os

import numpy as np
import pytest

from gale_b200 import workloads
from gale_b200.stokes import (BodyForce, MaterialViscosity, Mesh, RheologyMaterial, StokesProblem, UzawaSolver,
                              VelocityBC)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,degree", [((48, 32), 2), ((200, 8), 2), ((8, 200), 3), ((80, 24), 4), ((96, 96), 3),
                                      ((640, 320), 2)], ids=str)
def test_patches_match_graph_path(monkeypatch, n, degree):
    rng = np.random.default_rng(sum(n))
    mesh = Mesh(2, n, (0.0, 0.0), (n[0] / n[1], 1.0))
    x = workloads.random_points(mesh, 9, rng)
    mat = ((x[:, 0] - 0.5 * n[0] / n[1]) ** 2 + (x[:, 1] - 0.6) ** 2 < 0.04).astype(np.int32)
    G = StokesProblem(mesh)
    G.set_velocity_bc(VelocityBC(left={"vx": 0}, right={"vx": 0}, bottom={"vx": 0, "vy": 0}, top={"vx": 0.01, "vy": 0}))
    G.set_materials([RheologyMaterial([MaterialViscosity(1.0)], density=1.0),
                     RheologyMaterial([MaterialViscosity(50.0)], density=1.2)])
    G.set_body_force(BodyForce(gravity=1.0))
    G.set_points(x, mat)
    G.locate()
    G.build_operator("mixed")
    prm = UzawaSolver(precision="mixed", inner="mg", tolerance=1e-9, innerRtolFactor=0.01, smoothingDegree=degree,
                      maxIterations=5000)
    monkeypatch.setenv("GALE_B200_FUSED_FCG", "0")
    ug, pg, sg = G.solve(prm)
    monkeypatch.setenv("GALE_B200_FUSED_FCG", "1")
    uf, pf, sf = G.solve(prm)
    assert sf["uzawa_fused"] == 1 and sf["rel_residual"] <= 1e-9
    # the same preconditioner up to the order of FP32 sums: as test_fused holds the two paths
    assert np.linalg.norm(uf - ug) <= 1e-6 * np.linalg.norm(ug)
    pc = lambda q: q - q.mean()  # noqa: E731
    assert np.linalg.norm(pc(pf) - pc(pg)) <= 1e-6 * np.linalg.norm(pc(pg))
    assert abs(sf["outer_iterations"] - sg["outer_iterations"]) <= 2
    assert sf["inner_iterations"] <= 1.1 * sg["inner_iterations"] + 5
