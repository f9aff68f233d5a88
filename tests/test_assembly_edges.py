"""The operator build (gale_b200/csrc/gg_assembly.cu; needs a B200) on meshes and swarms at
the edges of its work split: single elements, element counts that fill no warp, 1 to 70
points per element, constant and Voronoi weights, both precisions."""
import numpy as np
import pytest

from gale_b200 import workloads
from gale_b200.stokes import (BodyForce, FrankKamenetskii, MaterialViscosity, Mesh, RheologyMaterial, StokesProblem,
                              free_slip)

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


@pytest.mark.parametrize("n,most,dvc", [((1, 1), 1, False), ((3, 5), 70, False), ((33, 1), 9, False), ((3, 5), 40, True),
                                        ((1, 1, 1), 5, False), ((2, 3, 5), 70, False), ((5, 2, 3), 30, True)],
                         ids=str)
def test_build_against_oracle(oracle_mod, n, most, dvc):
    dim = len(n)
    rng = np.random.default_rng(most + dim)
    mesh = Mesh(dim, n)
    cells = np.stack(np.meshgrid(*[np.arange(k) for k in n], indexing="ij"), -1).reshape(-1, dim)
    x = np.concatenate([(c + rng.uniform(0.02, 0.98, (rng.integers(1, most + 1), dim))) / n for c in cells])
    mat = rng.integers(0, 2, len(x), dtype=np.int32)
    T = rng.random(int(np.prod([k + 1 for k in n])))
    mats = [RheologyMaterial([FrankKamenetskii(eta0=10.0, theta=2.0)], density=1.0, alpha=0.1),
            RheologyMaterial([MaterialViscosity(30.0)], density=1.3)]

    def load(prob, points=True):
        prob.set_velocity_bc(free_slip(dim))
        prob.set_materials(mats)
        prob.set_body_force(BodyForce(gravity=2.0, rayleighNumber=3.0))
        prob.set_temperature(T)
        if points:
            prob.set_points(x, mat)
        return prob
    G = load(StokesProblem(mesh))
    if dvc:
        G.set_weights("dvc", 6)
    cell = G.locate()
    O = load(oracle_mod.OracleProblem(mesh), points=not dvc)
    if dvc:
        O.set_integration_points(cell, *G.integration_points(), mat)
    O.assemble()
    G.build_operator("mixed")
    v = rng.standard_normal(G.nnode * dim)
    f, h = G.rhs()
    fo, ho = O.rhs()
    # sums of at most 8 · 70 terms in the same order: 1e-12 as the full-size parity tests
    assert rel(f, fo) <= 1e-12 and rel(G.diagonals()[0], O.diagonals()[0]) <= 1e-12
    assert rel(G.diagonals()[1], O.diagonals()[1]) <= 1e-12
    y = O.apply_K(v)
    assert rel(G.apply_K(v), y) <= 1e-12
    assert rel(G.apply_K(v, "mixed"), y) <= 1e-5


@pytest.mark.parametrize("T", [None, 0.0], ids=["no T", "T=0"])
@pytest.mark.parametrize("gravity,ra,alpha,density", [(1.0, np.inf, 0.0, 1.0), (1.0, np.nan, 0.0, 1.0),
                                                      (0.0, 0.0, np.inf, 1.0), (0.0, 0.0, 0.0, np.nan)], ids=str)
def test_nonfinite_force_terms_stay_nonfinite(T, gravity, ra, alpha, density):
    """A weight that is zero times a factor that is not finite is NaN, with and without a
    temperature: an invalid body force is not taken for a zero one."""
    mesh = Mesh(2, (3, 4))
    G = StokesProblem(mesh)
    G.set_velocity_bc(free_slip(2))
    G.set_materials([RheologyMaterial([MaterialViscosity(1.0)], density=density, alpha=alpha)])
    G.set_body_force(BodyForce(gravity=gravity, rayleighNumber=ra))
    if T is not None:
        G.set_temperature(np.full(G.nnode, T))
    G.set_points(workloads.random_points(mesh, 5, np.random.default_rng(0)))
    G.locate()
    G.build_operator("fp64")
    f = G.rhs()[0].reshape(G.nnode, 2)
    # the free vertical components of the inner rows of nodes
    inner = np.arange(G.nnode).reshape(5, 4)[1:-1].ravel()
    assert np.isnan(f[inner, 1]).all()
