"""The element kernels' fixed-point stiffness (od_elements.cu) at the edges of its launch and of its scales.

* against the oracle, with element counts around a CTA's 128: within 1e-12 of the largest value (corotational, plastic) and
  1e-10 (invertible: nearly equal singular values turn an ulp of the decomposition into ulp / gap);
* elements whose exponents leave the fixed-point window (a Young's modulus of 1e70) take the same sums in FP64, with the
  same decomposition: the scaled values agree to a few roundings of the largest, 1e-14;
* a corotational element with a NaN among its nodes has NaN values, the others none (the invertible decomposition takes
  such an element for fully degenerate, clamps its singular values and stays finite)."""
import numpy as np
import pytest

from opendeformer_gb300 import api, meshgen
from oracle import restated
from tests.gpu_util import ctx

pytestmark = pytest.mark.gpu

KINDS = ["neohookean", "stvk", "corotational", "corotational_plastic"]


def material(kind, youngs):
    if kind == "corotational_plastic":
        return api.CorotationalPlasticMaterial(1000.0, youngs, 0.45, 1e-3, 0.5, 0.05, 0.1)
    return api.Material(kind, 1000.0, youngs, 0.45, 0.1)


def mesh(dims, per_cube=6):
    g = meshgen.tet_grid(*dims, h=0.05, jitter=0.15, seed=9, tets_per_cube=per_cube)
    u = np.random.default_rng(2).normal(scale=0.01, size=(g.n_nodes, 3))
    return g, meshgen.constrained_dofs_for_nodes(g.face_nodes(0, 0)), u


# 5, 6, 125, 126, 130 and 132 elements
@pytest.mark.parametrize("dims,per_cube", [((1, 1, 1), 5), ((1, 1, 1), 6), ((5, 5, 1), 5), ((7, 3, 1), 6), ((13, 2, 1), 5),
                                           ((11, 2, 1), 6)])
@pytest.mark.parametrize("kind", KINDS)
def test_element_values_match_the_oracle(kind, dims, per_cube):
    g, cd, u = mesh(dims, per_cube)
    s = api.Scene(ctx(), g.X, g.tets, g.facets, cd, material(kind, 1e5))
    o = restated.OracleScene(g.X, g.tets, g.facets, cd, kind, 1000.0, 1e5, 0.45, 0.1, plastic=(1e-3, 0.5, 0.05))
    s.set_displacements(u)
    o.set_displacements(u)
    bound = 1e-12 if kind.startswith("corotational") else 1e-10
    for a, b in zip(s.element_values(), o.element_values()):
        assert np.abs(a - b).max() <= bound * np.abs(b).max()


@pytest.mark.parametrize("kind", KINDS)
def test_fixed_point_and_fp64_stiffness_agree(kind):
    g, cd, u = mesh((5, 3, 2))
    out = []
    for youngs in (1e5, 1e70):
        s = api.Scene(ctx(), g.X, g.tets, g.facets, cd, material(kind, youngs))
        s.set_displacements(u)
        out.append([v / youngs for v in s.element_values()])
    for a, b in zip(*out):
        assert np.isfinite(b).all() and np.abs(a - b).max() <= 1e-14 * np.abs(b).max()


@pytest.mark.parametrize("kind", KINDS[2:])
def test_a_nan_stays_in_its_elements(kind):
    g, cd, u = mesh((5, 3, 2))
    u = u.copy()
    u[g.n_nodes - 1, 1] = np.nan
    s = api.Scene(ctx(), g.X, g.tets, g.facets, cd, material(kind, 1e5))
    s.set_displacements(u)
    K, f = s.element_values()
    hit = (g.tets == g.n_nodes - 1).any(axis=1)
    assert np.isnan(K[hit]).any(axis=1).all() and np.isnan(f[hit]).any(axis=1).all()
    assert np.isfinite(K[~hit]).all() and np.isfinite(f[~hit]).all()
