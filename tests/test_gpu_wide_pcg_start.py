"""Starts that are not zero in the fixed-point PCG of large systems (od_wide.cu), at a size whose CTAs differ enough in
length that some still form r = b - A x while others have gone on: 237,600 DOFs, the default there.  A start's residual
that is not b - A x would show in the true residual alone, which the recurrence keeps within 1e-12 ||b|| of its own.

The backward Euler steps warm-start their solves from the last one's solution from the second step on."""
import numpy as np
import pytest

from opendeformer_gb300 import api, meshgen
from tests.gpu_util import ctx

pytestmark = pytest.mark.gpu

DIMS = (96, 32, 24)


def mesh():
    g = meshgen.tet_grid(*DIMS, jitter=0.1, seed=1, tets_per_cube=5)
    return g, meshgen.constrained_dofs_for_nodes(g.face_nodes(0, 0))


@pytest.mark.parametrize("precond", ["none", "block_jacobi"])
def test_a_start_vector(precond):
    g, cd = mesh()
    s = api.Scene(ctx(), g.X, g.tets, g.facets, cd, api.InvertibleNeoHookeanMaterial(1000.0, 98640.0, 0.4506, 0.1))
    A = s.evaluate()[0] / 120.0 ** 2 + s.mass()
    rng = np.random.default_rng(0)
    b = rng.normal(size=s.dofs)
    solver = api.CGSolver(1e-8, 2000, api.Preconditioner(precond))
    x0 = rng.normal(scale=np.abs(b).max() / np.abs(A).max(), size=s.dofs)
    for start in (x0, s.pcg(A, b, None, api.CGSolver(1e-4, 2000, api.Preconditioner(precond)))[0]):
        x, st = s.pcg(A, b, start, solver)
        assert st.status == 0 and st.rel_residual <= 1e-8 + 1e-12
        true = np.linalg.norm(b - s.spmdv(A, x)) / np.linalg.norm(b)
        assert abs(true - st.rel_residual) <= 1e-12


def test_backward_euler_steps():
    g, cd = mesh()
    s = api.Scene(ctx(), g.X, g.tets, g.facets, cd, api.CorotationalHyperelasticMaterial(1000.0, 98640.0, 0.4506, 0.1))
    s.set_loads(body=(0.0, 0.0, -9800.0))
    solver = api.CGSolver(1e-8, 2000, api.BlockJacobiPreconditioner())
    s.setup_integrator(api.NonlinearImplicitBackwardEuler(0.01, 0.001, 1 / 60, solver))
    for _ in range(3):
        st = s.step(1)
        assert st.status == 0 and 0.0 < st.max_rel_residual <= 1e-8 + 1e-12
