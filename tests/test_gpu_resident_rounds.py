"""The chip-resident FP64 PCG (od_resident.cu) ends in the round it is told to, in all its warps: solves of one CTA (whose
sums meet nobody and so come soonest after a round's end) and of a cluster, stopped after every number of iterations up to
where they converge, over and over.  A warp that took a round's stop word for another's would leave early and the solve
would not end."""
import numpy as np
import pytest

from opendeformer_gb300 import api, meshgen
from tests.gpu_util import ctx

pytestmark = pytest.mark.gpu


# free block rows: 4, 12 and 36 (one CTA), 120 (four)
@pytest.mark.parametrize("dims", [(1, 1, 1), (3, 1, 1), (4, 2, 2), (10, 3, 2)])
def test_solves_stop_at_any_iteration(dims):
    g = meshgen.tet_grid(*dims, h=0.05, jitter=0.15, seed=4)
    cd = meshgen.constrained_dofs_for_nodes(g.face_nodes(0, 0))
    s = api.Scene(ctx(), g.X, g.tets, g.facets, cd, api.InvertibleNeoHookeanMaterial(1000.0, 98640.0, 0.4506, 0.1))
    A = s.evaluate()[0] / 240.0 ** 2 + s.mass()
    b = np.random.default_rng(2).normal(size=s.dofs)
    solver = lambda n: api.CGSolver(1e-8, n, api.JacobiPreconditioner())
    x, st = s.pcg(A, b, None, solver(1000))
    assert st.status == 0
    for n in range(st.iterations):
        _, part = s.pcg(A, b, None, solver(n))
        assert part.iterations == n and part.status == 3      # not converged
    for _ in range(300):
        again, more = s.pcg(A, b, None, solver(1000))
        assert more.iterations == st.iterations and np.array_equal(again, x)
