"""The chip-resident FP64 PCG (od_resident.cu) at the edges of its shapes: less than one group of block rows, the most
one CTA takes, clusters of 2, 4 and 16 CTAs (with CTAs that hold fewer groups than others), the grid, and the matrix in L2.

Bounds: the stop test is on the recursive residual, which a pipelined recurrence keeps within a few hundred roundings of
the true one over these some hundred iterations (and which below a tolerance of 1e-9 is verified), so ||b - A x|| <=
(tol + 1e-12) ||b|| with A x by the oracle; iteration counts as the other PCG paths' tests hold them (the larger of 2 and
3%)."""
import functools

import numpy as np
import pytest

from opendeformer_gb300 import api, meshgen
from oracle import restated
from tests.gpu_util import ctx

pytestmark = pytest.mark.gpu

# free block rows: 4; 36 and 40 (one CTA); 48 (two); 120 and 125 (four); 1620 (sixteen); 2400 (the grid)
MESHES = [(1, 1, 1), (4, 2, 2), (10, 1, 1), (4, 3, 2), (10, 3, 2), (5, 4, 4), (20, 8, 8), (24, 9, 9)]


@functools.lru_cache(maxsize=None)
def system(dims):
    g = meshgen.tet_grid(*dims, h=0.05, jitter=0.15, seed=4)
    cd = meshgen.constrained_dofs_for_nodes(g.face_nodes(0, 0))
    o = restated.OracleScene(g.X, g.tets, g.facets, cd, "neohookean", 1000.0, 98640.0, 0.4506, 0.1)
    o.set_displacements(np.random.default_rng(1).normal(scale=5e-4, size=(g.n_nodes, 3)))
    A = o.assemble()[0] / 240.0 ** 2 + o.mass()
    return g, cd, o, A, np.random.default_rng(2).normal(size=o.dofs)


def scene(g, cd):
    return api.Scene(ctx(), g.X, g.tets, g.facets, cd, api.InvertibleNeoHookeanMaterial(1000.0, 98640.0, 0.4506, 0.1))


@pytest.mark.parametrize("tol", [1e-9, 1e-10])
@pytest.mark.parametrize("smem", ["1", "0"])
@pytest.mark.parametrize("precond", ["none", "jacobi", "block_jacobi"])
@pytest.mark.parametrize("dims", MESHES)
def test_resident_pcg_at_its_edges(dims, precond, smem, tol, monkeypatch):
    monkeypatch.setenv("OD_GB300_PCG_SMEM", smem)
    g, cd, o, A, b = system(dims)
    s = scene(g, cd)
    x0 = np.random.default_rng(3).normal(scale=np.abs(b).max() / np.abs(A).max(), size=b.size)
    for start in (None, x0):
        x, st = s.pcg(A, b, start, api.CGSolver(tol, 5000, api.Preconditioner(precond)))
        assert st.status == 0
        true = np.linalg.norm(b - o.spmdv(A, x)) / np.linalg.norm(b)
        assert true <= tol + 1e-12
        assert abs(true - st.rel_residual) <= 1e-12
    _, its = o.pcg(A, b, tol=tol, maxit=5000, precond=precond)
    _, st = s.pcg(A, b, None, api.CGSolver(tol, 5000, api.Preconditioner(precond)))
    assert abs(st.iterations - its) <= max(2, 0.03 * its)


@pytest.mark.parametrize("dims", [(4, 2, 2), (20, 8, 8), (24, 9, 9)])
def test_resident_pcg_exits(dims):
    g, cd, _o, A, b = system(dims)
    s = scene(g, cd)
    x, st = s.pcg(A, np.zeros_like(b), None, api.CGSolver(1e-8, 100, api.BlockJacobiPreconditioner()))
    assert st.status == 0 and st.iterations == 0 and not x.any()
    _, st = s.pcg(A, b, None, api.CGSolver(1e-8, 3, api.BlockJacobiPreconditioner()))
    assert st.iterations == 3 and st.status == 3          # not converged
    bad = b.copy()
    bad[-1] = np.nan
    with pytest.raises(api.ODError) as e:
        s.pcg(A, bad, None, api.CGSolver(1e-8, 100, api.BlockJacobiPreconditioner()))
    assert e.value.status == 4                            # NaN
    x, st = s.pcg(A, b, None, api.CGSolver(1e-8, 1000, api.BlockJacobiPreconditioner()))
    assert st.status == 0 and np.isfinite(x).all()        # and the scene goes on
