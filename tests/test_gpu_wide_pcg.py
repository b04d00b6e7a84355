"""The fixed-point PCG of large systems (od_wide.cu) at its edges: the smallest systems it takes (one CTA), CTAs with
fewer groups than others, rows of very different lengths (five-tetrahedra cubes), a short last block, starts that are not
zero, scales at which no digits can be had, and a size at which the dispatch picks it.

Bounds: the stop test is on the recursive residual, which the recurrence form keeps within 1e-12 ||b|| of the true one
over these some tens of iterations, so ||b - A x|| <= (tol + 1e-12) ||b|| with A x by the oracle; iteration counts as the
other PCG paths' tests hold them (the larger of 2 and 3%)."""
import functools

import numpy as np
import pytest

from opendeformer_gb300 import api, meshgen
from oracle import restated
from tests.gpu_util import ctx

pytestmark = pytest.mark.gpu

# free block rows: 210 (one CTA); 361 (two, of six-tetrahedra cubes); 936 and 2,295 of five-tetrahedra cubes
MESHES = [(7, 5, 4, 6), (10, 5, 5, 6), (9, 7, 12, 5), (15, 8, 16, 5)]


@functools.lru_cache(maxsize=None)
def system(dims):
    g = meshgen.tet_grid(*dims[:3], h=0.05, jitter=0.15, seed=4, tets_per_cube=dims[3])
    cd = meshgen.constrained_dofs_for_nodes(g.face_nodes(0, 0))
    if dims == MESHES[1]:
        cd = cd[:-2]     # blocks that straddle nodes, a short last one
    o = restated.OracleScene(g.X, g.tets, g.facets, cd, "neohookean", 1000.0, 98640.0, 0.4506, 0.1)
    o.set_displacements(np.random.default_rng(1).normal(scale=5e-4, size=(g.n_nodes, 3)))
    A = o.assemble()[0] / 240.0 ** 2 + o.mass()
    return g, cd, o, A, np.random.default_rng(2).normal(size=o.dofs)


def scene(g, cd):
    return api.Scene(ctx(), g.X, g.tets, g.facets, cd, api.InvertibleNeoHookeanMaterial(1000.0, 98640.0, 0.4506, 0.1))


@pytest.mark.parametrize("tol", [1e-8, 1e-10])
@pytest.mark.parametrize("precond", ["none", "jacobi", "block_jacobi"])
@pytest.mark.parametrize("dims", MESHES)
def test_wide_pcg_at_its_edges(dims, precond, tol, monkeypatch):
    monkeypatch.setenv("OD_GB300_PCG_FORM", "wide")
    g, cd, o, A, b = system(dims)
    s = scene(g, cd)
    x0 = np.random.default_rng(3).normal(scale=np.abs(b).max() / np.abs(A).max(), size=b.size)
    solver = api.CGSolver(tol, 5000, api.Preconditioner(precond))
    for start in (None, x0):
        x, st = s.pcg(A, b, start, solver)
        assert st.status == 0
        true = np.linalg.norm(b - o.spmdv(A, x)) / np.linalg.norm(b)
        assert true <= tol + 1e-12
        assert abs(true - st.rel_residual) <= 1e-12
    _, its = o.pcg(A, b, tol=tol, maxit=5000, precond=precond)
    _, st = s.pcg(A, b, None, solver)
    assert abs(st.iterations - its) <= max(2, 0.03 * its)


@pytest.mark.parametrize("scale", [2.0 ** -700, 2.0 ** 500])
def test_wide_pcg_without_digits(scale, monkeypatch):
    """Matrix values far outside the digits' range: FP64 products, the same solution (the scales are powers of two)."""
    monkeypatch.setenv("OD_GB300_PCG_FORM", "wide")
    g, cd, o, A, b = system(MESHES[2])
    s = scene(g, cd)
    x, st = s.pcg(A * scale, b, None, api.CGSolver(1e-9, 2000, api.Preconditioner("none")))
    assert st.status == 0
    assert np.linalg.norm(b - o.spmdv(A, x * scale)) <= (1e-9 + 1e-12) * np.linalg.norm(b)


def test_wide_pcg_exits(monkeypatch):
    monkeypatch.setenv("OD_GB300_PCG_FORM", "wide")
    g, cd, _o, A, b = system(MESHES[2])
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


def test_wide_pcg_is_what_large_systems_take(monkeypatch):
    """237,600 DOFs, three groups a warp of the persistent kernel: the default is the wide form, bit for bit."""
    g = meshgen.tet_grid(96, 32, 24, jitter=0.1, seed=1, tets_per_cube=5)
    cd = meshgen.constrained_dofs_for_nodes(g.face_nodes(0, 0))
    out, A, b = {}, None, None
    for form in (None, "wide", "recur"):
        monkeypatch.delenv("OD_GB300_PCG_FORM", raising=False)
        if form:
            monkeypatch.setenv("OD_GB300_PCG_FORM", form)
        s = scene(g, cd)
        if A is None:
            A = s.evaluate()[0] / 120.0 ** 2 + s.mass()
            b = np.random.default_rng(0).normal(size=s.dofs)
        out[form] = s.pcg(A, b, None, api.CGSolver(1e-10, 1000, api.BlockJacobiPreconditioner()))
        s.close()
    assert all(st.status == 0 and st.rel_residual <= 1e-10 + 1e-12 for _, st in out.values())
    assert np.array_equal(out[None][0], out["wide"][0])
    assert abs(out["wide"][1].iterations - out["recur"][1].iterations) <= max(2, 0.03 * out["recur"][1].iterations)
