"""The IC(0) PCG of two launches (od_ic_pcg.cu) at its edges, in both forms: a system of one task, tasks with one and two
rows, the cluster's largest systems and the first beyond them, rows of more blocks than a task loads at once (a node that
is coupled to every other), factorisations that need a shift.

Bounds: the stop test is on the recursive residual, which these some tens of iterations keep within 1e-12 ||b|| of the
true one (A x by the oracle); iteration counts within the larger of 2 and 3% of the oracle's IC(0) PCG; the shift, one of
a discrete row of values, equals that of the separate launches."""
import functools

import numpy as np
import pytest

from opendeformer_gb300 import api, meshgen
from oracle import restated
from tests.gpu_util import ctx

pytestmark = pytest.mark.gpu

E, NU = 98640.0, 0.4506


def fan(m, last):
    """A patch of m x m squares, two triangles each, and one node above it that every tetrahedron shares."""
    X = np.array([[0.05 * i, 0.05 * j, 0.0] for j in range(m + 1) for i in range(m + 1)])
    at = lambda i, j: j * (m + 1) + i
    tri = [t for j in range(m) for i in range(m)
           for t in ((at(i, j), at(i + 1, j), at(i, j + 1)), (at(i + 1, j), at(i + 1, j + 1), at(i, j + 1)))]
    top = np.array([[0.025 * m, 0.025 * m, 0.05 * m]])
    X = np.vstack([X, top]) if last else np.vstack([top, X])
    a = len(X) - 1 if last else 0
    s = 0 if last else 1
    tets = np.array([(p + s, q + s, r + s, a) for p, q, r in tri], dtype=np.int32)
    facets = np.array([(p + s, r + s, q + s) for p, q, r in tri], dtype=np.int32)
    return X, tets, facets, np.arange(3 * s, 3 * s + 3)


@functools.lru_cache(maxsize=None)
def system(name):
    if name.startswith("fan"):
        X, tets, facets, cd = fan(int(name[3]), name.endswith("last"))
    else:
        dims = tuple(int(v) for v in name.split("x"))
        g = meshgen.tet_grid(*dims, h=0.05, jitter=0.15, seed=4)
        X, tets, facets = g.X, g.tets, g.facets
        cd = meshgen.constrained_dofs_for_nodes(g.face_nodes(0, 0))
        if dims == (5, 4, 4):
            cd = cd[:-2]     # blocks that straddle nodes, a short last one
    o = restated.OracleScene(X, tets, facets, cd, "neohookean", 1000.0, E, NU, 0.1)
    o.set_displacements(np.random.default_rng(1).normal(scale=2e-4, size=X.shape))
    A = o.assemble()[0] / 60.0 ** 2 + o.mass()
    return (X, tets, facets, cd), o, A, np.random.default_rng(2).normal(size=o.dofs)


def scene(mesh):
    return api.Scene(ctx(), *mesh, api.InvertibleNeoHookeanMaterial(1000.0, E, NU, 0.1))


# free block rows: 4; 36; 126; 2592 (870 tasks) and 2916 (976); fans of 36 and 64 nodes
@pytest.mark.parametrize("form", [None, "cluster", "grid"])
@pytest.mark.parametrize("name", ["1x1x1", "4x2x2", "5x4x4", "36x8x7", "36x8x8", "fan5first", "fan5last", "fan7last"])
def test_ic0_pcg_at_its_edges(name, form, monkeypatch):
    if form:
        monkeypatch.setenv("OD_GB300_IC0_PCG", form)
    mesh, o, A, b = system(name)
    s = scene(mesh)
    x0 = np.random.default_rng(3).normal(scale=np.abs(b).max() / np.abs(A).max(), size=b.size)
    for tol in (1e-8, 1e-11):
        for start in (None, x0):
            x, st = s.pcg(A, b, start, api.CGSolver(tol, 2000, api.IC0Preconditioner()))
            assert st.status == 0 and st.ic_shift == 0.0
            true = np.linalg.norm(b - o.spmdv(A, x)) / np.linalg.norm(b)
            assert true <= tol + 1e-12
            assert abs(true - st.rel_residual) <= 1e-12
        _, its = o.pcg(A, b, tol=tol, maxit=2000, precond="ic0")
        _, st = s.pcg(A, b, None, api.CGSolver(tol, 2000, api.IC0Preconditioner()))
        assert abs(st.iterations - its) <= max(2, 0.03 * its)


@pytest.mark.parametrize("form", ["cluster", "grid"])
@pytest.mark.parametrize("name", ["4x2x2", "5x4x4"])
def test_ic0_pcg_shift_and_exits(name, form, monkeypatch):
    mesh, o, A, b = system(name)
    # M - t K, a positive diagonal but not definite: the factorisation breaks down
    K = o.assemble()[0]
    shifts = []
    for f in (1e-5, -4.8e-7):
        bad = o.mass() + f * K
        for env in ("separate", form):
            monkeypatch.delenv("OD_GB300_IC0_FACTOR", raising=False)
            monkeypatch.delenv("OD_GB300_IC0_PCG", raising=False)
            monkeypatch.setenv(*(("OD_GB300_IC0_FACTOR", "coop") if env == "separate" else ("OD_GB300_IC0_PCG", form)))
            s = scene(mesh)
            _, st = s.pcg(bad, b, None, api.CGSolver(1e-8, 2, api.IC0Preconditioner()))
            shifts.append(st.ic_shift)
    assert shifts[0] == shifts[1] and shifts[2] == shifts[3]
    assert shifts[2] > 0.0
    x, st = s.pcg(A, np.zeros_like(b), None, api.CGSolver(1e-8, 100, api.IC0Preconditioner()))
    assert st.status == 0 and st.iterations == 0 and not x.any()
    _, st = s.pcg(A, b, None, api.CGSolver(1e-8, 3, api.IC0Preconditioner()))
    assert st.iterations == 3 and st.status == 3          # not converged
    nan = b.copy()
    nan[-1] = np.nan
    with pytest.raises(api.ODError) as e:
        s.pcg(A, nan, None, api.CGSolver(1e-8, 100, api.IC0Preconditioner()))
    assert e.value.status == 4                            # NaN
    x, st = s.pcg(A, b, None, api.CGSolver(1e-8, 1000, api.IC0Preconditioner()))
    assert st.status == 0 and np.isfinite(x).all()        # and the scene goes on
