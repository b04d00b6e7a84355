"""Solves whose plan finds no device memory (an allocation that is refused, from the host) take the form that needs less,
the first call as the later ones.

Bounds: those of the forms' own tests (true residual within 1e-12 of the tolerance, iterations within the larger of 2 and 3%
of the oracle's)."""
import numpy as np
import pytest

from opendeformer_gb300 import api, meshgen
from oracle import restated
from tests.gpu_util import ctx

pytestmark = pytest.mark.gpu


def check(precond, tol, monkeypatch, env=(), dims=(20, 8, 8)):
    g = meshgen.tet_grid(*dims, h=0.05, jitter=0.15, seed=4)
    cd = meshgen.constrained_dofs_for_nodes(g.face_nodes(0, 0))
    o = restated.OracleScene(g.X, g.tets, g.facets, cd, "neohookean", 1000.0, 98640.0, 0.4506, 0.1)
    o.set_displacements(np.random.default_rng(1).normal(scale=2e-4, size=g.X.shape))
    A = o.assemble()[0] / 60.0 ** 2 + o.mass()
    b = np.random.default_rng(2).normal(size=o.dofs)
    for name, value in env:
        monkeypatch.setenv(name, value)
    s = api.Scene(ctx(), g.X, g.tets, g.facets, cd, api.InvertibleNeoHookeanMaterial(1000.0, 98640.0, 0.4506, 0.1))
    monkeypatch.setenv("OD_GB300_PLAN_BYTES", "16384")
    _, its = o.pcg(A, b, tol=tol, maxit=2000, precond=precond)
    for _ in range(3):
        x, st = s.pcg(A, b, None, api.CGSolver(tol, 2000, api.Preconditioner(precond)))
        assert st.status == 0 and abs(st.iterations - its) <= max(2, 0.03 * its)
        assert np.linalg.norm(b - o.spmdv(A, x)) <= (tol + 1e-12) * np.linalg.norm(b)


def test_ic0_without_its_structure(monkeypatch):
    check("ic0", 1e-8, monkeypatch)


def test_large_systems_without_digits(monkeypatch):
    check("block_jacobi", 1e-10, monkeypatch, [("OD_GB300_PCG_FORM", "wide")])


@pytest.mark.parametrize("smem", ["0", "1"])
def test_chip_resident_systems_without_their_digits(smem, monkeypatch):
    """The grid form (2,400 block rows), its matrix in L2 or in shared memory."""
    check("block_jacobi", 1e-8, monkeypatch, [("OD_GB300_PCG_SMEM", smem)], (24, 9, 9))
