"""The elements as mixed-precision solves and batches evaluate them (OD_GB300_ELEMENT_DF=1), upright, inverted and flat,
against the oracle, and the switch itself: what it selects differs for flat elements, in the last places.

Bound: as for the FP64 path's flat elements, 16 2^-53 (s1 / s3)^2 of the largest value and at least 1e-12, twice that for
the reciprocal roots' own rounding."""
import numpy as np
import pytest

from opendeformer_gb300 import api
from oracle import restated
from tests.gpu_util import ctx, material

pytestmark = pytest.mark.gpu

FLAT = [0.8, 0.3, 0.112, 0.1105, 0.1095, 0.108, 0.03, 1e-2, 1e-3, 1.3e-4, -1e-3, -0.03, -0.1095, -0.3, -0.8]


@pytest.mark.parametrize("mat", ["neohookean", "stvk"])
def test_refined_elements_follow_the_oracle(mat, monkeypatch):
    rng = np.random.default_rng(5)
    X, tets, U = [], [], []
    for k, s in enumerate(FLAT):
        x = np.array([[0, 0, 0], [0.05, 0.004, 0.0], [0.003, 0.05, 0.002], [0.0, 0.005, 0.05]]) + 0.2 * k
        Q1, Q2 = (np.linalg.qr(rng.normal(size=(3, 3)))[0] for _ in range(2))
        Q1, Q2 = Q1 * np.sign(np.linalg.det(Q1)), Q2 * np.sign(np.linalg.det(Q2))
        U.append((x - x[0]) @ (Q1 @ np.diag([1.1, 0.9, s]) @ Q2 - np.eye(3)).T)
        X.append(x)
        tets.append(np.arange(4) + 4 * k)
    X, U, tets = np.vstack(X), np.vstack(U), np.array(tets, dtype=np.int32)
    facets = np.vstack([t[[[0, 2, 1], [0, 1, 3], [0, 3, 2], [1, 2, 3]]] for t in tets]).astype(np.int32)
    cd = np.zeros(0, dtype=np.int32)
    s = api.Scene(ctx(), X, tets, facets, cd, material(mat, 1000.0, 98640.0, 0.4506, 0.1))
    o = restated.OracleScene(X, tets, facets, cd, mat, 1000.0, 98640.0, 0.4506, 0.1)
    s.set_displacements(U)
    o.set_displacements(U)
    plain = s.evaluate()
    monkeypatch.setenv("OD_GB300_ELEMENT_DF", "1")
    K, f = s.evaluate()
    assert not np.array_equal(K, plain[0])
    Ko, fo = o.assemble()
    emap = o.pattern()[3]                       # no two elements share a node
    for k, flat in enumerate(FLAT):
        tol = 2 * max(1e-12, 16 * 2.0 ** -53 * (1.1 / flat) ** 2)
        at, dof = emap[k], np.arange(12 * k, 12 * k + 12)
        assert (at >= 0).all()
        assert np.abs(K[at] - Ko[at]).max() <= tol * np.abs(Ko[at]).max(), (flat, tol)
        assert np.abs(f[dof] - fo[dof]).max() <= tol * np.abs(fo[dof]).max(), (flat, tol)
