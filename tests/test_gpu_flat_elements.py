"""Invertible elements on both sides of the flatness at which their singular values are taken by the FP64 expressions
(smallest eigenvalue of F F^T 0.01 of the largest), Neo-Hookean and StVK, upright and inverted.

Bound: the smallest eigenvalue carries some roundings of the largest (a few 2^-53, doubled by F F^T's own), and scales a
row of V by its square root, so f and K follow the oracle's (the same expressions on the CPU) to 16 2^-53 (s1 / s3)^2, and
to 1e-12 like every element.  Above the threshold s1 / s3 of 0.1 the elements are clamped alike."""
import numpy as np
import pytest

from opendeformer_gb300 import api
from oracle import restated
from tests.gpu_util import ctx, material

pytestmark = pytest.mark.gpu

FLAT = [0.3, 0.112, 0.1105, 0.1095, 0.108, 0.03, 1e-2, 1e-3, 1.3e-4, -1e-3, -0.1095, -0.3]


@pytest.mark.parametrize("mat", ["neohookean", "stvk"])
def test_flat_elements_follow_the_oracle(mat):
    rng = np.random.default_rng(5)
    X, tets, U = [], [], []
    for k, s in enumerate(FLAT):
        x = np.array([[0, 0, 0], [0.05, 0.004, 0.0], [0.003, 0.05, 0.002], [0.0, 0.005, 0.05]]) + 0.2 * k
        Q1, Q2 = (np.linalg.qr(rng.normal(size=(3, 3)))[0] for _ in range(2))
        Q1, Q2 = Q1 * np.sign(np.linalg.det(Q1)), Q2 * np.sign(np.linalg.det(Q2))
        F = Q1 @ np.diag([1.1, 0.9, s]) @ Q2
        U.append((x - x[0]) @ (F - np.eye(3)).T)
        X.append(x)
        tets.append(np.arange(4) + 4 * k)
    X, U, tets = np.vstack(X), np.vstack(U), np.array(tets, dtype=np.int32)
    facets = np.vstack([t[[[0, 2, 1], [0, 1, 3], [0, 3, 2], [1, 2, 3]]] for t in tets]).astype(np.int32)
    cd = np.arange(3)
    s = api.Scene(ctx(), X, tets, facets, cd, material(mat, 1000.0, 98640.0, 0.4506, 0.1))
    o = restated.OracleScene(X, tets, facets, cd, mat, 1000.0, 98640.0, 0.4506, 0.1)
    s.set_displacements(U)
    o.set_displacements(U)
    K, f = s.element_values()
    Ko, fo = o.element_values()
    for k, flat in enumerate(FLAT):
        tol = max(1e-12, 16 * 2.0 ** -53 * (1.1 / flat) ** 2)
        assert np.abs(K[k] - Ko[k]).max() <= tol * np.abs(Ko[k]).max(), (flat, tol)
        assert np.abs(f[k] - fo[k]).max() <= tol * np.abs(fo[k]).max(), (flat, tol)
