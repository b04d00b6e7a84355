"""Corotational elements whose polar decomposition's dominant root lies close to another: flat in two directions, or
inverted with two singular values nearly alike, upright and inverted, by the derivative of the characteristic quartic at
the root (of F over its norm).

Bound: the FP64 closed form, which the oracle takes, leaves the root 2e-14 off there (180 2^-53), the rotation takes that
over the distance to the next root, and R K R^T twice it: both sides together 8 x 180 2^-53 / gap, 2048 2^-53 / gap with the
roundings of F; 1e-12 like every element else."""
import numpy as np
import pytest

from opendeformer_gb300 import api
from oracle import restated
from tests.gpu_util import ctx

pytestmark = pytest.mark.gpu

DERIVATIVES = [0.03, 0.049, 0.051, 0.06, 0.08, 0.12, 0.18, 0.3, 0.45, 0.499, 0.501, 0.6, 2.0]


def roots(s):
    s = s / np.linalg.norm(s)
    return np.array([s.sum(), s[0] - s[1] - s[2], s[1] - s[0] - s[2], s[2] - s[0] - s[1]])


def stretches(kind, derivative):
    """Singular values (the last negative: inverted) with that derivative at the dominant root, by bisection."""
    make = {"needle": lambda g: np.array([1.0, 0.6 * g, 0.4 * g]), "inverted": lambda g: np.array([1.0, 0.5 + g, -0.5])}[kind]
    lo, hi = 0.0, 0.45
    for _ in range(60):
        mid = 0.5 * (lo + hi)
        r = roots(make(mid))
        lo, hi = (mid, hi) if np.prod(r[0] - r[1:]) < derivative else (lo, mid)
    return make(mid)


@pytest.mark.parametrize("kind", ["needle", "inverted"])
@pytest.mark.parametrize("derivative", DERIVATIVES)
def test_close_roots_follow_the_oracle(kind, derivative):
    rng = np.random.default_rng(8)
    s = stretches(kind, derivative)
    gap = roots(s)[0] - roots(s)[1:].max()
    X, tets, U = [], [], []
    for k in range(48):
        x = np.array([[0, 0, 0], [0.05, 0.004, 0.0], [0.003, 0.05, 0.002], [0.0, 0.005, 0.05]])
        Q1, Q2 = (np.linalg.qr(rng.normal(size=(3, 3)))[0] for _ in range(2))
        Q1, Q2 = Q1 * np.sign(np.linalg.det(Q1)), Q2 * np.sign(np.linalg.det(Q2))
        X.append(x)
        U.append(x @ (Q1 @ np.diag(s) @ Q2 - np.eye(3)).T)
        tets.append(np.arange(4) + 4 * k)
    X, U, tets = np.vstack(X), np.vstack(U), np.array(tets, dtype=np.int32)
    facets = np.vstack([t[[[0, 2, 1], [0, 1, 3], [0, 3, 2], [1, 2, 3]]] for t in tets]).astype(np.int32)
    cd = np.arange(3)
    mat = api.Material("corotational", 1000.0, 98640.0, 0.4506, 1e-9)   # polar, whatever the volume
    a = api.Scene(ctx(), X, tets, facets, cd, mat)
    o = restated.OracleScene(X, tets, facets, cd, "corotational", 1000.0, 98640.0, 0.4506, 1e-9)
    a.set_displacements(U)
    o.set_displacements(U)
    tol = max(1e-12, 2048 * 2.0 ** -53 / gap)
    for got, want in zip(a.element_values(), o.element_values()):
        assert np.abs(got - want).max() <= tol * np.abs(want).max()
