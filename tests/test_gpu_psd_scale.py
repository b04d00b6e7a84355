"""The projection of an element's energy Hessian does not depend on the unit of its stiffness: elements whose Hessian (in
the singular values) is all but singular, on either side, with Young's moduli from 98,640 down to 2^-68 of that, where
products of three entries run through FP32's subnormal numbers.

Bound: the same operations on numbers that differ by a power of two, but for roots that FP32 starts at one scale and FP64
at another (some 2^-53 of the largest value): 1e-12.  An indefinite Hessian that is not projected is 1e-7 off."""
import numpy as np
import pytest

from opendeformer_gb300 import api
from tests.gpu_util import ctx

pytestmark = pytest.mark.gpu

E, NU = 98640.0, 0.4506
LAM, MU = NU * E / ((1 + NU) * (1 - 2 * NU)), E / (2 * (1 + NU))


def hessian(s):
    """Neo-Hookean d2E / ds2 in the singular values."""
    I3, l = np.prod(s * s), 2 * np.log(np.prod(s))
    g2, h5 = (-0.5 * MU + 0.25 * LAM * l) / I3, (0.5 * MU + 0.25 * LAM * (1 - l)) / I3 ** 2
    q, d = I3 / s, I3 * g2 / np.outer(s, s)
    return 4 * d + 4 * h5 * np.outer(q, q) + np.diag(MU - 2 * np.diag(d))


def singular_stretches():
    """Stretches at which the Hessian's determinant changes its sign with a positive leading minor, and near them."""
    rng, out = np.random.default_rng(0), []
    while len(out) < 16 * 21:
        s = rng.uniform(0.5, 1.5, 3)
        at = lambda x: s * np.array([1, 1, x])
        det = lambda x: np.linalg.det(hessian(at(x)))
        lo, hi = 0.6, 1.7
        if det(lo) * det(hi) >= 0:
            continue
        for _ in range(60):
            mid = 0.5 * (lo + hi)
            lo, hi = (mid, hi) if det(mid) * det(lo) > 0 else (lo, mid)
        H = hessian(at(lo))
        if H[0, 0] > 0 and H[0, 0] * H[1, 1] - H[0, 1] ** 2 > 0.01 * H[0, 0] ** 2:
            out += [at(lo) * np.array([1, 1, 1 + d]) for d in np.linspace(-2e-6, 2e-6, 21)]
    return out


def test_projection_at_any_scale():
    x = np.array([[0, 0, 0], [0.05, 0.004, 0.0], [0.003, 0.05, 0.002], [0.0, 0.005, 0.05]])
    stretch = singular_stretches()
    X = np.vstack([x for _ in stretch])
    U = np.vstack([x @ (np.diag(s) - np.eye(3)).T for s in stretch])
    tets = np.arange(4 * len(stretch), dtype=np.int32).reshape(-1, 4)
    facets = np.vstack([t[[[0, 2, 1], [0, 1, 3], [0, 3, 2], [1, 2, 3]]] for t in tets]).astype(np.int32)
    values = {}
    for k in [0, *range(60, 69)]:
        s = api.Scene(ctx(), X, tets, facets, np.arange(3), api.InvertibleNeoHookeanMaterial(1000.0, E * 2.0 ** -k, NU, 0.1))
        s.set_displacements(U)
        values[k] = s.element_values()[0] * 2.0 ** k
        s.close()
    for k, v in values.items():
        assert np.abs(v - values[0]).max() <= 1e-12 * np.abs(values[0]).max(), k
