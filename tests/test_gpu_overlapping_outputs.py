"""od_scene_evaluate into arrays that overlap: the forces are what stays where both go, bit for bit, as two copies in
that order leave it."""
import ctypes as C

import numpy as np
import pytest

from opendeformer_gb300 import api, meshgen
from tests.gpu_util import ctx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(1, 1, 1), (24, 9, 9)])
def test_forces_over_values(dims):
    g = meshgen.tet_grid(*dims, h=0.05, jitter=0.1, seed=2)
    cd = meshgen.constrained_dofs_for_nodes(g.face_nodes(0, 0))
    s = api.Scene(ctx(), g.X, g.tets, g.facets, cd, api.InvertibleNeoHookeanMaterial(1000.0, 98640.0, 0.4506, 0.1))
    s.set_displacements(np.random.default_rng(3).normal(scale=1e-3, size=(g.n_nodes, 3)))
    K, f = s.evaluate()
    p = lambda a: a.ctypes.data_as(C.POINTER(C.c_double))
    n, m = s.n_values, s.dofs
    for at in (0, 1, n // 2, n - m, n - 1, n):
        for _ in range(20):
            out = np.full(n + m, 7.0)
            want = out.copy()
            want[:n] = K
            want[at:at + m] = f
            assert api.load_library().od_scene_evaluate(s.h, p(out), p(out[at:])) == 0
            assert np.array_equal(out, want)
    # the forces first
    out = np.full(n + m, 7.0)
    want = out.copy()
    want[m // 2:m // 2 + n] = K
    want[:m] = f
    assert api.load_library().od_scene_evaluate(s.h, p(out[m // 2:]), p(out)) == 0
    assert np.array_equal(out, want)
