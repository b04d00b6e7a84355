"""State in and out: every bit of it, at the sizes of one block row, of a few CTAs and of many, for all three arrays
(one launch where the device reads the host's page tables), two of them and one, into memory that was never touched and
memory that is pinned."""
import numpy as np
import pytest

from opendeformer_gb300 import api, meshgen
from tests.gpu_util import ctx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(1, 1, 1), (4, 2, 2), (20, 8, 8), (40, 20, 20)])
def test_state_round_trip(dims):
    g = meshgen.tet_grid(*dims, h=0.05)
    cd = meshgen.constrained_dofs_for_nodes(g.face_nodes(0, 0))
    s = api.Scene(ctx(), g.X, g.tets, g.facets, cd, api.CorotationalHyperelasticMaterial(1000.0, 1e5, 0.45, 0.1))
    rng = np.random.default_rng(7)
    bits = [rng.integers(0, 2 ** 64, size=s.dofs, dtype=np.uint64) for _ in range(3)]   # NaN, infinities, denormals too
    d, v, a = (b.view(np.float64) for b in bits)
    s.set_state(d, v, a)
    for got, want in zip(s.state(), bits):
        assert np.array_equal(got.view(np.uint64), want)
    s.set_state(v=d)
    s.set_state(v, None, d)
    for got, want in zip(s.state(), (bits[1], bits[0], bits[0])):
        assert np.array_equal(got.view(np.uint64), want)
    torch = pytest.importorskip("torch")
    pinned = [torch.from_numpy(x.copy()).pin_memory().numpy() for x in (a, d, v)]
    s.set_state(*pinned)
    for got, want in zip(s.state(), (bits[2], bits[0], bits[1])):
        assert np.array_equal(got.view(np.uint64), want)
