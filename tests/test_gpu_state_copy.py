"""What the device reads from and writes to the host's arrays itself, where it reaches them.

State in and out: every bit of it, at the sizes of one block row, of a few CTAs and of many, for all three arrays
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
    # doubles at odd addresses: by copies, as any alignment
    odd = [np.frombuffer(bytearray(8 * s.dofs + 4), dtype=np.float64, offset=4) for _ in range(3)]
    for to, x in zip(odd, (v, a, d)):
        to[:] = x
    s.set_state(*odd)
    for got, want in zip(s.state(), (bits[1], bits[2], bits[0])):
        assert np.array_equal(got.view(np.uint64), want)
    torch = pytest.importorskip("torch")
    pinned = [torch.from_numpy(x.copy()).pin_memory().numpy() for x in (a, d, v)]
    s.set_state(*pinned)
    for got, want in zip(s.state(), (bits[2], bits[0], bits[1])):
        assert np.array_equal(got.view(np.uint64), want)


@pytest.mark.parametrize("drop", [0, 1])
@pytest.mark.parametrize("dims", [(1, 1, 1), (5, 4, 3)])
def test_evaluate_and_product_into_host_memory(dims, drop):
    """Touched, untouched, pinned and misaligned arrays receive the same bits; with `drop` a constrained DOF less, so that the last
    block row is padded and y goes by copies.  The product against the oracle's, within its rounding of some 20 terms."""
    import ctypes as C

    from oracle import restated
    torch = pytest.importorskip("torch")
    g = meshgen.tet_grid(*dims, h=0.05, jitter=0.1, seed=2)
    cd = meshgen.constrained_dofs_for_nodes(g.face_nodes(0, 0))
    cd = cd[:len(cd) - drop]
    args = (g.X, g.tets, g.facets, cd)
    s = api.Scene(ctx(), *args, api.InvertibleNeoHookeanMaterial(1000.0, 98640.0, 0.4506, 0.1))
    o = restated.OracleScene(*args, "neohookean", 1000.0, 98640.0, 0.4506, 0.1)
    rng = np.random.default_rng(3)
    s.set_displacements(rng.normal(scale=1e-3, size=(g.n_nodes, 3)))
    K, f = s.evaluate()
    p = lambda a: a.ctypes.data_as(C.POINTER(C.c_double))
    L = api.load_library()
    odd = lambda n: np.frombuffer(bytearray(8 * n + 4), dtype=np.float64, offset=4)
    for make in (lambda n: np.full(n, 7.0), np.empty, odd, lambda n: torch.empty(n, dtype=torch.float64).pin_memory().numpy()):
        k2, f2 = make(s.n_values), make(s.dofs)
        assert L.od_scene_evaluate(s.h, p(k2), p(f2)) == 0
        assert np.array_equal(k2, K) and np.array_equal(f2, f)
        f3 = make(s.dofs)
        assert L.od_scene_evaluate(s.h, None, p(f3)) == 0 and np.array_equal(f3, f)
    x, y = rng.normal(size=s.dofs), rng.normal(size=s.dofs)
    want = y + o.spmdv(K, x)
    scale = np.abs(K).max() * np.abs(x).max() * 60 + np.abs(y).max()
    for y0 in (y.copy(), torch.from_numpy(y.copy()).pin_memory().numpy()):
        assert L.od_scene_spmdv(s.h, p(K), p(x), p(y0)) == 0
        assert np.abs(y0 - want).max() <= 64 * 2.0 ** -53 * scale
