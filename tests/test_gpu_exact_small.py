"""Exact-Jacobian products on both sides of the node count at which they change
from one kernel per node to an element pass and a gather (12^3 has 2,197
nodes, 13^3 2,744), on a mesh with a tet that is skipped, a node that no tet
touches and per-element moduli.  Against the oracle's product: a node sums at
most 24 terms, each a few dozen FP64 operations on values of its own size, so
1e-12 of the largest entry; the same for the same mesh among copies of itself,
enough of them for the element pass."""
import numpy as np
import pytest

import oracle as O

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fm():
    import flexmesh_b200 as F

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return F


def cu(a):
    return torch.as_tensor(np.ascontiguousarray(a), device="cuda")


def mesh(N):
    xyz, conn = O.unit_cube(N)
    vol = O.volumes(xyz, conn)
    vol[len(vol) // 2] = 0.0  # stored as degenerate: skipped
    return np.concatenate([xyz, [2.0, 2.0, 2.0]]), conn, vol  # and a bare node


@pytest.mark.parametrize("N", [1, 3, 8, 12, 13])
def test_exact_apply_small_and_large(fm, N):
    xyz, conn, vol = mesh(N)
    rng = np.random.default_rng(N)
    ne, n = conn.size // 4, xyz.size
    E = np.exp(0.3 * rng.standard_normal(ne))
    mu, lam = E / 2.6, E * 0.3 / (1.3 * 0.4)
    u, v = 0.02 / N * rng.standard_normal(n), rng.standard_normal(n)
    one, two = fm.Context(0), fm.Context(0)
    one.set_mesh(xyz, conn, vol)
    one.set_material(1.0, 0.3, E)
    copies = 1 + 2400 // (n // 3)
    two.set_mesh(np.tile(xyz, copies), (conn.reshape(1, -1) + n // 3 * np.arange(
        copies, dtype=np.uint32)[:, None]).astype(np.uint32).reshape(-1), np.tile(vol, copies))
    two.set_material(1.0, 0.3, np.tile(E, copies))
    for t in (False, True):
        y = one.exact_apply(cu(u), cu(v), transpose=t)
        yo = O.exact_apply(xyz, conn, mu, lam, u, v, transpose=t,
                           active=(vol >= 1e-30).astype(np.uint8))
        assert np.abs(y.cpu().numpy() - yo).max() <= 1e-12 * np.abs(yo).max()
        y2 = two.exact_apply(cu(np.tile(u, copies)), cu(np.tile(v, copies)), transpose=t)
        for part in y2.view(copies, -1).cpu().numpy():
            assert np.abs(part - yo).max() <= 1e-12 * np.abs(yo).max()
