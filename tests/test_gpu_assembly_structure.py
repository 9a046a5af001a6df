"""Assembly on meshes whose node lists are irregular: skipped tets, nodes
without any tet, a tet that names a vertex twice, lists from one tet to the
kernels' limit of 32, node counts that are no multiple of a block.

The node pass takes each node's active tets from lists built once per mesh;
these are the shapes at which those lists and the shared-memory slots behind
them can go wrong.  K and f are compared with the oracle's assembly, FP64 to
1e-13 of the largest entry (sums of at most 32 terms, each a few dozen
roundings of 1.1e-16) and FP32 to 1e-5 (the same sums at 6e-8); the residual
entry point must return the same f bit for bit.  The exact-Jacobian products
gather over the same lists and are held to 1e-12 of their largest entry."""
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


def cube(N, skip=0.0, extra=0, seed=0):
    """unit cube with a fraction of its tets skipped and extra nodes no tet uses"""
    xyz, conn = O.unit_cube(N)
    rng = np.random.default_rng(seed)
    xyz = xyz + 0.05 / N * rng.standard_normal(xyz.size)
    vol = np.asarray(O.volumes(*O.unit_cube(N)), np.float64)
    vol[rng.random(vol.size) < skip] = 0.0
    xyz = np.concatenate([xyz, rng.standard_normal(3 * extra)])
    return xyz, conn, vol


def fan(m):
    """m tets around one edge: its two nodes have m incident tets each"""
    t = 2 * np.pi * np.arange(m) / m
    ring = np.stack([np.cos(t), np.sin(t), 0 * t], 1)
    xyz = np.concatenate([[[0, 0, -1.0], [0, 0, 1.0]], ring])
    conn = np.array([[0, 1, 2 + i, 2 + (i + 1) % m] for i in range(m)], np.uint32)
    return xyz.reshape(-1), conn.reshape(-1), np.ones(m)


def repeated():
    """a hex's tets and one more that names a vertex twice (skipped: it has
    no volume)"""
    xyz, conn, vol = cube(1)
    conn = np.concatenate([conn, np.array([0, 1, 1, 3], np.uint32)])
    return xyz, conn, np.concatenate([vol, [0.0]])


MESHES = {
    "one_hex": lambda: cube(1),
    "odd_skipped_isolated": lambda: cube(3, skip=0.3, extra=5, seed=1),
    "seven": lambda: cube(7, seed=2),
    "mostly_skipped": lambda: cube(4, skip=0.8, seed=3),
    "fan_3": lambda: fan(3),
    "fan_30": lambda: fan(30),
    "repeated_vertex": repeated,
}


@pytest.mark.parametrize("name", sorted(MESHES))
def test_assembly_on_irregular_lists(fm, name):
    xyz, conn, vol = MESHES[name]()
    ne, nu = conn.size // 4, 0.3
    rng = np.random.default_rng(7)
    E = np.exp(0.3 * rng.standard_normal(ne))
    mu = E / (2.0 * (1.0 + nu))
    lam = E * nu / ((1.0 + nu) * (1.0 - 2.0 * nu))
    u = 0.01 * rng.standard_normal(xyz.size)
    active = (vol >= 1e-30).astype(np.uint8)
    ctx = fm.Context(0)
    ctx.set_mesh(xyz, conn, vol)
    ctx.set_material(1.0, nu, E)
    rp, ci, sm = ctx.build_pattern(fm.FM_PATTERN_SOLVE, slot_map=True)
    Ko, fo = O.assemble(xyz, conn, mu, lam, nu, u, slot=sm, nnz=ci.size, active=active)
    K, f = ctx.assemble(cu(u), K=torch.full((ctx.nnz,), float("nan"), dtype=torch.float64,
                                            device="cuda"))
    assert np.abs(K.cpu().numpy() - Ko).max() <= 1e-13 * np.abs(Ko).max()
    assert np.abs(f.cpu().numpy() - fo).max() <= 1e-13 * np.abs(fo).max()
    K32, f32 = ctx.assemble(cu(u), prec=fm.FM_MIXED)
    assert np.abs(K32.cpu().numpy() - Ko).max() <= 1e-5 * np.abs(Ko).max()
    assert torch.equal(f32, f) and torch.equal(ctx.residual(cu(u)), f)
    # Dirichlet elimination against the oracle's
    mask = (rng.random(xyz.size) < 0.3).astype(np.uint8)
    ctx.set_bc(mask)
    Kb, _ = ctx.assemble(cu(u), apply_bc=True)
    Ke = Ko.copy()
    row = np.repeat(np.arange(xyz.size), np.diff(rp.astype(np.int64)))
    cut = (mask[row] | mask[ci.astype(np.int64)]) == 1
    Ke[cut] = (row[cut] == ci.astype(np.int64)[cut]).astype(np.float64)
    assert np.abs(Kb.cpu().numpy() - Ke).max() <= 1e-13 * np.abs(Ko).max()
    v = rng.standard_normal(xyz.size)
    for tr in (False, True):
        y = ctx.exact_apply(cu(u), cu(v), transpose=tr).cpu().numpy()
        yo = O.exact_apply(xyz, conn, mu, lam, u, v, transpose=tr, active=active)
        assert np.abs(y - yo).max() <= 1e-12 * np.abs(yo).max()
