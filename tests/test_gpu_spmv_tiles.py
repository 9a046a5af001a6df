"""The tiled SpMV at node counts around its tiles of 16 nodes, with nodes that
have no entries, and at the valences that change how many tiles are in flight
(up to the limit of 32 neighbours), against the oracle's product of the same
K: rows sum at most 96 products, so 1e-14 of the sum of their magnitudes.
The FP32 kernel is checked through mixed PCG on the cubes, clamped on their
bottom face: the FP64 residual of a solve to 1e-5 (preconditioned norm) must
fall below 1e-3."""
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


def fan(m, extra=0):
    """m tets around one edge (its nodes: m + 2 neighbours), extra bare nodes"""
    t = 2 * np.pi * np.arange(m) / m
    ring = np.stack([np.cos(t), np.sin(t), 0 * t], 1)
    xyz = np.concatenate([[[0, 0, -1.0], [0, 0, 1.0]], ring, np.zeros((extra, 3))])
    conn = np.array([[0, 1, 2 + i, 2 + (i + 1) % m] for i in range(m)], np.uint32)
    return xyz.reshape(-1), conn.reshape(-1)


MESHES = {
    "cube1": lambda: O.unit_cube(1),
    "cube2": lambda: O.unit_cube(2),
    "cube3_four_tiles": lambda: O.unit_cube(3),
    "cube11": lambda: O.unit_cube(11),
    "fan20": lambda: fan(20),
    "fan30": lambda: fan(30),
    "bare_tail": lambda: fan(5, extra=40),
}


@pytest.mark.parametrize("name", sorted(MESHES))
def test_spmv_tiles(fm, name):
    xyz, conn = MESHES[name]()
    rng = np.random.default_rng(3)
    ctx = fm.Context(0)
    ctx.set_mesh(xyz, conn)
    ctx.set_material(1.0, 0.3)
    cube = name.startswith("cube")
    mask = np.zeros(xyz.size, np.uint8)
    if cube:
        mask[np.repeat(xyz[2::3] < 1e-12, 3)] = 1
    else:
        mask[:9] = 1
    ctx.set_bc(mask)
    u = np.zeros(xyz.size)
    K, _ = ctx.assemble(cu(u), apply_bc=True)
    ctx.assemble_into_context(cu(u), apply_bc=True)
    rp, ci, _ = ctx.build_pattern(fm.FM_PATTERN_SOLVE)
    K = K.cpu().numpy()
    for _ in range(2):
        x = rng.standard_normal(xyz.size)
        y = ctx.spmv(cu(x)).cpu().numpy()
        yo, ya = O.spmv(rp, ci, K, x), O.spmv(rp, ci, np.abs(K), np.abs(x))
        assert (np.abs(y - yo) <= 1e-14 * np.maximum(ya, 1e-300)).all()
    if not cube:
        return
    ctx.assemble_into_context(cu(u), prec=fm.FM_MIXED, apply_bc=True)
    ctx.ilu0(fm.FM_MIXED)
    b = rng.standard_normal(xyz.size)
    b[mask == 1] = 0.0
    x, it, _ = ctx.pcg(cu(b), tol=1e-5, max_iter=500, prec=fm.FM_MIXED)
    r = b - O.spmv(rp, ci, K, x.cpu().numpy())
    assert it < 500 and np.linalg.norm(r) <= 1e-3 * np.linalg.norm(b)
