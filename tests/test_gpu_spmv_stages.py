"""The tiled SpMV's pipeline: meshes on which every CTA takes more tiles than it
has stages (stages are reused, both parities of their barriers come round),
with a ragged last tile, for each number of stages (FP64: 4 up to 11
neighbours, 3 up to 20, 2 beyond; FP32: 4 up to 21, 3 beyond, where rows are
also longer than the 64 columns that lanes hold in registers).

FP64: the product against the oracle's with the same K; rows sum at most 96
products, so 1e-14 of the sum of their magnitudes.  FP32: a mixed PCG solve
to 1e-6.  Three DOFs in five are fixed, which leaves small, well conditioned
clusters of free DOFs (no eigenvalue below 0.01), so FP32 keeps the true residual within about 1e-5 of
b; every row of b - K x must be below 1e-3 of its largest entry, where a tile
taken from a stale or wrong stage leaves residuals of the order of b."""
import numpy as np
import pytest

import oracle as O

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SMS = 148


@pytest.fixture(scope="module")
def fm():
    import flexmesh_b200 as F

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return F


def cu(a):
    return torch.as_tensor(np.ascontiguousarray(a), device="cuda")


def fans(m, copies):
    """disjoint copies of m tets around one edge (its nodes: m + 2 neighbours)"""
    t = 2 * np.pi * np.arange(m) / m
    ring = np.stack([np.cos(t), np.sin(t), 0 * t], 1)
    xyz = np.concatenate([[[0, 0, -1.0], [0, 0, 1.0]], ring])
    conn = np.array([[0, 1, 2 + i, 2 + (i + 1) % m] for i in range(m)])
    n = len(xyz)
    xyz = np.tile(xyz, (copies, 1))
    conn = (conn[None] + n * np.arange(copies)[:, None, None]).reshape(-1, 4)
    return xyz.reshape(-1), conn.astype(np.uint32).reshape(-1)


# mesh, nodes per disjoint part, stages in FP64 and FP32
MESHES = {
    "fan8": (lambda: fans(8, 5701), 10, 4, 4),
    "cube40": (lambda: O.unit_cube(40), 41 ** 3, 3, 4),
    "fan29": (lambda: fans(29, 1240), 31, 2, 3),
}


def fixed_dofs(n_dofs, part, rng):
    """three DOFs in five, and three nodes of each part (no part can move
    rigidly: random DOFs alone leave 15 of the 5,701 small fans singular)"""
    mask = (rng.random(n_dofs) < 0.6).astype(np.uint8)
    mask.reshape(-1, 3 * part)[:, :9] = 1
    return mask


@pytest.mark.parametrize("name", sorted(MESHES))
def test_stages_are_reused(fm, name):
    make, part, s64, s32 = MESHES[name]
    xyz, conn = make()
    tiles = (xyz.size // 3 + 15) // 16
    assert tiles >= SMS * max(s64 * (s64 + 2), s32 * (s32 + 2)) and (xyz.size // 3) % 16
    rng = np.random.default_rng(3)
    ctx = fm.Context(0)
    ctx.set_mesh(xyz, conn)
    ctx.set_material(1.0, 0.3)
    mask = fixed_dofs(xyz.size, part, rng)
    ctx.set_bc(mask)
    u = cu(np.zeros(xyz.size))
    K, _ = ctx.assemble(u, apply_bc=True)
    ctx.assemble_into_context(u, apply_bc=True)
    rp, ci, _ = ctx.build_pattern(fm.FM_PATTERN_SOLVE)
    K = K.cpu().numpy()
    for _ in range(2):
        x = rng.standard_normal(xyz.size)
        y = ctx.spmv(cu(x)).cpu().numpy()
        yo, ya = O.spmv(rp, ci, K, x), O.spmv(rp, ci, np.abs(K), np.abs(x))
        assert (np.abs(y - yo) <= 1e-14 * np.maximum(ya, 1e-300)).all()
    ctx.assemble_into_context(u, prec=fm.FM_MIXED, apply_bc=True)
    ctx.ilu0(fm.FM_MIXED)
    b = rng.standard_normal(xyz.size)
    x, it, _ = ctx.pcg(cu(b), tol=1e-6, max_iter=500, prec=fm.FM_MIXED)
    r = b - O.spmv(rp, ci, K, x.cpu().numpy())
    assert it < 500 and np.abs(r).max() <= 1e-3 * np.abs(b).max()
