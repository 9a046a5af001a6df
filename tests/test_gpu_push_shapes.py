"""The push solves on every branch of push_shape (fm_setup.hpp): one cluster
with 8 and with 10 / 12 warps per CTA, several clusters with 12 / 16 and 14 /
16, all of them; lattice cubes, one with its nodes renamed in blocks of 8, and
one numbered breadth first.  The per-node arithmetic does not depend on the
plan, so results must equal the grid-wide pipelined solves bit for bit."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from test_gpu_push import block, context, cu, trsv_kernels  # noqa: E402


@pytest.fixture(scope="module")
def fm():
    import flexmesh_b200 as F

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return F


def breadth_first(mesh):
    """the mesh with its nodes numbered by layers of neighbours of node 0"""
    P, xyz, conn, mask, val = mesh
    nn = xyz.size // 3
    c = conn.reshape(-1, 4).astype(np.int64)
    e = np.unique(np.repeat(c, 4, 1).ravel() * nn + np.tile(c, (1, 4)).ravel())
    ptr = np.concatenate([[0], np.cumsum(np.bincount(e // nn, minlength=nn))])
    nbr = e % nn
    perm = np.full(nn, -1, np.int64)
    perm[0], order = 0, [0]
    for n in order:
        for m in nbr[ptr[n]:ptr[n + 1]]:
            if perm[m] < 0:
                perm[m] = len(order)
                order.append(m)
    dof = (3 * perm[:, None] + np.arange(3)).reshape(-1)
    out = [np.empty_like(a) for a in (xyz, mask, val)]
    for o, a in zip(out, (xyz, mask, val)):
        o[dof] = a
    return P, out[0], perm[conn.astype(np.int64)].astype(np.uint32), out[1], out[2]


@pytest.mark.parametrize("N,seed,bfs", [(6, 0, False), (14, 0, False), (20, 0, False),
                                        (30, 0, False), (36, 0, False), (24, -5, False),
                                        (10, 0, True), (18, 0, True)])
def test_every_shape_gives_the_same_values(fm, monkeypatch, N, seed, bfs):
    mesh = block(N, seed)
    if bfs:
        mesh = breadth_first(mesh)
    n = mesh[1].size
    u = 0.005 / N * np.random.default_rng(N).standard_normal(n)
    u[mesh[3] == 1] = 0.0
    r = cu(np.random.default_rng(N + 1).standard_normal(n))
    res = []
    for push in (False, True):
        ctx = context(fm, monkeypatch, mesh, push)
        ctx.assemble_into_context(cu(u), apply_bc=True)
        ctx.ilu0()
        y, kern, calls = trsv_kernels(ctx, lambda: ctx.ilu0_apply(r))
        assert calls == 1 and kern == (3 if push else 4)
        x, it, _ = ctx.pcg(r, tol=1e-12, max_iter=40)
        ctx.assemble_into_context(cu(u), prec=fm.FM_MIXED, apply_bc=True)
        ctx.ilu0(fm.FM_MIXED)
        xm, itm, _ = ctx.pcg(r, tol=1e-7, max_iter=40, prec=fm.FM_MIXED)
        assert ctx.flags() & fm.FLAG_TIMEOUT == 0
        res.append((y, x, xm, it, itm))
    for a, b in zip(*res):
        assert torch.equal(a, b) if torch.is_tensor(a) else a == b
