"""PCG with the next iteration queued before the current one is judged: the
stop tests run on the device, so an iteration too many must leave no trace.
Iteration caps of 0, 1 and 2, a stop in the first iterations, the early exit
on entry, a start vector, and the |p.Ap| breakdown are the places where it
could.  Iteration counts must equal the oracle's and x agree to 1e-9 of its
largest entry (the caps stop at most 5 iterations in, where both sides
differ by roundings times the condition of a few steps).  Sizes around one
and several blocks of the reductions (256 DOFs) and around the node counts at
which the triangular solves change their cluster and warp counts."""
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


def system(fm, N):
    from flexmesh_b200 import configs

    P = configs.small_block(N)
    ctx = fm.Context(0)
    ctx.set_mesh(P.xyz, P.conn, P.elem_volume)
    ctx.set_material(1.0, P.nu)
    ctx.set_bc(P.mask, P.bc_value)
    rp, ci, _ = ctx.build_pattern(fm.FM_PATTERN_SOLVE)
    u = 0.001 * np.random.default_rng(N).standard_normal(P.xyz.size)
    K, _ = ctx.assemble(cu(u), apply_bc=True)
    ctx.assemble_into_context(cu(u), apply_bc=True)
    ctx.ilu0()
    b = np.random.default_rng(N + 1).standard_normal(P.xyz.size)
    b[P.mask == 1] = 0.0
    return ctx, rp, ci, K.cpu().numpy(), b


@pytest.mark.parametrize("N", [1, 3, 4, 9])
@pytest.mark.parametrize("cap,tol", [(0, 1e-10), (1, 1e-10), (2, 1e-10), (5, 1e-10),
                                     (50, 0.5), (50, 0.1)])
def test_caps_and_first_iterations(fm, N, cap, tol):
    ctx, rp, ci, val, b = system(fm, N)
    for x0 in (np.zeros_like(b), 0.3 * b):
        x, it, rr = ctx.pcg(cu(b), x=cu(x0.copy()), tol=tol, max_iter=cap)
        xo, ito, rro = O.pcg_ilu0(rp, ci, val, b, x0=x0, tol=tol, max_iter=cap)
        assert it == ito
        scale = max(np.abs(xo).max(), 1e-300)
        assert np.abs(x.cpu().numpy() - xo).max() <= 1e-9 * scale
    # a solve right after starts afresh
    x, it, _ = ctx.pcg(cu(b), tol=1e-11, max_iter=3000)
    r = b - O.spmv(rp, ci, val, x.cpu().numpy())
    assert np.abs(r).max() <= 1e-8 * np.abs(b).max()


def test_early_exit_on_entry(fm):
    ctx, rp, ci, val, b = system(fm, 4)
    x, it, _ = ctx.pcg(cu(b), tol=1e-12, max_iter=3000)
    y, it2, _ = ctx.pcg(cu(b), x=x.clone(), tol=1.0, max_iter=50)
    assert it2 == 0 and torch.equal(x, y)


def test_breakdown_leaves_x(fm):
    """A = 0: p.Ap = 0 in the first iteration; x is the start vector and the
    count the cap, as in the reference"""
    n = 300
    rp = np.arange(n + 1, dtype=np.uint32)
    ci = np.arange(n, dtype=np.uint32)
    val = np.zeros(n)
    b = np.random.default_rng(1).standard_normal(n)
    x0 = np.random.default_rng(2).standard_normal(n)
    ctx = fm.Context(0)
    x, it, _ = ctx.csr_pcg_ilu0(rp, ci, val, b, x0=x0, tol=1e-10, max_iter=7)
    xo, ito, _ = O.pcg_ilu0(rp, ci, val, b, x0=x0.copy(), tol=1e-10, max_iter=7)
    assert it == ito == 7
    assert np.array_equal(x, x0) and np.array_equal(xo, x0)
