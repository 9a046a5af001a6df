"""A context whose mesh changes: the product refuses the K of an earlier,
smaller mesh (its tiles are copied whole, past that K's end), and takes the new
one's; the oracle's product of the same K is the reference, rows of at most 57
products, so 1e-14 of the sum of their magnitudes."""
import numpy as np
import pytest

import oracle as O

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

FM_ERR_ARG = 1


@pytest.fixture(scope="module")
def fm():
    import flexmesh_b200 as F

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return F


def cu(a):
    return torch.as_tensor(np.ascontiguousarray(a), device="cuda")


def product_matches(fm, ctx, xyz):
    n = xyz.size
    K, _ = ctx.assemble(cu(np.zeros(n)))
    ctx.assemble_into_context(cu(np.zeros(n)), apply_bc=False)
    rp, ci, _ = ctx.build_pattern(fm.FM_PATTERN_SOLVE)
    x = np.random.default_rng(n).standard_normal(n)
    y, K = ctx.spmv(cu(x)).cpu().numpy(), K.cpu().numpy()
    yo, ya = O.spmv(rp, ci, K, x), O.spmv(rp, ci, np.abs(K), np.abs(x))
    return (np.abs(y - yo) <= 1e-14 * np.maximum(ya, 1e-300)).all()


def test_product_needs_a_k_of_this_mesh(fm):
    ctx = fm.Context(0)
    for N in (2, 7):  # no K at all, then one that is too small
        xyz, conn = O.unit_cube(N)
        ctx.set_mesh(xyz, conn)
        ctx.set_material(1.0, 0.3)
        with pytest.raises(fm.FMError) as e:
            ctx.spmv(cu(np.zeros(xyz.size)))
        assert e.value.status == FM_ERR_ARG
        assert product_matches(fm, ctx, xyz)
    xyz, conn = O.unit_cube(3)  # a smaller mesh again: its K fits
    ctx.set_mesh(xyz, conn)
    ctx.set_material(1.0, 0.3)
    assert product_matches(fm, ctx, xyz)
