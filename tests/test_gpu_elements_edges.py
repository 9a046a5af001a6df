"""Batched elements at batch sizes around a warp and a block of tets, with a
degenerate tet among them, against the oracle's element (1e-13 of the tet's
largest entry: a few dozen roundings).  Outputs are written in full: buffers
come back without a trace of what they held."""
import ctypes as C

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


@pytest.mark.parametrize("n", [1, 31, 32, 33, 127, 128, 129, 1000])
@pytest.mark.parametrize("offset", [0, 1])
def test_batch_edges(fm, n, offset):
    """offset 1: K and f eight bytes off a 16-byte boundary"""
    rng = np.random.default_rng(n)
    ref = np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0], [0, 0, 1]], float)
    x = (ref + 0.1 * rng.standard_normal((n, 4, 3))).reshape(n, 12)
    x[n // 2] = np.tile(x[n // 2, :3], 4)  # no volume: zeros
    u = 0.05 * rng.standard_normal((n, 12))
    E = np.exp(rng.standard_normal(n))
    ctx = fm.Context(0)
    K = torch.full((144 * n + 1 + offset,), float("nan"), dtype=torch.float64, device="cuda")
    f = torch.full((12 * n + 1 + offset,), float("nan"), dtype=torch.float64, device="cuda")
    t = [torch.as_tensor(a, device="cuda") for a in (x, u, E)]
    st = fm.lib().fm_elements(ctx._h, n, *[C.c_void_p(a.data_ptr()) for a in t], 0.3,
                              C.c_void_p(K.data_ptr() + 8 * offset),
                              C.c_void_p(f.data_ptr() + 8 * offset))
    assert st == 0
    # nothing beyond the outputs is touched
    assert bool(torch.isnan(K[144 * n + offset:]).all()) and bool(torch.isnan(K[:offset]).all())
    assert bool(torch.isnan(f[12 * n + offset:]).all()) and bool(torch.isnan(f[:offset]).all())
    K = K[offset:offset + 144 * n].cpu().numpy().reshape(n, 144)
    f = f[offset:offset + 12 * n].cpu().numpy().reshape(n, 12)
    for e in range(n):
        if e == n // 2:
            assert not K[e].any() and not f[e].any()
            continue
        Ko, fo = O.element(x[e], u[e], E[e], 0.3)
        Ko, fo = np.asarray(Ko).reshape(-1), np.asarray(fo).reshape(-1)
        assert np.abs(K[e] - Ko).max() <= 1e-13 * np.abs(Ko).max()
        assert np.abs(f[e] - fo).max() <= 1e-13 * np.abs(Ko).max()
