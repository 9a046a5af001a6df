"""Generic CSR PCG on both sides of the rules that choose its kernels: levels
wider than the single CTA's block with up to 4 and 8 entries per row and side,
shallow matrices that the warp-per-row solves take, and rows much longer than
the mean (4, 8 and 32 lanes per row of the product).  Diagonally dominant
matrices, so the iterates of both sides differ by roundings only (a row of 500
terms rounds 500 times: 500 x 2^-53 < 1e-13 of its terms): equal counts, x to
1e-12 of its largest entry."""
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


def matrix(n, pairs, seed=5):
    """SPD matrix with the given off-diagonal pairs (i > j, each once)"""
    rng = np.random.default_rng(seed)
    p = np.array(pairs, np.int64).reshape(-1, 2)
    v = -0.5 - rng.random(len(p))
    i = np.concatenate([p[:, 0], p[:, 1], np.arange(n)])
    j = np.concatenate([p[:, 1], p[:, 0], np.arange(n)])
    off = np.bincount(i[:2 * len(p)], -np.concatenate([v, v]), minlength=n)
    a = np.concatenate([v, v, 1.2 * off + 1.0])
    o = np.lexsort((j, i))
    rp = np.concatenate([[0], np.cumsum(np.bincount(i, minlength=n))])
    return rp.astype(np.uint32), j[o].astype(np.uint32), a[o], rng.standard_normal(n)


def band(n, k, step):
    return [(i, i - step * q) for q in range(1, k + 1) for i in range(step * q, n)]


def red_black(g):
    at = np.arange(g * g).reshape(g, g)
    par = np.add.outer(np.arange(g), np.arange(g)) % 2
    at[np.nonzero(par == 0)] = np.arange((g * g + 1) // 2)
    at[np.nonzero(par == 1)] = np.arange((g * g + 1) // 2, g * g)
    e = [(at[1:].ravel(), at[:-1].ravel()), (at[:, 1:].ravel(), at[:, :-1].ravel())]
    return [(max(a, b), min(a, b)) for x, y in e for a, b in zip(x, y)]


def arrows(m, k):
    return [(q * m + m - 1, q * m + j) for q in range(k) for j in range(m - 1)]


CASES = {
    # one CTA, levels wider than its block (512 threads), up to 4 and 8 entries
    "wide_three_per_side": (6000, band(6000, 3, 1100)),
    "wide_four_per_side": (5200, band(5200, 4, 513)),
    "wide_six_per_side": (8000, band(8000, 6, 1100)),
    "wide_eight_per_side": (9300, band(9300, 8, 1000)),
    # the rule's two sides
    "diagonal_7000": (7000, []),
    "diagonal_27000": (27000, []),
    "red_black_60": (3600, red_black(60)),
    "red_black_120": (14400, red_black(120)),
    "two_levels": (26000, band(26000, 2, 14336)),
    # long rows: 32 lanes, and 8 where there are too many rows for 32
    "arrow_500": (500, arrows(500, 1)),
    "arrows_60": (480, arrows(60, 8)),
    "arrows_200": (50000, arrows(200, 250)),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_csr_routes(fm, name):
    n, pairs = CASES[name]
    rp, ci, val, b = matrix(n, pairs)
    ctx = fm.Context(0)
    for x0 in (np.zeros(n), 0.3 * b):  # the second call reuses the pattern's streams
        xo, ito, _ = O.pcg_ilu0(rp, ci, val, b, x0=x0.copy(), tol=1e-10, max_iter=200)
        x, it, _ = ctx.csr_pcg_ilu0(rp, ci, val, b, x0=x0, tol=1e-10, max_iter=200)
        assert it == ito
        assert np.abs(x - xo).max() <= 1e-12 * np.abs(xo).max()
