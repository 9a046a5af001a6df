"""Generic CSR PCG on matrices around the edges of the single-CTA solves:
up to 2, 4 and 8 entries per row and side (and 9, beyond them), one row, level
widths below, at and beyond the block, a vector at the shared-memory limit
and one past it, unsorted columns.  Diagonally dominant matrices (condition
below 10), so the iterates of both sides differ by roundings only: equal
counts, x to 1e-12 of its largest entry."""
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


def symmetric(n, pairs, seed, shuffle=False):
    """SPD matrix with the given off-diagonal pairs (i > j)"""
    rng = np.random.default_rng(seed)
    a = {}
    for i, j in pairs:
        if i != j:
            a[(i, j)] = a[(j, i)] = -0.5 - rng.random()
    rows = [[] for _ in range(n)]
    for (i, j), v in a.items():
        rows[i].append((j, v))
    rp, ci, val = [0], [], []
    for i in range(n):
        off = sum(-v for _, v in rows[i])
        r = sorted(rows[i] + [(i, 1.2 * off + 1.0)])
        if shuffle:
            r = [r[k] for k in rng.permutation(len(r))]
        ci += [c for c, _ in r]
        val += [v for _, v in r]
        rp.append(len(ci))
    return (np.array(rp, np.uint32), np.array(ci, np.uint32), np.array(val, np.float64),
            rng.standard_normal(n))


def band(n, k, step=1):
    return [(i, i - step * q) for i in range(n) for q in range(1, k + 1) if i >= step * q]


def star(n, m, seed):
    """every row from m on reads k < 4 of the first m rows: one wide level"""
    rng = np.random.default_rng(seed)
    return [(i, int(j)) for i in range(m, n) for j in rng.choice(m, 1)]


CASES = {
    "one_row": (1, [], False),
    "two_rows": (2, band(2, 1), False),
    "tridiagonal": (1000, band(1000, 1), False),
    "two_per_side": (777, band(777, 2, 31), False),
    "three_per_side": (500, band(500, 3, 17), False),
    "eight_per_side": (400, band(400, 8, 9), True),
    "nine_per_side": (300, band(300, 9, 5), False),
    "diagonal": (2050, [], False),
    "wide_shift": (5000, band(5000, 1, 1100), False),
    "at_the_limit": (27000, band(27000, 2, 7000), True),
    "past_the_limit": (28600, band(28600, 2, 7000), False),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_small_csr_pcg(fm, name):
    n, pairs, shuffle = CASES[name]
    rp, ci, val, b = symmetric(n, pairs, 5, shuffle)
    # the oracle's ILU wants ascending columns
    order = np.concatenate([rp[i] + np.argsort(ci[rp[i]:rp[i + 1]], kind="stable")
                            for i in range(n)]).astype(np.int64)
    xo, ito, _ = O.pcg_ilu0(rp, ci[order], val[order], b, tol=1e-10, max_iter=200)
    ctx = fm.Context(0)
    for k in range(2):  # the second call reuses the pattern's streams
        x, it, _ = ctx.csr_pcg_ilu0(rp, ci, val, b, tol=1e-10, max_iter=200)
        assert it == ito
        assert np.abs(x - xo).max() <= 1e-12 * np.abs(xo).max()
    # other values on the same pattern
    x, _, _ = ctx.csr_pcg_ilu0(rp, ci, 2.0 * val, b, tol=1e-10, max_iter=200)
    assert np.abs(2.0 * x - xo).max() <= 1e-9 * np.abs(xo).max()
