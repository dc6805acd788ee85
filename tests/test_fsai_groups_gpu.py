"""GPU FSAI rows at the edges of the lane groups that build them (patterns of
up to 4, 8, 16 and 32 entries, row counts that leave part of a warp or a CTA
idle), against the CPU restatement of the construction."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def banded(n, K, seed, ispm, arrow=False):
    """SPD matrix whose longest lower pattern has K entries: each row couples to
    up to K - 1 earlier rows at random within a band (arrow: to row 0 too, whose
    own row then holds n entries), diagonal 1.05 times the row sum."""
    rng = np.random.default_rng(seed)
    M = np.zeros((n, n))
    for i in range(1, n):
        m = min(i, K - 1 if rng.random() < 0.7 else int(rng.integers(0, K)))
        lo = max(0, i - 3 * K)
        j = rng.choice(np.arange(lo, i), size=min(m, i - lo), replace=False)
        if arrow and j.size:
            j[0] = 0
        M[i, j] = -rng.uniform(0.1, 1.0, j.size)
    M = M + M.T
    M[np.arange(n), np.arange(n)] = 1.05 * np.abs(M).sum(1) + (M == 0).all(1)
    r, c = np.nonzero(M)
    rp = np.zeros(n + 1, np.int32)
    np.add.at(rp, r + 1, 1)
    return ispm.csr_matrix(n, n, np.cumsum(rp).astype(np.int32), c.astype(np.int32), M[r, c])


@pytest.mark.parametrize("n,K,arrow", [(1, 1, False), (31, 4, False), (130, 4, True),
                                       (33, 5, False), (200, 8, True), (17, 9, False),
                                       (300, 16, True), (65, 17, False), (257, 32, True)])
def test_rows_match_oracle(ispm, oracle, cuda, n, K, arrow):
    A = banded(n, K, 100 * n + K, ispm, arrow)
    if n > 100:  # one row whose local matrix is indefinite: a Jacobi row
        k = A.row_ptr[n - 1] + np.searchsorted(A.cols[A.row_ptr[n - 1]:A.row_ptr[n]], n - 1)
        A.elms[k] *= 1e-3
    st = {}
    G1, G2 = ispm.fsai_sym_gpu(A, np.float64, stats=st)
    rp, ci, v, jac = oracle.fsai_rows_f64(A.row_ptr, A.cols, A.elms, np.arange(n))
    assert np.array_equal(G1.row_ptr, rp) and np.array_equal(G1.cols, ci)
    assert np.diff(rp).max() <= K
    assert st["fallbacks"] == jac
    # both sides factor local matrices of condition below 2.05 / 0.05 times the
    # spread of the diagonal (under 40): K eps 1600 < 1e-11 for K <= 32
    scale = np.repeat(np.maximum.reduceat(np.abs(v), rp[:-1]), np.diff(rp))
    assert np.all(np.abs(G1.elms - v) <= 1e-11 * scale)
