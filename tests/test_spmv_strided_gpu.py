"""Diagonal blocks with one thread a row or fewer: the strided walk (two and four
rows a thread in the launch shape) has the bits of the walk with one row a thread
(H = 1) for FP64 vectors; for FP32 ones, whose H = 1 walk adds columns and
diagonals in another order, and with several threads a row it stays within the
forward error of a sum in another order.  Boundary slices, unaligned vectors,
rectangular matrices, more than 32 diagonals, explicit columns among the
diagonals, and sizes either side of each shape's one resident wave."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NEAR = (-1201, -33, -1, 0, 1, 33, 1201)
MANY = tuple(range(-20, 19)) + (64, 4000)


def matrix(ispm, n_rows, n_cols, offsets, seed, extra):
    rng = np.random.default_rng(seed)
    r = np.arange(n_rows, dtype=np.int64)[:, None]
    c = r + np.asarray(offsets, dtype=np.int64)[None, :]
    key = (r * n_cols + c)[(c >= 0) & (c < n_cols)]
    if extra:
        rows = np.arange(0, n_rows, 53, dtype=np.int64)
        key = np.concatenate([key, rows * n_cols + (rows * 7919) % n_cols])
    key = np.unique(key)
    row_ptr = np.zeros(n_rows + 1, dtype=np.int32)
    np.cumsum(np.bincount(key // n_cols, minlength=n_rows), out=row_ptr[1:])
    return ispm.csr_matrix(n_rows, n_cols, row_ptr, (key % n_cols).astype(np.int32),
                           rng.uniform(-1, 1, key.size))


CASES = [(500, 500, NEAR, True, 64), (3000, 2900, NEAR, True, 128), (9001, 9100, MANY, False, 256),
         (40000, 40000, MANY, True, 64), (90000, 90000, NEAR, False, 256),
         (140001, 140001, NEAR, False, 64), (330000, 330000, NEAR, True, 64),
         (470000, 470000, NEAR, True, 128), (740001, 740000, NEAR, False, 256),
         (1500000, 1500000, NEAR, True, 64), (1500001, 1499000, NEAR, True, 256)]


@pytest.mark.parametrize("T,E", [(np.float64, np.float64), (np.float64, np.float32),
                                 (np.float32, np.float32)], ids=["f64", "f64f32", "f32"])
@pytest.mark.parametrize("case", CASES, ids=lambda c: "%dx%d-%d-S%d" % (c[0], c[1], len(c[2]), c[4]))
def test_strided_rows_match_one_thread_a_row(ispm, cuda, case, T, E):
    n_rows, n_cols, offsets, extra, S = case
    A = matrix(ispm, n_rows, n_cols, offsets, 3, extra)
    B = ispm.csr_to_slell(ispm.csr_matrix(A.n_rows, A.n_cols, A.row_ptr, A.cols,
                                          A.elms.astype(E)), S, 1, 0, 1)
    dB = B.upload()
    td = cuda.float64 if T == np.float64 else cuda.float32
    rng = np.random.default_rng(9)
    xb = cuda.from_numpy(rng.uniform(-1, 1, n_cols + 1).astype(T)).cuda()
    bound = None
    for shift in (0, 1):
        x = xb[shift:shift + n_cols]

        def product(N, H, v):
            y = cuda.full((B.n_rows + 8,), float("nan"), dtype=td, device="cuda")
            ispm.launch_spmv_kernel(ispm.spmv_launch_params(N, S, H, 1, 1), dB, v, y)
            h = y.cpu().numpy()
            assert np.all(np.isnan(h[B.n_rows:]))
            return h[:B.n_rows]

        want = product(S, 1, x)
        assert np.all(np.isfinite(want))
        # k terms in two orders differ by at most 2 gamma_k sum |a x|
        if bound is None:
            k = int(np.diff(A.row_ptr).max()) + 1
            bound = 2 * k * (2.0 ** -53 if T == np.float64 else 2.0 ** -24) * 1.001
        ax = np.abs(A.elms.astype(E).astype(np.float64) * x.cpu().numpy()[A.cols])
        absrow = np.zeros(B.n_rows)
        absrow[:n_rows] = np.bincount(np.repeat(np.arange(n_rows), np.diff(A.row_ptr)), ax,
                                      minlength=n_rows)
        for N, H in ((S // 2, 2), (S // 4, 4), (S, 4), (1024, 4)):
            got = product(N, H, x)
            if T == np.float64 and N * H == S:
                assert np.array_equal(got, want), (shift, H)
            assert np.all(np.abs(got.astype(np.float64) - want) <= bound * absrow + 1e-300), (shift, N, H)
