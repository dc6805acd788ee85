"""Solves that run as one cooperative launch: every shape of the walk (rows a
thread, threads a row), ragged sizes, explicit columns, no preconditioner, and
a batch with more lanes than CTAs.  Each solve is judged by its true residual
against the FP64 CSR oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def residual(oracle, A, b, x):
    r = b - oracle.csr_spmv_f64(A.row_ptr, A.cols, A.elms, x)
    return np.linalg.norm(r) / np.linalg.norm(b)


@pytest.mark.parametrize("inner", [np.float32, np.float64], ids=["mixed", "fp64"])
@pytest.mark.parametrize("dims,points", [((3, 4, 5), 7), ((8, 8, 8), 27), ((17, 19, 23), 27),
                                         ((33, 31, 37), 7), ((58, 57, 59), 7),
                                         ((69, 68, 67), 7), ((55, 56, 57), 27)])
def test_boxes(ispm, oracle, cuda, gen, dims, points, inner):
    A = gen._box_lognormal(dims, points, 1.0, sum(dims), 1.0)
    b = oracle.csr_spmv_f64(A.row_ptr, A.cols, A.elms,
                            np.random.default_rng(1).uniform(-1, 1, A.n_rows))
    for prec in ("fsai_gpu", "given"):  # given without a pair: none
        S = ispm.PCGSolver(A, inner=inner, tol=1e-10, prec=prec)
        x, st = S.solve_host(b)
        assert st["converged"] and residual(oracle, A, b, x) <= 1e-10 * 1.001, (prec, st)
        # the reported residual is the FP64 one, and a phase ends the history
        assert abs(st["true_relres"] - S.history()[-1]) == 0.0
        if prec == "given" and A.n_rows > 50000:
            break


@pytest.mark.parametrize("inner,variant", [(np.float32, "auto"), (np.float64, "auto"),
                                           (np.float64, "classic")])
def test_explicit_columns(ispm, oracle, cuda, gen, inner, variant):
    A = gen.unstructured(21, seed=4)
    b = oracle.csr_spmv_f64(A.row_ptr, A.cols, A.elms,
                            np.random.default_rng(2).uniform(-1, 1, A.n_rows))
    its = []
    for reorder in ("none", "auto"):
        S = ispm.PCGSolver(A, inner=inner, tol=1e-10, prec="fsai_gpu", reorder=reorder,
                           variant=variant)
        x, st = S.solve_host(b)
        assert st["converged"] and residual(oracle, A, b, x) <= 1e-10 * 1.001, st
        its.append(st["iterations"])
    assert abs(its[0] - its[1]) <= 0.2 * its[0] + 2


@pytest.mark.parametrize("count,inner", [(3, np.float64), (700, np.float32)])
def test_batches(ispm, oracle, cuda, gen, count, inner):
    """Three uneven systems (groups of several CTAs), and more lanes than the
    GPU holds CTAs (lanes queue in groups of one)."""
    rng = np.random.default_rng(count)
    kinds = [gen._box_lognormal(d, p, 1.0, 7, 0.5) for d, p in (((5, 6, 7), 7), ((4, 4, 9), 27),
                                                                ((24, 25, 26), 7))]
    systems = kinds if count == 3 else [kinds[k % 2] for k in range(count - 1)] + [kinds[2]]
    B = ispm.BatchSolver(systems, 1, inner=inner, tol=1e-9)
    bs = [oracle.csr_spmv_f64(A.row_ptr, A.cols, A.elms, rng.uniform(-1, 1, A.n_rows))
          for A in systems]
    bs[1] = np.zeros_like(bs[1])  # solved at once by x = 0
    xs, lanes, tot = B.solve_host(bs)
    assert tot["converged"] and not np.any(xs[1])
    for A, b, x in zip(systems, bs, xs):
        if np.any(b):
            assert residual(oracle, A, b, x) <= 1e-9 * 1.001


def test_large_batch_shares_launches(ispm, oracle, cuda, gen):
    """A batch past the L2 line keeps the shared launches: systems of several
    shapes in one launch a product, several right-hand sides."""
    systems = [gen._box_lognormal((64, 62, 60), 27, 1.0, 1, 1.0),
               gen._box_lognormal((96, 97, 98), 7, 1.0, 2, 1.0),
               gen._box_lognormal((9, 10, 11), 27, 1.0, 3, 1.0)]
    n_rhs = [1, 2, 3]
    B = ispm.BatchSolver(systems, n_rhs, inner=np.float32, tol=1e-9)
    rng = np.random.default_rng(3)
    bs = [np.stack([oracle.csr_spmv_f64(A.row_ptr, A.cols, A.elms, rng.uniform(-1, 1, A.n_rows))
                    for _ in range(r)]) for A, r in zip(systems, n_rhs)]
    xs, lanes, tot = B.solve_host(bs)
    assert tot["converged"] and B.launches > 20  # (one launch would be the persistent path)
    for A, b, x in zip(systems, bs, xs):
        for k in range(b.shape[0]):
            assert residual(oracle, A, b[k], x[k]) <= 1e-9 * 1.001
