"""A one-launch solve whose bounded wait runs out: the kernel returns, the call
reports ISPM_ERR_TIMEOUT with stats that say so, and the object solves again
once the limit is back.  (A limit of no cycles: every CTA but the last to
arrive at a meeting gives up at its first look.)"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def stale(ispm):
    st = ispm.solve_stats()
    st.iterations, st.converged, st.status, st.true_relres = 99, 1, 0, 1e-30
    return st


def timed_out(ispm, st):
    return (st.status == ispm.ERR_TIMEOUT and not st.converged and st.iterations == 0
            and np.isnan(st.true_relres) and st.seconds > 0)


@pytest.mark.parametrize("inner", [np.float32, np.float64])
@pytest.mark.parametrize("mesh", ["box", "renumbered", "few"])
def test_solver(ispm, cuda, gen, inner, mesh):
    A = {"box": lambda: gen._box_lognormal((40, 41, 39), 27, 1.0, 3, 1e-2),
         "few": lambda: gen._box_lognormal((16, 17, 15), 7, 1.0, 3, 1e-2),
         "renumbered": lambda: gen.unstructured(20, seed=4)}[mesh]()
    S = ispm.PCGSolver(A, inner=inner, tol=1e-10, prec="fsai_gpu")
    assert S.one_launch
    b = cuda.zeros(S.rows, dtype=cuda.float64, device="cuda")
    b[:A.n_rows] = cuda.from_numpy(np.random.default_rng(1).uniform(-1, 1, A.n_rows)).cuda()
    x, x1 = cuda.zeros_like(b), cuda.full_like(b, 7.0)
    want = S.solve(b, x)
    L = ispm.lib_handle()
    limit = lambda c: L.ispm_solver_set_wait_limit(S._h, C.c_longlong(c))
    assert limit(0) == 0
    st = stale(ispm)
    assert L.ispm_solver_solve(S._h, b.data_ptr(), x1.data_ptr(), C.byref(st),
                               None) == ispm.ERR_TIMEOUT
    assert timed_out(ispm, st)
    cuda.cuda.synchronize()
    assert not bool((x1 == 7.0).any())  # (also in the caller's order)
    assert limit(-1) == 0
    again = S.solve(b, x1)
    assert again["iterations"] == want["iterations"] and cuda.equal(x, x1)


def test_batch(ispm, cuda, gen):
    systems = [gen._box_lognormal((24, 23, 22), 27, 1.0, 3, 1e-2), gen.poisson7(12)]
    n_rhs = [1, 2]
    _, bs = gen.batch_rhs(systems, n_rhs, seed=4)
    B = ispm.BatchSolver(systems, n_rhs, inner=np.float32, tol=1e-8)
    assert B.one_launch
    xs, lanes, _ = B.solve_host(bs)
    L = ispm.lib_handle()
    assert L.ispm_batch_set_wait_limit(B._h, C.c_longlong(0)) == 0
    b = cuda.ones(B.rows, dtype=cuda.float64, device="cuda")
    x = cuda.zeros_like(b)
    st = (ispm.solve_stats * B.lanes)(*[stale(ispm) for _ in range(B.lanes)])
    tot = stale(ispm)
    assert L.ispm_batch_solve(B._h, b.data_ptr(), x.data_ptr(), st, C.byref(tot),
                              None) == ispm.ERR_TIMEOUT
    assert timed_out(ispm, tot) and all(timed_out(ispm, s) for s in st)
    assert L.ispm_batch_set_wait_limit(B._h, C.c_longlong(-1)) == 0
    xs2, lanes2, tot2 = B.solve_host(bs)
    assert tot2["converged"]
    assert all(np.array_equal(p, q) for p, q in zip(xs, xs2))
