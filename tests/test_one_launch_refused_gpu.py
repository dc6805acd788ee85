"""A one-launch solve whose cooperative launch the device refuses (the CTAs
cannot all be resident where a process has a part of the SMs) is solved by the
step kernels instead; any other launch error is the solve's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOO_LARGE, OUT_OF_RESOURCES, INVALID_VALUE = 720, 701, 1  # cudaError_t


@pytest.mark.parametrize("error", [TOO_LARGE, OUT_OF_RESOURCES])
@pytest.mark.parametrize("inner", [np.float32, np.float64])
def test_solver(ispm, cuda, gen, inner, error):
    for A in (gen._box_lognormal((17, 18, 15), 27, 1.0, 5, 1e-2), gen.unstructured(14, seed=4)):
        b = np.random.default_rng(1).uniform(-1, 1, A.n_rows)
        kw = dict(inner=inner, tol=1e-10, prec="fsai_gpu")
        ref = ispm.PCGSolver(A, **kw)
        ref.one_launch = False
        x0, st0 = ref.solve_host(b)
        S = ispm.PCGSolver(A, **kw)
        assert S.one_launch
        assert ispm.lib_handle().ispm_solver_refuse_launch(S._h, error) == 0
        for _ in range(2):
            x, st = S.solve_host(b)
            assert st["converged"] and not S.one_launch
            assert st["iterations"] == st0["iterations"] and np.array_equal(x, x0)


def test_other_launch_errors_fail(ispm, cuda, gen):
    A = gen.poisson7(12)
    b = np.ones(A.n_rows)
    S = ispm.PCGSolver(A, prec="fsai_gpu")
    x0, _ = S.solve_host(b)
    ispm.lib_handle().ispm_solver_refuse_launch(S._h, INVALID_VALUE)
    with pytest.raises(ispm.IspmError) as e:
        S.solve_host(b)
    assert e.value.status == ispm.ERR_CUDA and S.one_launch
    x, st = S.solve_host(b)
    assert st["converged"] and np.array_equal(x, x0)


@pytest.mark.parametrize("inner", [np.float32, np.float64])
def test_batch(ispm, cuda, gen, inner):
    systems, n_rhs, _ = gen.batch_systems(4, seed=5, lo=6, hi=16)
    _, bs = gen.batch_rhs(systems, n_rhs, seed=4)
    ref = ispm.BatchSolver(systems, n_rhs, inner=inner)
    ref.one_launch = False
    xs0, _, _ = ref.solve_host(bs)
    B = ispm.BatchSolver(systems, n_rhs, inner=inner)
    assert B.one_launch
    ispm.lib_handle().ispm_batch_refuse_launch(B._h, TOO_LARGE)
    xs, _, tot = B.solve_host(bs)
    assert tot["converged"] and not B.one_launch and B.launches > 20
    assert all(np.array_equal(p, q) for p, q in zip(xs, xs0))
