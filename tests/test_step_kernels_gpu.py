"""The two ways a small system is solved -- one cooperative launch, and chunks of
step kernels (ispm_solver_set_one_launch / ispm_batch_set_one_launch) -- each
made to take every way it can end; and the step kernels' own three forms
(graph, while node, eager), which must agree bit for bit.  Solutions are
judged by their true residual against the FP64 CSR oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

WAYS = pytest.mark.parametrize("one_launch", [True, False], ids=["one_launch", "steps"])
INNER = pytest.mark.parametrize("inner", [np.float32, np.float64], ids=["mixed", "fp64"])


@pytest.fixture(scope="module")
def system(gen, oracle):
    A = gen._box_lognormal((17, 18, 15), 27, 1.0, 5, 1e-2)
    b = oracle.csr_spmv_f64(A.row_ptr, A.cols, A.elms,
                            np.random.default_rng(1).uniform(-1, 1, A.n_rows))
    return A, b


def residual(oracle, A, b, x):
    r = b - oracle.csr_spmv_f64(A.row_ptr, A.cols, A.elms, x)
    return np.linalg.norm(r) / np.linalg.norm(b)


def solver(ispm, A, one_launch, **kw):
    S = ispm.PCGSolver(A, **kw)
    assert S.one_launch
    S.one_launch = one_launch
    assert S.one_launch == one_launch
    return S


@pytest.mark.parametrize("prec", ["fsai_gpu", "given"])  # given without a pair: none
@pytest.mark.parametrize("inner,variant", [(np.float32, "classic"), (np.float64, "classic"),
                                           (np.float64, "pipelined"),
                                           (np.float32, "pipelined")])
def test_graph_loop_and_eager_agree(ispm, oracle, cuda, system, inner, variant, prec):
    A, b = system
    tol = 1e-9 if variant == "classic" or inner == np.float64 else 1e-5
    out = []
    for use_graph in (True, False, 2):
        S = ispm.PCGSolver(A, inner=inner, tol=tol, prec=prec, variant=variant,
                           use_graph=use_graph, check_every=4)
        # (FP32 pipelined solves have no one-launch form)
        assert S.one_launch == (variant == "classic" or inner == np.float64)
        S.one_launch = False
        out.append(S.solve_host(b))
    for x, st in out:
        assert st["converged"] and residual(oracle, A, b, x) <= tol * 1.001, st
        assert np.array_equal(x, out[0][0]) and st["iterations"] == out[0][1]["iterations"]
        assert st["refinements"] == out[0][1]["refinements"]


@INNER
@pytest.mark.parametrize("prec", ["fsai_gpu", "given"])
def test_both_ways_solve_alike(ispm, oracle, cuda, system, inner, prec):
    A, b = system
    S = solver(ispm, A, True, inner=inner, tol=1e-10, prec=prec)
    its = []
    for on in (True, False, True):
        S.one_launch = on
        x, st = S.solve_host(b)
        assert st["converged"] and residual(oracle, A, b, x) <= 1e-10 * 1.001, (on, st)
        its.append(st["iterations"])
    assert its[0] == its[2] and abs(its[0] - its[1]) <= 0.1 * its[0] + 4


@WAYS
@INNER
@pytest.mark.parametrize("prec", ["fsai_gpu", "given"])
def test_iteration_cap(ispm, cuda, system, inner, prec, one_launch):
    A, b = system
    for use_graph in (True, 2):
        S = solver(ispm, A, one_launch, inner=inner, tol=1e-14, prec=prec, max_iters=5,
                   use_graph=use_graph)
        x, st = S.solve_host(b)
        assert not st["converged"] and st["status"] == ispm.ERR_NOT_CONVERGED
        assert 0 < st["iterations"] <= 5 and np.all(np.isfinite(x))


@WAYS
@INNER
def test_breakdown(ispm, cuda, inner, one_launch):
    n = 64
    d = np.where(np.arange(n) % 2 == 0, 2.0, -2.0)
    A = ispm.csr_matrix(n, n, np.arange(n + 1, dtype=np.int32), np.arange(n, dtype=np.int32), d)
    for use_graph in (True, 2):
        S = solver(ispm, A, one_launch, inner=inner, tol=1e-10, max_refinements=5,
                   use_graph=use_graph)
        x, st = S.solve_host(np.ones(n))
        assert st["status"] == ispm.ERR_BREAKDOWN and np.all(np.isfinite(x))


@WAYS
@INNER
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_non_finite_and_zero_right_hand_sides(ispm, oracle, cuda, system, inner, bad, one_launch):
    A, b = system
    S = solver(ispm, A, one_launch, inner=inner, tol=1e-10, prec="fsai_gpu")
    bb = b.copy()
    bb[123] = bad
    with pytest.raises(ispm.IspmError) as e:
        S.solve_host(bb)
    assert e.value.status == ispm.ERR_INVALID
    x, st = S.solve_host(np.zeros_like(b))
    assert st["converged"] and st["iterations"] == 0 and not np.any(x)
    x, st = S.solve_host(b)
    assert st["converged"] and residual(oracle, A, b, x) <= 1e-10 * 1.001


@WAYS
@INNER
@pytest.mark.parametrize("order", ["none", "rcm"])
def test_updated_values(ispm, oracle, cuda, gen, inner, order, one_launch):
    """The captured graph holds the FP16 factor's scale by value: the values
    change by 64, and with them the scale."""
    A1 = gen.unstructured(14, 0.05, 3, 0.1, 10.0, 1.01)
    w = np.random.default_rng(8).uniform(4.0, 16.0, A1.n_rows)
    rows = np.repeat(np.arange(A1.n_rows), np.diff(A1.row_ptr))
    A2 = ispm.csr_matrix(A1.n_rows, A1.n_rows, A1.row_ptr, A1.cols,
                         A1.elms * w[rows] * w[A1.cols])
    b = np.random.default_rng(9).uniform(-1, 1, A1.n_rows)
    kw = dict(inner=inner, tol=1e-10, prec="fsai_gpu", reorder=order)
    S = solver(ispm, A1, one_launch, refresh=True, **kw)
    S.solve_host(b)
    S.update_values(A2.elms)
    x, st = S.solve_host(b)
    assert st["converged"] and residual(oracle, A2, b, x) <= 1e-10 * 1.001
    x_new, st_new = solver(ispm, A2, one_launch, **kw).solve_host(b)
    assert st["iterations"] == st_new["iterations"]
    assert np.allclose(x, x_new, rtol=0, atol=1e-13 * np.abs(x_new).max())


@INNER
@pytest.mark.parametrize("dims,points", [((3, 4, 5), 7), ((8, 8, 8), 27), ((17, 19, 23), 27),
                                         ((33, 31, 37), 7), ((58, 57, 59), 7),
                                         ((69, 68, 67), 7), ((55, 56, 57), 27)])
def test_small_systems_take_one_launch(ispm, cuda, gen, dims, points, inner):
    A = gen._box_lognormal(dims, points, 1.0, sum(dims), 1.0)
    for prec in ("fsai_gpu", "given"):
        assert ispm.PCGSolver(A, inner=inner, prec=prec).one_launch
    U = gen.unstructured(21, seed=4)
    assert ispm.PCGSolver(U, inner=inner, prec="fsai_gpu").one_launch
    systems = [A] * 3 if A.n_rows < 20000 else [A]
    assert ispm.BatchSolver(systems, 1, inner=inner).one_launch


def test_one_launch_is_refused_where_it_cannot_be(ispm, cuda, gen):
    A = gen.poisson7(8)
    S = ispm.PCGSolver(A, inner=np.float32, variant="pipelined", prec="fsai_gpu")
    assert not S.one_launch
    with pytest.raises(ispm.IspmError) as e:
        S.one_launch = True
    assert e.value.status == ispm.ERR_INVALID
    S.one_launch = False


# ---- batches

def batch(ispm, systems, n_rhs, one_launch, **kw):
    B = ispm.BatchSolver(systems, n_rhs, **kw)
    assert B.one_launch
    B.one_launch = one_launch
    return B


def check_lanes(ispm, oracle, B, systems, n_rhs, bs, xs, lanes, tol):
    for lane in range(B.lanes):
        info = B.lane_info(lane)
        k, j = info["system"], info["rhs"]
        b = np.asarray(bs[k]).reshape(n_rhs[k], -1)[j]
        x = np.asarray(xs[k]).reshape(n_rhs[k], -1)[j]
        st = lanes[lane]
        if not np.all(np.isfinite(b)):
            assert st["status"] == ispm.ERR_INVALID and not st["converged"]
            assert st["iterations"] == 0
        elif not np.any(b):
            assert st["converged"] and st["iterations"] == 0 and not np.any(x)
        else:
            assert st["converged"] and residual(oracle, systems[k], b, x) <= tol * 1.001, st


@INNER
@pytest.mark.parametrize("prec", ["fsai_gpu", "none"])
def test_batch_graph_and_eager_agree(ispm, oracle, cuda, gen, inner, prec):
    systems, n_rhs, _ = gen.batch_systems(5, seed=5, lo=6, hi=16)
    _, bs = gen.batch_rhs(systems, n_rhs, seed=4)
    out = []
    for use_graph in (True, False):
        B = batch(ispm, systems, n_rhs, False, inner=inner, tol=1e-8, prec=prec,
                  use_graph=use_graph)
        xs, lanes, tot = B.solve_host(bs)
        assert tot["converged"] and B.launches > 20
        check_lanes(ispm, oracle, B, systems, n_rhs, bs, xs, lanes, 1e-8)
        out.append((xs, [l["iterations"] for l in lanes]))
    assert out[0][1] == out[1][1]
    for a, b in zip(out[0][0], out[1][0]):
        assert np.array_equal(a, b)


@WAYS
@INNER
@pytest.mark.parametrize("prec", ["fsai_gpu", "none"])
def test_batch_lanes_that_stop_early(ispm, oracle, cuda, gen, inner, prec, one_launch):
    """A zero, a NaN and an infinite right-hand side, a tiny system and a 1 x 1
    one beside larger ones."""
    one = ispm.csr_matrix(1, 1, np.array([0, 1], np.int32), np.array([0], np.int32),
                          np.array([4.0]))
    systems = [gen.poisson7(4), gen.lognormal_stencil(20, 27, 1.5, 5), one,
               gen.lognormal_stencil(9, 7, 1.0, 8)]
    n_rhs = [3, 2, 1, 2]
    rng = np.random.default_rng(0)
    bs = [rng.uniform(-1, 1, (r, A.n_rows)) for A, r in zip(systems, n_rhs)]
    bs[0][1] = 0.0
    bs[0][2, 7] = np.nan
    bs[3][1, 100] = np.inf
    B = batch(ispm, systems, n_rhs, one_launch, inner=inner, tol=1e-8, prec=prec)
    xs, lanes, tot = B.solve_host(bs)
    assert (B.launches == 1) == one_launch and not tot["converged"]
    check_lanes(ispm, oracle, B, systems, n_rhs, bs, xs, lanes, 1e-8)


@WAYS
@INNER
def test_batch_of_one_lane_and_its_cap(ispm, oracle, cuda, gen, inner, one_launch):
    A = gen.lognormal_stencil(12, 27, 1.0, 8)
    b = np.random.default_rng(1).uniform(-1, 1, A.n_rows)
    B = batch(ispm, [A], 1, one_launch, inner=inner, tol=1e-8)
    xs, lanes, tot = B.solve_host([b])
    assert tot["converged"] and B.lanes == 1 and (B.launches == 1) == one_launch
    check_lanes(ispm, oracle, B, [A], [1], [b], xs, lanes, 1e-8)
    B = batch(ispm, [A], 1, one_launch, inner=inner, tol=1e-14, max_iters=5)
    xs, lanes, tot = B.solve_host([b])
    assert lanes[0]["status"] == ispm.ERR_NOT_CONVERGED and 0 < lanes[0]["iterations"] <= 5
    assert np.all(np.isfinite(xs[0]))
