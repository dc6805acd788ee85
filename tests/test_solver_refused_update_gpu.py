"""A value update whose FP16 factor would need a scale outside FP32's range is
refused and leaves the factor (its elements and its scale) as it was; the next
update works."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def elements(cuda, S, which):
    """The device elements of G (2) or G^T (3), as bits."""
    v, _ = S.operator(which)

    class Array:
        __cuda_array_interface__ = {"shape": (int(v.n_elms),), "typestr": "<i2", "version": 2,
                                    "data": (v.elms, False)}

    return cuda.as_tensor(Array(), device="cuda").clone()


@pytest.mark.parametrize("dims,points", [((12, 13, 11), 27), ((40, 9, 10), 7)])
@pytest.mark.parametrize("scale", [2.0**-600, 2.0**600], ids=["tiny", "huge"])
def test_refused_update_keeps_the_factor(ispm, oracle, cuda, gen, dims, points, scale):
    A = gen._box_lognormal(dims, points, 1.0, 3, 1e-2)
    other = gen._box_lognormal(dims, points, 1.0, 4, 1e-2).elms  # (another factor, not a multiple)
    b = np.random.default_rng(1).uniform(-1, 1, A.n_rows)
    S = ispm.PCGSolver(A, inner=np.float32, tol=1e-10, prec="fsai_gpu", refresh=True)
    x0, st0 = S.solve_host(b)
    before = [elements(cuda, S, k) for k in (2, 3)]
    assert all(bool((e != 0).any()) for e in before)
    with pytest.raises(ispm.IspmError) as e:
        S.update_values(other * scale)
    assert e.value.status == ispm.ERR_INVALID
    for k, e0 in zip((2, 3), before):
        assert cuda.equal(elements(cuda, S, k), e0)
    S.update_values(A.elms)
    x, st = S.solve_host(b)
    assert st["iterations"] == st0["iterations"] and np.array_equal(x, x0)
