"""The factor's device elements, written once into a solver without refresh and
through maps into one with it: the same bits, in every element type and slice
shape."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def elements(cuda, S, which):
    v, _ = S.operator(which)
    t = {0: "<f4", 1: "<f8"}.get(v.elm_dtype, "<i2")

    class Array:
        __cuda_array_interface__ = {"shape": (int(v.n_elms),), "typestr": t, "version": 2,
                                    "data": (v.elms, False)}

    return cuda.as_tensor(Array(), device="cuda").cpu().numpy()


@pytest.mark.parametrize("kw", [dict(inner=np.float64), dict(inner=np.float32),
                                dict(inner=np.float32, factor_f16=False),
                                dict(inner=np.float32, factor_f16=False, factor_bf16=True)],
                         ids=["f64", "f16", "f32", "bf16"])
def test_once_and_mapped_agree(ispm, cuda, gen, kw):
    assert (ispm.F32, ispm.F64) == (0, 1)
    for A in (gen._box_lognormal((12, 13, 11), 27, 1.0, 3, 1e-2), gen.unstructured(14, seed=4),
              gen.poisson7(3)):
        once = ispm.PCGSolver(A, prec="fsai_gpu", **kw)
        mapped = ispm.PCGSolver(A, prec="fsai_gpu", refresh=True, **kw)
        for which in (2, 3):
            a, b = elements(cuda, once, which), elements(cuda, mapped, which)
            assert a.size and np.any(a) and np.array_equal(a, b)
