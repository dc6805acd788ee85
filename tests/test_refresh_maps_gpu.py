"""New values into a plan's device matrix for every kind of slice: runs of the
CSR through shared memory, slices too wide for it (gathered slot by slot),
odd boxes, variable heights and blocked columns.  The product must then have
the bits of a plan made from the new values."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def matrices(gen):
    wide = gen.random_csr(1100, 900, 5, mean_len=55.0, max_len=64)  # slices over 8,192 entries
    return {"box7": gen._box_lognormal((7, 9, 11), 7, 1.0, 1, 1e-3),
            "box27": gen._box_lognormal((13, 12, 15), 27, 1.0, 2, 1e-3),
            "graph": gen.unstructured(11, seed=3),
            "ragged": gen.random_csr(3000, 3100, 4, mean_len=9.0),
            "banded": gen.random_csr(2000, 2000, 6, mean_len=7.0, band=40),
            "wide": wide, "short": gen.random_csr(40, 40, 7, mean_len=3.0)}


@pytest.mark.parametrize("name", ["box7", "box27", "graph", "ragged", "banded", "wide", "short"])
@pytest.mark.parametrize("E,V", [(np.float64, np.float64), (np.float32, np.float64),
                                 (np.float64, np.float32), (np.float32, np.float32)],
                         ids=["64from64", "32from64", "64from32", "32from32"])
def test_refreshed_product_has_the_same_bits(ispm, cuda, gen, name, E, V):
    A = matrices(gen)[name]
    rng = np.random.default_rng(8)
    new = rng.standard_normal(A.elms.size).astype(V)
    csr = lambda v: ispm.csr_matrix(A.row_ptr.size - 1, A.n_cols, A.row_ptr, A.cols, v)
    x = cuda.from_numpy(rng.uniform(-1, 1, A.n_cols)).cuda()
    ys = []
    for values, fresh in ((A.elms, False), (new, True)):
        p = ispm.spmv_plan(csr(np.ascontiguousarray(values.astype(E))), T=np.float64)
        if not fresh:
            for _ in range(2):  # the second call reuses the map
                ispm.plan_refresh_values(p, csr(np.ascontiguousarray(A.elms)),
                                         cuda.from_numpy(new).cuda())
        y = cuda.full((p.host_matrix.n_rows,), 7.0, dtype=cuda.float64, device="cuda")
        p.execute_spmv(x, y)
        ys.append(y.cpu().numpy())
    assert np.array_equal(ys[0], ys[1])
