"""Solves on a stream that does not wait for the legacy one, right after the
solver was made or its values were updated (the FP16 factor's scale changes
with them): what they read has landed."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(9, 8, 7), (30, 31, 29)])
def test_solves_right_after_updates(ispm, cuda, gen, dims):
    A = gen._box_lognormal(dims, 7, 1.0, 3, 1e-2)
    stream = cuda.cuda.Stream()  # (non-blocking)
    b = None
    want = None
    for made in range(4):
        S = ispm.PCGSolver(A, inner=np.float32, tol=1e-10, prec="fsai_gpu", refresh=True)
        if b is None:
            b = cuda.zeros(S.rows, dtype=cuda.float64, device="cuda")
            b[:A.n_rows] = cuda.from_numpy(np.random.default_rng(1).uniform(-1, 1, A.n_rows)).cuda()
            x = cuda.zeros_like(b)
            cuda.cuda.synchronize()
        for k in range(12):
            st = S.solve(b, x, stream=stream.cuda_stream)
            stream.synchronize()
            # A times a power of four: the same iterates, scaled
            got = (st["iterations"], (x * 4.0 ** (k % 3)).cpu().numpy())
            want = got if want is None else want
            assert st["converged"] and got[0] == want[0] and np.array_equal(got[1], want[1]), k
            S.update_values(A.elms * 4.0 ** ((k + 1) % 3))
