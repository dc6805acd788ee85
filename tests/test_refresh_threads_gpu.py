"""Refreshes of plans with different chunk sizes from several threads: each
launch finds the shared memory it asks for, whatever the others ask for
meanwhile."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def uniform_rows(ispm, n, width):
    """n rows of `width` neighbouring columns."""
    rp = (np.arange(n + 1) * width).astype(np.int32)
    first = np.minimum(np.arange(n), n - width)
    cols = (first[:, None] + np.arange(width)).astype(np.int32).ravel()
    return ispm.csr_matrix(n, n, rp, cols, np.random.default_rng(width).standard_normal(n * width))


def test_threads_with_different_chunks(ispm, cuda):
    jobs = []
    for width in (195, 203, 211, 220, 228, 237, 246, 255):  # 32-row slices of 49 to 65 KB
        A = uniform_rows(ispm, 2048, width)
        plan = ispm.spmv_plan(A, T=np.float64)
        jobs.append((plan, A, cuda.from_numpy(A.elms).cuda(), cuda.cuda.Stream()))
    assert all(p.host_matrix.slice_height * (A.elms.size // A.n_rows) * 8 > 48 * 1024
               for p, A, *_ in jobs)  # (what the test is about)
    for plan, A, v, s in jobs:
        ispm.plan_refresh_values(plan, A, v, stream=s.cuda_stream)
    cuda.cuda.synchronize()
    errors = []
    go = threading.Barrier(len(jobs))

    def work(plan, A, v, s):
        try:
            go.wait()
            for _ in range(2000):
                ispm.plan_refresh_values(plan, A, v, stream=s.cuda_stream)
        except ispm.IspmError as e:
            errors.append(str(e))

    threads = [threading.Thread(target=work, args=j) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    cuda.cuda.synchronize()
    assert not errors, errors[0]
