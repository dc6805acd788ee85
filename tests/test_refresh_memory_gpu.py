"""A value refresh that finds no device memory for its map says so, leaves no
CUDA error for the next launch, and works once there is memory."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def fill(torch):
    """Take the device memory in ever smaller blocks."""
    held, size = [], torch.cuda.mem_get_info()[0]
    while size >= 1 << 20:
        try:
            held.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
        except torch.cuda.OutOfMemoryError:
            size = size // 2 if size > 20 << 20 else (1 << 20 if size > 1 << 20 else 0)
    return held


def test_no_memory_for_the_map(ispm, cuda, gen):
    A = gen._box_lognormal((64, 64, 64), 27, 1.0, 1, 1e-3)  # a map of 14 MB
    plan = ispm.spmv_plan(A, T=np.float64)
    vals = cuda.from_numpy(2.0 * A.elms).cuda()
    x = cuda.ones(plan.host_matrix.n_cols, dtype=cuda.float64, device="cuda")
    y, y2 = (cuda.zeros(plan.host_matrix.n_rows, dtype=cuda.float64, device="cuda")
             for _ in range(2))
    plan.execute_spmv(x, y)
    cuda.cuda.synchronize()
    held = fill(cuda)
    try:
        with pytest.raises(ispm.IspmError) as e:
            ispm.plan_refresh_values(plan, A, vals)
        assert e.value.status == ispm.ERR_NOMEM
        plan.execute_spmv(x, y2)  # (the values are the old ones)
        cuda.cuda.synchronize()
    finally:
        del held
        cuda.cuda.empty_cache()
    assert cuda.equal(y, y2)
    ispm.plan_refresh_values(plan, A, vals)
    plan.execute_spmv(x, y2)
    assert cuda.equal(2.0 * y, y2)
