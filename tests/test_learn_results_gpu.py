"""Results handed to the host are the same from the first call to the many
hundredth, whatever memory they come through, and for several objects used
from several threads at once."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_results_over_many_calls(ispm, cuda):
    import ispm.learn as learn
    jobs = []
    for seed in (1, 2, 3):
        rng = np.random.default_rng(seed)
        n = 130 + seed
        f = cuda.from_numpy(rng.uniform(0, 1, (n, learn.N_IN)).astype(np.float32)).cuda()
        t = cuda.from_numpy(rng.uniform(-3, 3, (n, 2)).astype(np.float32)).cuda()
        jobs.append((learn.MLP(learn.init_params(seed)), f.to(cuda.bfloat16), t,
                     cuda.cuda.Stream()))
    cuda.cuda.synchronize()
    bad = []

    def work(m, f, t, s):
        p0 = m.params()
        loss0, g0 = m.loss_grad(f, t, stream=s.cuda_stream)
        for k in range(700):
            loss, g = m.loss_grad(f, t, stream=s.cuda_stream)
            if loss != loss0 or not np.array_equal(g, g0) or not np.array_equal(m.params(), p0):
                bad.append(k)
                return

    threads = [threading.Thread(target=work, args=j) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
