"""The network and the row features on every device of a process, whichever
was used first."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_every_device(ispm, cuda, gen):
    import ispm.learn as learn
    if cuda.cuda.device_count() < 2:
        pytest.skip("one device")
    A = gen._box_lognormal((12, 13, 14), 27, 1.0, 1, 1e-3)
    out = []
    for dev in (0, 1, 0):
        with cuda.cuda.device(dev):
            f = learn.row_features(A, (12, 13, 14))
            m = learn.MLP(learn.init_params(3))
            loss, g = m.loss_grad(f, cuda.ones((A.n_rows, 2), device=f.device))
            out.append((f.float().cpu(), m.forward(f).cpu(), loss, g))
    for f, y, loss, g in out[1:]:
        assert cuda.equal(f, out[0][0]) and cuda.equal(y, out[0][1])
        assert loss == out[0][2] and np.array_equal(g, out[0][3])
