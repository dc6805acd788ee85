"""The network and feature kernels at the edges of their tiles: row counts
around a warp's and a CTA's rows, feature rows that are only 4-byte aligned,
matrix rows too long for the feature kernel's buffer."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lo():
    import learn_oracle
    return learn_oracle


@pytest.fixture(scope="module")
def learn(ispm, cuda):
    import ispm.learn as L
    return L


def _features(lo, M, offset):
    """BF16 rows on the GPU whose first value sits `offset` values into an allocation."""
    import torch
    X = lo.bf16(np.random.default_rng(M).normal(0, 1, (M, 32)).astype(np.float32))
    buf = torch.zeros(M * 32 + 8, dtype=torch.bfloat16, device="cuda")
    buf[offset:offset + M * 32] = torch.from_numpy(
        lo.bf16_bits(X).view(np.int16).copy()).cuda().view(torch.bfloat16).ravel()
    return X, buf[offset:offset + M * 32].view(M, 32)


@pytest.mark.parametrize("M", [15, 33, 127, 129, 148 * 2 * 128 + 1])
@pytest.mark.parametrize("weighted", [False, True])
def test_step_matches_oracle_and_any_alignment(lo, learn, M, weighted):
    import torch
    rng = np.random.default_rng(M + 1)
    p = rng.normal(0, 0.25, lo.N_PARAMS).astype(np.float32)
    T = rng.normal(0, 1, (M, 2)).astype(np.float32)
    Wt = rng.uniform(0.5, 2.0, (M, 2)).astype(np.float32) if weighted else None
    Td = torch.from_numpy(T).cuda()
    Wd = torch.from_numpy(Wt).cuda() if weighted else None
    got = []
    for offset in (0, 2):  # 16-byte copies, then 4-byte ones: the same bits
        X, Xd = _features(lo, M, offset)
        net = learn.MLP(p)
        y = net.forward(Xd).cpu().numpy()
        loss, g = net.loss_grad(Xd, Td, Wd)
        got.append((y, loss, g))
    assert got[0][1] == got[1][1]
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][2], got[1][2])
    yo, lo_loss, go = lo.forward_backward(p, X, T, Wt if weighted else np.ones_like(T))
    # the oracle rounds to BF16 at the same points; an FP32 sum next to a
    # rounding boundary may fall on the other side: 2^-8 of single activations
    y, loss, g = got[0]
    assert np.abs(y - yo).max() <= 2e-3 * (np.abs(yo).max() + 1e-3) + 1e-2 * np.abs(yo).max()
    assert abs(loss - lo_loss) <= 1e-4 * lo_loss
    assert np.linalg.norm(g - go) <= 1e-2 * np.linalg.norm(go)


@pytest.mark.parametrize("n", [1, 127, 128, 129, 400])
@pytest.mark.parametrize("long_rows", [False, True])
def test_features_match_oracle(ispm, lo, learn, n, long_rows):
    rng = np.random.default_rng(n)
    # up to 80 entries a row: more than 28 on average do not fit the buffer
    lens = rng.integers(40, 81, n) if long_rows else rng.integers(1, 29, n)
    cols, rp = [], np.zeros(n + 1, np.int32)
    n_cols = n + 100
    for i in range(n):
        c = np.unique(np.append(rng.choice(n_cols, lens[i], replace=False), i))
        cols.append(c)
        rp[i + 1] = rp[i] + c.size
    ci = np.concatenate(cols).astype(np.int32)
    v = rng.uniform(0.1, 2.0, ci.size) * rng.choice([-1.0, 1.0], ci.size)
    v[ci == np.repeat(np.arange(n), np.diff(rp))] = rng.uniform(1.0, 3.0, n)
    A = ispm.csr_matrix(n, n_cols, rp, ci, v)
    F = learn.row_features(A).view(__import__("torch").int16).cpu().numpy().view(np.uint16)
    ref = lo.bf16_bits(lo.row_features(rp, ci, v, 0, 0))
    diff = np.abs(F.astype(np.int32) - ref.astype(np.int32))
    # host and device logarithms may round differently: one BF16 unit, rarely
    assert diff.max() <= 1 and np.count_nonzero(diff) <= max(1, 0.001 * diff.size)
