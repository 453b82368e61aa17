"""The integer form of the FP64 products with the spin matrix (signsum_f64.cu): columns of
very different sizes, columns of zeros, columns that leave the integer form (infinities,
NaN, entries near the ends of the exponent range), the table blocks' edges (26 groups of
four sites) and chunks of more than 256 samples.

Tolerance: a column's sum of k entries is off by at most k 2^-53 sum |entry| in FP64 and
k 2^-55 max |entry| in units; both are below k^2 2^-53 max |entry| of that column, 1e-11
for k <= 300 and, for O^T v, sums over spans of 256 samples; the spans add n / 256
roundings of at most n max |entry|: 150,000 samples, 1e-13 n max |entry|."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _spins(n, N, g):
    return torch.as_tensor(np.where(g.random((n, N)) < 0.5, 1, -1).astype(np.int8))


@pytest.mark.parametrize("N,M,n", [(5, 3, 9), (100, 70, 40), (104, 33, 21), (105, 64, 70),
                                   (257, 40, 2500)])
def test_columns_keep_their_own_scale(N, M, n):
    import netket_gb300 as nk
    g = np.random.default_rng(N + M + n)
    x = _spins(n, N, g)
    scale = 10.0 ** g.integers(-200, 200, size=M)
    scale[0] = 0.0
    scale[-1] = 1e-305  # below the integer form's exponents
    W, b = g.normal(size=(N, M)) * scale, g.normal(size=M) * scale
    W[N // 2] *= 1e-12  # rows far below their columns' largest
    flat = torch.as_tensor(np.concatenate([b, W.ravel(), g.normal(size=N)])).cuda()
    _, theta, _ = nk.kernels.rbm_forward(flat, x.cuda(), N, M, want_theta=True, want_tanh=True)
    ref = x.numpy().astype(np.longdouble) @ W.astype(np.longdouble) + b.astype(np.longdouble)
    size = np.maximum(np.abs(W).max(0), np.abs(b))
    assert (np.abs(theta.cpu().numpy() - ref) <= 1e-11 * size).all()


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
def test_values_that_are_not_finite_stay_in_their_columns(bad):
    import netket_gb300 as nk
    N, M, n = 30, 70, 50
    g = np.random.default_rng(1)
    x = _spins(n, N, g)
    W, b = g.normal(size=(N, M)), g.normal(size=M)
    W[7, 3] = bad
    flat = torch.as_tensor(np.concatenate([b, W.ravel(), np.zeros(N)])).cuda()
    _, theta, _ = nk.kernels.rbm_forward(flat, x.cuda(), N, M, want_theta=True, want_tanh=True)
    theta = theta.cpu().numpy()
    assert not np.isfinite(theta[:, 3]).any()
    keep = np.arange(M) != 3
    np.testing.assert_allclose(theta[:, keep], (x.numpy() @ W + b)[:, keep], rtol=0, atol=1e-11)


@pytest.mark.parametrize("N,M,n,tiny", [(3, 2, 150000, False), (33, 40, 5000, True),
                                        (70, 31, 33, False)])
def test_ot_v_spans_and_scales(N, M, n, tiny):
    import netket_gb300 as nk
    g = np.random.default_rng(N + n)
    x = _spins(n, N, g)
    t = np.tanh(g.normal(size=(n, M)))
    t[:, 0] = 0.0
    t[:, -1] *= 1e-290 if tiny else 1e-30
    v = g.standard_t(2, size=n)
    out = nk.kernels.ot_v(torch.as_tensor(t).cuda(), x.cuda(), N, M, torch.as_tensor(v).cuda())
    w = v[:, None] * t
    xd = x.numpy().astype(np.float64)
    size = np.abs(w).max(0)
    tol = max(1e-11, 1e-13 * n)
    out = out.cpu().numpy()
    assert (np.abs(out[:M] - w.sum(0)) <= tol * size).all()
    assert (np.abs(out[M:M + N * M].reshape(N, M) - xd.T @ w) <= tol * size).all()
    assert (np.abs(out[M + N * M:] - xd.T @ v) <= tol * np.abs(v).max()).all()
