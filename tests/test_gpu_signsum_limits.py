"""FP64 log-amplitudes (signsum_f64.cu) of hidden layers so wide that a lane's product of
1 + e^(-2|theta|) <= 2 passes 2^512 and 2^1024 (a lane of a cluster holds M / 64 units).

Tolerance: a factor of the product is off by an exponential and a rounding, 2^-52; theta by
2^-53 (|b| + sum |W|) for each of N + 2 additions; the sums over hidden units and over sites
round each partial sum, at most 2^-53 of the result's size for each addition of a lane
(M / 32), of the sites (N) and of the warps' trees (10)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
L = np.longdouble


def _problem(N, M, n, std):
    g = np.random.default_rng(N + M + n)
    flat = g.normal(size=M + N * M + N) * std
    return flat, (2 * g.integers(0, 2, size=(n, N), dtype=np.int8) - 1).astype(np.int8)


def _rows(n):
    """The samples that are compared: the first and the last 50."""
    return np.unique(np.r_[0:min(n, 50), max(0, n - 50):n])


def _log_psi(flat, x, N, M):
    b, W = flat[:M].astype(L), flat[M:M + N * M].reshape(N, M)
    theta = b + x.astype(L) @ W.astype(L)
    a = np.abs(theta)
    vis = x.astype(L) @ flat[M + N * M:].astype(L)
    return (a + np.log1p(np.exp(-2 * a)) - np.log(L(2))).sum(1) + vis


def _check(flat, x, N, M):
    import netket_gb300 as nk
    rows = _rows(len(x))
    ref = _log_psi(flat, x[rows], N, M)
    got = nk.kernels.rbm_forward(torch.as_tensor(flat).cuda(), torch.as_tensor(x).cuda(), N, M)[0]
    got = got[torch.as_tensor(rows).cuda()]
    W = np.abs(flat[M:M + N * M].reshape(N, M)).sum(0) + np.abs(flat[:M])
    size = float(np.abs(ref).max()) + np.abs(flat[M + N * M:]).sum()
    tol = 2.0**-52 * M + 2.0**-53 * ((N + 2) * W.sum() + (M / 32 + N + 10) * size)
    assert np.abs(got.cpu().numpy() - ref).max() <= tol


@pytest.mark.parametrize("M", [32704, 32705, 32769, 65536, 70000, 140001])
@pytest.mark.parametrize("std", [0.0, 0.01, 0.3])
def test_log_psi_of_very_wide_layers(M, std):
    flat, x = _problem(4, M, 9, std)
    _check(flat, x, 4, M)
