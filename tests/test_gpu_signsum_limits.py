"""FP64 log-amplitudes and O v (signsum_f64.cu) at the limits of their dispatch: hidden
layers so wide that a lane's product of 1 + e^(-2|theta|) <= 2 passes 2^512 and 2^1024 (a
lane of a cluster holds M / 64 units), as many sites as the tables of sign indices take and
one more, and the forms with fewer samples per warp that many sites ask for.

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


@pytest.mark.parametrize("N,M,n", [(16384, 1, 3), (16384, 33, 2), (16385, 1, 3), (16385, 3, 70),
                                   (2048, 2, 9800), (2049, 2, 9800), (4097, 2, 9800),
                                   (8193, 2, 9800)])
def test_many_sites(N, M, n):
    """16,384 sites take the tables, 16,385 the general kernel; 2,048, 4,096 and 8,192 are the
    most that eight, four and two samples per warp take (9,800 samples fill the SMs with
    eight each)."""
    import netket_gb300 as nk
    flat, x = _problem(N, M, n, 0.01)
    _check(flat, x, N, M)
    t = np.tanh(np.random.default_rng(1).normal(size=(n, M)))
    b, W, a = flat[:M], flat[M:M + N * M].reshape(N, M), flat[M + N * M:]
    got = nk.kernels.o_v(torch.as_tensor(t).cuda(), torch.as_tensor(x).cuda(), N, M,
                         torch.as_tensor(flat).cuda()).cpu().numpy()
    size, rows = np.abs(flat).sum(), _rows(n)
    got, t, xd = got[rows], t[rows], x[rows].astype(np.float64)
    np.testing.assert_allclose(got, (t * (b + xd @ W)).sum(1) + xd @ a, rtol=0,
                               atol=2.0**-53 * N * size)


def test_energies_beyond_the_tables():
    """16,385 sites: the FP64 energies take the general kernels."""
    import netket_gb300 as nk
    N, M, n = 16385, 1, 3
    flat, x = _problem(N, M, n, 0.01)
    hi = nk.hilbert.Spin(0.5, N)
    edges = [(i, i + 1) for i in range(0, 40)]
    H = nk.operator.Ising(hi, nk.graph.Graph(edges=edges, n_nodes=N), h=0.5, J=1.0)
    e = nk.kernels.local_energies_fused(H, torch.as_tensor(flat).cuda(),
                                        torch.as_tensor(x).cuda(), N, M).cpu().numpy()
    W, a = flat[M:M + N], flat[M + N:]
    theta = flat[0] + x.astype(np.float64) @ W
    d = -2.0 * x
    ratio = np.cosh(theta[:, None] + d * W) / np.cosh(theta)[:, None] * np.exp(d * a)
    ref = sum(x[:, i].astype(float) * x[:, j] for i, j in edges) - 0.5 * ratio.sum(1)
    np.testing.assert_allclose(e, ref, rtol=1e-10)
