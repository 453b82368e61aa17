"""FP64 local energies (eloc_f64.cu) against extended precision where the table form loses
most: weights of one sign, for which a lane's product moves far from 1 and the flipped row's
sum of weights far beyond the log-ratio (up to 150: from about 300 on, e^(2 sum) leaves the
double range and the log_cosh route takes over).

Tolerance: six times the rms of independent roundings.  With a = 4 |W| log2 e of eight
neighbours' sum S <= 8, a lane's product of eight factors in units of 2^-(63 - S) is off by at
most 1.2 units / sqrt(3) of the last factor's size 2^-S, M / 8 times over: 0.7 2^(2 S - 63)
sqrt(M / 8).  The tables' exponentials are off by 2^-53 at most, 2^-54 rms, and theta by 2^-54
|theta| rms, of which 2 |W| sech^2 theta enters: 2^-54 (1 + 2 |W|), M times over."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
L = np.longdouble


def _log_cosh(t):
    a = np.abs(t)
    return a + np.log1p(np.exp(-2 * a))


def _ising(flat, x, N, M):
    """sum_k psi(x with k flipped) / psi(x) and sum of x_i x_i+1 on the open chain."""
    b, W, a = flat[:M].astype(L), flat[M:M + N * M].reshape(N, M).astype(L), flat[M + N * M:]
    xl = x.astype(L)
    theta = b + sum(xl[:, i:i + 1] * W[i] for i in range(N))
    base = _log_cosh(theta)
    flips = sum(np.exp((_log_cosh(theta - 2 * xl[:, k:k + 1] * W[k]) - base).sum(1)
                       - 2 * xl[:, k] * a[k].astype(L)) for k in range(N))
    return flips, (xl[:, 1:] * xl[:, :-1]).sum(1)


def _energies(flat, x, N, M):
    import netket_gb300 as nk
    H = nk.operator.Ising(nk.hilbert.Spin(0.5, N), nk.graph.Chain(N, pbc=False), h=1.0, J=1.0)
    return nk.kernels.local_energies_fused(H, torch.as_tensor(flat).cuda(),
                                           torch.as_tensor(x).cuda(), N, M).cpu().numpy()


@pytest.mark.parametrize("N,M,weight,bias", [
    (16, 512, 0.13, 3.0), (16, 512, 0.13, 0.0), (16, 512, 0.13, -3.0), (64, 256, 0.13, 3.0),
    (64, 256, 0.1, -3.0), (12, 264, 0.09, 3.0), (6, 3000, 0.05, 0.0), (6, 2500, 0.06, 2.0)])
def test_weights_of_one_sign(N, M, weight, bias):
    n = 24
    g = np.random.default_rng(N + M)
    flat = g.normal(size=M + N * M + N) * 0.01
    flat[M:M + N * M] = weight * (0.9 + 0.2 * g.random(N * M))
    flat[:M] += np.where(np.arange(M) % 2, bias, -bias) if bias > 0 else bias
    x = (2 * g.integers(0, 2, size=(n, N)) - 1).astype(np.int8)
    flips, diag = _ising(flat, x, N, M)
    assert np.isfinite(flips.astype(float)).all()
    S = np.ceil(8 * 5.7708 * 1.1 * weight)
    assert S <= 7
    rms = 0.7 * 2.0**(2 * S - 63) * np.sqrt(M / 8) + 2.0**-54 * np.sqrt(M) * (1 + 2 * weight)
    tol = 6 * rms
    err = np.abs(_energies(flat, x, N, M) - (diag - flips)) / np.maximum(1, flips)
    assert err.max() <= tol


@pytest.mark.parametrize("N,M", [(8, 40), (70, 33)])
@pytest.mark.parametrize("bias", [np.inf, -np.inf, np.nan])
def test_infinite_theta_gives_nan(N, M, bias):
    """A hidden bias that is not finite: psi(x') / psi(x) is a quotient of infinities, and no
    energy may look finite."""
    import netket_gb300 as nk
    g = np.random.default_rng(1)
    flat = g.normal(size=M + N * M + N) * 0.1
    flat[3] = bias
    x = (2 * g.integers(0, 2, size=(40, N)) - 1).astype(np.int8)
    x[:, :2] = 1, -1
    assert np.isnan(_energies(flat, x, N, M)).all()
    H = nk.operator.Heisenberg(nk.hilbert.Spin(0.5, N), nk.graph.Chain(N))
    e = nk.kernels.local_energies_fused(H, torch.as_tensor(flat).cuda(), torch.as_tensor(x).cuda(),
                                        N, M)
    assert bool(torch.isnan(e).all())
