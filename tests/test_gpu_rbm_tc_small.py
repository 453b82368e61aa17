"""Log-amplitudes of the tensor-core forward pass without tanh near the initial weights, where
the result is a sum of thousands of small log cosh: its error has to follow theta, not the 2^-22
of an exponential or a logarithm near 1.

Tolerance: cosh - 1 is off by |theta| 2^-22 + 2^-22 (cosh - 1) for a unit (an exponential, a
reciprocal and three roundings), theta by 2^-22 (|b| + sum |W|), of which tanh theta <= |theta|
enters; the FP32 sums add 2^-24 of the largest partial sum for each addition of a lane
(M / 256 + N / 32 + 5)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,M,n", [(8, 64, 2048), (16, 128, 1000), (36, 144, 999), (64, 256, 512),
                                   (100, 400, 300), (16, 33, 500)])
@pytest.mark.parametrize("std", [0.001, 0.01, 0.03])
def test_small_weights(N, M, n, std):
    import netket_gb300 as nk
    g = torch.Generator().manual_seed(N * M)
    flat = (torch.randn(M + N * M + N, generator=g) * std).cuda()
    x = torch.where(torch.rand(n, N, generator=g) < 0.5, 1, -1).to(torch.int8).cuda()
    d, xd = flat.double(), x.double()
    b, W, a = d[:M], d[M:M + N * M].view(N, M), d[M + N * M:]
    theta = xd @ W + b
    terms = theta.abs() + torch.log1p(torch.exp(-2 * theta.abs())) - 0.6931471805599453
    ref = terms.sum(1) + xd @ a
    lp, _, _ = nk.kernels.rbm_forward(flat, x, N, M, use_tc=True)
    unit = b.abs() + W.abs().sum(0)
    tol = 2.0**-22 * (theta.abs() * (1 + unit) + terms).sum(1) + \
        2.0**-24 * (M / 256 + N / 32 + 5) * (terms.sum(1) + a.abs().sum())
    assert bool(((lp.double() - ref).abs() <= tol).all())
