"""Log-amplitudes of the tensor-core forward pass without tanh (logpsi_cosh_kernel) at the
edges of its eight units per lane and of its wide loads, with theta below and beyond 10.

Tolerance: a hidden unit's cosh is off by 2^-21 (two exponentials of 2^-22), theta by
2^-20 (|b| + sum |W|) (two FP16 halves, FP32 sums), each of |tanh theta| <= 1 into the
result; the FP32 sums of M / 8 logarithms add (M / 8) 2^-24 of the result's size."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,M,n,std", [(5, 1, 3, 0.3), (16, 31, 9, 0.3), (16, 32, 8, 2.0),
                                       (33, 255, 17, 0.2), (40, 256, 7, 3.0), (9, 260, 100, 0.1),
                                       (64, 514, 33, 1.0)])
@pytest.mark.parametrize("keep", [False, True])
def test_logpsi_matches_fp64(N, M, n, std, keep):
    import netket_gb300 as nk
    g = torch.Generator().manual_seed(N * M)
    flat = (torch.randn(M + N * M + N, generator=g) * std).cuda()
    x = torch.where(torch.rand(n, N, generator=g) < 0.5, 1, -1).to(torch.int8).cuda()
    d, xd = flat.double(), x.double()
    b, W, a = d[:M], d[M:M + N * M].view(N, M), d[M + N * M:]
    theta = xd @ W + b
    ref = (torch.logaddexp(theta, -theta) - 0.6931471805599453).sum(1) + xd @ a
    lp, th, _ = nk.kernels.rbm_forward(flat, x, N, M, want_theta=keep, use_tc=True)
    size = float((b.abs() + W.abs().sum(0)).sum()) + float(a.abs().sum())
    tol = M * 2.0**-21 + 2.0**-20 * size + M / 8 * 2.0**-24 * float(ref.abs().max())
    assert float((lp.double() - ref).abs().max()) <= tol
    if keep:
        unit = b.abs() + W.abs().sum(0)
        assert bool(((th.double() - theta).abs() <= 2.0**-20 * unit).all())
