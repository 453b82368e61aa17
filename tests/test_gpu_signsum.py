"""The FP64 products with the spin matrix by tables of signed sums (signsum_f64.cu)
against plain FP64 matrix products, at the edges of their tiles: groups of four
sites and samples, 32 hidden units, the register forms of the sites (N + 1 = 32, 64
and 128 and one more) and sample counts between the launch forms.  Tolerance 1e-12
of the largest entry: sums of at most 5,000 terms of FP64 rounding."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _problem(N, M, n):
    g = torch.Generator().manual_seed(N * M + n)
    flat = torch.randn(M + N * M + N, generator=g, dtype=torch.float64).cuda() * 0.2
    x = torch.where(torch.rand(n, N, generator=g) < 0.5, 1, -1).to(torch.int8).cuda()
    return flat, x


def _close(got, ref):
    torch.testing.assert_close(got, ref, rtol=1e-12, atol=1e-12 * float(ref.abs().max()))


@pytest.mark.parametrize("N,M,n", [(1, 1, 1), (3, 33, 7), (4, 32, 8), (31, 5, 65), (32, 31, 300),
                                   (63, 64, 2432), (64, 40, 2433), (127, 33, 4863),
                                   (129, 65, 100), (257, 20, 37), (288, 3, 17)])
def test_products_match_plain_fp64(N, M, n):
    import netket_gb300 as nk
    flat, x = _problem(N, M, n)
    xd = x.double()
    b, W, a = flat[:M], flat[M:M + N * M].view(N, M), flat[M + N * M:]
    theta = xd @ W + b
    lp, th, t = nk.kernels.rbm_forward(flat, x, N, M, want_theta=True, want_tanh=True)
    ref = (torch.logaddexp(theta, -theta) - 0.6931471805599453).sum(1) + xd @ a
    _close(th, theta)
    # of the kernel's own theta: near 0 tanh keeps theta's rounding, relative to itself
    torch.testing.assert_close(t, torch.tanh(th), rtol=1e-12, atol=1e-15)
    _close(lp, ref)
    _close(nk.kernels.rbm_forward(flat, x, N, M)[0], ref)
    O = torch.cat([t, (xd[:, :, None] * t[:, None, :]).reshape(n, -1), xd], 1)
    _close(nk.kernels.o_v(t, x, N, M, flat), O @ flat)
    v = lp - lp.mean() + 0.5
    _close(nk.kernels.ot_v(t, x, N, M, v), O.T @ v)


def test_logpsi_many_sites():
    """More sites than the tables hold in shared memory take the tiled kernel."""
    import netket_gb300 as nk
    flat, x = _problem(500, 17, 33)
    theta = x.double() @ flat[17:17 + 8500].view(500, 17) + flat[:17]
    ref = (torch.logaddexp(theta, -theta) - 0.6931471805599453).sum(1) + x.double() @ flat[8517:]
    _close(nk.kernels.rbm_forward(flat, x, 500, 17)[0], ref)
