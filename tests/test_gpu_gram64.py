"""FP64 Gram matrix on the tensor cores (gram64_tc.cu) against the dense FP64 product
of the centred Jacobian, at the edges of its tiles (128 rows, 64 columns, 32 hidden
units per stage, 512 per exact sum) and with t at the ends of its range.  Entries
are sums of at most (M + N M + N) products of FP64 numbers of magnitude at most 1:
tolerance 1e-13 of the largest entry before centring, N M / n."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _dense(t, x, shift):
    n = x.shape[0]
    xd = x.double()
    O = torch.cat([t, (xd[:, :, None] * t[:, None, :]).reshape(n, -1), xd], 1)
    obar = O.mean(0)
    O = (O - obar) / n ** 0.5
    return obar, torch.tril(O @ O.T + shift * torch.eye(n, dtype=torch.float64, device="cuda"))


def _gram(t, x, obar, shift, want_f32=False):
    import netket_gb300 as nk
    n, N = x.shape
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    T64, T32 = nk.kernels.gram_structured(t.contiguous(), x, N, t.shape[1], obar, shift, 0,
                                          want_f32=want_f32, status=status)
    assert int(status.item()) == 0
    return torch.tril(T64), T32


@pytest.mark.parametrize("N,M,n", [(1, 32, 1600), (33, 31, 1601), (40, 20, 900), (64, 33, 513), (100, 400, 640),
                                   (288, 65, 400), (8, 512, 385), (6, 513, 384), (5, 1100, 300)])
@pytest.mark.parametrize("kind", ["small", "spread", "ends"])
def test_against_dense(N, M, n, kind):
    g = torch.Generator().manual_seed(N + M + n)
    x = torch.where(torch.rand(n, N, generator=g) < 0.5, 1, -1).to(torch.int8).cuda()
    r = torch.randn(n, M, generator=g, dtype=torch.float64).cuda()
    if kind == "small":
        t = torch.tanh(0.05 * r)
    elif kind == "spread":
        t = torch.tanh(r)
    else:  # +-1, the largest digit sums, and tiny values
        t = torch.where(r > 1.0, 1e-9 * r, torch.where(r > 0.2, 1.0, -1.0))
    obar, ref = _dense(t, x, 1e-3)
    T, T32 = _gram(t, x, obar, 1e-3, want_f32=True)
    scale = (N + 1) * M / n
    torch.testing.assert_close(T, ref, rtol=0.0, atol=1e-13 * scale)
    torch.testing.assert_close(torch.tril(T32), T.float(), rtol=0.0, atol=0.0)


@pytest.mark.parametrize("bad", [1.5, float("nan")])
def test_values_beyond_tanh_take_the_plain_kernel(bad):
    """t is any FP64 matrix to the entry point: values above 1 and NaN give what
    the CUDA-core kernel gives."""
    g = torch.Generator().manual_seed(1)
    N, M, n = 20, 64, 600
    x = torch.where(torch.rand(n, N, generator=g) < 0.5, 1, -1).to(torch.int8).cuda()
    t = torch.tanh(torch.randn(n, M, generator=g, dtype=torch.float64)).cuda()
    t[17, 5] = bad
    obar, ref = _dense(t, x, 1e-3)
    T, _ = _gram(t, x, obar, 1e-3)
    torch.testing.assert_close(T, ref, rtol=1e-11, atol=1e-11, equal_nan=True)
