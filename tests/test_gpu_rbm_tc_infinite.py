"""FP32 log-amplitudes of a batch that takes the tensor-core forward pass, with infinite weights:
infinite where one hidden unit's theta is, NaN where infinities of both signs meet, as the
CUDA-core forward pass has them."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1024, 1023])
@pytest.mark.parametrize("entries", [[(3, 5, 1.0)], [(0, 0, -1.0)], [(3, 5, 1.0), (9, 5, 1.0)],
                                     [(3, 5, 1.0), (9, 77, -1.0)]])
def test_infinite_weights(M, entries):
    import netket_gb300 as nk
    N, n = 16, 4200
    g = torch.Generator().manual_seed(1)
    flat = torch.randn(M + N * M + N, generator=g) * 0.1
    for i, j, sign in entries:
        flat[M + i * M + j] = sign * float("inf")
    flat = flat.cuda()
    x = torch.where(torch.rand(n, N, generator=g) < 0.5, 1, -1).to(torch.int8).cuda()
    ref = nk.kernels.rbm_forward(flat, x, N, M, use_tc=False)[0]
    assert n * M >= nk.kernels.TC_MIN_WORK
    lp = nk.models.RBM(alpha=M / N, param_dtype=torch.float32).apply(flat, x)
    assert not bool(torch.isfinite(ref).any())
    assert torch.equal(torch.isnan(lp), torch.isnan(ref)) and torch.equal(lp == ref, ref == ref)
    theta = nk.kernels.rbm_forward(flat, x, N, M, want_theta=True, use_tc=True)[1]
    want = nk.kernels.rbm_forward(flat, x, N, M, want_theta=True, use_tc=False)[1]
    torch.testing.assert_close(theta, want, rtol=1e-5, atol=1e-5, equal_nan=True)
