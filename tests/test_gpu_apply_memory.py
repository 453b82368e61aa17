"""RBM.apply on more FP32 states than the tensor-core forward pass holds theta of at once
(1 GiB of theta and spins): the memory that it asks for, and the values on both sides of a
part's edge.  Tolerance as for any FP32 sum over M hidden units: M 2^-21 + 2^-20 of the sum of
|b| + sum |W| + |a|."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_theta_is_formed_in_parts():
    import netket_gb300 as nk
    N, M = 16, 4096
    n = 3 * (1 << 28) // (M + N) + 5
    g = torch.Generator().manual_seed(1)
    flat = (torch.randn(M + N * M + N, generator=g) * 0.05).cuda()
    x = torch.where(torch.rand(n, N, generator=g) < 0.5, 1, -1).to(torch.int8).cuda()
    model = nk.models.RBM(alpha=M // N, param_dtype=torch.float32)
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    lp = model.apply(flat, x)
    assert lp.shape == (n,)
    assert torch.cuda.max_memory_allocated() - before < 1.2 * 2**30 + 8 * n + 2**24
    rows = (1 << 28) // (M + N)
    at = torch.tensor([0, 1, rows - 1, rows, rows + 1, 2 * rows - 1, 2 * rows, 3 * rows - 1,
                       3 * rows, n - 1])
    d, xd = flat.double(), x[at.cuda()].double()
    theta = xd @ d[M:M + N * M].view(N, M) + d[:M]
    ref = (torch.logaddexp(theta, -theta) - 0.6931471805599453).sum(1) + xd @ d[M + N * M:]
    tol = M * 2.0**-21 + 2.0**-20 * float(d.abs().sum())
    assert float((lp[at.cuda()].double() - ref).abs().max()) <= tol
