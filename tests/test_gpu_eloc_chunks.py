"""The workspace of the FP64 local energies (theta and q of a chunk of samples) for wide layers:
its size, and energies on both sides of a chunk's edge, which are those of a call by itself."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,M", [(4, 2048), (4, 2049), (4, 6000), (4, 12000)])
def test_workspace_is_bounded(N, M):
    from netket_gb300 import _native as nat
    size = nat.lib().vmck_rbm_eloc_f64_workspace_size
    tables = size(N, M, 0)
    assert 8 * (size(N, M, 10**7) - tables) <= 2**29
    assert size(N, M, 100) - tables == 2 * 100 * M


@pytest.mark.parametrize("M,n", [(6000, 5700), (3000, 11300)])
def test_chunk_edges(M, n):
    import netket_gb300 as nk
    N = 4
    g = np.random.default_rng(M)
    flat = torch.as_tensor(g.normal(size=M + N * M + N) * 0.02).cuda()
    x = torch.as_tensor((2 * g.integers(0, 2, size=(n, N)) - 1).astype(np.int8)).cuda()
    x[:, :2] = torch.tensor([1, -1], dtype=torch.int8)
    hi = nk.hilbert.Spin(0.5, N)
    at = (1 << 25) // M
    assert at < n
    rows = torch.tensor([0, at - 2, at - 1, at, at + 1, n - 1])
    for H in (nk.operator.Ising(hi, nk.graph.Chain(N), h=1.0, J=1.0),
              nk.operator.Heisenberg(hi, nk.graph.Chain(N))):
        e = nk.kernels.local_energies_fused(H, flat, x, N, M)
        for r in rows.tolist():
            one = nk.kernels.local_energies_fused(H, flat, x[r:r + 1].contiguous(), N, M)
            torch.testing.assert_close(one, e[r:r + 1], rtol=1e-13, atol=0.0)
