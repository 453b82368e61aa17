"""FP32 local energies of eloc_f32.cu against the general kernels they replace (which
the entry points run when the log-amplitudes are asked for as well): every
log-ratio is the same FP32 value, so the energies agree to the rounding of an FP64
sum of at most 600 terms, 1e-13 of the sum of magnitudes.  Widths around the 32
partial sums and the four-wide loads, sample counts that leave groups without a
sample, weights in shared memory and through L1, and terms with several elements
per row, unchanged configurations and one- and two-site terms together."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _general(op, flat, x, N, M):
    import netket_gb300 as nk
    nat = nk._native
    n = x.shape[0]
    e = torch.empty(n, dtype=torch.float64, device="cuda")
    lp = torch.empty(n, dtype=torch.float32, device="cuda")
    if isinstance(op, nk.operator.Ising):
        nat.check(nat.lib().vmck_rbm_eloc_ising(
            nat.stream(), nat.F32, nat.ptr(flat), N, M, nat.ptr(x), n, nat.ptr(op._edges_dev()),
            len(op.edges), op.h, op.J, nat.ptr(e), nat.ptr(lp)))
    else:
        st = op.device_struct()
        nat.check(nat.lib().vmck_rbm_eloc_local(nat.stream(), nat.F32, nat.ptr(flat), N, M,
                                                nat.ptr(x), n, ctypes.byref(st), nat.ptr(e),
                                                nat.ptr(lp)))
    return e


def _check(op, N, M, n, std=0.2, total_sz=None):
    import netket_gb300 as nk
    g = torch.Generator().manual_seed(N + M)
    flat = (torch.randn(M + N * M + N, generator=g) * std).cuda()
    x = nk.hilbert.Spin(0.5, N, total_sz=total_sz).random_state(seed=3, size=n)
    got = nk.kernels.local_energies_fused(op, flat, x, N, M)
    ref = _general(op, flat, x, N, M)
    scale = float(ref.abs().max())
    torch.testing.assert_close(got, ref, rtol=1e-13, atol=1e-13 * scale)


@pytest.mark.parametrize("N,M,n", [(2, 1, 1), (5, 31, 3), (9, 32, 1030), (16, 33, 1024),
                                   (33, 100, 1500), (100, 400, 1100), (64, 259, 40),
                                   (100, 512, 1030), (256, 256, 30), (128, 40, 8000),
                                   (33, 100, 31000)])
def test_ising(N, M, n):
    import netket_gb300 as nk
    hi = nk.hilbert.Spin(0.5, N)
    _check(nk.operator.Ising(hi, nk.graph.Chain(N, pbc=N > 2), h=0.9, J=-1.2), N, M, n)


@pytest.mark.parametrize("L,M,n,std", [(4, 7, 5, 0.2), (4, 32, 1027, 0.01), (6, 66, 1024, 0.3),
                                       (6, 144, 100, 3.0), (10, 400, 1100, 0.05),
                                       (10, 402, 33, 0.05), (10, 800, 20, 0.05),
                                       (10, 66, 3751, 0.3), (10, 400, 3800, 0.05)])
def test_heisenberg(L, M, n, std):
    import netket_gb300 as nk
    hi = nk.hilbert.Spin(0.5, L * L, total_sz=0)
    g = nk.graph.Square(L, max_neighbor_order=2)
    H = nk.operator.Heisenberg(hi, g, J=[1.0, 0.5], sign_rule=[True, False])
    _check(H, L * L, M, n, std, total_sz=0)


@pytest.mark.parametrize("n", [3, 1500])
def test_one_and_two_site_terms(n):
    """Full 4 x 4 and 2 x 2 matrices: up to three elements per row, one or both
    spins changed, 140 terms (more than one round of a warp's share), a constant."""
    import netket_gb300 as nk
    N = 70
    rng = np.random.default_rng(1)
    hi = nk.hilbert.Spin(0.5, N)
    ops, on = [], []
    for i in range(N):
        m = rng.normal(size=(4, 4))
        ops.append(m + m.T)
        on.append([i, (i + 1) % N])
        m = rng.normal(size=(2, 2))
        ops.append(m + m.T)
        on.append([i])
    _check(nk.operator.LocalOperator(hi, ops, on, constant=0.3), N, 90, n)
