"""FP64 local energies from flip-factor tables (eloc_f64.cu) against the oracle at
the sizes where the kernels can go wrong: hidden widths around the 32 lanes, a
sample count that leaves the last group of four ragged, operators of one to four
sites, and parameters whose products leave the double range, which take the
log_cosh route.  Tolerance 1e-10 relative, the accuracy stated for FP64 paths: a
product of M factors of a few ulp is within 1e-13, and the log_cosh route within
|theta| M ulp = 400 * 70 * 2e-16 = 6e-12."""
import numpy as np
import pytest
import torch

from gpu_common import oracle_local, oracle_params
from oracle import operator as oop
from oracle import rbm as orbm

pytestmark = pytest.mark.gpu


def _flat(N, M, seed, std, bias=0.0):
    g = torch.Generator().manual_seed(seed)
    flat = torch.randn(M + N * M + N, generator=g, dtype=torch.float64) * std
    flat[M - 1] += bias
    return flat.cuda()


def _check(H, get_conn, flat, x, N, M):
    import netket_gb300 as nk
    ref = orbm.local_energies(oracle_params(flat, N, M), x.cpu().numpy(), get_conn)
    e = nk.kernels.local_energies_fused(H, flat, x, N, M).cpu().numpy()
    np.testing.assert_allclose(e, ref, rtol=1e-10, atol=1e-10 * np.abs(ref).max())


# bias -400: exp(-2 theta) overflows and every element takes the log_cosh route
@pytest.mark.parametrize("N,M,n,bias", [(2, 1, 1, 0.0), (7, 31, 5, 0.0), (12, 32, 4, 0.0),
                                        (13, 33, 7, 0.0), (20, 70, 203, 0.0), (12, 70, 9, -400.0)])
def test_ising(N, M, n, bias):
    import netket_gb300 as nk
    hi, g = nk.hilbert.Spin(0.5, N), nk.graph.Chain(N, pbc=N > 2)
    H = nk.operator.Ising(hi, g, h=0.7, J=-1.3)
    x = hi.random_state(seed=5, size=n)
    edges = np.array(g.edges())
    _check(H, lambda s: oop.ising_get_conn_padded(s, edges, 0.7, -1.3),
           _flat(N, M, 3, 0.4, bias), x, N, M)


@pytest.mark.parametrize("sites", [1, 2, 3, 4])
@pytest.mark.parametrize("M,n,bias", [(1, 3, 0.0), (33, 50, 0.0), (70, 9, -400.0)])
def test_local_operator(sites, M, n, bias):
    """Real symmetric terms with diagonal and off-diagonal elements on 1 .. sites
    sites, so that elements of one group of four differ in their sites."""
    import netket_gb300 as nk
    N = 8
    hi = nk.hilbert.Spin(0.5, N)
    rng = np.random.default_rng(sites)
    ops, on = [], []
    for k in range(1, sites + 1):
        m = rng.normal(size=(2**k, 2**k))
        for start in (0, 3):
            ops.append(m + m.T)
            on.append([(start + 2 * q) % N for q in range(k)])
    H = nk.operator.LocalOperator(hi, ops, on, constant=0.25)
    x = hi.random_state(seed=6, size=n)
    _check(H, oracle_local(H).get_conn_padded, _flat(N, M, 4, 0.4, bias), x, N, M)
