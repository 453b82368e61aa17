"""The fixed-point form of the FP64 local energies (eloc_f64.cu) against the oracle where
it changes course: hidden widths around the 32 lanes and the eight factors of a lane
between two scalings, weights that ask for four or two factors or for the FP64 form in
some rows, theta at the ends of q, eight, four and two samples per CTA, sites shared by
two CTAs (from 64 sites on), more samples than a chunk.

Tolerance 1e-11 relative: M <= 4,000 factors within 2^-53 are 5e-13, the oracle's
log_cosh sums M |theta| 2^-53 <= 600 x 40 x 1.1e-16 = 3e-12."""
import numpy as np
import pytest
import torch

from gpu_common import oracle_local, oracle_params
from oracle import operator as oop
from oracle import rbm as orbm

pytestmark = pytest.mark.gpu


def _flat(N, M, std, bias, seed):
    g = torch.Generator().manual_seed(seed)
    flat = torch.randn(M + N * M + N, generator=g, dtype=torch.float64) * std
    flat[:M] += bias * torch.where(torch.arange(M) % 2 == 0, 1.0, -1.0)
    return flat.cuda()


def _check(H, get_conn, flat, x, N, M):
    import netket_gb300 as nk
    ref = orbm.local_energies(oracle_params(flat, N, M), x.cpu().numpy(), get_conn)
    e = nk.kernels.local_energies_fused(H, flat, x, N, M).cpu().numpy()
    np.testing.assert_allclose(e, ref, rtol=1e-11, atol=1e-11 * np.abs(ref).max())


@pytest.mark.parametrize("N,M,n,std,bias", [
    (6, 31, 40, 0.05, 0.0), (9, 33, 1500, 0.1, 0.0), (5, 257, 30, 0.05, 0.0),
    (7, 520, 13, 0.02, 0.0), (8, 300, 20, 0.15, 0.0), (11, 64, 21, 0.6, 0.0),
    (4, 2000, 9, 0.01, 0.0), (3, 4000, 5, 0.01, 0.0), (4, 8, 16390, 0.1, 0.0),
    (6, 40, 1300, 0.1, 30.0), (64, 40, 50, 0.05, 0.0), (65, 33, 2500, 0.03, 0.0)])
def test_ising(N, M, n, std, bias):
    import netket_gb300 as nk
    hi, g = nk.hilbert.Spin(0.5, N), nk.graph.Chain(N, pbc=N > 2)
    H = nk.operator.Ising(hi, g, h=0.7, J=-1.3)
    x = hi.random_state(seed=5, size=n)
    edges = np.array(g.edges())
    _check(H, lambda s: oop.ising_get_conn_padded(s, edges, 0.7, -1.3),
           _flat(N, M, std, bias, 3), x, N, M)


@pytest.mark.parametrize("sites", [1, 2])
@pytest.mark.parametrize("M,n,std,bias", [(31, 7, 0.05, 0.0), (257, 20, 0.05, 0.0),
                                          (300, 9, 0.1, 0.0), (64, 30, 0.6, 0.0),
                                          (8, 16390, 0.1, 0.0), (40, 9, 0.1, 30.0)])
def test_local_operator(sites, M, n, std, bias):
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
    H = nk.operator.LocalOperator(hi, ops, on)
    x = hi.random_state(seed=7, size=n)
    o = oracle_local(H)
    _check(H, o.get_conn_padded, _flat(N, M, std, bias, 11), x, N, M)
