"""The filtered Metropolis kernels at the limits of their dispatch, against the plain kernel bit
for bit: every lane's bit word in use (1,024 sites, 1,024 clusters), one more (the plain kernel
on both sides: the rule refuses), and M = 2,049."""
import numpy as np
import pytest
import torch

from test_gpu_sampler_filter import _both, _model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("N,M", [(1024, 3), (1024, 33), (1024, 300), (1025, 3), (8, 2049)])
def test_local(monkeypatch, dtype, N, M):
    import netket_gb300 as nk
    model, flat = _model(nk, N, M, 0.1, dtype)
    hi = nk.hilbert.Spin(0.5, N)
    _both(monkeypatch, lambda: nk.sampler.MetropolisLocal(hi, n_chains=5, sweep_size=200), model,
          flat, chain_length=2, n_discard=1)


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("N,M,C", [(1024, 3, 1024), (46, 20, 1024), (46, 300, 1024), (46, 20, 1025),
                                   (1025, 3, 64)])
def test_exchange(monkeypatch, dtype, N, M, C):
    import netket_gb300 as nk
    model, flat = _model(nk, N, M, 0.1, dtype)
    hi = nk.hilbert.Spin(0.5, N, total_sz=0.0 if N % 2 == 0 else 0.5)
    if N < 100:
        cl = np.argwhere(np.triu(np.ones((N, N)), 1))[:C]
    else:
        cl = np.stack([np.arange(C), (np.arange(C) + 1) % N], 1)
    assert len(cl) == C
    _both(monkeypatch,
          lambda: nk.sampler.MetropolisExchange(hi, clusters=cl, n_chains=5, sweep_size=200), model,
          flat, chain_length=2, n_discard=1)
