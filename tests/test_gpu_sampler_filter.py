"""The filtered Metropolis kernel (sampler_filter.cu) decides every proposal as the
plain warp-per-chain kernel does: samples, acceptance counters and log-probabilities
are identical, at the edges of its register forms (M = 32 r and one more), of its
bit words (N and the number of clusters around 32 and 1024), with weights from the
initialiser's to ones whose amplitudes differ by e^100, with repeated and
one-site clusters, and with more chains than fit one wave."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _both(monkeypatch, make, model, flat, chain_length=3, n_discard=2):
    out = []
    for plain in ("0", "1"):
        monkeypatch.setenv("VMCK_EXCHANGE_GENERIC", plain)
        sampler = make()
        st = sampler.init_state(model, flat, seed=17)
        for _ in range(2):  # the second call continues the chains
            s, st = sampler.sample(model, flat, state=st, chain_length=chain_length,
                                   n_discard=n_discard)
        out.append((s, st.σ, st.log_prob, st.n_accepted_proc))
    for a, b in zip(*out):
        assert torch.equal(a, b)
    return out[0]


def _model(nk, N, M, std, dtype):
    model = nk.models.RBM(alpha=M / N + 1e-9, kernel_init_std=std, hidden_bias_init_std=std,
                          visible_bias_init_std=std)
    assert model.n_hidden(N) == M
    return model, model.init_flat(N + M, N).to(dtype)


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("std", [0.01, 0.3, 3.0])
@pytest.mark.parametrize("N,M", [(1, 1), (16, 16), (31, 32), (33, 33), (32, 65), (20, 129),
                                 (24, 257), (20, 417), (10, 512)])
def test_local(monkeypatch, dtype, std, N, M):
    import netket_gb300 as nk
    model, flat = _model(nk, N, M, std, dtype)
    hi = nk.hilbert.Spin(0.5, N)
    _both(monkeypatch, lambda: nk.sampler.MetropolisLocal(hi, n_chains=37, sweep_size=40), model,
          flat)


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("std", [0.01, 0.3, 3.0])
@pytest.mark.parametrize("N,M,order", [(4, 4, 1), (16, 32, 2), (34, 33, 1), (32, 128, 2),
                                       (66, 200, 3), (100, 400, 2), (36, 500, 2)])
def test_exchange(monkeypatch, dtype, std, N, M, order):
    import netket_gb300 as nk
    model, flat = _model(nk, N, M, std, dtype)
    hi = nk.hilbert.Spin(0.5, N, total_sz=0)
    g = nk.graph.Chain(N, max_neighbor_order=order)
    s = _both(monkeypatch,
              lambda: nk.sampler.MetropolisExchange(hi, graph=g, d_max=order, n_chains=37), model,
              flat)[0]
    assert torch.all(s.to(torch.int32).sum(-1) == 0)


def test_exchange_all_pairs_and_waves(monkeypatch):
    """990 clusters on 45 sites (every pair; 31 bit words), more chains than one
    wave of blocks holds, an odd magnetisation."""
    import netket_gb300 as nk
    N = 45
    model, flat = _model(nk, N, 45, 0.1, torch.float32)
    hi = nk.hilbert.Spin(0.5, N, total_sz=0.5)
    cl = np.argwhere(np.triu(np.ones((N, N)), 1))
    _both(monkeypatch,
          lambda: nk.sampler.MetropolisExchange(hi, clusters=cl, n_chains=5001, sweep_size=9),
          model, flat, chain_length=1, n_discard=1)


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_exchange_repeated_clusters(monkeypatch, dtype):
    """Clusters given twice, in both orders, and a cluster of one site twice."""
    import netket_gb300 as nk
    N = 8
    model, flat = _model(nk, N, 24, 0.3, dtype)
    hi = nk.hilbert.Spin(0.5, N, total_sz=0)
    cl = [(0, 1), (1, 0), (0, 1), (2, 2), (2, 3), (3, 4), (4, 5), (5, 6), (6, 7), (7, 0), (1, 2)]
    _both(monkeypatch, lambda: nk.sampler.MetropolisExchange(hi, clusters=cl, n_chains=33), model,
          flat)


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("N,M,rule,chains,std", [
    (200, 250, 0, 5, 0.05), (200, 256, 1, 3, 0.01), (140, 512, 0, 37, 0.3), (120, 513, 1, 37, 0.01),
    (16, 1024, 1, 300, 0.3), (24, 1027, 0, 19, 0.01), (24, 2048, 1, 37, 0.1)])
def test_weights_through_l2(monkeypatch, dtype, N, M, rule, chains, std):
    """Weights too large for shared memory: the edges of the register forms (M =
    256, 512, 1024, 2048 and beyond), rows that are not 16-byte aligned, fewer and
    more chains than a block holds."""
    import netket_gb300 as nk
    model, flat = _model(nk, N, M, std, dtype)
    if rule == 0:
        hi = nk.hilbert.Spin(0.5, N)
        make = lambda: nk.sampler.MetropolisLocal(hi, n_chains=chains, sweep_size=40)
    else:
        hi = nk.hilbert.Spin(0.5, N, total_sz=0)
        g = nk.graph.Chain(N, max_neighbor_order=2)
        make = lambda: nk.sampler.MetropolisExchange(hi, graph=g, d_max=2, n_chains=chains,
                                                     sweep_size=40)
    _both(monkeypatch, make, model, flat)
