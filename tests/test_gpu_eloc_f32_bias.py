"""FP32 local energies (eloc_f32.cu) of an operator with one- and two-site terms where a visible
bias is infinite: an element that leaves the site alone does not meet it."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [7, 5000])
def test_infinite_visible_bias_of_an_untouched_site(n):
    import netket_gb300 as nk
    N, M = 8, 24
    rng = np.random.default_rng(1)
    ops, on = [], []
    for k, sites in ((1, [1]), (1, [5]), (2, [2, 3]), (2, [6, 4])):  # not site 0
        m = rng.normal(size=(2**k, 2**k))
        ops.append(m + m.T)
        on.append(sites)
    hi = nk.hilbert.Spin(0.5, N)
    H = nk.operator.LocalOperator(hi, ops, on)
    flat = torch.randn(M + N * M + N, generator=torch.Generator().manual_seed(2)).cuda() * 0.2
    x = hi.random_state(seed=3, size=n)
    ref = nk.kernels.local_energies_fused(H, flat, x, N, M)
    flat[M + N * M] = float("inf")
    e = nk.kernels.local_energies_fused(H, flat, x, N, M)
    assert bool(torch.isfinite(ref).all()) and torch.equal(e, ref)
