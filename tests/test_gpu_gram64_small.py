"""The FP64 Gram matrix on the tensor cores (gram64_tc.cu) at tanh(theta) near 0, on its diagonal
and for configurations that were sampled twice, against extended precision.

There T's entries are (A (1 + N) + N - g - g' + c) / n with A = sum t^2 small.  What is left out of
A's digit products is 2^-55.8 rms per hidden unit, of either sign: sqrt(M) of them times 1 + N, with
five roundings of the assembly, 2^-53 of N + A (1 + N) each.  Tolerance: six times that for an
entry, and six times that over sqrt(n) for the mean over the diagonal, where nothing of one sign
may be left (squares of digits would be: M (1 + N) 2^-57.6)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
L = np.longdouble


@pytest.mark.parametrize("N,M,n", [(8, 64, 130), (36, 144, 200), (100, 400, 150), (30, 700, 140)])
@pytest.mark.parametrize("size", [1e-4, 1e-3, 0.03])
def test_equal_rows(N, M, n, size):
    import netket_gb300 as nk
    g = np.random.default_rng(N + M)
    x = (2 * g.integers(0, 2, size=(n, N)) - 1).astype(np.int8)
    t = np.tanh(size * g.normal(size=(n, M)))
    half = n // 2
    x[half:2 * half], t[half:2 * half] = x[:half], t[:half]
    td, xd = torch.as_tensor(t).cuda(), torch.as_tensor(x).cuda()
    obar = nk.kernels.column_means(td, xd, N, M)
    T = nk.kernels.gram_structured(td, xd, N, M, obar, 0.0, 0)[0].cpu().numpy()
    tl, xl, ob = t.astype(L), x.astype(L), obar.cpu().numpy().astype(L)
    gv = (tl * (ob[:M] + xl @ ob[M:M + N * M].reshape(N, M))).sum(1) + xl @ ob[M + N * M:]
    A = (tl * tl).sum(1)
    ref = A * (1 + N) + N - 2 * gv + (ob * ob).sum()
    rms = 2.0**-55.8 * np.sqrt(M) * (1 + N) + 5 * 2.0**-53 * (N + A.astype(float) * (1 + N))
    for entries, at in ((np.diag(T), slice(None)),
                        (T[np.arange(half) + half, np.arange(half)], slice(half))):
        err = entries * L(n) - ref[at]
        assert (np.abs(err) <= 6 * rms[at]).all()
        assert abs(err.mean()) <= 6 * rms[at].max() / np.sqrt(len(err))
