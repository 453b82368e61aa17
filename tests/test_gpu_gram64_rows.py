"""The FP64 Gram matrix on the tensor cores (gram64_tc.cu) with rows of t of very different sizes,
against extended precision: each row's digits follow its own largest entry.

One site, so that T's entries, (A (1 + x x') + x x' - g - g' + c) / n with A = t.t', show the error
of A: what is left out of the digit products is 2^-55.8 rms per hidden unit of the rows' largest
entries' product, and the assembly rounds five times, 2^-53 of 1 + |A| (1 + x x') + |g| + |g'| +
c.  Tolerance: six times that."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
L = np.longdouble


@pytest.mark.parametrize("sizes", [(1e-3,), (1e-3, 1.0, 1e-9, 1e-200, 0.0, 1e-310), (0.49, 0.51, 1.0)])
@pytest.mark.parametrize("M", [33, 4100])
def test_row_sizes(sizes, M):
    import netket_gb300 as nk
    N, n = 1, 200
    g = np.random.default_rng(M)
    x = (2 * g.integers(0, 2, size=(n, N)) - 1).astype(np.int8)
    t = (2 * g.random(size=(n, M)) - 1) * np.array(sizes)[np.arange(n) % len(sizes)][:, None]
    t[np.arange(n) % len(sizes) == 1, 3] = sizes[-1] if len(sizes) == 3 else 0.7
    td, xd = torch.as_tensor(t).cuda(), torch.as_tensor(x).cuda()
    obar = torch.zeros(M + N * M + N, dtype=torch.float64, device="cuda")
    T = nk.kernels.gram_structured(td, xd, N, M, obar, 0.0, 0)[0].cpu().numpy()
    rows = np.r_[0:12, n - 12:n]
    tl, xl = t[rows].astype(L), x[rows].astype(L)
    A, B = tl @ tl.T, xl @ xl.T
    ref = A * (1 + B) + B
    top = np.abs(t[rows]).max(1)
    rms = 2.0**-55.8 * np.sqrt(M) * np.outer(top, top) * 4 * (1 + B.astype(float)) \
        + 5 * 2.0**-53 * (1 + np.abs(A.astype(float)) * (1 + B.astype(float)))
    low = np.tril(np.ones_like(rms, dtype=bool))
    err = np.abs(T[np.ix_(rows, rows)] * L(n) - ref)
    assert (err <= 6 * rms)[low].all()


def test_small_rows_of_wide_layers():
    """12,000 hidden units of size 1e-3: digits of fixed units leave out more than T's rounding."""
    import netket_gb300 as nk
    N, M, n = 1, 12000, 130
    g = np.random.default_rng(5)
    x = (2 * g.integers(0, 2, size=(n, N)) - 1).astype(np.int8)
    t = 1e-3 * g.normal(size=(n, M))
    t[n // 2:], x[n // 2:] = t[:n // 2], x[:n // 2]
    td, xd = torch.as_tensor(t).cuda(), torch.as_tensor(x).cuda()
    obar = torch.zeros(M + N * M + N, dtype=torch.float64, device="cuda")
    T = nk.kernels.gram_structured(td, xd, N, M, obar, 0.0, 0)[0].cpu().numpy()
    A = (t.astype(L)**2).sum(1)
    err = np.abs(np.diag(T) * L(n) - (2 * A + 1))
    assert (err <= 30 * 2.0**-53 * (1 + 2 * A.astype(float))).all()
