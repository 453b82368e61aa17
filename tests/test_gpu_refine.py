"""The refined solve's symmetric residual and triangular solves at the sizes where a tile
or a block is cut off, against FP64 numpy.

A = 4 I + a random symmetric part of norm <= 2, some of whose entries are exact zeros,
minus zero, 1e-25 (below the range that the double-float split takes without its rare
cases) or whole rows of zeros.  Only the lower triangle is set.

Tolerances.  ||A|| ||A^-1|| <= 3, so the FP32 factor contracts the error by more than
1e4 per iteration and the iteration ends at the floor of its residual.  Double-float
sums of n <= 1,000 terms: at most n 2^-44 sum |a||x| ~ n sqrt(n) 2^-44 ||A|| ||x|| in
the worst case, 2e-9 at n = 1,000; with roundings of either sign 2^-44 sqrt(n) ~ 2e-12.
The mixed solve stops below a residual of 1e-10, so its solution is within
cond(A) 1e-10 <= 3e-10; the residual that it reports is within 1e-10 of the true one, and
the FP64 solution within 1e-12 (same reasoning with 2^-53); a lost tile, slot or triangle is an error of 1e-3 or more."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def nk():
    import netket_gb300
    return netket_gb300


def _matrix(n):
    rng = np.random.default_rng(n)
    B = rng.normal(size=(n, n))
    B = (B + B.T) / (2.0 * np.sqrt(n) + 2.0)
    B[rng.random((n, n)) < 0.05] = 0.0
    B[rng.random((n, n)) < 0.05] = -0.0
    B[rng.random((n, n)) < 0.05] = 1e-25
    B[n // 3] = 0.0
    L = np.tril(B)
    S = L + np.tril(L, -1).T
    S *= 2.0 / max(2.0, np.abs(np.linalg.eigvalsh(S)).max())
    return S + 4.0 * np.eye(n), rng.normal(size=n)


@pytest.mark.parametrize("n", [1, 2, 63, 64, 65, 127, 128, 129, 255, 257, 1000])
def test_refined_solution_and_residual(nk, n):
    A, b = _matrix(n)
    ref = np.linalg.solve(A, b)
    At = torch.as_tensor(np.tril(A) + np.triu(np.full((n, n), np.nan), 1), device="cuda")
    A32 = torch.as_tensor(A, device="cuda").float().contiguous()
    bt = torch.as_tensor(b, device="cuda")
    st = torch.zeros(1, dtype=torch.int32, device="cuda")
    x, res = nk.kernels.cholesky_solve_refined(At, A32, bt, st, max_iter=8, tol=1e-10)
    assert st.item() == 0
    xs = x.cpu().numpy()
    assert np.linalg.norm(xs - ref) <= 3e-10 * np.linalg.norm(ref)
    assert abs(res.item() - np.linalg.norm(b - A @ xs) / np.linalg.norm(b)) <= 1e-10
    st = torch.zeros(1, dtype=torch.int32, device="cuda")
    x = nk.kernels.cholesky_solve(torch.as_tensor(A, device="cuda"), bt, st)
    assert st.item() == 0
    assert np.linalg.norm(x.cpu().numpy() - ref) <= 1e-12 * np.linalg.norm(ref)
