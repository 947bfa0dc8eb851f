"""The CSR Krylov solves (tcad_csr_krylov: state on the device, an iteration
without the host) at the sizes where they can go wrong -- fewer rows than a
block, a row past one, restarts of one column and of more than 256, 1 x 1, 3 x 3
and 6 x 6 blocks, iteration caps, a start at the solution -- against a direct
solve of the same matrix."""
import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as spl

pytestmark = pytest.mark.gpu


def _system(n, seed=0):
    """A nonsymmetric diagonally dominant matrix (condition number below 10)."""
    rng = np.random.default_rng(seed)
    k = min(5, n - 1)
    rows = np.repeat(np.arange(n), k)
    cols = rng.integers(0, n, rows.size)
    A = sp.csr_matrix((rng.uniform(-1, 1, rows.size), (rows, cols)), shape=(n, n))
    A.setdiag(0)
    A = A + sp.diags(np.asarray(abs(A).sum(axis=1)).ravel() * 1.5 + 1.0)
    return A.tocsr(), rng.standard_normal(n)


@pytest.mark.parametrize("method", ["gmres", "bicgstab"])
@pytest.mark.parametrize("n,bs", [(2, None), (3, 3), (31, None), (255, 3), (257, None), (258, 6),
                                  (3072, 3), (151554, 6), (200001, 3)])
def test_csr_krylov_against_direct(method, n, bs):
    from tcad_b200.linsolve import solve_linear
    A, b = _system(n)
    x, info = solve_linear(A, b, method=method, rtol=1e-12, block_size=bs)
    # ||A x - b|| <= 1e-12 ||b|| with ||A^-1|| <= 1 and ||b|| <= ||A|| ||x||
    ref = spl.spsolve(A.tocsc(), b) if n < 4000 else None
    assert np.linalg.norm(A @ x - b) <= 1.01e-12 * np.linalg.norm(b)
    if ref is not None:
        assert np.linalg.norm(x - ref) <= 1e-11 * np.linalg.norm(ref)
    assert info["iterations"] <= n + 2


@pytest.mark.parametrize("restart", [1, 2, 7, 300])
def test_gmres_restarts(restart):
    from tcad_b200.linsolve import solve_linear
    A, b = _system(2000, 3)
    A = A - 0.4 * sp.diags(A.diagonal())        # slower: several cycles
    x, info = solve_linear(A, b, method="gmres", rtol=1e-11, restart=restart, maxiter=3000)
    assert np.linalg.norm(A @ x - b) <= 1.01e-11 * np.linalg.norm(b)


@pytest.mark.parametrize("method", ["gmres", "bicgstab"])
def test_caps_starts_and_breakdown(method):
    from tcad_b200.linsolve import LinearSolveError, solve_linear
    A, b = _system(600, 5)
    x, info = solve_linear(A, b, method=method, rtol=1e-12)
    again, info2 = solve_linear(A, b, method=method, rtol=1e-10, x0=x)
    assert info2["iterations"] == 0 and np.array_equal(again, x)
    with pytest.raises(LinearSolveError):
        solve_linear(A, b, method=method, rtol=1e-14, maxiter=1, restart=2)
    z, _ = solve_linear(A, np.zeros(600), method=method)
    assert np.array_equal(z, np.zeros(600))
