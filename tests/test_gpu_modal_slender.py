"""Eigenvalues of slender and flat models, where a linear solve's recurrence
residual (1e-12) and the true one (1e-9 to 1e-7) part: the projected stiffness
from the right-hand sides is as good as the one from products with K.  Both
converge to the eigenvalues of the assembled K and M, here from a subspace
iteration in extended precision.

Bound: the rounding of the product K v by rows of 27 blocks, 81 eps |v|' |K| |v|,
relative to v' K v."""
import numpy as np
import pytest
import scipy.linalg as sl

from fast_b200 import decks, gpu

pytestmark = pytest.mark.gpu

LD = np.longdouble


def _full(low):
    a = low.toarray()
    return a + np.tril(a, -1).T


def _factor(K):
    n = len(K)
    L = K.astype(LD)
    for j in range(n):
        L[j, j] = np.sqrt(L[j, j])
        i = np.nonzero(L[j + 1:, j])[0] + j + 1
        L[i, j] /= L[j, j]
        L[np.ix_(i, i)] -= np.outer(L[i, j], L[i, j])
    return np.tril(L)


def _solve(L, B):
    X = B.copy()
    n = len(L)
    below = [np.nonzero(L[j + 1:, j])[0] + j + 1 for j in range(n)]
    for j in range(n):
        X[j] /= L[j, j]
        X[below[j]] -= np.outer(L[below[j], j], X[j])
    for j in range(n - 1, -1, -1):
        X[j] = (X[j] - L[below[j], j] @ X[below[j]]) / L[j, j]
    return X


def _reference(K, M, modes):
    """(eigenvalues, relative rounding of v' K v) of the lowest modes."""
    L, Kl, Ml = _factor(K), K.astype(LD), M.astype(LD)
    X = np.random.default_rng(0).standard_normal((len(K), 3 * modes)).astype(LD)
    for _ in range(12):
        Y = _solve(L, Ml @ X)
        _, Phi = sl.eigh((Y.T @ (Kl @ Y)).astype(float), (Y.T @ (Ml @ Y)).astype(float))
        X = Y @ Phi.astype(LD)
        X /= np.sqrt((X * (Ml @ X)).sum(0))
    X = X[:, :modes]
    e = (X * (Kl @ X)).sum(0)
    A = np.abs(X).astype(float)
    return e / (X * (Ml @ X)).sum(0), 81 * 2.0 ** -52 * (A * (np.abs(K) @ A)).sum(0) / e.astype(float)


@pytest.mark.parametrize("n,L", [((40, 1, 1), (40.0, 1.0, 1.0)), ((8, 8, 1), (10.0, 10.0, 0.05))])
def test_slender_eigenvalues(n, L):
    rng = np.random.default_rng(5)
    X, conn, _ = decks.box_mesh("hex8", n, L)
    X = X + rng.uniform(-0.03, 0.03, X.shape) * np.asarray(L) / np.asarray(n) * (X > 1e-9)
    fixed = np.zeros(X.shape, bool)
    fixed[X[:, 0] < 1e-9] = True
    ne = len(conn)
    d = decks.Deck("hex8", X, conn, np.full(ne, 1000.0), np.full(ne, 0.3), (2, 2, 2), fixed, matrix_type="sparse",
                   rho=np.full(ne, 1e-3))
    s = gpu.GpuSystem(0)
    s.upload(d)
    s.assemble()
    s.assemble_mass()
    K, M = _full(s.lower_csr()), _full(s.lower_csr(gpu.ASM_M))
    ref, bound = _reference(K, M, 4)
    # the linear solves are the case described: recurrence below 1e-12, true residual far above
    u, _ = s.solve(M @ np.ones(len(M)), tol=1e-12)
    _, rep = s.solve(M @ u, tol=1e-12)
    assert rep["rel_residual"] < 1e-12 and rep["true_rel_residual"] > 1e-10
    lam, modes, r = s.modal(4, tol=1e-6, max_iter=40, lin_tol=1e-12)
    assert r["converged"] == 1
    assert np.all(np.abs(lam / ref - 1.0).astype(float) <= bound), (lam / ref - 1.0, bound)
    # products with K (a looser linear tolerance): the same eigenvalues, whether or not its measure settles
    lam2, _, _ = s.modal(4, tol=1e-6, max_iter=12, lin_tol=1.001e-12, raise_on_fail=False)
    assert np.all(np.abs(lam2 / ref - 1.0).astype(float) <= bound), (lam2 / ref - 1.0, bound)
    s.close()
