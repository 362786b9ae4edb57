"""A mixed solve whose FP32 iteration breaks down goes on in FP64 from its
best FP64 iterate, not from what the breakdown left behind: one hex8 element
(10 equations), where 50 FP32 iterations run far past convergence."""
import numpy as np
import pytest

from fast_b200 import decks, gpu


@pytest.mark.gpu
@pytest.mark.parametrize("precond", [gpu.PRECOND_JACOBI, gpu.PRECOND_BLOCK_JACOBI])
@pytest.mark.parametrize("persistent", [0, 65536])
def test_one_element_mixed(precond, persistent):
    for seed in range(6):
        rng = np.random.default_rng([seed, 1, 1, 1])
        X, conn, _ = decks.box_mesh("hex8", (1, 1, 1), (0.25, 0.25, 0.25))
        fixed = np.zeros(X.shape, bool)
        fixed[X[:, 0] < 1e-9] = True
        fixed[X[:, 1] < 1e-9, 1] = True
        X = X + rng.uniform(-0.02, 0.02, X.shape)
        d = decks.Deck("hex8", X, conn, np.full(1, 1000.0), np.full(1, 0.3), (2, 2, 2), fixed)
        f = rng.standard_normal(d.num_eq())
        s = gpu.GpuSystem(0)
        s.set_option(gpu.OPT_PERSISTENT_MAX_NODES, persistent)
        s.upload(d)
        s.assemble()
        u, rep = s.solve(f, tol=1e-11, precision=gpu.PREC_MIXED, precond=precond)
        low = s.lower_csr().toarray()
        K = low + np.tril(low, -1).T
        # residual 1e-11 |f| and the product's rounding
        bound = 2e-11 * np.linalg.norm(f) + 24 * np.finfo(float).eps * np.linalg.norm(np.abs(K) @ np.abs(u))
        assert rep["converged"] and np.linalg.norm(f - K @ u) <= bound
        assert np.abs(u - np.linalg.solve(K, f)).max() <= 1e-8 * np.abs(u).max()
