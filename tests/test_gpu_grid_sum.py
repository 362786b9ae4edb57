"""Grid sums of the persistent PCG kernel whose partials cancel: an indefinite
matrix of two uncoupled equations, diag(1, -1), whose nodes lie in different
blocks.  p.K p and z.r are 1 - f1^2, far below their partials, or zero."""
import numpy as np
import pytest

from fast_b200 import decks, gpu

pytestmark = pytest.mark.gpu


def _two_equations(persistent):
    X, conn, _ = decks.box_mesh("hex8", (9, 9, 10), (1.0, 1.0, 1.0))   # 1,100 nodes: 35 blocks, no cluster
    fixed = np.ones(X.shape, bool)
    fixed[[0, len(X) - 1], 0] = False
    ne = len(conn)
    d = decks.Deck("hex8", X, conn, np.full(ne, 1000.0), np.full(ne, 0.3), (2, 2, 2), fixed, matrix_type="sparse")
    s = gpu.GpuSystem(0)
    s.set_option(gpu.OPT_PERSISTENT_MAX_NODES, persistent)
    s.upload(d)
    s.assemble()
    for i, v in ((0, 1.0), (1, -1.0)):
        s.add(i, i, -s.get(i, i))
        s.add(i, i, v)
    assert s.neq == 2
    return s


@pytest.mark.parametrize("f1", [1.0 + 2.0 ** -20, 1.0 - 2.0 ** -20, 1.0 + 2.0 ** -31, 1.0 - 2.0 ** -31, 1.0])
def test_cancelling_sums_end(f1):
    f = np.array([1.0, f1])
    got = []
    for persistent in (0, 65536):
        s = _two_equations(persistent)
        u, rep = s.solve(f, tol=1e-10, raise_on_nonconv=False)
        got.append((u, rep["converged"], rep["iterations"]))
        s.close()
    (u0, c0, i0), (u1, c1, i1) = got
    assert c0 == c1 and i0 == i1
    if f1 == 1.0:
        assert not c1                       # z.r = 0: a breakdown
    else:
        # alpha = (1 - f1^2) / (1 - f1^2) = 1: exact after one iteration
        assert c1 and i1 == 1 and np.array_equal(u1, u0) and np.array_equal(u1, f * np.array([1.0, -1.0]))
