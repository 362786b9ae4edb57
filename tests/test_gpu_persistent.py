"""The persistent PCG kernel against the kernel-per-step iteration at the
sizes where its parts change: one block, one cluster, many blocks, rows that
do not fit in shared memory, blocks with more rows than threads, node lists
that overflow, and sums far from 1."""
import numpy as np
import pytest

from fast_b200 import decks, gpu

pytestmark = pytest.mark.gpu

TOL = 1e-10
TOL_U = 1e-8   # the two paths' solutions (each solved to TOL)


def _box(kind, n, shuffle=False, scale=1.0, free_only=None):
    rng = np.random.default_rng(sum(n))
    X, conn, _ = decks.box_mesh(kind, n, tuple(v / 8 for v in n))
    X = X + rng.uniform(-0.04, 0.04, X.shape) / (16 if kind == "hex20" else 8)
    fixed = np.zeros(X.shape, bool)
    fixed[X[:, 2] < 0.02] = True
    if shuffle:
        perm = rng.permutation(len(X))
        inv = np.argsort(perm)
        X, fixed, conn = X[perm], fixed[perm], inv[conn].astype(np.int32)
    if free_only is not None:
        fixed[:] = True
        fixed.reshape(-1)[free_only] = False
    ne = len(conn)
    g = 2 if kind == "hex8" else 3
    d = decks.Deck(kind, X, conn, scale * 1000.0 * np.exp(0.3 * rng.standard_normal(ne)), np.full(ne, 0.3), (g, g, g),
                   fixed, matrix_type="sparse")
    return d, rng.standard_normal(d.num_eq())


@pytest.mark.parametrize("kind,n,kw,limit", [
    ("hex8", (1, 1, 1), {}, 65536),                    # 8 nodes: one block
    ("hex8", (1, 1, 1), {"free_only": [14]}, 65536),   # one equation: exact after one iteration (sums of zero)
    ("hex8", (2, 2, 3), {}, 65536),                    # 36 nodes: two blocks in a cluster
    ("hex8", (9, 9, 9), {}, 65536),                    # 1,000 nodes: a full cluster
    ("hex8", (9, 9, 10), {}, 65536),                   # 1,100 nodes: past the cluster, 35 blocks
    ("hex20", (7, 6, 5), {}, 65536),
    ("hex8", (9, 9, 10), {"scale": 1e25}, 65536),      # p.K p and z.r far from 1
    ("hex8", (9, 9, 10), {"scale": 1e-25}, 65536),
    ("hex20", (18, 17, 15), {}, 65536),                # matrix larger than the SMs' shared memory (FP64)
    ("hex8", (39, 39, 38), {"shuffle": True}, 65536),  # scattered numbering: the node list overflows
    ("hex8", (46, 46, 45), {}, 10 ** 6),               # 101,614 nodes: no list, more rows than threads
])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_persistent_path_agrees_with_kernel_path(kind, n, kw, limit, precision):
    d, f = _box(kind, n, **kw)
    prec = gpu.PREC_FP64 if precision == "fp64" else gpu.PREC_MIXED
    got = {}
    for nodes in (0, limit):
        s = gpu.GpuSystem(0)
        s.set_option(gpu.OPT_PERSISTENT_MAX_NODES, nodes)
        s.upload(d)
        s.assemble()
        u, rep = s.solve(f, tol=TOL, precision=prec)
        u2, rep2 = s.solve(f, tol=TOL, precision=prec)
        assert rep["converged"] and np.array_equal(u, u2) and rep == rep2   # the same bits every run
        r = f - s.mult_vect(u)
        assert np.linalg.norm(r) <= 1.5 * TOL * np.linalg.norm(f)
        got[nodes] = (u, rep)
        s.close()
    (u0, r0), (u1, r1) = got[0], got[limit]
    assert abs(r0["iterations"] - r1["iterations"]) <= max(2, r0["iterations"] // 50)
    assert np.abs(u1 - u0).max() <= TOL_U * np.abs(u0).max()
