"""How long a mixed solve waits for FP32 before FP64 takes over
(reliable_scalar): FP64 residuals formed (`outer`) in models where CG's residual
does not halve for hundreds of iterations."""
import numpy as np
import pytest

from fast_b200 import decks, gpu

pytestmark = pytest.mark.gpu


def _model(kind, n, L, sigma=0.5, seed=11):
    rng = np.random.default_rng(seed)
    X, conn, _ = decks.box_mesh(kind, n, L)
    h = np.asarray(L) / np.asarray(n) / (2 if kind == "hex20" else 1)
    Y = X + rng.uniform(-0.05, 0.05, X.shape) * h
    fixed = np.zeros(X.shape, bool)
    fixed[np.abs(X[:, 0]) < 1e-9] = True
    ne = len(conn)
    g = 2 if kind == "hex8" else 3
    d = decks.Deck(kind, Y, conn, 1000.0 * np.exp(sigma * rng.standard_normal(ne)), np.full(ne, 0.3), (g, g, g),
                   fixed, matrix_type="sparse")
    f = np.zeros(d.num_eq())
    q = d.node_eq()[np.abs(X[:, 0] - L[0]) < 1e-9, 2]
    f[q[q > 0] - 1] = -1.0 / len(q)
    return d, f


def test_no_restarts_on_the_matrix_free_operator():
    """After tensor-core assembly the assembled FP32 matrix may restart its
    recurrence 40 times before it gives up (each after 10 residuals at the
    least); the matrix-free operator is the FP64 one rounded, and does not."""
    d, f = _model("hex20", (100, 5, 5), (100.0, 5.0, 5.0))
    s = gpu.GpuSystem(0)
    s.set_option(gpu.OPT_MATRIX_FREE, 0)
    s.upload(d)
    s.assemble(gpu.ASM_K_TF32)
    u, rep = s.solve(f, tol=1e-8, precision=gpu.PREC_MIXED)
    assert rep["converged"] and rep["escalated"] & 1 and rep["outer"] < 400
    s.close()


@pytest.mark.parametrize("least", [0, 10 ** 12])
def test_escalated_solve_leaves_the_fp64_stiffness(least):
    """A mixed solve on the tensor-core stiffness that FP32 cannot finish
    assembles the FP64 one, matrix-free or not: FP64 solves and products are
    refused before it and taken after it."""
    d, f = _model("hex20", (60, 3, 3), (60.0, 3.0, 3.0))
    s = gpu.GpuSystem(0)
    s.set_option(gpu.OPT_MATRIX_FREE, least)
    s.upload(d)
    s.assemble(gpu.ASM_K_TF32)
    for call in (lambda: s.solve(f, tol=1e-8), lambda: s.mult_vect(f)):
        with pytest.raises(gpu.FastGpuError) as e:
            call()
        assert e.value.rc == -4
    u, rep = s.solve(f, tol=1e-10, precision=gpu.PREC_MIXED)
    assert rep["converged"] and rep["escalated"] & 2
    v, rep = s.solve(f, tol=1e-10)
    assert rep["converged"]
    y = s.mult_vect(f)
    s.assemble()
    assert np.array_equal(s.mult_vect(f), y)
    w, _ = s.solve(f, tol=1e-10)
    assert np.array_equal(v, w)
    s.close()


def test_matrix_free_is_decided_once():
    """A solve that began on an assembled matrix stays on it, also where it
    assembles the FP64 stiffness on the way: here on the tensor-core matrix, after
    a transient analysis that was refused has changed the FP64 slot."""
    d, f = _model("hex20", (60, 3, 3), (60.0, 3.0, 3.0))
    d.rho = np.full(len(d.conn), 1e-3)
    s = gpu.GpuSystem(0)
    s.set_option(gpu.OPT_MATRIX_FREE, 0)
    s.upload(d)
    s.assemble(gpu.ASM_K_TF32)
    with pytest.raises(gpu.FastGpuError) as e:
        s.newmark(f, 2, 1e-3)
    assert e.value.rc == -4
    before = s.launch_count()
    u, rep = s.solve(f, tol=1e-10, precision=gpu.PREC_MIXED)
    assert rep["converged"] and rep["escalated"] & 2
    # the persistent kernel: far fewer launches than the two an iteration of a matrix-free solve
    assert s.launch_count() - before < rep["iterations"]
    v, rep = s.solve(f, tol=1e-10, precision=gpu.PREC_MIXED)
    assert rep["converged"] and np.linalg.norm(u - v) <= 1e-6 * np.linalg.norm(v)
    s.close()


@pytest.mark.parametrize("kind,n,L", [("hex8", (200, 2, 2), (200.0, 2.0, 2.0)), ("hex20", (60, 3, 3), (60.0, 3.0, 3.0)),
                                      ("hex8", (60, 60, 1), (60.0, 60.0, 0.5))])
def test_persistent_kernel_gives_up_after_ten(kind, n, L):
    """The first residual and ten without a halving."""
    d, f = _model(kind, n, L)
    s = gpu.GpuSystem(0)
    s.upload(d)
    s.assemble()
    u, rep = s.solve(f, tol=1e-8, precision=gpu.PREC_MIXED)
    assert rep["converged"] and rep["escalated"] == 1 and rep["outer"] == 11
    s.close()


@pytest.mark.parametrize("least", [0, 10 ** 12])
def test_large_system_waits_out_a_plateau(least):
    """On a large system (matrix-free or kernel by kernel) a plateau of ten
    residuals is no reason to give up."""
    d, f = _model("hex8", (60, 60, 60), (1.0, 1.0, 1.0), sigma=2.0)
    s = gpu.GpuSystem(0)
    s.set_option(gpu.OPT_MATRIX_FREE, least)
    s.upload(d)
    s.assemble()
    u, rep = s.solve(f, tol=1e-8, precision=gpu.PREC_MIXED)
    assert rep["converged"] and rep["escalated"] == 0 and rep["outer"] > 11
    s.close()
