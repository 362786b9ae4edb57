"""Matrix-free solves (fast_gpu_set_option FAST_OPT_MATRIX_FREE) against
solves on the assembled matrix: the sizes around a batch of 32 elements, both
element kinds, precisions, preconditioners and starts, and the calls after
which the assembled matrix has to be used or the operator rebuilt."""
import numpy as np
import pytest

from fast_b200 import decks, gpu

pytestmark = pytest.mark.gpu

ALWAYS, NEVER = 0, 10 ** 12
TOL = 1e-11
TOL_U = 1e-8   # two solutions of residual TOL; the boxes' condition numbers stay below 1e3 / sqrt(TOL)


def _deck(kind, n, seed=0, jitter=0.08):
    rng = np.random.default_rng([seed, *n])
    X, conn, _ = decks.box_mesh(kind, n, tuple(0.25 * v for v in n))
    fixed = np.zeros(X.shape, bool)
    fixed[X[:, 0] < 1e-9] = True
    fixed[X[:, 1] < 1e-9, 1] = True            # a face on rollers: supports in one direction
    X = X + rng.uniform(-jitter, jitter, X.shape) * (0.125 if kind == "hex20" else 0.25)
    g = 2 if kind == "hex8" else 3
    d = decks.Deck(kind, X, conn, 1000.0 * np.exp(0.5 * rng.standard_normal(len(conn))),
                   rng.uniform(0.0, 0.4, len(conn)), (g, g, g), fixed, matrix_type="sparse")
    return d, rng.standard_normal(d.num_eq())


def _system(d, least):
    s = gpu.GpuSystem(0)
    s.upload(d)
    s.set_option(gpu.OPT_MATRIX_FREE, least)
    s.assemble()
    return s


def _product_rounding(s, u):
    """Rounding of one product K u by rows of at most 81 blocks: 3 * 81 eps |K| |u|."""
    low = abs(s.lower_csr())
    full = low + low.T
    full.setdiag(low.diagonal())
    return 243 * np.finfo(float).eps * np.linalg.norm(full @ np.abs(u))


def _close(a, b, tol=TOL_U):
    assert np.abs(a - b).max() <= tol * np.abs(b).max()


@pytest.mark.parametrize("kind,n", [("hex8", (1, 1, 1)), ("hex8", (31, 1, 1)), ("hex8", (4, 4, 2)), ("hex8", (11, 3, 1)),
                                    ("hex8", (13, 12, 11)), ("hex20", (1, 1, 1)), ("hex20", (4, 4, 2)),
                                    ("hex20", (11, 3, 1)), ("hex20", (9, 8, 7))])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("precond", [gpu.PRECOND_JACOBI, gpu.PRECOND_BLOCK_JACOBI])
def test_solutions_agree(kind, n, precision, precond):
    d, f = _deck(kind, n)
    opt = dict(tol=TOL, precond=precond, precision=gpu.PREC_FP64 if precision == "fp64" else gpu.PREC_MIXED)
    ref = _system(d, NEVER)
    u0, r0 = ref.solve(f, **opt)
    s = _system(d, ALWAYS)
    u1, r1 = s.solve(f, **opt)
    u2, r2 = s.solve(f, **opt)
    assert np.array_equal(u1, u2) and r1 == r2                   # the same bits every run
    assert r0["converged"] and r1["converged"]   # (the counts of slender bars differ with the rounding of K.u)
    r = f - s.mult_vect(u1)                                      # against the assembled matrix
    assert np.linalg.norm(r) <= 2 * TOL * np.linalg.norm(f) + _product_rounding(s, u1)
    _close(u1, u0)
    w, rw = s.solve(f, u0=u1 * (1 + 1e-5 * np.cos(np.arange(len(u1)))), **opt)  # warm start
    assert rw["converged"]
    _close(w, u0)


def test_operator_follows_the_model():
    d, f = _deck("hex20", (5, 4, 3))
    rng = np.random.default_rng(5)
    s, ref = _system(d, ALWAYS), _system(d, NEVER)
    for k in range(4):
        E = d.E * np.exp(0.3 * rng.standard_normal(d.num_elems))
        X = d.coords + 0.004 * rng.standard_normal(d.coords.shape)
        for q in (s, ref):
            if k % 2 == 0:
                q.update_material(E)
            if k >= 1:
                q.update_coords(X)
            q.assemble()
        prec = gpu.PREC_MIXED if k < 3 else gpu.PREC_FP64       # FP64 operands after FP32 ones and the other way round
        _close(s.solve(f, tol=TOL, precision=prec)[0], ref.solve(f, tol=TOL, precision=prec)[0])
    # an edited matrix is solved as edited
    for q in (s, ref):
        q.add(7, 7, 1e5)
    u = s.solve(f, tol=TOL)[0]
    _close(u, ref.solve(f, tol=TOL)[0])
    assert np.linalg.norm(f - s.mult_vect(u)) <= 2 * TOL * np.linalg.norm(f)
    # and a fresh assembly takes the operator back
    for q in (s, ref):
        q.assemble()
    _close(s.solve(f, tol=TOL)[0], ref.solve(f, tol=TOL)[0])


def test_tensor_core_stiffness_and_other_loads():
    d, f = _deck("hex20", (6, 5, 4))
    s, ref = _system(d, ALWAYS), _system(d, NEVER)
    s.assemble(gpu.ASM_K_TF32)
    u = s.solve(f, tol=TOL, precision=gpu.PREC_MIXED)[0]
    _close(u, ref.solve(f, tol=TOL)[0])
    z, rep = s.solve(np.zeros_like(f), tol=TOL, precision=gpu.PREC_MIXED)      # PCGSolver's early exit
    assert rep["converged"] and not z.any()
    _, rep = s.solve(f, tol=TOL, precision=gpu.PREC_MIXED, maxit=3, raise_on_nonconv=False)
    assert not rep["converged"] and rep["iterations"] == 3


def test_mass_edited_matrix_keeps_the_assembled_solve():
    d, f = _deck("hex8", (6, 5, 4))
    d.rho = np.full(d.num_elems, 2.0)
    out = []
    for least in (ALWAYS, NEVER):
        s = _system(d, least)
        s.assemble_mass()
        s.add_mat(50.0)
        out.append(s.solve(f, tol=TOL)[0])
    _close(out[0], out[1])
