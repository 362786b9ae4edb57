"""Independent hex8 problems solved matrix-free an iteration at a time against
the same problems solved a cluster of blocks each on the assembled matrix:
members around a batch of 32 elements and a tile of 256 nodes, elements of
different members interleaved, starts, preconditioners, loads of zero, and
contexts whose problems or values change."""
import numpy as np
import pytest

from fast_b200 import decks, gpu

pytestmark = pytest.mark.gpu

LOCKSTEP, CLUSTERS = 0, 10 ** 12
TOL = 1e-11
TOL_U = 1e-8   # two solutions of residual TOL; the members' condition numbers stay below 1e3 / sqrt(TOL)


def _members(boxes, seed=0, shuffle=True):
    rng = np.random.default_rng([seed, len(boxes)])
    Xs, cs, fs, off = [], [], [], [0]
    for n in boxes:
        X, conn, _ = decks.box_mesh("hex8", n, tuple(0.25 * v for v in n))
        fixed = np.zeros(X.shape, bool)
        fixed[X[:, 0] < 1e-9] = True
        Xs.append(X + rng.uniform(-0.02, 0.02, X.shape))
        cs.append(conn + off[-1])
        fs.append(fixed)
        off.append(off[-1] + len(X))
    conn = np.concatenate(cs)
    if shuffle:
        conn = conn[rng.permutation(len(conn))]
    ne = len(conn)
    d = decks.Deck("hex8", np.concatenate(Xs), conn, 1000.0 * np.exp(0.5 * rng.standard_normal(ne)),
                   rng.uniform(0.0, 0.4, ne), (2, 2, 2), np.concatenate(fs), matrix_type="sparse")
    return d, np.asarray(off), rng.standard_normal(d.num_eq())


def _system(d, off, least):
    s = gpu.GpuSystem(0)
    s.upload(d)
    s.set_problems(off)
    s.set_option(gpu.OPT_MATRIX_FREE, least)
    s.assemble()
    return s


def _eqs(d, off, k):
    e = d.node_eq()[off[k]:off[k + 1]].ravel()
    return e[e > 0] - 1


def _same(a, b, d, off):
    (u0, c0, i0, r0), (u1, c1, i1, r1) = a, b
    assert (np.asarray(c0) == np.asarray(c1)).all()
    assert (np.asarray(r1)[np.asarray(c1)] < TOL).all()
    for k in range(len(off) - 1):
        e = _eqs(d, off, k)
        assert np.abs(u0[e] - u1[e]).max() <= TOL_U * max(np.abs(u0[e]).max(), 1e-300)
        assert (int(i0[k]) == 0) == (int(i1[k]) == 0)


BOXES = [[(1, 1, 1)], [(31, 1, 1), (1, 1, 1), (4, 4, 2)], [(7, 7, 3), (8, 7, 3), (3, 11, 1), (2, 2, 2)],
         [(13, 6, 5), (1, 2, 1), (4, 3, 11), (6, 6, 6), (33, 1, 1)]]


@pytest.mark.parametrize("boxes", BOXES)
@pytest.mark.parametrize("precond", [gpu.PRECOND_JACOBI, gpu.PRECOND_BLOCK_JACOBI])
@pytest.mark.parametrize("warm", [False, True])
def test_solutions_agree(boxes, precond, warm):
    d, off, f = _members(boxes)
    f[_eqs(d, off, len(boxes) - 1)] *= 0.0 if len(boxes) > 1 else 1.0   # one member has nothing to do
    u0 = np.random.default_rng(5).standard_normal(len(f)) * 1e-3 if warm else None
    ref = _system(d, off, CLUSTERS).solve_batch(f, tol=TOL, precond=precond, u0=u0)
    s = _system(d, off, LOCKSTEP)
    got = s.solve_batch(f, tol=TOL, precond=precond, u0=u0)
    _same(ref, got, d, off)
    again = s.solve_batch(f, tol=TOL, precond=precond, u0=u0)
    assert again[0].tobytes() == got[0].tobytes() and (np.asarray(again[2]) == np.asarray(got[2])).all()


def test_iteration_limit_and_state():
    d, off, f = _members(BOXES[3])
    s = _system(d, off, LOCKSTEP)
    for maxit in (1, 9, 33):
        u, conv, its, res = s.solve_batch(f, tol=TOL, maxit=maxit, raise_on_nonconv=False)
        ref = _system(d, off, CLUSTERS).solve_batch(f, tol=TOL, maxit=maxit, raise_on_nonconv=False)
        run = ~np.asarray(ref[1], bool) & ~np.asarray(conv, bool)
        assert (np.asarray(its)[run] == maxit).all() and (np.asarray(ref[2])[run] == maxit).all()
        assert maxit > 9 or run.any()
        # (after 33 iterations a change of summation order alone, in FP64 on a
        # CPU, moves these members' residuals by up to 2.5 %; after 9 by 1e-14)
        if maxit <= 9:
            assert np.allclose(np.asarray(res)[run], np.asarray(ref[3])[run], rtol=1e-4)


def test_values_and_problems_change():
    d, off, f = _members(BOXES[3], seed=2)
    s, ref = _system(d, off, LOCKSTEP), _system(d, off, CLUSTERS)
    _same(ref.solve_batch(f, tol=TOL), s.solve_batch(f, tol=TOL), d, off)
    E = np.asarray(d.E) * np.random.default_rng(3).uniform(0.5, 2.0, len(d.E))
    X = d.coords * 1.25
    for t in (s, ref):
        t.update_material(E)
        t.update_coords(X)
        t.assemble()
    _same(ref.solve_batch(f, tol=TOL), s.solve_batch(f, tol=TOL), d, off)
    both = np.array([off[0], off[2], off[-1]])    # members joined: other batches, other tiles
    for t in (s, ref):
        t.set_problems(both)
    _same(ref.solve_batch(f, tol=TOL), s.solve_batch(f, tol=TOL), d, both)
    # the whole context as one system, on the same batches
    one, two = s.solve(f, tol=TOL)[0], ref.solve(f, tol=TOL)[0]
    assert np.abs(one - two).max() <= TOL_U * np.abs(two).max()


@pytest.mark.parametrize("boxes,lockstep", [([(2, 2, 2)] * 3, False), ([(12, 12, 12)] * 3, True), ([(2, 2, 2)] * 900, True)])
def test_default_route(boxes, lockstep):
    """The default takes the route that its rule names, with the same results."""
    d, off, f = _members(boxes, shuffle=False)
    s = gpu.GpuSystem(0)
    s.upload(d)
    s.set_problems(off)
    s.assemble()
    got = s.solve_batch(f, tol=TOL)
    same = _system(d, off, LOCKSTEP if lockstep else CLUSTERS).solve_batch(f, tol=TOL)
    other = _system(d, off, CLUSTERS if lockstep else LOCKSTEP).solve_batch(f, tol=TOL)
    assert got[0].tobytes() == same[0].tobytes()
    _same(other, got, d, off)
