"""A change of stream between the calls that leave a copy from the pinned
staging buffer on its way (new coordinates, moduli, displacements) and the
next call: the same bits as on one stream."""
import numpy as np
import pytest

from fast_b200 import decks, gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(6, 5, 4), (40, 40, 38)])   # 48 KB of coordinates and less; 1.5 MB
def test_stream_changes_between_calls(n):
    import torch
    X, conn, _ = decks.box_mesh("hex8", n, (1.0, 1.0, 1.0))
    fixed = np.zeros(X.shape, bool)
    fixed[X[:, 2] < 1e-9] = True
    ne = len(conn)
    d = decks.Deck("hex8", X, conn, np.full(ne, 1000.0), np.full(ne, 0.3), (2, 2, 2), fixed, matrix_type="sparse",
                   total_lagrangian=True)
    one, many = gpu.GpuSystem(0), gpu.GpuSystem(0)
    one.upload(d)
    many.upload(d)
    streams = [torch.cuda.Stream() for _ in range(3)]
    for seed in range(6):
        rng = np.random.default_rng(seed)
        Xs = X + rng.uniform(-0.05, 0.05, X.shape) / max(n)
        E, nu = 1000.0 * np.exp(0.3 * rng.standard_normal(ne)), rng.uniform(0.1, 0.4, ne)
        u = 0.01 / max(n) * rng.standard_normal(d.num_eq())
        out = []
        for s in (one, many):
            k = seed

            def switch():
                nonlocal k
                k += 1
                if s is many:
                    s.set_stream(streams[k % 3].cuda_stream if k % 4 else None)
            for call in (lambda: s.update_coords(Xs), lambda: s.update_material(E, nu), lambda: s.set_displacement(u)):
                call()
                switch()
            s.assemble()
            switch()
            s.set_displacement(u)
            switch()
            out.append((s.internal_force(), s.mult_vect(u)))
            switch()
        assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
    # a stream may be gone when it is left
    many.set_stream(streams[0].cuda_stream)
    many.update_material(E)
    many.synchronize()
    del streams
    many.set_stream(None)
    many.assemble()
    one.close()
    many.close()


def test_first_batched_solve_on_a_callers_stream():
    """The tables of an ensemble's first solve are uploaded on the stream that
    reads them: the first solve of a fresh context gives the second one's bits."""
    import torch
    off = [0]
    rng = np.random.default_rng(3)
    Xs, cs, fs = [], [], []
    for n in [(3 + k % 5, 3 + k % 3, 2 + k % 4) for k in range(64)]:
        X, conn, _ = decks.box_mesh("hex8", n, (1.0, 1.0, 1.0))
        fixed = np.zeros(X.shape, bool)
        fixed[X[:, 0] < 1e-9] = True
        Xs.append(X)
        cs.append(conn + off[-1])
        fs.append(fixed)
        off.append(off[-1] + len(X))
    conn = np.concatenate(cs)
    ne = len(conn)
    d = decks.Deck("hex8", np.concatenate(Xs), conn, 1000.0 * np.exp(0.3 * rng.standard_normal(ne)),
                   np.full(ne, 0.3), (2, 2, 2), np.concatenate(fs), matrix_type="sparse")
    f = rng.standard_normal(d.num_eq())
    first = None
    for k in range(8):
        stream = torch.cuda.Stream()
        s = gpu.GpuSystem(0)
        s.set_stream(stream.cuda_stream)
        s.set_option(gpu.OPT_MATRIX_FREE, 0)
        s.upload(d)
        s.set_problems(np.asarray(off))
        s.assemble()
        u = s.solve_batch(f, tol=1e-10)[0]
        assert np.array_equal(u, s.solve_batch(f, tol=1e-10)[0])
        first = u if first is None else first
        assert np.array_equal(u, first)
        s.close()
