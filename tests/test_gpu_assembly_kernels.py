"""Hex stiffness and mass kernels and the product with an assembled matrix
against the CPU oracle: every Gauss rule, numberings without order, supports in
single directions, and a hub whose axis nodes couple to more than 128 others."""
import numpy as np
import pytest

from fast_b200 import decks, gpu
from oracle import fem_oracle as fo

pytestmark = pytest.mark.gpu

# sums of at most 64 products of factors accurate to a few ulp, over at most 24
# elements: below 1e3 eps of the largest entry
TOL = 1e-12


def _wheel(kind, sectors, layers):
    """Elements around a common axis: quads (axis, r = 1, r = 1.5, r = 1)."""
    nat = np.asarray(decks.KINDS[kind][1], float)
    index, X, conn = {}, [], []
    for k in range(layers):
        for s in range(sectors):
            t0, t1 = 2 * np.pi * s / sectors, 2 * np.pi * (s + 1) / sectors
            tm = 0.5 * (t0 + t1)
            q = np.array([[0, 0], [np.cos(t0), np.sin(t0)], [1.5 * np.cos(tm), 1.5 * np.sin(tm)],
                          [np.cos(t1), np.sin(t1)]])
            row = []
            for x, y, z in nat:
                w = 0.25 * np.array([(1 - x) * (1 - y), (1 + x) * (1 - y), (1 + x) * (1 + y), (1 - x) * (1 + y)])
                p = np.array([*(w @ q), 0.6 * k + 0.3 * (1 + z)])
                key = tuple(np.round(p, 9) + 0.0)
                if key not in index:
                    index[key] = len(X)
                    X.append(p)
                row.append(index[key])
            conn.append(row)
    return np.array(X), np.array(conn, np.int32)


def _deck(kind, ngp, mesh, seed=0):
    rng = np.random.default_rng(seed)
    if mesh == "wheel":
        X, conn = _wheel(kind, 12, 2)
    else:
        X, conn, _ = decks.box_mesh(kind, mesh, tuple(0.5 * v for v in mesh))
    p = rng.permutation(len(X))            # nodes and elements in no order
    Xp = np.empty_like(X)
    Xp[p] = X + rng.uniform(-0.01, 0.01, X.shape)
    conn = p[conn][rng.permutation(len(conn))].astype(np.int32)
    fixed = rng.random(X.shape) < 0.05
    fixed[0] = True
    ne = len(conn)
    return decks.Deck(kind, Xp, conn, 1000.0 * np.exp(0.5 * rng.standard_normal(ne)), rng.uniform(0.0, 0.4, ne),
                      (ngp, ngp, ngp), fixed, rho=rng.uniform(0.5, 2.0, ne), matrix_type="sparse")


def _full(s, what):
    low = s.lower_csr(what)
    full = (low + low.T).tolil()
    full.setdiag(low.diagonal())
    return full.tocsr()


@pytest.mark.parametrize("mesh", [(1, 1, 1), (3, 2, 2), (5, 4, 3), "wheel"])
@pytest.mark.parametrize("kind,ngp", [("hex8", 1), ("hex8", 2), ("hex8", 3), ("hex20", 2), ("hex20", 3), ("hex20", 4)])
def test_assembled_matrices_match_oracle(kind, ngp, mesh):
    d = _deck(kind, ngp, mesh)
    s = gpu.GpuSystem(0)
    s.upload(d)
    x = np.random.default_rng(1).standard_normal(d.num_eq())
    for what, ref in ((gpu.ASM_K, fo.assemble(d)), (gpu.ASM_M, fo.mass_matrix(d))):
        (s.assemble if what == gpu.ASM_K else s.assemble_mass)()
        A = _full(s, what)
        ref = ref.tocsr()
        top = abs(ref).max()
        assert abs(A - ref).max() <= TOL * top
        y = s.mult_vect(x, what)
        assert np.abs(y - A @ x).max() <= TOL * np.abs(abs(A) @ np.abs(x)).max()
    # assembled again: the same bits, and the product after a solve's layout is there
    K0 = s.lower_csr(gpu.ASM_K).data.tobytes()
    M0 = s.lower_csr(gpu.ASM_M).data.tobytes()
    s.assemble()
    s.assemble_mass()
    assert s.lower_csr(gpu.ASM_K).data.tobytes() == K0 and s.lower_csr(gpu.ASM_M).data.tobytes() == M0


def test_mass_reports_an_inverted_element():
    d = _deck("hex20", 3, (2, 2, 1))
    s = gpu.GpuSystem(0)
    s.upload(d)
    X = d.coords.copy()
    X[:, 2] *= -1.0
    s.update_coords(X)
    with pytest.raises(gpu.FastGpuError):
        s.assemble_mass()
    s.update_coords(d.coords)
    s.assemble_mass()


@pytest.mark.parametrize("gather", [0, 1])
@pytest.mark.parametrize("tl", [False, True])
@pytest.mark.parametrize("mesh", [(1, 1, 1), (5, 4, 3), (16, 8, 1), (43, 3, 1), "wheel"])
def test_hex8_internal_force_matches_oracle(mesh, tl, gather):
    """Around a block of 128 elements, per node and colour by colour."""
    d = _deck("hex8", 2, mesh)
    d.total_lagrangian = tl
    rng = np.random.default_rng(7)
    u = 0.05 * rng.standard_normal(d.num_eq())
    eq = d.node_eq()
    full = np.where(eq > 0, u[np.maximum(eq, 1) - 1], 0.0)
    want, size = np.zeros(d.num_eq() + 1), np.zeros(d.num_eq() + 1)
    for e, en in enumerate(d.conn):
        f = (fo.elem_tl if tl else fo.elem_intforce)(8, d.ngp, d.coords[en], d.E[e], d.nu[e], full[en].ravel())
        g = np.asarray([v for v in f if np.ndim(v) == 1 and np.size(v) == 24][0])
        np.add.at(want, eq[en].ravel(), g)
        np.add.at(size, eq[en].ravel(), np.abs(g))
    s = gpu.GpuSystem(0)
    s.upload(d)
    s.set_option(gpu.OPT_FORCE_GATHER, gather)
    s.set_displacement(u)
    got = s.internal_force()
    assert np.abs(got - want[1:]).max() <= TOL * size[1:].max()


def test_large_host_arrays_arrive_whole():
    """Copies of more than 3 MB are shared among threads: a system updated to
    other moduli and coordinates equals one uploaded with them, bit for bit."""
    import dataclasses
    rng = np.random.default_rng(3)
    X, conn, _ = decks.box_mesh("hex8", (75, 74, 73), (75.0, 74.0, 73.0))
    fixed = np.zeros(X.shape, bool)
    fixed[X[:, 0] < 1e-9] = True
    ne = len(conn)
    d = decks.Deck("hex8", X, conn, np.full(ne, 1000.0), np.full(ne, 0.3), (2, 2, 2), fixed, matrix_type="sparse")
    assert 8 * ne > 3 << 20
    E, X2 = rng.uniform(500.0, 2000.0, ne), X + rng.uniform(-0.05, 0.05, X.shape)
    x = rng.standard_normal(d.num_eq())
    y = []
    for upd in (True, False):
        s = gpu.GpuSystem(0)
        s.upload(d if upd else dataclasses.replace(d, E=E, coords=X2))
        if upd:
            s.update_material(E)
            s.update_coords(X2)
        s.assemble()
        y.append(s.mult_vect(x))
        s.close()
    assert y[0].tobytes() == y[1].tobytes() and np.abs(y[0]).min() >= 0.0 and np.isfinite(y[0]).all()
