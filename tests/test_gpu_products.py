"""fast_gpu_mult_vect from the blocks as assembled and from the solve layout:
the same bits, whether a solve has made the layout, many products have, or
nothing has; rows of 8 to 343 blocks, odd numbers of rows, every lane count."""
import numpy as np
import pytest

from fast_b200 import decks, gpu

pytestmark = pytest.mark.gpu


def _box(kind, n):
    rng = np.random.default_rng(sum(n))
    X, conn, _ = decks.box_mesh(kind, n, tuple(0.25 * v for v in n))
    X = X + rng.uniform(-0.01, 0.01, X.shape)
    fixed = np.zeros(X.shape, bool)
    fixed[X[:, 0] < 0.02] = True
    g = 2 if kind == "hex8" else 3
    return decks.Deck(kind, X, conn, 1000.0 * np.exp(0.5 * rng.standard_normal(len(conn))),
                      rng.uniform(0.0, 0.4, len(conn)), (g, g, g), fixed, matrix_type="sparse",
                      rho=np.full(len(conn), 1e-3))


DECKS = {
    "hex8 1x1x1": lambda: _box("hex8", (1, 1, 1)),
    "hex8 4x3x2": lambda: _box("hex8", (4, 3, 2)),
    "hex8 12x11x9": lambda: _box("hex8", (12, 11, 9)),
    "hex20 1x1x1": lambda: _box("hex20", (1, 1, 1)),
    "hex20 7x5x4": lambda: _box("hex20", (7, 5, 4)),
    "tied column": lambda: decks.tied_column((5, 5, 3), (3, 3, 2), (5, 5, 2), (5, 5, 2)),
}


@pytest.mark.parametrize("lanes", [4, 8, 16, 32])
@pytest.mark.parametrize("name", list(DECKS))
def test_products_have_the_same_bits(name, lanes):
    d = DECKS[name]()
    x = np.random.default_rng(5).standard_normal(d.num_eq())
    whats = (gpu.ASM_K,) if name == "tied column" else (gpu.ASM_K, gpu.ASM_M)
    s = gpu.GpuSystem(0)
    s.set_option(gpu.OPT_SPMV_LANES_FP64, lanes)
    s.set_option(gpu.OPT_MATRIX_FREE, 10 ** 12)
    s.upload(d)
    s.assemble()
    if gpu.ASM_M in whats:
        s.assemble_mass()
    first = {w: s.mult_vect(x, w) for w in whats}
    for w in whats:
        for _ in range(16):                       # past the number after which the layout is made
            assert np.array_equal(s.mult_vect(x, w), first[w])
    s.assemble()
    assert np.array_equal(s.mult_vect(x), first[gpu.ASM_K])
    s.solve(x, tol=1e-2)                          # makes the layout
    assert np.array_equal(s.mult_vect(x), first[gpu.ASM_K])
    low = s.lower_csr()
    full = low + low.T
    full.setdiag(low.diagonal())
    # rows of at most 343 blocks in FP64
    assert np.all(np.abs(full @ x - first[gpu.ASM_K]) <= 3 * 343 * 2.0 ** -52 * (abs(full) @ np.abs(x)))
    s.close()


def test_no_product_with_an_edited_slot_behind_the_tensor_core_stiffness():
    """While the tensor-core stiffness is the context's, the FP64 slot is not:
    no product with it, also when a refused transient analysis has filled it."""
    d = _box("hex20", (4, 3, 2))
    x = np.ones(d.num_eq())
    s = gpu.GpuSystem(0)
    s.upload(d)
    s.assemble(gpu.ASM_K_TF32)
    for call in (lambda: s.mult_vect(x), lambda: s.newmark(x, 2, 1e-3), lambda: s.mult_vect(x)):
        with pytest.raises(gpu.FastGpuError) as e:
            call()
        assert e.value.rc == -4
    s.close()
