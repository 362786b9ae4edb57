"""What a call does where an allocation of device memory fails: the same
result another way where one exists, and nothing half allocated is used
afterwards."""
import numpy as np
import pytest

from fast_b200 import decks, gpu

pytestmark = pytest.mark.gpu


def _box(kind, n, rho=None):
    rng = np.random.default_rng(sum(n))
    X, conn, _ = decks.box_mesh(kind, n, tuple(v / 8 for v in n))
    X = X + rng.uniform(-0.04, 0.04, X.shape) / (16 if kind == "hex20" else 8)
    fixed = np.zeros(X.shape, bool)
    fixed[X[:, 2] < 0.02] = True
    ne = len(conn)
    g = 2 if kind == "hex8" else 3
    d = decks.Deck(kind, X, conn, 1000.0 * np.exp(0.3 * rng.standard_normal(ne)), np.full(ne, 0.3), (g, g, g), fixed,
                   matrix_type="sparse", rho=None if rho is None else np.full(ne, rho))
    return d, rng.standard_normal(d.num_eq())


# the persistent kernel's list indices (3.3 MB) and second z (2 MB): room for none, one, both
@pytest.mark.parametrize("leave", [0, 4 << 20, 32 << 20])
def test_persistent_kernel_buffers(leave):
    from tests.device_memory import short_of_memory
    d, f = _box("hex8", (39, 39, 38))
    s = gpu.GpuSystem(0)
    s.set_option(gpu.OPT_MATRIX_FREE, 10 ** 12)
    s.upload(d)
    s.assemble()
    warm = gpu.GpuSystem(0)          # loads the kernels
    warm.set_option(gpu.OPT_MATRIX_FREE, 10 ** 12)
    warm.upload(d)
    warm.assemble()
    want, rep = warm.solve(f, tol=1e-10)
    warm.close()
    s.set_option(gpu.OPT_PERSISTENT_MAX_NODES, 0)
    steps, _ = s.solve(f, tol=1e-10)
    with short_of_memory(leave):
        for _ in range(3):           # raising the limit again must not use half of the buffers
            s.set_option(gpu.OPT_PERSISTENT_MAX_NODES, 65536)
            u, r = s.solve(f, tol=1e-10)
            assert r["converged"]
            assert np.array_equal(u, steps) or np.array_equal(u, want)
            if leave == 0:
                assert np.array_equal(u, steps)
    u, r = s.solve(f, tol=1e-10)     # memory is back: so is the kernel
    assert np.array_equal(u, want) and r == rep
    s.close()


@pytest.mark.parametrize("precision", [gpu.PREC_FP64, gpu.PREC_MIXED])
def test_matrix_free_solve_falls_back(precision):
    """No memory for the matrix-free operands: the assembled matrix, whose
    layout is there, solves; matrix-free again once there is memory."""
    from tests.device_memory import short_of_memory
    d, f = _box("hex20", (14, 13, 12))
    s = gpu.GpuSystem(0)
    s.upload(d)
    s.set_option(gpu.OPT_PERSISTENT_MAX_NODES, 0)
    s.assemble()

    def solve():
        before = s.launch_count()
        u, r = s.solve(f, tol=1e-10, precision=precision)
        return u, r, (s.launch_count() - before) / r["iterations"]

    s.set_option(gpu.OPT_MATRIX_FREE, 0)
    free, rf, per_free = solve()
    assert per_free < 3.0
    s.set_option(gpu.OPT_MATRIX_FREE, 10 ** 12)
    asm, ra, per_asm = solve()
    assert per_asm >= 3.0
    s.upload(d)                        # the operands go, the layouts too
    s.assemble()
    assert np.array_equal(solve()[0], asm)
    s.set_option(gpu.OPT_MATRIX_FREE, 0)
    for leave in (0, 12 << 20):        # 2,184 elements: 4 MB of geometry, 2 MB of element forces
        with short_of_memory(leave):
            u, r, per = solve()
            assert np.array_equal(u, asm) or np.array_equal(u, free)
            if leave == 0:
                assert np.array_equal(u, asm) and r == ra and per >= 3.0
    u, r, per = solve()
    assert np.array_equal(u, free) and r == rf
    s.close()


def test_ensemble_falls_back():
    from tests.device_memory import short_of_memory
    from tests.test_gpu_batch_lockstep import _members
    d, off, f = _members([(10, 9, 8)] * 40)
    s = gpu.GpuSystem(0)
    s.upload(d)
    s.set_problems(off)
    s.assemble()
    s.set_option(gpu.OPT_MATRIX_FREE, 0)
    free = s.solve_batch(f, tol=1e-10)[0]
    s.set_option(gpu.OPT_MATRIX_FREE, 10 ** 12)
    asm = s.solve_batch(f, tol=1e-10)[0]
    s.set_problems(off)                # the operands go, the layout stays
    s.set_option(gpu.OPT_MATRIX_FREE, 0)
    with short_of_memory():
        assert np.array_equal(s.solve_batch(f, tol=1e-10)[0], asm)
    assert np.array_equal(s.solve_batch(f, tol=1e-10)[0], free)
    s.close()


@pytest.mark.parametrize("n,kept", [((24, 24, 24), True), ((70, 70, 69), False)])   # 44 MB and 1.08 GB of pair numbers
def test_mass_assembly_keeps_little(n, kept):
    """A large array of mass numbers per node pair is given back; the next
    assembly gives the same bits, and without room for it the element-wise
    scatter takes its place."""
    import torch
    from tests.device_memory import short_of_memory
    d, f = _box("hex20", n, rho=1e-3)
    x = np.random.default_rng(1).standard_normal(d.num_eq())
    s = gpu.GpuSystem(0)
    s.upload(d)
    s.assemble()
    s.assemble_mass()                     # M itself is there from here on
    y = s.mult_vect(x, gpu.ASM_M)
    s.upload(d)
    s.assemble()
    s._ck(s.L.fast_gpu_zero(s.ctx, gpu.ASM_M), "zero")
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    s.assemble_mass()
    torch.cuda.synchronize()
    used = before - torch.cuda.mem_get_info()[0]
    size = 8 * 400 * n[0] * n[1] * n[2]
    assert used >= size if kept else used < 4 << 20
    assert np.array_equal(s.mult_vect(x, gpu.ASM_M), y)
    s.assemble_mass()
    assert np.array_equal(s.mult_vect(x, gpu.ASM_M), y)
    if not kept:
        with short_of_memory():
            s.assemble_mass()
        z = s.mult_vect(x, gpu.ASM_M)
        assert np.abs(z - y).max() <= 1e-13 * np.abs(y).max()   # another order of at most 8 sums a block, 81 blocks a row
    s.close()
