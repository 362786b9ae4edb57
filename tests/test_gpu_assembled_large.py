"""Large models solved on the assembled matrix, where the default is the
matrix-free operator: the persistent PCG kernel beyond its node list (FP64
overflow, more nodes than the list takes, more rows than threads per block),
and the kernel-per-step iteration on the full-size box.  Newton, transient and
multi-block models of these sizes take the same kernels."""
import numpy as np
import pytest

from fast_b200 import gpu
from tests.test_gpu_full_size import BOUND, box, errors  # noqa: F401
from tests.test_gpu_persistent import TOL, TOL_U, _box

pytestmark = pytest.mark.gpu

NEVER = 10 ** 12


@pytest.mark.parametrize("n,kw,limit", [
    ((39, 39, 38), {"shuffle": True}, 65536),   # scattered numbering: the node list overflows
    ((46, 46, 45), {}, 10 ** 6),                # 101,614 nodes: no list, more rows than threads
    ((40, 40, 40), {}, 10 ** 6),                # 68,921 nodes: no list, fewer rows than threads
])
@pytest.mark.parametrize("precision", [gpu.PREC_FP64, gpu.PREC_MIXED])
def test_persistent_kernel_on_large_systems(n, kw, limit, precision):
    d, f = _box("hex8", n, **kw)
    got = {}
    for nodes in (0, limit):
        s = gpu.GpuSystem(0)
        s.set_option(gpu.OPT_MATRIX_FREE, NEVER)
        s.set_option(gpu.OPT_PERSISTENT_MAX_NODES, nodes)
        s.upload(d)
        s.assemble()
        before = s.launch_count()
        u, rep = s.solve(f, tol=TOL, precision=precision)
        launches = s.launch_count() - before
        # kernel by kernel: three an iteration; the persistent kernel: one for at least 50
        assert rep["converged"]
        assert launches >= 3 * rep["iterations"] if nodes == 0 else launches < rep["iterations"]
        u2, rep2 = s.solve(f, tol=TOL, precision=precision)
        assert np.array_equal(u, u2) and rep == rep2
        r = f - s.mult_vect(u)
        assert np.linalg.norm(r) <= 1.5 * TOL * np.linalg.norm(f)
        got[nodes] = (u, rep)
        s.close()
    (u0, r0), (u1, r1) = got[0], got[limit]
    assert abs(r0["iterations"] - r1["iterations"]) <= max(2, r0["iterations"] // 50)
    assert np.abs(u1 - u0).max() <= TOL_U * np.abs(u0).max()


@pytest.mark.parametrize("path", ["fp64", "mixed", "mixed_tf32"])
def test_full_hex20_box_on_the_assembled_matrix(box, path):  # noqa: F811
    s, f, z = box
    s.set_option(gpu.OPT_MATRIX_FREE, NEVER)
    s.assemble(gpu.ASM_K_TF32) if path == "mixed_tf32" else s.assemble()
    before = s.launch_count()
    u, rep = s.solve(f, tol=1e-10, precision=gpu.PREC_FP64 if path == "fp64" else gpu.PREC_MIXED)
    assert s.launch_count() - before >= 3 * rep["iterations"]   # matrix-free: two
    assert rep["converged"] and rep["true_rel_residual"] < 1e-10, rep
    e_sample, e_check = errors(u, z)
    assert e_sample < BOUND[1e-10] and e_check < BOUND[1e-10], (e_sample, e_check)
