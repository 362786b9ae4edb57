"""check_every of FP64 solves in the persistent kernel: a launch takes 512
iterations, or the caller's period (from 64 on); the same bits either way."""
import numpy as np
import pytest

from fast_b200 import decks, gpu

pytestmark = pytest.mark.gpu


def test_callers_period_is_kept():
    d = decks.cantilever_hex8(40, 4, 4, L=(20.0, 1.0, 1.0))
    f = gpu.face_load_vector(d)
    s = gpu.GpuSystem(0)
    s.upload(d)
    s.assemble()
    s.solve(f, tol=1e-10)   # layouts

    def launches(check_every):
        before = s.launch_count()
        u, r = s.solve(f, tol=1e-10, check_every=check_every)
        return s.launch_count() - before, u, r["iterations"]

    n0, u0, its = launches(0)
    assert its > 256
    for period in (1, 64, 128):
        n, u, i = launches(period)
        # one launch a period, and one in flight when the last one is seen to have ended
        extra = -(-its // max(period, 64)) - (-(-its // 512))
        assert abs(n - n0 - extra) <= 1 and i == its and np.array_equal(u, u0)
    s.close()
