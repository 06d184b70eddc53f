"""What goes on without the memory it would have liked: the arranged failures are cudaMalloc's own (they
set CUDA's last error), and the calls that have another way take it and succeed."""
import numpy as np
import pytest

import galfast_b200 as G
from test_gpu_integrate_pixels import beam

pytestmark = pytest.mark.gpu


@pytest.fixture
def lib_hook(lib):
    yield lib
    lib.gf_debug_fail_allocations(-1, 0)


def test_integrate_by_pixels_falls_back_to_the_crawl(lib_hook):
    """2.8e7 bins a model: whichever of the pixel integrate's tables cannot be had, the crawl gives the counts."""
    w = beam(lib_hook, 10.0, 45.0, 5.0, 16.0, 19.0, 0.2)
    ctx = G.Context(0)
    sky = G.Skygen(ctx, w)
    want = [sky.integrate_counts(m, per_pixel=True) for m in range(3)]
    sky.close()
    ctx.close()
    failed = 0
    for after in range(7):
        ctx = G.Context(0)
        sky = G.Skygen(ctx, w)
        assert lib_hook.gf_debug_fail_allocations(after, 1) == 0
        e, ec, pp = sky.integrate_counts(1, per_pixel=True)
        lib_hook.gf_debug_fail_allocations(-1, 0)
        failed += e != want[1][0]                  # (the sums of the crawl are added in another order)
        assert e == pytest.approx(want[1][0], rel=1e-12) and ec == pytest.approx(want[1][1], rel=1e-12)
        np.testing.assert_allclose(pp, want[1][2], rtol=1e-6)
        # the next calls are the usual ones
        for m in range(3):
            assert sky.integrate_counts(m)[0] == pytest.approx(want[m][0], rel=1e-14)
        sky.close()
        ctx.close()
    assert failed >= 3
