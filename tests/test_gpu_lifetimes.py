"""A generator that outlives its context: it can be destroyed, in any order with others, and says so when it is used."""
import pytest

import galfast_b200 as G
from test_gpu_integrate_pixels import beam

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("radius", [1.0, 5.0])       # by streams, and by pixels with block words
@pytest.mark.parametrize("order", [(0, 1), (1, 0)])
def test_generators_outlive_their_context(lib, radius, order):
    w = beam(lib, 10.0, 45.0, radius, 16.0, 19.0, 0.2)
    ctx = G.Context(0)
    skies = [G.Skygen(ctx, w), G.Skygen(ctx, w)]
    table = G.DeviceTable(ctx, 100000, 0)
    ctx.rng_init(w.seed48, w.nstreams)
    want = [skies[0].integrate_counts(m)[0] for m in range(3)]
    drawn = skies[0].draw_sources(1, table)[0]
    table.free()
    ctx.close()
    for k in order:
        with pytest.raises(G.GalfastError, match="error -6"):
            skies[k].integrate_counts(0)
        skies[k].close()
    # another context is not touched by any of it
    ctx = G.Context(0)
    sky, table = G.Skygen(ctx, w), G.DeviceTable(ctx, 100000, 0)
    ctx.rng_init(w.seed48, w.nstreams)
    assert [sky.integrate_counts(m)[0] for m in range(3)] == want
    assert sky.draw_sources(1, table)[0] == drawn
    table.free()
    sky.close()
    ctx.close()
