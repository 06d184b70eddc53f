"""A generator's draw through block words (25 million bins a model and more), a warp a stream, against
the oracle: every batch's rows and the state of every stream after it.  Batches of one window and of
many, few streams and many, batches that end inside a stream and resume there, cuts that differ
between pixels, distance limits, a negative density, luminosity functions with zero rows, and the
modules' draws from the same streams between batches.  Positions and states are compared bit for bit."""
import pytest

from galfast_b200 import workloads as W
from oracle import oracle as O
from test_gpu_integrate_pixels import beam
from test_gpu_parity import MODULE_COLS, SKY_COLS, assert_same, draw_all, run_both

pytestmark = pytest.mark.gpu

CASES = {
    "one_batch": (1 << 18, lambda lib: beam(lib, 10.0, 45.0, 5.0, 16.0, 19.0, 0.2)),
    "batches": (20000, lambda lib: beam(lib, 10.0, 45.0, 5.0, 16.0, 19.0, 0.2)),
    "few_streams": (7777, lambda lib: beam(lib, 10.0, 45.0, 5.0, 16.0, 19.0, 0.2, nthreads=97)),
    "many_streams": (30000, lambda lib: beam(lib, 10.0, 45.0, 5.0, 16.0, 19.0, 0.2, nthreads=65472)),
    "cuts": (20000, lambda lib: beam(lib, 30.0, 7.0, 5.0, 16.0, 19.0, 0.2, ext_E=0.12)),
    "distances": (10000, lambda lib: beam(lib, 60.0, 35.0, 5.0, 16.0, 19.0, 0.2, dmin=300.0, dmax=4000.0)),
    "negative": (10000, lambda lib: beam(lib, 60.0, 35.0, 5.0, 16.0, 19.0, 0.2, f=(1.0, -0.12, 0.005))),
    "zero_lf": (10000, lambda lib: beam(lib, 60.0, 35.0, 5.0, 16.0, 19.0, 0.2, zero_lf=True)),
    "few_rows": (5000, lambda lib: beam(lib, 75.0, 20.0, 8.6, 20.0, 20.25, 0.1)),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_batches_equal_oracle(ctx, lib, multipliers, name):
    capacity, make = CASES[name]
    w = make(lib)
    nb, total = draw_all(ctx, w, multipliers, capacity)
    assert total > 1000 and (nb == 3) == (name == "one_batch")


def test_catalog_with_modules_equals_oracle(ctx, lib, multipliers):
    w = W.build_workload(lib, foot=W.cap_footprint(10.0, 45.0, 5.0), dx_deg=0.2, m0=16.0, m1=19.0, seed48=5, capacity=20000)
    gs, os_, gb, ob = run_both(ctx, w, multipliers)
    assert len(gb) == len(ob) > 3
    for (gm, go, g), (om, oo, o) in zip(gb, ob):
        assert (gm, go) == (om, oo)
        assert_same(g, o, SKY_COLS)
        # the modules skip clipped rows: the oracle's table keeps what the batch before left there
        vis = {k: (g[k][..., g["hidden"] == 0], o[k][..., o["hidden"] == 0]) for k in MODULE_COLS}
        assert_same({k: v[0] for k, v in vis.items()}, {k: v[1] for k, v in vis.items()}, MODULE_COLS, exact=False)
