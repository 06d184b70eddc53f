"""The batched draw's block words and parked lanes, where they can go wrong: pixels whose cuts
differ inside a row, cuts of more and fewer bins than a block's unconditional steps, pixels at
the projection's edge, grids of fewer blocks than streams and of few magnitude rows, distance
limits, dense bins (several stars in most blocks), densities without a bound, and draw tables
cut into segments.  Every catalog equals the oracle's, row for row and bit for bit."""
import numpy as np
import pytest

import galfast_b200 as G
from galfast_b200 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu

COLS = ["lb", "DM", "absmag", "XYZ", "Am", "comp", "hidden", "vcyl"]


def beam(lib, l, b, r, m0, m1, seed, dmin=0.0, dmax=0.0, f=None, nthreads=7680, dx=0.2, **kw):
    w = W.build_workload(lib, foot=W.cap_footprint(l, b, r), dx_deg=dx, m0=m0, m1=m1, seed48=seed, capacity=1 << 20,
                         nthreads=nthreads, **kw)
    w.sky.dmin, w.sky.dmax = dmin, dmax
    if f is not None:
        for i, v in enumerate(f):
            w.models[i].f = v
    return w


CASES = {
    # strong extinction near the plane: the cut changes along the pixels and takes many rows
    "cuts": lambda lib: beam(lib, 30.0, 7.0, 2.0, 16.0, 19.0, 11, ext_E=0.12),
    # the edge of the projection disk (b = 0 for the polar projections)
    "edge": lambda lib: beam(lib, 200.0, 0.3, 1.0, 16.0, 18.0, 12, ext_E=0.0),
    # 5 magnitude rows (120 blocks a pixel), one row of which is cut
    "few_rows": lambda lib: beam(lib, 75.0, 20.0, 1.5, 20.0, 20.25, 13),
    # a single pixel, fewer blocks than streams
    "one_pixel": lambda lib: beam(lib, 10.0, 60.0, 0.05, 17.0, 19.0, 14),
    # streams that are no multiple of a warp, more blocks than any
    "streams_33": lambda lib: beam(lib, 120.0, 50.0, 0.8, 17.0, 19.0, 15, nthreads=33),
    # anchors inside [dmin, dmax) only
    "distances": lambda lib: beam(lib, 60.0, 35.0, 1.5, 16.0, 19.0, 16, dmin=300.0, dmax=4000.0),
    # several stars in most blocks of the faint end
    "dense": lambda lib: beam(lib, 60.0, 12.0, 0.9, 17.0, 19.5, 17, f=(30.0, 4.0, 0.2), dx=0.3),
    # a negative density: no bound holds for it, and it draws nothing
    "no_bound": lambda lib: beam(lib, 60.0, 35.0, 0.8, 17.0, 19.0, 18, f=(1.0, -0.12, 0.005)),
}


def oracle_rows(w, multipliers):
    out = {}
    O.run_catalog(w, multipliers, threads=8, sink=lambda m, t, off: out.setdefault(m, []).append(t.as_dict(COLS)))
    return {m: {c: np.concatenate([p[c] for p in v], axis=-1) for c in COLS} for m, v in out.items()}


def batched_rows(ctx, ws):
    got = {}
    G.run_catalog_multi(ctx, ws, sink=lambda j, m, rows: got.setdefault((j, m), []).append({c: rows[c] for c in COLS}))
    return {k: {c: np.concatenate([p[c] for p in v], axis=-1) for c in COLS} for k, v in got.items()}


@pytest.mark.parametrize("name", sorted(CASES))
def test_drawn_rows_equal_oracle(ctx, lib, multipliers, name):
    w = CASES[name](lib)
    want = oracle_rows(w, multipliers)
    got = batched_rows(ctx, [w])
    assert {m for _, m in got} == set(want)
    for m, cols in want.items():
        seen = cols["hidden"] == 0          # the modules leave the rows that the clipper hid as they find them
        for c in COLS:
            a, b = got[(0, m)][c], cols[c]
            assert a.shape == b.shape, (m, c)
            assert np.array_equal(a[..., seen], b[..., seen]) if c == "vcyl" else np.array_equal(a, b), (m, c)
    if name == "dense":
        assert sum(len(v["DM"]) for v in want.values()) > 20000


def test_any_failed_allocation_leaves_the_rows(lib):
    """A failed allocation of the draw tables cuts them into segments (every other one is retried
    after the caches are freed): whichever fails, the rows are the same."""
    ws = [CASES[n](lib) for n in ("cuts", "edge", "few_rows")]
    ctx = G.Context(0)
    want = batched_rows(ctx, ws)
    ctx.close()
    try:
        for after in range(0, 64, 3):
            ctx = G.Context(0)
            assert lib.gf_debug_fail_allocations(after, 1) == 0
            got = batched_rows(ctx, ws)
            lib.gf_debug_fail_allocations(-1, 0)
            ctx.close()
            assert got.keys() == want.keys()
            for k in want:
                for c in COLS:
                    assert np.array_equal(got[k][c], want[k][c]), (after, k, c)
    finally:
        lib.gf_debug_fail_allocations(-1, 0)
