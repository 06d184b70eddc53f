"""A magnitude grid so fine that a row of its slot densities does not fit a CTA's shared memory (54298
slots): the many-request path crawls it, as does the draw of a single request, and both give the oracle's
catalog row for row."""
import numpy as np
import pytest

import galfast_b200 as G
from galfast_b200 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu

COLS = ["lb", "DM", "absmag", "XYZ", "Am", "comp", "hidden"]


def test_grid_above_the_slots_of_the_block_words_crawls(ctx, lib, multipliers):
    w = W.build_workload(lib, foot=W.cap_footprint(60.0, 40.0, 0.12), dx_deg=0.1, m0=8.0, m1=24.8, M0=14.0, M1=16.4, seed48=21,
                         capacity=1 << 20, with_modules=False)
    w.sky.dm = 0.0012
    for m, f in zip(w.models, (0.1, 0.1, 0.1)):
        m.f, m.lf_n = f, 0                 # a flat luminosity function does not narrow the grid
    inf = G.Skygen(ctx, w).info(0)
    assert (inf.nm, inf.nM) == (14000, 2000) and 1 < w.npixels < 16
    want = {}
    O.run_catalog(w, multipliers, threads=8, sink=lambda m, t, off: want.setdefault(m, []).append(t.as_dict(COLS)))
    assert sum(len(v[0]["DM"]) for v in want.values()) > 500
    many, one = {}, {}
    G.run_catalog_multi(ctx, [w, w], sink=lambda j, m, r: many.setdefault((j, m), []).append({c: r[c] for c in COLS}))
    G.run_catalog(ctx, w, sink=lambda m, t, off: one.setdefault(m, []).append(t.as_dict(COLS)))
    for m, v in want.items():
        for got in (many[0, m], many[1, m], one[m]):
            for c in COLS:
                assert np.array_equal(np.concatenate([p[c] for p in got], axis=-1), np.concatenate([p[c] for p in v], axis=-1)), (m, c)


@pytest.mark.parametrize("radius,words", [(0.85, False), (1.35, True)])       # 0.01 mag rows: about 230 and 580 pixels
def test_few_pixels_of_a_fine_grid_crawl(ctx, lib, multipliers, radius, words):
    """Both have 1e8 bins and more; the fewer pixels leave the pixel integrate and the block words a few warps only."""
    w = W.build_workload(lib, foot=W.cap_footprint(60.0, 40.0, radius), dx_deg=0.1, m0=16.0, m1=19.0, seed48=22, capacity=1 << 20,
                         with_modules=False)
    w.sky.dm = 0.01
    assert (w.npixels >= 512) == words and w.npixels > 200
    ctx.profile()
    ctx.profile_read()
    one = {}
    G.run_catalog(ctx, w, sink=lambda m, t, off: one.setdefault(m, []).append(t.as_dict(COLS)))
    phases = ctx.profile_read()
    ctx.profile(False)
    assert ("slot_density" in phases) == words
    want = {}
    O.run_catalog(w, multipliers, threads=8, sink=lambda m, t, off: want.setdefault(m, []).append(t.as_dict(COLS)))
    assert sorted(one) == sorted(want) == [0, 1, 2]
    for m, v in want.items():
        for c in COLS:
            assert np.array_equal(np.concatenate([p[c] for p in one[m]], axis=-1), np.concatenate([p[c] for p in v], axis=-1)), (m, c)
