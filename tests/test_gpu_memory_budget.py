"""The draw tables of a request count in the memory that was given to it: with a budget the batched draw
cuts them into segments and a request that runs alone does without block words, and a server reserves
them.  The rows are the same.  One request of some 70000 pixels, whose tables take 0.3 GB for 9000 stars."""
import numpy as np
import pytest

import galfast_b200 as G
from test_gpu_integrate_pixels import beam

pytestmark = pytest.mark.gpu

MB = 1 << 20
COLS = ["lb", "DM", "absmag", "XYZ"]


def wide(lib, capacity):
    w = beam(lib, 60.0, 40.0, 15.0, 12.0, 18.0, 0.1, f=(0.02, 0.002, 0.0001), with_modules=False)
    w.capacity = capacity
    return w


def run(w, budget):
    """Rows by model, and the device memory that the call took and its context keeps."""
    import torch
    ctx = G.Context(0)
    free = torch.cuda.mem_get_info()[0]
    got = {}
    try:
        ctx.set_multi_budget(budget)
        G.run_catalog_multi(ctx, [w], sink=lambda j, m, r: got.setdefault(m, []).append({c: r[c] for c in COLS}))
        return {m: {c: np.concatenate([p[c] for p in v], axis=-1) for c in COLS} for m, v in got.items()}, free - torch.cuda.mem_get_info()[0]
    finally:
        ctx.close()


def assert_same(a, b):
    assert sorted(a) == sorted(b)
    for m in a:
        for c in COLS:
            assert np.array_equal(a[m][c], b[m][c]), (m, c)


@pytest.mark.parametrize("capacity", [1 << 18, 1000])      # batched, and alone in many batches
def test_budget_bounds_the_draw_tables(lib, capacity):
    w = wide(lib, capacity)
    assert 60000 < w.npixels < 80000
    want, whole = run(w, 0)
    got, cut = run(w, 64 * MB)
    assert_same(want, got)
    assert all(v["DM"].size > 1000 for v in want.values())
    # block words of 2880 blocks for a fourth of the pixels at least: 200 MB, of which 64 stay for the batched form
    assert whole - cut > 130 * MB


def test_server_reserves_the_words_of_a_request_that_runs_alone(lib):
    w = wide(lib, 1000)
    want, _ = run(w, 0)
    for budget in (64 * MB, 8 << 30):
        srv = G.Server(0, workers=1, memory_budget=budget, max_batch=4, keep_rows=True)
        rid = srv.submit(w)
        srv.drain()
        info, status, rows = srv.info(), srv.status[rid], srv.rows[rid]
        srv.close()
        assert status == 0
        assert_same(want, {m: {c: np.concatenate([p[c] for p in v], axis=-1) for c in COLS} for m, v in rows.items()})
        if budget == 64 * MB:
            assert info["peak_reserved"] == 0 and info["peak_running"] == 0
        else:
            assert info["peak_reserved"] > w.npixels // 4 * 2880 * 4 and info["peak_running"] == 1
