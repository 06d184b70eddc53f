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


COLS = ["lb", "DM", "absmag", "XYZ", "Am"]
GF_E_OOM = -2


def draw_batch(ctx, sky, capacity):
    """One batch of model 1 into a table of that capacity: (rows, done), or None when the device has no memory."""
    table = G.DeviceTable(ctx, capacity, 0)
    try:
        n, done = sky.draw_sources(1, table)
    except G.GalfastError as e:
        assert "error %d:" % GF_E_OOM in str(e)
        return None
    else:
        rows = table.download().as_dict(COLS)
        return rows, done
    finally:
        table.free()


def draw(ctx, w, lib_hook, capacities, fail_in, after):
    """The batches of capacities in turn, the after-th allocation of batch fail_in failing; a batch that ran out of
    memory is drawn again.  Returns the rows and whether one did."""
    sky = G.Skygen(ctx, w)
    ctx.rng_init(w.seed48, w.nstreams)
    sky.integrate_counts(1)
    out, oom = [], False
    try:
        for k, c in enumerate(capacities):
            if k == fail_in:
                # the table's own allocations come first (20 columns, no bands)
                table_allocations = 18
                assert lib_hook.gf_debug_fail_allocations(table_allocations + after, 1) == 0
            got = draw_batch(ctx, sky, c)
            lib_hook.gf_debug_fail_allocations(-1, 0)
            if got is None:
                oom = True
                # (with the smallest of the tables: nothing may be left of one that could not grow)
                got = draw_batch(ctx, sky, min(capacities))
                assert got is not None
                out.append(got[0])
                break
            out.append(got[0])
        return out, oom
    finally:
        sky.close()


@pytest.mark.parametrize("fail_in,capacities", [(0, [6000, 6000]), (1, [6000, 90000])])
def test_generator_draws_without_the_memory_of_its_block_words(lib_hook, fail_in, capacities):
    w = beam(lib_hook, 10.0, 45.0, 5.0, 16.0, 19.0, 0.2)
    ctx = G.Context(0)
    want, oom = draw(ctx, w, lib_hook, capacities, -1, 0)
    assert not oom
    ctx.close()
    outcomes = []
    for after in range(0, 28):
        ctx = G.Context(0)
        got, oom = draw(ctx, w, lib_hook, capacities, fail_in, after)
        ctx.close()
        outcomes.append(oom)
        for k, rows in enumerate(got):
            n = rows["DM"].shape[-1]
            whole = want[k]["DM"].shape[-1]
            assert n == whole or (oom and k == len(got) - 1)
            if n == whole:
                for c in COLS:
                    assert np.array_equal(rows[c], want[k][c]), (after, k, c)
    # the tables of the block words and of the records are done without or got at the second try; a few small ones are not
    assert sum(outcomes) <= 6 and not all(outcomes)


def test_what_a_context_keeps_goes_back_before_an_allocation_fails(lib_hook):
    """A catalog leaves blocks and block words with its context; the allocation that fails after it takes them back first."""
    w = beam(lib_hook, 10.0, 45.0, 5.0, 16.0, 19.0, 0.2)
    for what in ("table", "generator"):
        ctx = G.Context(0)
        want = G.run_catalog(ctx, w)
        assert lib_hook.gf_debug_fail_allocations(0, 1) == 0
        if what == "table":
            G.DeviceTable(ctx, 1000, 5).free()
        else:
            # 3.5e6 pixels: more than any kept block holds, so that the first allocation is a new one
            big = beam(lib_hook, 10.0, 45.0, 5.0, 16.0, 19.0, 0.2)
            n = 3500000 // big.npixels
            big.pixels, big.ammin, big.npixels = bytearray(bytes(big.pixels) * n), np.tile(big.ammin, n), big.npixels * n
            G.Skygen(ctx, big).close()
        lib_hook.gf_debug_fail_allocations(-1, 0)
        got = G.run_catalog(ctx, w)
        assert list(got.generated[:3]) == list(want.generated[:3])
        ctx.close()
