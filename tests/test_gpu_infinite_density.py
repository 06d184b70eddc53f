"""Requests whose expected counts are no numbers: a density that overflows to infinity, over a luminosity
function with zero rows (infinity times zero).  Such a request does not reach the batched draw; it is
refused with GF_E_INVALID where a bin with stars has an infinite count, on the single and on the
many-request path, and where every product is no number it has no stars, as on the CPU path."""
import ctypes as C

import numpy as np
import pytest

import galfast_b200 as G
from galfast_b200 import _abi as A
from galfast_b200 import workloads as W

pytestmark = pytest.mark.gpu

GF_E_INVALID = -1
OVERFLOWS = 2e38           # times the disk's normalisation (about e^3)


def request(lib, half_deg, zero_knots):
    """A square about the pole; the thin disk's luminosity function is zero in its first knots."""
    half = np.deg2rad(half_deg)
    foot = A.Footprint()
    foot.kind, foot.proj = A.GF_FOOT_LAMBERT_RECT, 0
    foot.a, foot.b, foot.c, foot.d = -half, half, -half, half
    w = W.build_workload(lib, foot=foot, dx_deg=0.25, m0=15.0, m1=20.0, capacity=1 << 20, with_modules=False)
    M, phi = W.lf_table()
    phi = phi.copy()
    phi[:zero_knots] = 0.0
    w.keep += [M, phi]
    w.models[0].f = OVERFLOWS
    w.models[0].lf_M, w.models[0].lf_phi = (v.ctypes.data_as(C.POINTER(C.c_double)) for v in (M, phi))
    w.models[0].lf_n = len(M)
    return w


def rows(ctx, ws, multi):
    got = {}
    if multi:
        G.run_catalog_multi(ctx, ws, sink=lambda j, m, r: got.setdefault((j, m), []).append(r["lb"].copy()))
    else:
        for j, w in enumerate(ws):
            G.run_catalog(ctx, w, sink=lambda m, t, off, j=j: got.setdefault((j, m), []).append(t.as_dict(["lb"])["lb"]))
    return {k: np.concatenate(v, axis=-1) for k, v in got.items() if sum(x.shape[-1] for x in v)}


@pytest.mark.parametrize("half_deg", [1.0, 5.0])       # the crawl, and block words over 3.8e7 bins a model
def test_infinite_counts_are_refused(ctx, lib, half_deg):
    w = request(lib, half_deg, 30)
    e, _, _ = G.Skygen(ctx, w).integrate_counts(0)
    assert np.isnan(e)
    job = w.job(G.Job)
    assert lib.gf_catalog_run(ctx.h, C.byref(job), G.BatchCallback(), None, None) == GF_E_INVALID
    fine = request(lib, 1.0, 0)
    fine.models[0].f = 1.0
    jobs = (G.Job * 2)(fine.job(G.Job), job)
    assert lib.gf_catalog_run_multi(ctx.h, jobs, 2, G.MultiCallback(), None, None) == GF_E_INVALID
    # the context goes on
    a, b = rows(ctx, [fine, fine], True), rows(ctx, [fine, fine], False)
    assert sorted(a) == sorted(b) and len(a) == 6 and all(np.array_equal(a[k], b[k]) for k in a)


@pytest.mark.parametrize("half_deg", [1.0, 5.0])
def test_counts_that_are_no_numbers_draw_nothing(ctx, lib, half_deg):
    w = request(lib, half_deg, 1000)
    fine = request(lib, 1.0, 0)
    fine.models[0].f = 1.0
    a, b = rows(ctx, [fine, w], True), rows(ctx, [fine, w], False)
    assert sorted(a) == sorted(b) == [(0, 0), (0, 1), (0, 2), (1, 1), (1, 2)]
    assert all(np.array_equal(a[k], b[k]) for k in a)
