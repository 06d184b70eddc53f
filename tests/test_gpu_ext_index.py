"""Requests whose pixels name a beam extinction that is not there are refused on the host, whatever kind of
extinction they say they have."""
import ctypes as C

import pytest

import galfast_b200 as G
from galfast_b200 import _abi as A
from galfast_b200 import workloads as W

pytestmark = pytest.mark.gpu

GF_E_INVALID = -1


@pytest.mark.parametrize("index", [-1, 1 << 30])
@pytest.mark.parametrize("kind", [A.GF_EXT_SCREEN_CSCB, 7])
def test_extinction_indexes_out_of_range_are_refused(ctx, lib, kind, index):
    w = W.build_workload(lib, foot=W.cap_footprint(60.0, 40.0, 0.5), dx_deg=0.1, m0=16.0, m1=19.0, with_modules=False)
    pix = (G.PencilBeam * w.npixels).from_buffer_copy(w.pixels)
    pix[w.npixels - 1].extIdx = index
    job = w.job(G.Job)
    job.ext.kind = kind
    job.pixels = C.cast(pix, C.POINTER(G.PencilBeam))
    jobs = (G.Job * 2)(w.job(G.Job), job)
    assert lib.gf_catalog_run_multi(ctx.h, jobs, 2, G.MultiCallback(), None, None) == GF_E_INVALID
    assert lib.gf_catalog_run(ctx.h, C.byref(job), G.BatchCallback(), None, None) == GF_E_INVALID
