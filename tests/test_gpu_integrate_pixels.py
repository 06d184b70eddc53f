"""The pixel-by-pixel integrate, where it can go wrong: fewer pixels than a warp's 64 and just
more, a single partly covered pixel, grids of few and many magnitude rows, cuts that differ
within a group, distance limits, a negative density, and luminosity functions with zero rows
(their bins take the general conversion).  Totals and covered totals equal the oracle's per-stream
sums to 1e-12 (the same bins; FP64 additions in another order: at most a few 1e-13)."""
import numpy as np
import pytest

import galfast_b200 as G
from galfast_b200 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def beam(lib, l, b, r, m0, m1, dx, dmin=0.0, dmax=0.0, f=None, zero_lf=False, **kw):
    w = W.build_workload(lib, foot=W.cap_footprint(l, b, r), dx_deg=dx, m0=m0, m1=m1, seed48=5, capacity=1 << 18, **kw)
    w.sky.dmin, w.sky.dmax = dmin, dmax
    for i, v in enumerate(f or ()):
        w.models[i].f = v
    if zero_lf:
        import ctypes as C
        M, phi = W.lf_table()
        phi = np.where((M > 6.0) & (M < 8.0), 0.0, phi)
        w.keep += [M, phi]
        for m in w.models:
            m.lf_M = M.ctypes.data_as(C.POINTER(C.c_double))
            m.lf_phi = phi.ctypes.data_as(C.POINTER(C.c_double))
    return w


CASES = {
    "one_pixel": lambda lib: beam(lib, 10.0, 60.0, 0.05, 17.0, 19.0, 0.2),
    "pixels_60": lambda lib: beam(lib, 10.0, 60.0, 0.8, 17.0, 19.0, 0.2),
    "pixels_70": lambda lib: beam(lib, 10.0, 60.0, 0.87, 17.0, 18.0, 0.2),
    "pixels_350": lambda lib: beam(lib, 10.0, 45.0, 2.0, 17.0, 17.5, 0.2),
    "few_rows": lambda lib: beam(lib, 75.0, 20.0, 1.5, 20.0, 20.25, 0.2),
    "more_m_than_M_rows": lambda lib: beam(lib, 75.0, 40.0, 0.5, 10.0, 24.0, 0.2, M0=5.0, M1=9.0),
    "cuts": lambda lib: beam(lib, 30.0, 7.0, 2.0, 16.0, 19.0, 0.2, ext_E=0.12),
    "distances": lambda lib: beam(lib, 60.0, 35.0, 1.0, 16.0, 19.0, 0.2, dmin=300.0, dmax=4000.0),
    "negative": lambda lib: beam(lib, 60.0, 35.0, 0.8, 17.0, 19.0, 0.2, f=(1.0, -0.12, 0.005)),
    "zero_lf": lambda lib: beam(lib, 60.0, 35.0, 0.8, 17.0, 19.0, 0.2, zero_lf=True),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_expected_counts_equal_oracle(ctx, lib, name):
    w = CASES[name](lib)
    stats = G.run_catalog_multi(ctx, [w], sink=lambda *a: 0)[0]
    sky = O.OracleSkygen(w)
    for i in range(len(w.models)):
        e, ec, _ = sky.integrate_counts(i)
        assert stats.expected[i] == pytest.approx(e, rel=1e-12), i
        assert stats.expected_covered[i] == pytest.approx(ec, rel=1e-12), i
