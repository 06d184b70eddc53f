"""The expected counts of a generator (gf_skygen_integrate) with 25 million bins a model and more, which
take the pixel-by-pixel integrate.  The totals and the sum of the pixels' covered counts equal the
oracle's per-stream sums to 1e-12 (the same bins; FP64 additions in another order); a pixel's covered
count equals the oracle's, which adds the ten bins of a block in float (10 x 2^-24), to 1e-6.  The
last case lies just below that number of bins."""
import numpy as np
import pytest

import galfast_b200 as G
from oracle import oracle as O
from test_gpu_integrate_pixels import beam

pytestmark = pytest.mark.gpu

CASES = {
    "plain": (lambda lib: beam(lib, 10.0, 45.0, 5.0, 16.0, 19.0, 0.2), True),
    "cuts": (lambda lib: beam(lib, 30.0, 7.0, 5.0, 16.0, 19.0, 0.2, ext_E=0.12), True),
    "distances": (lambda lib: beam(lib, 60.0, 35.0, 5.0, 16.0, 19.0, 0.2, dmin=300.0, dmax=4000.0), True),
    "few_rows": (lambda lib: beam(lib, 75.0, 20.0, 8.6, 20.0, 20.25, 0.1), True),
    "fewer_bins": (lambda lib: beam(lib, 10.0, 45.0, 4.3, 16.0, 19.0, 0.2), False),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_pixel_counts_equal_oracle(ctx, lib, name):
    make, many = CASES[name]
    w = make(lib)
    sky, want = G.Skygen(ctx, w), O.OracleSkygen(w)
    assert (w.npixels * sky.info(0).nm * sky.info(0).nM >= 25000000) == many
    for i in range(len(w.models)):
        e, ec, pp = sky.integrate_counts(i, per_pixel=True)
        oe, oc, op = want.integrate_counts(i, per_pixel=True)
        assert e == pytest.approx(oe, rel=1e-12) and ec == pytest.approx(oc, rel=1e-12), i
        np.testing.assert_allclose(pp, op, rtol=1e-6)
        assert pp.sum() == pytest.approx(oc, rel=1e-12), i
        assert sky.integrate_counts(i)[0] == pytest.approx(e, rel=1e-14)
