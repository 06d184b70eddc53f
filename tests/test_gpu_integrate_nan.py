"""Expected counts that are no positive numbers, in the pixel-by-pixel integrate: densities that are none in some pixels
and rows of a luminosity function that are none, and factors of both signs.  The same pixels as on the CPU path have no number, and the others
its counts."""
import ctypes as C

import numpy as np
import pytest

import galfast_b200 as G
from galfast_b200 import _abi as A
from galfast_b200 import workloads as W
from oracle import oracle as O
from test_gpu_integrate_pixels import beam
from test_gpu_parity import draw_all

pytestmark = pytest.mark.gpu


def counts(ctx, w, model):
    sky, osk = G.Skygen(ctx, w), O.OracleSkygen(w)
    assert w.npixels >= 512 and w.npixels * sky.info(model).nm * sky.info(model).nM >= 25000000
    return sky.integrate_counts(model, per_pixel=True), osk.integrate_counts(model, per_pixel=True)


def assert_same(got, want):
    (e, ec, pp), (oe, oc, op) = got, want
    assert np.array_equal(np.isnan(pp), np.isnan(op))
    fine = ~np.isnan(op)
    np.testing.assert_allclose(pp[fine], op[fine], rtol=1e-6)
    assert np.isnan(e) == np.isnan(oe) and np.isnan(ec) == np.isnan(oc)


# whole runs of ten bins, and a grid of five rows, whose runs are all shorter
GRIDS = {"deep": (180.0, 45.0, 5.0, 16.0, 19.0, 0.2), "few_rows": (180.0, 20.0, 8.6, 20.0, 20.25, 0.1)}


@pytest.mark.parametrize("grid", sorted(GRIDS))
def test_densities_that_are_no_numbers(ctx, lib, grid):
    """A bulge whose index is no integer: the density is none where the second coordinate of its frame is negative."""
    w = beam(lib, *GRIDS[grid])
    m = w.models[2]
    m.type, m.n, m.l, m.ba, m.ca, m.f = A.GF_MODEL_LCBULGE, 1.3, 2000.0, 1.0, 1.0, 0.01
    got, want = counts(ctx, w, 2)
    assert 0.2 < np.isnan(want[2]).mean() < 0.8
    assert_same(got, want)


@pytest.mark.parametrize("grid", sorted(GRIDS))
@pytest.mark.parametrize("knots", [(40, 42), (119, 121)])
def test_luminosity_functions_that_are_no_numbers(ctx, lib, grid, knots):
    w = beam(lib, *GRIDS[grid])
    M, phi = W.lf_table()
    phi = phi.copy()
    phi[slice(*knots)] = np.nan
    w.models[1].lf_M, w.models[1].lf_phi = (v.ctypes.data_as(C.POINTER(C.c_double)) for v in (M, phi))
    got, want = counts(ctx, w, 1)
    assert np.isnan(want[0]) and np.isnan(want[2]).any()         # (pixels whose rows are all cut have 0)
    assert_same(got, want)


def test_bins_without_a_number_draw_nothing(ctx, lib, multipliers):
    """Every batch and stream state equals the CPU path's: such a bin takes its uniform and has no stars."""
    w = beam(lib, 180.0, 45.0, 5.0, 16.0, 19.0, 0.2)
    m = w.models[2]
    m.type, m.n, m.l, m.ba, m.ca, m.f = A.GF_MODEL_LCBULGE, 1.3, 2000.0, 1.0, 1.0, 1e-6
    _, total = draw_all(ctx, w, multipliers, 20000)
    assert total > 10000


@pytest.mark.parametrize("grid", sorted(GRIDS))
def test_negative_densities_over_luminosity_functions_of_both_signs(ctx, lib, grid):
    """Products of two negative factors are among the bins, beside negative ones."""
    w = beam(lib, *GRIDS[grid])
    M, phi = W.lf_table()
    phi = phi * np.where(M < 9.0, -1.0, 0.5)
    w.models[1].lf_M, w.models[1].lf_phi = (v.ctypes.data_as(C.POINTER(C.c_double)) for v in (M, phi))
    w.models[1].f = -0.12
    (e, ec, pp), (oe, oc, op) = counts(ctx, w, 1)
    # sums with cancellation: a part in 1e6 of what the same grid counts with positive factors
    w.models[1].f = 0.12
    phi[:] = np.abs(phi)
    sky = G.Skygen(ctx, w)
    pe, pc, ppos = sky.integrate_counts(1, per_pixel=True)
    assert np.all(np.abs(pp - op) <= 1e-6 * ppos)
    assert abs(e - oe) <= 1e-11 * pe and abs(ec - oc) <= 1e-11 * pc
