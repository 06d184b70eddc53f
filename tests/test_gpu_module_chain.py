"""The postprocessing modules over as many rows and streams as a large batch has, on contexts of their
own (so that the tables of stream powers are made anew), against the oracle: the whole chain on 4000003
rows, and the modules that draw on some rows of every stream, with a warp and with a thread to a chunk of 256
rows.  Stream states and columns must be equal bit for bit (the same portable math on both sides)."""
import ctypes as C

import numpy as np
import pytest

import galfast_b200 as G
from galfast_b200 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu

NS = 65536


class DeviceColumn:
    def __init__(self, ptr, shape, dtype, pitch):
        item = np.dtype(dtype).itemsize
        self.__cuda_array_interface__ = {"data": (int(ptr), False), "shape": shape, "version": 3, "strides": (pitch * item, item),
                                         "typestr": np.dtype(dtype).newbyteorder("<").str}


def column(table, host, name):
    import torch
    a = host.arrays[name]
    return torch.as_tensor(DeviceColumn(getattr(table, name), a.shape, a.dtype, int(table.capacity)), device="cuda")


def upload(dev, host, names):
    import torch
    for name in names:
        column(dev.t, host, name).copy_(torch.from_numpy(host.arrays[name]))
    torch.cuda.synchronize()
    dev.t.size = host.t.size = host.capacity


def stars(n, nbands, l0, b0, seed):
    """Rows of one component in a 10 deg field, 14 < r < 24, under a csc|b| screen."""
    rng = np.random.default_rng(seed)
    host = G.HostTable(n, nbands)
    a = host.arrays
    l, b = np.sort(rng.uniform(l0 - 5, l0 + 5, n)), rng.uniform(b0 - 5, b0 + 5, n)
    M = rng.uniform(3, 15, n)
    DM = rng.uniform(14, 24, n) - M
    D = 10.0 ** (0.2 * DM + 1.0)
    lr, br = np.deg2rad(l), np.deg2rad(b)
    a["lb"][:] = l, b
    a["absmag"][0], a["DM"][0] = M, DM
    a["XYZ"][:] = D * np.cos(lr) * np.cos(br), D * np.sin(lr) * np.cos(br), D * np.sin(br)
    a["Am"][0] = a["AmInf"][0] = 0.05 / np.sin(br)
    return host


def test_chain_on_four_million_rows_equals_oracle(lib, multipliers):
    n, nb, l0, b0 = 4000003, 6, 150.0, 35.0
    w = W.build_workload(lib, foot=W.cap_footprint(l0, b0, 4.9), dx_deg=1.0, m0=14.0, m1=24.0, nbands=nb, m5=W.LSST_M5, perr_seed=7)
    host = stars(n, nb, l0, b0, 11)
    state = O.seed_streams(123, multipliers, NS)
    ctx = G.Context(0)
    ph, pe = C.c_void_p(), C.c_void_p()
    dev = G.DeviceTable(ctx, n, nb)
    try:
        upload(dev, host, ["lb", "absmag", "DM", "XYZ", "Am", "AmInf", "comp", "hidden"])
        ctx.rng_init(123, NS)
        G.check(lib.gf_photometry_create(ctx.h, C.byref(w.phot), C.byref(ph)))
        G.check(lib.gf_photoerr_create(ctx.h, C.byref(w.perr), C.byref(pe)))
        t = C.byref(dev.t)
        G.check(lib.gf_module_clipper(ctx.h, C.byref(w.foot), w.sky.proj, t, 0, n))
        G.check(lib.gf_module_fixedfeh(ctx.h, C.byref(w.feh), t, 0, n))
        G.check(lib.gf_module_bond2010(ctx.h, C.byref(w.kin), t, 0, n))
        G.check(lib.gf_module_photometry(ctx.h, ph, t, 0, n))
        G.check(lib.gf_module_photoerrors(ctx.h, pe, 0, t, 0, n))
        G.check(lib.gf_module_vel2pm(ctx.h, C.byref(w.v2pm), t, 0, n))
        G.check(lib.gf_module_gal2other(ctx.h, w.gal2other, t, 0, n))
        ctx.sync()
        L, th = O.load("p"), C.addressof(host.t)
        L.or_set_threads(8)
        assert L.or_module_clipper(C.addressof(w.foot), None, th, 0, n) == 0
        assert L.or_module_fixedfeh(C.addressof(w.feh), th, 0, n) == 0
        assert L.or_module_bond2010(C.addressof(w.kin), state.ctypes.data, NS, th, 0, n) == 0
        assert L.or_module_photometry(C.addressof(w.phot), th, 0, n) == 0
        assert L.or_module_photoerrors(C.addressof(w.perr), 0, th, 0, n) == 0
        assert L.or_module_vel2pm(C.addressof(w.v2pm), th, 0, n) == 0
        assert L.or_module_gal2other(w.gal2other, th, 0, n) == 0
        assert np.array_equal(ctx.rng_state(), state)
        for name in ("hidden", "FeH", "vcyl", "mags", "photoflags", "obsmags", "pm", "radec"):
            got = column(dev.t, host, name).cpu().numpy()
            assert np.array_equal(got, host.arrays[name], equal_nan=got.dtype.kind == "f"), name
    finally:
        lib.gf_photometry_destroy(ph)
        lib.gf_photoerr_destroy(pe)
        dev.free()
        ctx.close()


@pytest.mark.parametrize("chunks", [30999, 44999, NS])       # a warp a chunk; the multiples, then all modules, a thread a chunk
def test_rows_of_every_stream_equal_oracle(lib, multipliers, chunks):
    """24 visible rows in each chunk of 256, of several components: the powers of every stream are used (a run is
    832 uniforms, the rows take some 200), the other rows stay as they are."""
    n = 256 * chunks - 5
    host = G.HostTable(n, 0)
    a = host.arrays
    rng = np.random.default_rng(3)
    a["hidden"][0] = 1
    rows = np.minimum(256 * np.arange(chunks)[:, None] + np.sort(rng.integers(0, 256, (chunks, 24)), axis=1), n - 1).ravel()
    a["hidden"][0, rows] = 0
    a["comp"][0, rows] = rng.integers(0, 4, len(rows))
    a["XYZ"][:, rows] = rng.normal(size=(3, len(rows))) * 3000.0
    a["absmag"][0, rows] = rng.uniform(3, 15, len(rows))
    L = O.load("p")
    modules = [("gf_module_feh", L.or_module_feh, W.feh_config()), ("gf_module_gaussfeh", L.or_module_gaussfeh, W.gaussfeh_config(comp_mask=0b100)),
               ("gf_module_multiples", L.or_module_multiples, W.multiples_config(lib, comp_mask=0b011, fraction=W.MULT_FRACTION, lf=W.MULT_LF)),
               ("gf_module_bond2010", L.or_module_bond2010, W.bond2010_config())]
    state = O.seed_streams(77, multipliers, NS)
    ctx = G.Context(0)
    dev = G.DeviceTable(ctx, n, 0)
    try:
        upload(dev, host, ["hidden", "comp", "XYZ", "absmag"])
        ctx.rng_init(77, NS)
        for fn, orfn, cfg in modules:
            G.check(getattr(lib, fn)(ctx.h, C.byref(cfg), C.byref(dev.t), 0, n))
            assert orfn(C.addressof(cfg), state.ctypes.data, NS, C.addressof(host.t), 0, n) == 0
            assert np.array_equal(ctx.rng_state(), state), fn
        for name in ("FeH", "FeH_comp", "absmag", "absmagSys", "absmagSysNcomp", "vcyl"):
            got = column(dev.t, host, name).cpu().numpy()
            assert np.array_equal(got, a[name], equal_nan=got.dtype.kind == "f"), name
    finally:
        dev.free()
        ctx.close()
