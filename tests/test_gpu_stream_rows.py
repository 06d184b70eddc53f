"""The modules that draw from the streams (256 rows to a stream: Bond2010, the metallicities,
unresolved multiples), called on rows of the test's own, against the oracle: row counts
around a warp, a chunk and a run of uniforms, rows that draw nothing among the others,
mixed components, and stream states in and out of the range in which a stream can be
jumped ahead.  Draw positions and stream states must be equal; the columns are computed
with the same portable math, so they are too."""
import ctypes as C

import numpy as np
import pytest

import galfast_b200 as G
from galfast_b200 import _abi as A
from galfast_b200 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu

NS = 64
COLS = ["FeH", "FeH_comp", "vcyl", "absmag", "absmagSys", "absmagSysNcomp", "hidden"]


class DeviceColumn:
    def __init__(self, ptr, shape, dtype):
        self.__cuda_array_interface__ = {"data": (int(ptr), False), "shape": shape, "version": 3,
                                         "typestr": np.dtype(dtype).newbyteorder("<").str}


def columns(n, rng):
    """Rows of three components, some hidden."""
    D = 10.0 ** rng.uniform(1.5, 4.5, n)
    u = rng.normal(size=(3, n))
    host = G.HostTable(n, 0)
    a = host.arrays
    a["XYZ"][:] = (u / np.linalg.norm(u, axis=0) * D).astype(np.float32)
    a["absmag"][0] = rng.uniform(3, 15, n).astype(np.float32)
    a["comp"][0] = rng.integers(0, 4, n)          # component 3: in no module's mask
    a["hidden"][0] = rng.uniform(size=n) < 0.2
    host.t.size = n
    return host


def states(kind, multipliers, rng):
    st = O.seed_streams(int(rng.integers(1, 1 << 31)), multipliers, NS).reshape(3, NS).copy()
    if kind == "outside":
        # multipliers below and above the jump's range, carries at and above the multiplier
        st[0, ::4] = 13
        st[1, ::4] = rng.integers(1, 12, len(st[1, ::4]))
        st[0, 1::4] = 0xfffffff5
        st[0, 2::4] = 701
        st[1, 2::4] = 802
    return np.ascontiguousarray(st.reshape(-1))


@pytest.mark.parametrize("kind", ["seeded", "outside"])
@pytest.mark.parametrize("begin,n", [(0, 1), (3, 31), (0, 255), (0, 256), (5, 257), (0, 1000), (0, 8191)])
def test_rows_that_draw_from_streams_equal_oracle(ctx, lib, multipliers, kind, begin, n):
    import torch
    rng = np.random.default_rng(1000 * n + begin + (kind == "outside"))
    end = begin + n
    host = columns(end, rng)
    state = states(kind, multipliers, rng)
    L = O.load("p")
    modules = [("gf_module_feh", L.or_module_feh, W.feh_config()),
               ("gf_module_gaussfeh", L.or_module_gaussfeh, W.gaussfeh_config(comp_mask=0b100)),
               ("gf_module_gaussfeh", L.or_module_gaussfeh, W.gaussfeh_config(mean=(-1.0,), sigma=(0.3,), wt=(1.0,), comp_mask=0b1)),
               ("gf_module_multiples", L.or_module_multiples, W.multiples_config(lib, algo=A.GF_MULT_LF_M2_GT_M1, comp_mask=0b011,
                                                                                 fraction=W.MULT_FRACTION, lf=W.MULT_LF)),
               ("gf_module_multiples", L.or_module_multiples, W.multiples_config(lib, algo=A.GF_MULT_EQUAL_MASS, comp_mask=0b100,
                                                                                 fraction=W.MULT_FRACTION)),
               ("gf_module_bond2010", L.or_module_bond2010, W.bond2010_config())]
    dev = G.DeviceTable(ctx, end, 0)
    try:
        for name in ("XYZ", "absmag", "comp", "hidden"):
            src = host.arrays[name]
            torch.as_tensor(DeviceColumn(getattr(dev.t, name), src.shape, src.dtype), device="cuda").copy_(torch.from_numpy(src))
        torch.cuda.synchronize()
        dev.t.size = end
        ctx.rng_init(1, NS)
        ctx.set_rng_state(state)
        for fn, orfn, cfg in modules:
            assert orfn(C.addressof(cfg), state.ctypes.data, NS, C.addressof(host.t), begin, end) == 0
            G.check(getattr(lib, fn)(ctx.h, C.byref(cfg), C.byref(dev.t), begin, end))
            assert np.array_equal(ctx.rng_state(), state), fn
            got = dev.download()
            for name in COLS:
                a, b = got.arrays[name][:, begin:end], host.arrays[name][:, begin:end]
                assert np.array_equal(a, b, equal_nan=a.dtype.kind == "f"), (fn, name)
    finally:
        dev.free()
