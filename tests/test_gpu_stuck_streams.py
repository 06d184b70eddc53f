"""Streams that never leave their state.  The two fixed points of a stream are refused where a caller
sets states; a module that meets such a stream all the same (a multiplier of 0 marks a stream that is
not used) gives up after a bounded number of pairs and reports it, and the context goes on."""
import ctypes as C

import numpy as np
import pytest

import galfast_b200 as G
from galfast_b200 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu

NS, N = 64, 2000
GF_E_INVALID, GF_E_TIMEOUT = -1, -4


@pytest.mark.parametrize("point", ["zero", "last"])
def test_fixed_points_are_refused(ctx, lib, multipliers, point):
    ctx.rng_init(5, NS)
    before = ctx.rng_state()
    st = before.reshape(3, NS).copy()
    st[1, 7], st[2, 7] = (0, 0) if point == "zero" else (st[0, 7] - 1, 0xffffffff)
    flat = np.ascontiguousarray(st.reshape(-1))
    ptr = flat.ctypes.data_as(C.POINTER(C.c_uint32))
    assert lib.gf_rng_set_state(ctx.h, ptr, NS) == GF_E_INVALID
    assert np.array_equal(ctx.rng_state(), before)
    one = (C.c_uint32 * 3)(*[int(v) for v in st[:, 7]])
    mu, out = (C.c_float * 1)(0.5), (C.c_uint32 * 1)()
    assert lib.gf_rng_poisson(ctx.h, one, mu, 1, out) == GF_E_INVALID
    # the neighbours of the fixed points are states like any other
    st[1, 7], st[2, 7] = (0, 1) if point == "zero" else (st[0, 7] - 1, 0xfffffffe)
    flat = np.ascontiguousarray(st.reshape(-1))
    assert lib.gf_rng_set_state(ctx.h, flat.ctypes.data_as(C.POINTER(C.c_uint32)), NS) == 0


def test_a_stream_without_accepted_pairs_is_reported(ctx, lib, multipliers):
    dev, cfg = G.DeviceTable(ctx, N, 0), W.bond2010_config()
    try:
        ctx.rng_init(9, NS)
        good = ctx.rng_state()
        st = good.reshape(3, NS).copy()
        st[:, 3] = 0
        ctx.set_rng_state(np.ascontiguousarray(st.reshape(-1)))
        dev.t.size = N
        # rows at the origin's distance: what matters is which streams are drawn from
        host = G.HostTable(N, 0)
        host.arrays["XYZ"][:] = 100.0
        import torch
        for name, ncomp in (("XYZ", 3), ("comp", 1), ("hidden", 1)):
            a = host.arrays[name]
            src = torch.from_numpy(np.ascontiguousarray(a)).cuda()
            col = torch.as_tensor(_Column(getattr(dev.t, name), a.shape, a.dtype), device="cuda")
            col.copy_(src)
        torch.cuda.synchronize()
        assert lib.gf_module_bond2010(ctx.h, C.byref(cfg), C.byref(dev.t), 0, N) == 0
        assert lib.gf_ctx_sync(ctx.h) == GF_E_TIMEOUT
        assert lib.gf_ctx_sync(ctx.h) == 0
        # the other streams' rows and states are the oracle's; with the states set again all are
        full = good.copy()
        assert O.load("p").or_module_bond2010(C.addressof(cfg), full.ctypes.data, NS, C.addressof(host.t), 0, N) == 0
        got = dev.download().arrays["vcyl"]
        drawn = np.r_[0:768, 1024:N]
        assert np.array_equal(got[:, drawn], host.arrays["vcyl"][:, drawn])
        now, others = ctx.rng_state().reshape(3, NS), np.arange(NS) != 3
        assert np.array_equal(now[:, others], full.reshape(3, NS)[:, others]) and not now[:, 3].any()
        ctx.set_rng_state(good)
        G.check(lib.gf_module_bond2010(ctx.h, C.byref(cfg), C.byref(dev.t), 0, N))
        assert np.array_equal(ctx.rng_state(), full)
        assert np.array_equal(dev.download().arrays["vcyl"], host.arrays["vcyl"])
    finally:
        dev.free()


class _Column:
    def __init__(self, ptr, shape, dtype):
        self.__cuda_array_interface__ = {"data": (int(ptr), False), "shape": shape, "version": 3,
                                         "typestr": np.dtype(dtype).newbyteorder("<").str}
