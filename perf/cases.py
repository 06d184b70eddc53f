"""The work that users of galfast_b200 have it do, as cases that can be timed.

Every case goes through the package's public entry points: one request at a time
(gf_catalog_run), many requests per pass (gf_catalog_run_multi, kept on the device, and
gf_catalog_run_multi_host), the expected counts of a footprint (gf_skygen_integrate) and the
postprocessing modules on rows that the caller holds (gf_module_*).  Sizes are those of the
configurations in galfast_b200/workloads.py and of the tests, from a half-degree pencil beam
to a few hundred beams together and a survey stripe of many output batches.

A case fixes what is asked for: the footprints, the magnitude limits, the pixels.  The seed
gives the models' parameters, the random streams and the rows.  A catalog is kept as a
program keeps it, in columns of the caller's that hold the rows as they come.
"""
import ctypes as C
import math
import weakref

import numpy as np
import torch

import galfast_b200 as G
from galfast_b200 import _abi as A
from galfast_b200 import workloads as W

D2R = math.pi / 180.0
# what a catalog's user keeps of each row
CATALOG = ["comp", "radec", "DM", "absmag", "mags", "obsmags", "vcyl", "pm"]
COLUMN = {name: (dt, ncomp) for name, dt, ncomp in G.COLUMNS}
TYPESTR = {np.float64: "<f8", np.float32: "<f4", np.int32: "<i4"}
TORCH = {np.float64: torch.float64, np.float32: torch.float32, np.int32: torch.int32}
RG, Z0 = 8000.0, 25.0


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # one small pencil beam, read back to the host: a request where set-up and launches count
        {"name": "cap_single", "kind": "request", "area": "cap", "l": 75.0, "b": 40.0, "size": 0.7, "dx": 0.1, "m0": 14.0,
         "m1": 20.0, "capacity": 1 << 20, "sink": "host", "options": "plain"},
        # configuration 1: 10 x 10 deg at the galactic pole, 0.25 deg pixels, 15 < r < 21
        {"name": "patch_100deg2", "kind": "request", "area": "patch", "l": 0.0, "b": 90.0, "size": 5.0, "dx": 0.25, "m0": 15.0,
         "m1": 21.0, "capacity": 1 << 20, "sink": "host", "options": "plain"},
        # configuration 2's form on a stripe of the sky: one large request that fills several output batches
        {"name": "survey_stripe", "kind": "request", "area": "stripe", "l": 100.0, "b": 38.0, "size": 30.0, "dx": 0.1, "m0": 14.0,
         "m1": 22.0, "capacity": 1 << 19, "sink": "device", "options": "plain"},
        # 3-D extinction maps, a density cube, metallicity and unresolved multiples: the options together
        {"name": "maps_cube_multiples", "kind": "request", "area": "patch", "l": 0.0, "b": 90.0, "size": 4.0, "dx": 0.2, "m0": 15.0,
         "m1": 21.0, "capacity": 1 << 20, "sink": "device", "options": "maps"},
        # configuration 4, the batched form: a handful of beams, an ordinary batch, a large one
        {"name": "beams_8", "kind": "beams", "first": 0, "requests": 8, "sink": "device"},
        {"name": "beams_64", "kind": "beams", "first": 0, "requests": 64, "sink": "device"},
        {"name": "beams_256", "kind": "beams", "first": 0, "requests": 256, "sink": "device"},
        # the same delivered to host memory
        {"name": "beams_24_to_host", "kind": "beams", "first": 64, "requests": 24, "sink": "host"},
        # configuration 5's requests: caps and rectangles, deep, ugriz and ugrizy mixed
        {"name": "served_12", "kind": "served", "stream": 99, "requests": 12, "area_max": 120.0, "sink": "device"},
        # expected counts of every pixel, without drawing (planning a run)
        {"name": "expected_counts", "kind": "counts", "area": "patch", "l": 0.0, "b": 90.0, "size": 7.0, "dx": 0.1, "m0": 14.0,
         "m1": 22.0, "options": "plain"},
        # the postprocessing modules on rows that the caller holds on the device
        {"name": "modules_20k", "kind": "modules", "rows": 20001, "nbands": 5, "comp": 2},
        {"name": "modules_4m", "kind": "modules", "rows": 4000003, "nbands": 6, "comp": 0},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    """One more case of the same ranges, each kind about as often as the list has it."""
    kind = rng.choice(["request", "request", "request", "options", "beams", "beams", "beams", "to_host", "served",
                       "counts", "modules", "modules"])
    if kind == "request":
        area = rng.choice(["cap", "patch", "stripe"])
        size = _log(rng, 0.5, 6.0) if area == "cap" else _log(rng, 1.0, 5.0) if area == "patch" else _log(rng, 3.0, 28.0)
        south = rng.choice([-1.0, 1.0])
        return {"kind": "request", "area": area, "l": round(rng.uniform(40.0, 320.0), 2),
                "b": round(south * (90.0 if area == "patch" else rng.uniform(30.0, 60.0)), 2), "size": round(size, 3),
                "dx": rng.choice([0.1, 0.2, 0.25]), "m0": rng.choice([14.0, 15.0]), "m1": round(rng.uniform(19.0, 22.0), 2),
                "capacity": int(_log(rng, 2e5, 4e6)), "sink": rng.choice(["host", "device"]), "options": "plain"}
    if kind == "options":
        return {"kind": "request", "area": "patch", "l": 0.0, "b": rng.choice([-90.0, 90.0]), "size": round(_log(rng, 1.0, 4.0), 3),
                "dx": rng.choice([0.2, 0.25]), "m0": 15.0, "m1": round(rng.uniform(19.5, 21.0), 2), "capacity": 1 << 20,
                "sink": "device", "options": "maps"}
    if kind == "beams":
        return {"kind": "beams", "first": rng.randint(300, 3800), "requests": int(_log(rng, 1.0, 200.0)), "sink": "device"}
    if kind == "to_host":
        return {"kind": "beams", "first": rng.randint(300, 3800), "requests": int(_log(rng, 2.0, 32.0)), "sink": "host"}
    if kind == "served":
        return {"kind": "served", "stream": rng.randint(100, 10000), "requests": rng.randint(2, 12),
                "area_max": round(_log(rng, 10.0, 120.0), 1), "sink": "device"}
    if kind == "counts":
        return {"kind": "counts", "area": "patch", "l": 0.0, "b": rng.choice([-90.0, 90.0]), "size": round(_log(rng, 0.5, 7.0), 3),
                "dx": rng.choice([0.1, 0.2]), "m0": 14.0, "m1": round(rng.uniform(19.0, 23.0), 2), "options": "plain"}
    return {"kind": "modules", "rows": int(_log(rng, 1e3, 4e6)), "nbands": rng.choice([5, 6]), "comp": rng.choice([0, 1, 2])}


# ---------------------------------------------------------------------------
# what a program has in hand: the library context, its requests, its catalog
# ---------------------------------------------------------------------------
_shared = None


def _context():
    """A program keeps one context for its requests: the one in use, or a new one."""
    global _shared
    ctx = _shared() if _shared is not None else None
    if ctx is None:
        ctx = G.Context(0)
        _shared = weakref.ref(ctx)
    return ctx


def _footprint(case):
    size = case["size"]
    if case["area"] == "cap":
        return W.cap_footprint(case["l"], case["b"], size)
    if case["area"] == "stripe":                # 2 size by size / 2 deg in galactic longitude and latitude
        return W.lb_rect_footprint(case["l"], case["l"] + 2 * size, case["b"] - size / 4, case["b"] + size / 4)
    foot = A.Footprint()                        # 2 size by 2 size about a galactic pole
    foot.kind = A.GF_FOOT_LAMBERT_RECT
    foot.proj = 0 if case["b"] > 0 else 1
    foot.a, foot.b, foot.c, foot.d = -size * D2R, size * D2R, -size * D2R, size * D2R
    return foot


def _variation(rng):
    """What the seed gives a request: the thin disk's height, the halo's axis ratio, its streams."""
    return dict(thin_h=float(rng.uniform(250, 350)), halo_q=float(rng.uniform(0.55, 0.75)),
                seed48=int(rng.integers(1, 1 << 31)), perr_seed=int(rng.integers(1, 1 << 31)))


def _request(case, seed):
    rng = np.random.default_rng(1000003 * seed + 17)
    L = G.lib()
    w = W.build_workload(L, foot=_footprint(case), dx_deg=case["dx"], m0=case["m0"], m1=case["m1"],
                         capacity=case.get("capacity", 1 << 20), **_variation(rng))
    if case["options"] == "maps":
        W.use_extinction_maps(L, w)
        w.models[1] = W.density_cube_model(1, f=0.12 * math.exp(RG / 2600.0), lf=W.lf_table(), keep=w.keep)
        w.feh, w.feh_ivezic = None, W.feh_config()
        w.multiples = W.multiples_config(L, fraction=W.MULT_FRACTION, lf=W.MULT_LF)
    return w


def _parameters(case):
    """The footprints of a case of many requests: lists of (l, b, deg^2, pixels, r limit) and their parameters."""
    if case["kind"] == "beams":
        reqs = W.config4_requests(case["first"] + case["requests"])[case["first"]:]
    else:
        reqs = W.config5_requests(case["requests"], 1000.0, seed=case["stream"], area=(1.0, case["area_max"]), rmax=(20.0, 24.0))
    where = [(q["l"], q["b"], q.get("area", math.pi * q.get("r", 0.0) ** 2), q["rmax"]) for q in reqs]
    return reqs, where


def _requests(case, seed):
    rng = np.random.default_rng(1000003 * seed + 29)
    reqs, _ = _parameters(case)
    vary = [_variation(rng) for _ in reqs]
    L = G.lib()
    if case["kind"] == "beams":
        return W.config4_workloads(L, [dict(q, h=v["thin_h"], q=v["halo_q"], seed48=v["seed48"], perr_seed=v["perr_seed"])
                                       for q, v in zip(reqs, vary)], capacity=1 << 24)
    return W.config5_workloads(L, [dict(q, seed48=v["seed48"], perr_seed=v["perr_seed"]) for q, v in zip(reqs, vary)])


class _Device:
    """Device memory of the library, as torch.as_tensor reads it; it holds its owner while a tensor does."""

    def __init__(self, ptr, shape, dtype, pitch, owner):
        item = np.dtype(dtype).itemsize
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (int(ptr), False), "shape": shape, "typestr": TYPESTR[dtype], "version": 3,
                                         "strides": None if len(shape) == 1 else (pitch * item, item)}


def _width(table, name):
    dt, ncomp = COLUMN[name]
    return int(table.nbands) if ncomp == "bands" else ncomp


def _column(table, name, rows, owner=None):
    """The first `rows` rows of a column of a device table: (rows,) or (components, rows)."""
    k = _width(table, name)
    shape = (rows,) if k == 1 else (k, rows)
    return torch.as_tensor(_Device(getattr(table, name), shape, COLUMN[name][0], int(table.capacity), owner), device="cuda")


class _Catalog:
    """The caller's columns, on the device or in host memory, with room for about 1.6 times the expected rows."""

    def __init__(self, case, nbands):
        self.room = int(1.6 * _expected_rows(case)) + 20000
        self.device = case["sink"] == "device"
        self.col = {}
        for name in CATALOG:
            dt, ncomp = COLUMN[name]
            shape = (nbands if ncomp == "bands" else ncomp, self.room)
            self.col[name] = torch.zeros(shape, dtype=TORCH[dt], device="cuda") if self.device else np.zeros(shape, dtype=dt)
        self.rows = 0

    def _place(self, rows):
        if self.rows + rows > self.room:
            raise RuntimeError("more rows than the catalog has room for")
        at = self.rows
        self.rows += rows
        return slice(at, at + rows)

    def from_device(self, table, rows):
        """Rows of a device table, copied before the library goes on with it."""
        at = self._place(rows)
        for name in CATALOG:
            k = _width(table, name)
            if self.device:
                self.col[name][:k, at].copy_(_column(table, name, rows).view(k, rows) if k == 1 else _column(table, name, rows))
        torch.cuda.current_stream().synchronize()

    def from_host(self, table, rows):
        """Rows of a table in host memory."""
        at = self._place(rows)
        pitch = int(table.capacity)
        for name in CATALOG:
            k, ct = _width(table, name), np.ctypeslib.as_ctypes_type(COLUMN[name][0])
            src = np.ctypeslib.as_array(C.cast(getattr(table, name), C.POINTER(ct)), shape=(k * pitch,)).reshape(k, pitch)
            self.col[name][:k, at] = src[:, :rows]


# ---------------------------------------------------------------------------
# rows for the modules
# ---------------------------------------------------------------------------
def _rows(case, seed):
    """Stars of one component as the generator leaves them: positions in a 10 deg field ordered by
    longitude, magnitudes 14 < r < 24 and the extinction of a csc|b| screen."""
    g = torch.Generator(device="cuda").manual_seed(seed * 7919 + 5)
    n = case["rows"]

    def u(lo, hi):
        return torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * (hi - lo) + lo

    l0, b0 = 20.0 + 13.0 * (seed % 23), 35.0
    l = torch.sort(u(l0 - 5.0, l0 + 5.0)).values
    b = u(b0 - 5.0, b0 + 5.0)
    M = u(3.0, 15.0).float()
    DM = (u(14.0, 24.0) - M.double()).float()
    D = 10.0 ** (0.2 * DM.double() + 1.0)
    lr, br = l * D2R, b * D2R
    xyz = torch.stack([D * torch.cos(lr) * torch.cos(br), D * torch.sin(lr) * torch.cos(br), D * torch.sin(br)]).float()
    Am = (0.05 / torch.sin(br).abs()).float()
    return {"lb": torch.stack([l, b]), "absmag": M, "DM": DM, "XYZ": xyz, "Am": Am, "l0": l0, "b0": b0}


def _prepare_modules(case, seed):
    L, ctx = G.lib(), G.Context(0)
    rows, nb, n = _rows(case, seed), case["nbands"], case["rows"]
    w = W.build_workload(L, foot=W.cap_footprint(rows["l0"], rows["b0"], 4.9), dx_deg=1.0, m0=14.0, m1=24.0, nbands=nb,
                         m5=W.SDSS_M5 if nb == 5 else W.LSST_M5, perr_seed=seed + 1)
    t = G.DeviceTable(ctx, n, nb)
    for name in ("lb", "absmag", "DM", "XYZ", "Am"):
        _column(t.t, name, n).copy_(rows[name])
    _column(t.t, "AmInf", n).copy_(rows["Am"])
    _column(t.t, "comp", n).fill_(case["comp"])
    _column(t.t, "hidden", n).zero_()
    t.t.size = n
    ctx.rng_init(seed * 31 + 7, 65536)
    ph, pe = C.c_void_p(), C.c_void_p()
    G.check(L.gf_photometry_create(ctx.h, C.byref(w.phot), C.byref(ph)))
    G.check(L.gf_photoerr_create(ctx.h, C.byref(w.perr), C.byref(pe)))
    weakref.finalize(t, _free_modules, ctx, t.t, ph, pe)
    torch.cuda.synchronize()
    return {"w": w, "ctx": ctx, "table": t, "phot": ph, "perr": pe}


def _free_modules(ctx, table, phot, perr):
    L = G.lib()
    L.gf_photometry_destroy(phot)
    L.gf_photoerr_destroy(perr)
    L.gf_table_free(ctx.h, C.byref(table))


# ---------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------
def prepare(case, seed):
    if case["kind"] == "modules":
        s = _prepare_modules(case, seed)
    elif case["kind"] == "counts":
        s = {"ctx": _context(), "w": _request(case, seed)}
        s["sky"] = G.Skygen(s["ctx"], s["w"])
    elif case["kind"] == "request":
        s = {"ctx": _context(), "w": _request(case, seed), "catalog": _Catalog(case, 5)}
    else:
        s = {"ctx": _context(), "w": _requests(case, seed), "catalog": _Catalog(case, 5 if case["kind"] == "beams" else 6)}
        s["ctx"].set_host_columns(G.COL_CATALOG | G.COL["comp"])
    s["case"] = case
    return s


def run(s):
    return {"request": _run_request, "beams": _run_many, "served": _run_many, "counts": _run_counts,
            "modules": _run_modules}[s["case"]["kind"]](s)


def _run_request(s):
    """One catalog: gf_catalog_run, its batches kept as they come."""
    cat, rows = s["catalog"], np.zeros(len(s["w"].models), dtype=np.int64)
    cat.rows = 0
    if s["case"]["sink"] == "host":
        def sink(model, host, row_offset):
            cat.from_host(host.t, host.size)
            rows[model] += host.size
            return 0

        G.run_catalog(s["ctx"], s["w"], sink)
    else:
        def batch(user, model, tptr, row_offset):
            t = tptr.contents
            cat.from_device(t, int(t.size))
            rows[model] += int(t.size)
            return 0

        job, stats, cb = s["w"].job(G.Job), G.CatalogStats(), G.BatchCallback(batch)
        G.check(G.lib().gf_catalog_run(s["ctx"].h, C.byref(job), cb, None, C.byref(stats)))
    return {"rows": rows, **cat.col}


def _run_many(s):
    """Many catalogs: gf_catalog_run_multi, or its form that delivers to host memory."""
    w, cat = s["w"], s["catalog"]
    n = len(w)
    rows = np.zeros((n, len(w[0].models)), dtype=np.int64)
    cat.rows = 0
    if cat.device:
        def device_sink(model, tptr, begin, count):
            t = tptr.contents
            rows[:, model] += np.ctypeslib.as_array(count, shape=(n,))
            cat.from_device(t, int(t.size))
            return 0

        G.run_catalog_multi(s["ctx"], w, device_sink=device_sink)
    else:
        def piece(user, model, tptr, begin, count):
            t = tptr.contents
            rows[:, model] += np.ctypeslib.as_array(count, shape=(n,))
            cat.from_host(t, int(t.size))
            return 0

        jobs, stats = (G.Job * n)(*[x.job(G.Job) for x in w]), (G.CatalogStats * n)()
        G.check(G.lib().gf_catalog_run_multi_host(s["ctx"].h, jobs, n, 0, G.MultiHostCallback(piece), None, stats))
    return {"rows": rows, **cat.col}


def _run_counts(s):
    """Expected stars of each model, and of each pixel."""
    out = {}
    for m in range(len(s["w"].models)):
        e, ec, pp = s["sky"].integrate_counts(m, per_pixel=True)
        out["model%d" % m] = {"totals": np.array([e, ec]), "per_pixel": pp}
    return out


def _run_modules(s):
    """The module chain in pipeline order on rows [0, n)."""
    L, w, n = G.lib(), s["w"], s["case"]["rows"]
    h, t = s["ctx"].h, C.byref(s["table"].t)
    G.check(L.gf_module_clipper(h, C.byref(w.foot), w.sky.proj, t, 0, n))
    G.check(L.gf_module_fixedfeh(h, C.byref(w.feh), t, 0, n))
    G.check(L.gf_module_bond2010(h, C.byref(w.kin), t, 0, n))
    G.check(L.gf_module_photometry(h, s["phot"], t, 0, n))
    G.check(L.gf_module_photoerrors(h, s["perr"], 0, t, 0, n))
    G.check(L.gf_module_vel2pm(h, C.byref(w.v2pm), t, 0, n))
    G.check(L.gf_module_gal2other(h, w.gal2other, t, 0, n))
    s["ctx"].sync()
    names = ("hidden", "FeH", "vcyl", "mags", "photoflags", "obsmags", "pm", "radec")
    return {name: _column(s["table"].t, name, n, s["table"]) for name in names}


# ---------------------------------------------------------------------------
# what the work cannot do without
# ---------------------------------------------------------------------------
def _footprints(case):
    """(l, b, deg^2, pixels, m0, m1) of each request of a case."""
    if case["kind"] in ("beams", "served"):
        return [(l, b, area, area * 100.0, 14.0, m1) for l, b, area, m1 in _parameters(case)[1]]
    size = case["size"]
    area = {"cap": math.pi * size ** 2, "patch": 4 * size ** 2, "stripe": size ** 2 * math.cos(case["b"] * D2R)}[case["area"]]
    l = case["l"] + (size if case["area"] == "stripe" else 0.0)
    return [(l, case["b"], area, area / case["dx"] ** 2, case["m0"], case["m1"])]


def _expected_rows(case):
    """About how many stars a case draws: the models' counts at a few points of each footprint."""
    total = 0.0
    for l, b, area, _, m0, m1 in _footprints(case):
        r = min(0.6 * math.sqrt(area / math.pi), 0.5 * abs(b))
        pts = [(l, b), (l, b - math.copysign(r, b)), (l, b + math.copysign(min(r, 90 - abs(b)), b)), (l - r, b), (l + r, b)]
        lr, br = (np.array([p[k] for p in pts]) * D2R for k in (0, 1))
        grid = _grid(m0, m1)
        total += area * D2R ** 2 * sum(float((c * grid["S"][-1]).sum(1).mean()) for c in
                                       _counts(grid, np.cos(lr), np.sin(lr), np.cos(br), np.sin(br), *_MODELS))
    return total


def work(case):
    """Every bin of the magnitude grids takes its expected count (4 products, a sum) and, in a catalog, a
    uniform and its test (a product, two sums); every row is placed, gets its module columns and is written."""
    if case["kind"] == "modules":
        n, nb = case["rows"], case["nbands"]
        return {"bytes": n * (16 + 4 + 4 + 12 + 4 + 4 + 4 + 4 + 12 + 8 * nb + 4 + 12 + 16), "flops": n * (250.0 + 60.0 * nb)}
    bins = sum(3 * p * round((m1 - m0) / 0.05) * 240 for _, _, _, p, m0, m1 in _footprints(case))
    pixels = sum(p for _, _, _, p, _, _ in _footprints(case))
    if case["kind"] == "counts":
        return {"bytes": 3 * pixels * (52 + 8), "flops": 5 * bins}
    rows = _expected_rows(case)
    return {"bytes": rows * (4 + 16 + 4 + 4 + 8 * 5 + 12 + 12) + 52 * pixels, "flops": 8 * bins + 600 * rows}


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------
_MODELS = (("disk", 1.0, 2600.0, 300.0), ("disk", 0.12, 3600.0, 900.0), ("halo", 0.005, -2.77, 0.64))


def _grid(m0, m1):
    """The (m, M) grid of 0.05 mag: its rows, and along each line of constant distance the sum of the
    luminosity function (at its nearest of 1024 samples) over the m rows below k, for every k."""
    dm, nm, nM = np.float32(0.05), round((m1 - m0) / 0.05), 240
    M1 = np.float32(15.0 - 0.025)
    knots = np.round(np.arange(121) * 0.1 + 3.0, 10)
    phi = 10.0 ** (-3.5 + 1.5 * (knots - 3.0) / 12.0)
    X = np.concatenate([[knots[0] - 1.2e-4], knots, [knots[-1] + 1.2e-4]])       # zero just outside the knots
    lf = np.interp(np.linspace(X[0], X[-1], 1024), X, np.concatenate([[0.0], phi, [0.0]])).astype(np.float32)
    at = (M1 - np.arange(nM, dtype=np.float32) * dm - np.float32(X[0])) * np.float32(1023.0 / (X[-1] - X[0])) + np.float32(0.5)
    lfM = lf[np.clip(at.astype(np.int64), 0, 1023)].astype(np.float64)
    rows = np.float32(m0 + 0.5 * 0.05) + dm * np.arange(nm, dtype=np.float32)
    S = np.zeros((nm + 1, nm + nM - 1))
    for i in range(nm):
        S[i + 1] = S[i]
        S[i + 1, i:i + nM] += lfM
    D = 10.0 ** (0.2 * (float(rows[0]) - float(M1) + np.arange(nm + nM - 1) * float(dm)) + 1.0)
    return {"rows": rows, "S": S, "D": D, "vol": D ** 3 * 0.46051701859880914 * float(dm) ** 2}


def _counts(grid, cl, sl, cb, sb, *models):
    """Per unit solid angle and unit luminosity function: rho(D) D^3 (ln 10 / 5) dm dM of each model, (directions, distances)."""
    D = grid["D"][None]
    sina = -Z0 / RG
    cosa = math.sqrt(1 - sina * sina)
    x, y, z = D * (cl * cb)[:, None] - RG, D * (sl * cb)[:, None], D * sb[:, None]
    R, gz = np.hypot(-cosa * x + sina * z, y), sina * x + cosa * z
    R0, gz0 = cosa * RG, -sina * RG
    for kind, f, p, q in models:
        if kind == "disk":
            rho = np.exp((R0 - R) / p + (abs(gz0) - np.abs(gz)) / q)
        else:
            rho = ((R ** 2 + (gz / q) ** 2) / (R0 ** 2 + (gz0 / q) ** 2)) ** (0.5 * p)
        yield f * rho * grid["vol"][None]


def exact(case, seed):
    """In 64 bits: the expected counts, and the modules' columns that are functions of the rows.
    A drawn catalog has no such value: which stars it holds follows from its random streams."""
    if case["kind"] == "counts":
        return _exact_counts(case, seed)
    if case["kind"] == "modules":
        return _exact_modules(case, seed)
    return None


def _exact_counts(case, seed):
    """Sums over (m, M) of LF(M) rho(D) D^3 dA (ln 10 / 5) dm dM for the bins with m + Am <= m1."""
    w = _request(case, seed)
    pix = np.frombuffer(w.pixels, dtype=np.float32).reshape(w.npixels, 12)
    cl, cb, sl, sb, covered, dA = (pix[:, k].astype(np.float64) for k in (0, 1, 2, 3, 4, 6))
    am = w.ammin[pix.view(np.int32)[:, 10]]
    grid = _grid(case["m0"], case["m1"])
    cut = grid["rows"][None] + am[:, None] > np.float32(case["m1"])
    below = np.where(cut.any(1), cut.argmax(1), len(grid["rows"]))
    models = [("disk", c.f, c.l, c.h) if c.type == A.GF_MODEL_EXP_DISK else ("halo", c.f, c.n, c.ca) for c in w.models]
    out = {}
    for k, c in enumerate(_counts(grid, cl, sl, cb, sb, *models)):
        per = (c * grid["S"][below]).sum(1) * dA
        out["model%d" % k] = {"totals": np.array([per.sum(), (per * covered).sum()]), "per_pixel": per * covered}
    return out


def _exact_modules(case, seed):
    """Magnitudes from the colours' cubic relations as tabulated, and equatorial coordinates; rows that
    the clipper hides keep zeros.  Velocities and errors are drawn and have no such value."""
    rows, nb = _rows(case, seed), case["nbands"]
    l, b = (v.cpu().numpy() * D2R for v in rows["lb"])
    M, DM, Am = (rows[k].cpu().numpy().astype(np.float64) for k in ("absmag", "DM", "Am"))
    l0, b0 = rows["l0"] * D2R, rows["b0"] * D2R
    seen = np.sin(b) * np.sin(b0) + np.cos(b) * np.cos(b0) * np.cos(l - l0) >= math.cos(4.9 * D2R)
    coef, AE = W.color_coefficients(nb), (W.SDSS_AE if nb == 5 else W.LSST_AE)
    j = np.clip(((M.astype(np.float32) - np.float32(3.0)) * np.float32(100.0) + np.float32(0.5)).astype(np.int64), 0, 1200)
    t = (3.0 + 0.01 * j - 9.0) / 6.0
    colour = [sum(c[k] * t ** k for k in range(4)) for c in coef]
    mags = np.zeros((nb, len(M)))
    for k in range(nb):
        mags[k] = M + sum(colour[k:2]) - sum(colour[2:k]) + DM + Am * (AE[k] / AE[2])
    se, ce, lg, ag = 0.45598511375586859, 0.88998740217659689, 32.932 * D2R, 192.859508333 * D2R
    sb, cb, s, c = np.sin(b), np.cos(b), np.sin(l - lg), np.cos(l - lg)
    radec = np.stack([np.mod(np.arctan2(cb * c, sb * ce - cb * se * s) + ag, 2 * math.pi), np.arcsin(cb * ce * s + sb * se)]) / D2R
    return {"hidden": None, "FeH": np.zeros(len(M)), "vcyl": None, "mags": mags * seen, "photoflags": None, "obsmags": None,
            "pm": None, "radec": radec * seen}
