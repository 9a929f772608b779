"""The work that programs built on this framework have it do, as timed cases.

A case names an operation (`op`) and its sizes; prepare() makes what such a program holds before the
call (device tensors, the table, the plan, the captured graph, the workspace) and run() is one pass
through the public entry points of tconvolve.

  call    one-call gridding or degridding of samples seen once: raw.grid_raw / raw.degrid_raw
  plan    one gridding or degridding pass of a binning plan that the program keeps (raw.Plan)
  batch   the captured bin + grid + degrid step of several jobs that share a table (batch.Batch)
  track   the variable-support path: samples of the 36-antenna track, a kernel width per w-plane,
          on a plan that uses the sample-parallel passes (raw.VarPlan)
  hogbom  a minor cycle of Hogbom CLEAN on device images (hogbom.deconvolve_device)
  fft     the image transform, forward and back (major.fft_exec)
  cycle   an imaging cycle: grid, dirty image, CLEAN, model transform, degrid
  table   set-up of the convolution table and its stored form (raw.init_c, raw.convert_c)

Sizes: the attic benchmark's constants (160000 samples, 33 w-planes, 4096^2 grid, 2000 m baseline,
5-wavelength cells: support 64) and its 1024^2 case (16000 samples, support 22), the continuum and
spectral runs of current/tConvolveMPI, tHogbomCleanOMP's 1000 iterations on images of 1024^2 and
4096^2, tMajorACC's 100 minor iterations; the drawn cases spread over the ranges between and around
them, with ragged sample counts and odd grid sides.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "askap-benchmarks_b200"))

from tconvolve import _lib, batch, current, hogbom, major, raw  # noqa: E402

FREQ0 = 1.4e9 / 2.998e8
BASELINE = 2000
PASSES = _lib.PASS_BIN | _lib.PASS_GRID | _lib.PASS_DEGRID


def listed():
    return [
        # smallest: a short observation snapshot gridded in one call, new samples each time
        # (latency, launches and binning count); 45^2 footprints on 1024^2
        dict(name="call_grid_16k_c64", op="call", way="grid", n=16000, g=1024, cell=40.0, w=9, form="c64"),
        # one-call degridding with a ragged sample count on an odd grid, real-table form
        dict(name="call_degrid_odd_r32", op="call", way="degrid", n=37123, g=1501, cell=20.0, w=17, form="r32"),
        # the reference's default problem, one kept plan, plain complex64 table: gridding
        dict(name="grid_4096_c64", op="plan", way="grid", n=160000, g=4096, cell=5.0, w=33, form="c64"),
        # the same problem degridded with the exact real table, the benchmark's headline form
        dict(name="degrid_4096_r32", op="plan", way="degrid", n=160000, g=4096, cell=5.0, w=33, form="r32"),
        # a batched step over jobs of uneven size (channels or Taylor terms), one graph launch
        dict(name="batch_12_r32", op="batch", jobs=12, n_min=10000, n_max=60000, form="r32", w=33),
        # spectral-line imaging: 3.8 M samples of a 12 h track, kernels 7..19 wide, all samples
        dict(name="spectral_grid", op="track", way="grid", run=1, part=1.0, form="c64"),
        # continuum imaging: 5.4 M samples, kernels 7..121 wide, the prediction direction
        dict(name="continuum_degrid", op="track", way="degrid", run=0, part=1.0, form="c64"),
        # CLEAN minor cycles at the small and the large image size
        dict(name="hogbom_1024", op="hogbom", width=1024, psf=1024, iters=1000, sources=20),
        dict(name="hogbom_4096", op="hogbom", width=4096, psf=4096, iters=1000, sources=20),
        # grid to image and back: one transform each way at the default grid
        dict(name="fft_4096", op="fft", way="round", g=4096),
        # one imaging cycle at a medium size (all samples on the w = 0 plane), 100 minor iterations
        dict(name="cycle_2048", op="cycle", n=60000, g=2048, cell=10.0, w=1, iters=100, form="r32"),
        # table set-up of the default problem: 35 M entries made, normalised, stored as real floats
        dict(name="table_33_planes", op="table", cell=5.0, w=33, form="r32"),
    ]


def _support(cell):
    return int(1.5 * math.sqrt(BASELINE * cell * FREQ0) / cell)


def _least_side(cell):
    """A grid side on which every footprint of the generator's +-1000 m samples lies inside (its
    rows run from the sample's cell up)."""
    return 2 * (int(1000 * FREQ0 / cell) + 2 * _support(cell) + 4)


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sky_samples(rng, n_hi):
    """A ragged sample count, a cell size and a grid side (odd ones among them) that holds it."""
    cell = math.exp(rng.uniform(math.log(5.0), math.log(100.0)))
    lo = max(_least_side(cell), 128)
    return dict(n=_log(rng, 2000, n_hi), cell=round(cell, 2), g=min(4096, lo + 1 + _log(rng, 1, lo)))


def draw(rng):
    op = rng.choice(["call", "plan", "plan", "batch", "track", "track", "hogbom", "hogbom", "fft", "cycle", "table"])
    if op in ("call", "plan"):
        form = rng.choice(["c64", "c64", "r32", "r32", "cbf16", "rbf16", "cf16", "rf16"])
        way = rng.choice(["grid", "degrid"])
        return dict(op=op, way=way, form=form, w=rng.choice([1, 5, 9, 17, 33]),
                    **_sky_samples(rng, 60000 if op == "call" else 160000))
    if op == "batch":
        return dict(op=op, jobs=rng.randint(2, 24), n_min=_log(rng, 2000, 10000), n_max=_log(rng, 10000, 30000),
                    form=rng.choice(["r32", "c64", "rbf16"]), w=rng.choice([9, 17, 33]))
    if op == "track":
        return dict(op=op, way=rng.choice(["grid", "degrid"]), run=rng.choice([0, 1, 1]),
                    part=round(math.exp(rng.uniform(math.log(0.02), 0.0)), 4), form=rng.choice(["c64", "c64", "cbf16"]))
    if op == "hogbom":
        width = _log(rng, 128, 4096)
        width -= rng.choice([0, 0, width % 4, width % 16])
        psf = rng.choice([width, width, width | 1, max(32, width // 2), min(4096, 2 * width)])
        return dict(op=op, width=width, psf=psf, iters=_log(rng, 50, 1000), sources=rng.randint(3, 60))
    if op == "fft":
        g = rng.choice([128, 256, 512, 1024, 2048, 4096, 2 * _log(rng, 64, 2048)])
        return dict(op=op, way=rng.choice(["round", "forward", "backward"]), g=g)
    if op == "cycle":
        cell = rng.choice([10.0, 20.0, 40.0])
        g = rng.choice([s for s in (512, 1024, 2048) if s >= _least_side(cell)])
        return dict(op=op, n=_log(rng, 4000, 60000), g=g, cell=cell, w=1,
                    iters=_log(rng, 20, 200), form=rng.choice(["r32", "c64"]))
    return dict(op=op, cell=round(math.exp(rng.uniform(math.log(5.0), math.log(100.0))), 2), w=rng.randint(3, 33),
                form=rng.choice(["c64", "r32", "cbf16", "rbf16", "rf16"]))


# ---- inputs ----------------------------------------------------------------------------------
def _gen(seed, salt=0):
    return torch.Generator(device="cuda").manual_seed(1000003 * int(seed) + salt)


def _normal(n, seed, salt=0):
    return torch.view_as_complex(torch.randn(n, 2, generator=_gen(seed, salt), device="cuda"))


def _table(cell, w, form):
    """(table, c_type, c_scale, geometry) in a stored form; the complex64 table is let go."""
    support, over, w_cell, c_len = raw.c_geometry(FREQ0, cell, BASELINE, w)
    c64, _ = raw.init_c(FREQ0, cell, BASELINE, w)
    code = _lib.CTYPE_BY_NAME[form]
    if form == "c64":
        return c64, code, 1.0, (support, over, w_cell, c_len)
    tab, scale, _ = raw.convert_c(c64, code)
    return tab, code, scale, (support, over, w_cell, c_len)


def _samples(n, cell, w, g, geo, seed):
    support, over, w_cell, _ = geo
    u, v, ww = raw.init_uvw(n, BASELINE, 1 + int(seed))
    freq = torch.tensor([FREQ0], dtype=torch.float64, device="cuda")
    return raw.init_offsets(u, v, ww, freq, cell, w_cell, w, g, support, over)


def _batch_sizes(case):
    """Jobs with sample counts spread over the range and sides 2304 and 4096."""
    lo, hi, k = case["n_min"], case["n_max"], case["jobs"]
    n = [int(lo * (hi / lo) ** ((j * 0.618034) % 1.0)) for j in range(k)]
    return [(m, 4096 if j % 3 == 0 else 2304) for j, m in enumerate(n)]


def _track_part(case, total, seed):
    n = max(1, int(case["part"] * total))
    at = (int(seed) * 7919 * 631) % (total - n + 1)
    return at, n


def _track_inputs(case, seed):
    """Samples (a stretch of the track), planes and table of one run type, on the device."""
    b = current.Benchmark()
    b.setRunType(case["run"])
    b.init()
    geo = b.geometry()
    at, n = _track_part(case, b.nVisibilitiesGridded(), seed)
    iu, iv, wp, co = (torch.from_numpy(a[at:at + n].copy()).cuda() for a in b.offsets())
    s_size, off0 = b.planes()
    c64 = torch.from_numpy(b.C()).cuda()
    g, c_len = int(geo.g_size), int(geo.c_len)
    b.close()
    return dict(iu=iu, iv=iv, wp=wp, co=co, s_size=s_size, off0=off0, c64=c64, g=g, c_len=c_len, n=n)


def _psf_value(r2, s):
    """The point-spread shape of workload.synthetic_psf at squared radius r2."""
    q = 1.0 + r2 / (s * s)
    return (1.0 - r2 / (2.0 * s * s)) / (q * q)


def _clean_inputs(case, seed):
    """A dirty image of point sources with sidelobes plus noise (as workload.synthetic_dirty) and
    the PSF image; float32 on the device."""
    w, p = case["width"], case["psf"]
    s = max(2.0, w / 64.0)
    host = np.random.default_rng(int(seed))
    d = torch.arange(w, dtype=torch.float64, device="cuda")
    img = 1e-3 * (torch.rand(w, w, generator=_gen(seed), device="cuda", dtype=torch.float64) - 0.5)
    for _ in range(case["sources"]):
        x, y = host.integers(int(0.1 * w), int(0.9 * w), 2)
        r2 = (d[:, None] - int(y)) ** 2 + (d[None, :] - int(x)) ** 2
        img += (0.1 + 0.9 * host.random()) * _psf_value(r2, s)
    e = torch.arange(p, dtype=torch.float64, device="cuda") - p // 2
    psf = _psf_value(e[:, None] ** 2 + e[None, :] ** 2, s)
    return img.float().reshape(-1), psf.float().reshape(-1)


def _cycle_inputs(case, seed):
    """Visibilities of a point-source sky (its transform at each sample's cell, plus noise)."""
    g = case["g"]
    tab, code, scale, geo = _table(case["cell"], case["w"], case["form"])
    iu, iv, coff = _samples(case["n"], case["cell"], case["w"], g, geo, seed)
    host = np.random.default_rng(int(seed))
    sky = torch.zeros(g, g, dtype=torch.complex64, device="cuda")
    for _ in range(20):
        x, y = host.integers(int(0.3 * g), int(0.7 * g), 2)
        sky[int(y), int(x)] += float(0.1 + 0.9 * host.random())
    uv = torch.fft.fftshift(torch.fft.fft2(torch.fft.fftshift(sky)))
    vis = uv[iv.long(), iu.long()] + 0.05 * _normal(case["n"], seed, 7)
    # a footprint's rows run from its sample's iv up: centre them on the sample, as its columns are
    return tab, code, scale, geo, iu, iv - geo[0], coff, vis.contiguous()


def prepare(case, seed):
    op = case["op"]
    s = dict(case=case)
    if op in ("call", "plan"):
        tab, code, scale, geo = _table(case["cell"], case["w"], case["form"])
        iu, iv, coff = _samples(case["n"], case["cell"], case["w"], case["g"], geo, seed)
        s.update(tab=tab, code=code, scale=scale, support=geo[0], iu=iu, iv=iv, coff=coff)
        if case["way"] == "grid":
            s["data"] = _normal(case["n"], seed)
            s["grid"] = torch.zeros(case["g"] ** 2, dtype=torch.complex64, device="cuda")
        else:
            s["grid"] = _normal(case["g"] ** 2, seed)
            s["out"] = torch.zeros(case["n"], dtype=torch.complex64, device="cuda")
        if op == "plan":  # the tuning that the autotuner takes for the default problem
            s["plan"] = raw.Plan(iu, iv, coff, geo[0], case["g"], geo[3], tuning=(16, 64, 0, 64))
    elif op == "batch":
        sizes = _batch_sizes(case)
        tab, code, scale, geo = _table(5.0, case["w"], case["form"])
        parts = [_samples(n, 5.0, case["w"], g, geo, 97 * int(seed) + j) for j, (n, g) in enumerate(sizes)]
        iu, iv, coff = (torch.cat([p[k] for p in parts]) for k in range(3))
        grids = [torch.zeros(g * g, dtype=torch.complex64, device="cuda") for _, g in sizes]
        data = _normal(iu.numel(), seed)
        vis = torch.zeros_like(data)
        plan = batch.Batch(sizes, grids, iu, iv, coff, geo[0], geo[3], tuning=(16, 64, 0, 128))
        s.update(tab=tab, scale=scale, grids=grids, data=data, vis=vis, plan=plan, iu=iu, iv=iv, coff=coff,
                 graph=plan.capture(PASSES, data, tab, code, vis, scale))
    elif op == "track":
        s.update(_track_inputs(case, seed))
        code = _lib.CTYPE_BY_NAME[case["form"]]
        tab, scale = (s["c64"], 1.0) if case["form"] == "c64" else raw.convert_c(s["c64"], code)[:2]
        # the tuner's choices for the two runs: tile rows, group MiB, split, degrid split, passes
        tuning = (8, -1, 512, 128, 3) if case["run"] == 0 else (8, 32, 1024, 256, 3)
        plan = raw.VarPlan(s["iu"], s["iv"], s["co"], s["wp"], s["s_size"], s["off0"], s["g"], s["c_len"], tuning=tuning)
        s.update(tab=tab, code=code, scale=scale, plan=plan)
        if case["way"] == "grid":
            s["data"] = _normal(s["n"], seed)
            s["grid"] = torch.zeros(s["g"] ** 2, dtype=torch.complex64, device="cuda")
        else:
            s["grid"] = _normal(s["g"] ** 2, seed)
            s["out"] = torch.zeros(s["n"], dtype=torch.complex64, device="cuda")
    elif op == "hogbom":
        dirty, psf = _clean_inputs(case, seed)
        s.update(dirty=dirty, psf=psf, model=torch.zeros_like(dirty), residual=torch.empty_like(dirty),
                 work=hogbom.Workspace(case["width"]))
    elif op == "fft":
        s["grid"] = torch.empty(case["g"] ** 2, dtype=torch.complex64, device="cuda")
        if case["way"] == "round":
            s["model"] = torch.randn(case["g"] ** 2, generator=_gen(seed), device="cuda")
            s["image"] = torch.empty_like(s["model"])
        else:
            s["source"] = _normal(case["g"] ** 2, seed)
    elif op == "cycle":
        tab, code, scale, geo, iu, iv, coff, vis = _cycle_inputs(case, seed)
        g = case["g"]
        plan = raw.Plan(iu, iv, coff, geo[0], g, geo[3], tuning=(16, 64, 0, 64))
        grid = torch.zeros(g * g, dtype=torch.complex64, device="cuda")
        psf = torch.empty(g * g, dtype=torch.float32, device="cuda")
        plan.grid(torch.ones_like(vis), tab, code, grid, scale)
        major.image_from_grid(grid, g, 1.0, psf)
        norm = 1.0 / float(psf.max())
        psf *= norm
        s.update(tab=tab, code=code, scale=scale, support=geo[0], iu=iu, iv=iv, coff=coff, vis=vis, plan=plan, grid=grid,
                 psf=psf, norm=norm, dirty=torch.empty_like(psf), model=torch.empty_like(psf), residual=torch.empty_like(psf),
                 pred=torch.empty_like(vis), work=hogbom.Workspace(g))
    else:
        s["seed"] = int(seed)
        # tables of neighbouring cell sizes: each seed sets up another
        s["cell"] = case["cell"] * (1.0 + 1e-4 * (int(seed) % 97))
    return s


def run(s):
    case = s["case"]
    op = case["op"]
    if op == "call":
        if case["way"] == "grid":
            raw.grid_raw(s["data"], s["support"], s["tab"], s["code"], s["scale"], s["coff"], s["iu"], s["iv"],
                         s["grid"], case["g"])
            return s["grid"]
        raw.degrid_raw(s["grid"], case["g"], s["support"], s["tab"], s["code"], s["scale"], s["coff"], s["iu"],
                       s["iv"], s["out"])
        return s["out"]
    if op in ("plan", "track"):
        if case["way"] == "grid":
            s["plan"].grid(s["data"], s["tab"], s["code"], s["grid"], s["scale"])
            return s["grid"]
        s["plan"].degrid(s["grid"], s["tab"], s["code"], s["out"], s["scale"])
        return s["out"]
    if op == "batch":
        s["graph"].launch()
        return [s["vis"]] + s["grids"]
    if op == "hogbom":
        s["model"].zero_()
        hogbom.deconvolve_device(s["dirty"], case["width"], s["psf"], case["psf"], s["model"], s["residual"],
                                 case["iters"], work=s["work"])
        return {"model": s["model"], "residual": s["residual"]}
    if op == "fft":
        if case["way"] == "round":  # the model's grid, then the image of that grid
            major.grid_from_image(s["model"], case["g"], s["grid"])
            major.image_from_grid(s["grid"], case["g"], case["g"] ** -2.0, s["image"])
            return s["image"]
        s["grid"].copy_(s["source"])  # the transform is in place
        major.fft_exec(s["grid"], case["g"], case["way"] == "forward")
        return s["grid"]
    if op == "cycle":
        g = case["g"]
        s["grid"].zero_()
        s["plan"].grid(s["vis"], s["tab"], s["code"], s["grid"], s["scale"])
        major.image_from_grid(s["grid"], g, s["norm"], s["dirty"])
        s["model"].zero_()
        hogbom.deconvolve_device(s["dirty"], g, s["psf"], g, s["model"], s["residual"], case["iters"],
                                 threshold=0.0, work=s["work"])
        major.grid_from_image(s["model"], g, s["grid"])
        s["plan"].degrid(s["grid"], s["tab"], s["code"], s["pred"], s["scale"])
        return {"dirty": s["dirty"], "model": s["model"], "residual": s["residual"], "pred": s["pred"]}
    c64, sum_c = raw.init_c(FREQ0, s["cell"], BASELINE, case["w"])
    if case["form"] == "c64":
        return {"c": c64, "sum": sum_c}
    tab, scale, _ = raw.convert_c(c64, _lib.CTYPE_BY_NAME[case["form"]])
    view = {"r32": torch.float32, "rbf16": torch.bfloat16, "cbf16": torch.bfloat16, "rf16": torch.float16}
    return {"c": c64, "tab": tab.view(view[case["form"]]), "scale": scale, "sum": sum_c}


# ---- what a pass cannot do without -------------------------------------------------------------
def _grid_work(n, s, g, entry, real, c_len, way):
    """Samples (value, position, table offset), the grid and the table once; a complex
    multiply-add (by a real or a complex entry) per sample and footprint point."""
    grid = 8.0 * min(g * g, n * s * s)
    return dict(bytes=20.0 * n + grid * (2 if way == "grid" else 1) + entry * min(c_len, n * s * s),
                flops=(4.0 if real else 8.0) * n * s * s)


def _entry(form):
    return float(_lib.lib().tcv_ctype_bytes(_lib.CTYPE_BY_NAME[form]))


def work(case):
    op = case["op"]
    if op in ("call", "plan"):
        s = 2 * _support(case["cell"]) + 1
        form, c_len = case["form"], s * s * 64 * case["w"]
        return _grid_work(case["n"], s, case["g"], _entry(form), form[0] == "r", c_len, case["way"])
    if op == "batch":
        s = 2 * _support(5.0) + 1
        out = dict(bytes=_entry(case["form"]) * s * s * 64 * case["w"], flops=0.0)
        for n, g in _batch_sizes(case):
            for way in ("grid", "degrid"):
                w = _grid_work(n, s, g, 0.0, case["form"][0] == "r", 0, way)
                out = {k: out[k] + w[k] for k in out}
        return out
    if op == "track":
        # mean squared kernel width of the runs' samples: 380 (continuum), 86 (spectral)
        total, mean, c_len, g = ((5443200, 379.5, 38906416, 6440), (3827520, 85.7, 1456576, 1034))[case["run"]]
        n = max(1, int(case["part"] * total))
        return dict(bytes=22.0 * n + 8.0 * g * g * (2 if case["way"] == "grid" else 1) + _entry(case["form"]) * c_len,
                    flops=8.0 * n * mean)
    if op == "hogbom":
        w, p = case["width"], case["psf"]
        overlap = min(w * w, (0.75 * min(w, p)) ** 2)  # a mean over the peaks' places
        return dict(bytes=4.0 * (3 * w * w + p * p), flops=2.0 * case["iters"] * overlap)
    if op == "fft":
        n = float(case["g"]) ** 2
        passes = 2 if case["way"] == "round" else 1
        return dict(bytes=(24.0 if passes == 2 else 16.0) * n, flops=passes * 5.0 * n * math.log2(n))
    if op == "cycle":
        n, g, s = case["n"], case["g"], 2 * _support(case["cell"]) + 1
        real, e = case["form"][0] == "r", _entry(case["form"])
        c_len = s * s * 64 * case["w"]
        both = [_grid_work(n, s, g, e, real, c_len, way) for way in ("grid", "degrid")]
        fl = sum(b["flops"] for b in both) + 2 * 5.0 * g * g * math.log2(g * g) + 2.0 * case["iters"] * (0.75 * g) ** 2
        return dict(bytes=sum(b["bytes"] for b in both) + 24.0 * g * g, flops=fl)
    s = 2 * _support(case["cell"]) + 1
    c_len = s * s * 64 * case["w"]
    return dict(bytes=c_len * (8.0 + (0.0 if case["form"] == "c64" else _entry(case["form"]))), flops=30.0 * c_len)


# ---- the same results in 64 bits, by torch alone -----------------------------------------------
def _stored(tab, form, scale):
    """A stored table as complex128 values (rounding to the stored form is part of the input)."""
    if form == "c64":
        return tab.to(torch.complex128)
    kind = {"r32": torch.float32, "rbf16": torch.bfloat16, "cbf16": torch.bfloat16, "rf16": torch.float16, "cf16": torch.float16}
    v = tab.view(kind[form]).double() * scale
    return torch.view_as_complex(v.view(-1, 2)) if form[0] == "c" else v.to(torch.complex128)


def _footprints(iu, iv, coff, width, g):
    """Flat grid and table indices of every footprint point: samples x width^2 (columns centred on
    iu, rows from iv on)."""
    k = torch.arange(width * width, device="cuda")
    at = (iv.long()[:, None] + (k // width)[None, :]) * g + (iu.long()[:, None] - width // 2) + (k % width)[None, :]
    return at, coff.long()[:, None] + k[None, :]


def _chunks(n, width):
    step = max(1, 60_000_000 // (width * width))
    return [slice(a, min(n, a + step)) for a in range(0, n, step)]


def _grid64(data, tab, iu, iv, coff, width, grid, g):
    flat = torch.view_as_real(grid)
    for c in _chunks(iu.numel(), width):
        at, ci = _footprints(iu[c], iv[c], coff[c], width, g)
        flat.index_add_(0, at.reshape(-1), torch.view_as_real((data[c].to(torch.complex128)[:, None] * tab[ci]).reshape(-1)))


def _degrid64(grid, tab, iu, iv, coff, width, g):
    out = torch.empty(iu.numel(), dtype=torch.complex128, device="cuda")
    for c in _chunks(iu.numel(), width):
        at, ci = _footprints(iu[c], iv[c], coff[c], width, g)
        out[c] = (grid[at] * tab[ci]).sum(1)
    return out


def _clean64(dirty, w, psf, p, iters, threshold, gain=0.1):
    """HogbomGolden::deconvolve in 64 bits; images as flat float32 inputs, 64-bit model and residual."""
    gain = float(np.float32(gain))
    psf = psf.double().view(p, p)
    peak = int(psf.abs().argmax())
    py, px = peak // p, peak % p
    res = dirty.double().view(w, w).clone()
    model = torch.zeros_like(res)
    for _ in range(iters):
        k = int(res.abs().argmax())
        v, y, x = float(res.view(-1)[k]), k // w, k % w
        if abs(v) < threshold:
            break
        model[y, x] += gain * v
        x0, y0 = max(0, x - px), max(0, y - py)
        x1, y1 = min(w, x + p - px), min(w, y + p - py)
        res[y0:y1, x0:x1] -= gain * v * psf[y0 - y + py:y1 - y + py, x0 - x + px:x1 - x + px]
    return model.view(-1), res.view(-1)


def _image64(grid, g, scale):
    x = torch.fft.fftshift(grid.view(g, g))
    return (torch.fft.fftshift(torch.fft.ifft2(x, norm="forward")).real * scale).reshape(-1)


def _spectrum64(image, g):
    x = torch.fft.fftshift(image.view(g, g).to(torch.complex128))
    return torch.fft.fftshift(torch.fft.fft2(x)).reshape(-1)


def exact(case, seed):
    op = case["op"]
    if op == "table":
        return None  # scaled by a running 32-bit sum whose order decides its value (it saturates)
    s = prepare(case, seed)
    if op in ("call", "plan"):
        tab, width = _stored(s["tab"], case["form"], s["scale"]), 2 * s["support"] + 1
        if case["way"] == "degrid":
            return _degrid64(s["grid"].to(torch.complex128), tab, s["iu"], s["iv"], s["coff"], width, case["g"])
        grid = torch.zeros(case["g"] ** 2, dtype=torch.complex128, device="cuda")
        _grid64(s["data"], tab, s["iu"], s["iv"], s["coff"], width, grid, case["g"])
        return grid
    if op == "batch":
        tab, width = _stored(s["tab"], case["form"], s["scale"]), 2 * _support(5.0) + 1
        grids, vis, at = [], [], 0
        for n, g in _batch_sizes(case):
            p = slice(at, at + n)
            grid = torch.zeros(g * g, dtype=torch.complex128, device="cuda")
            _grid64(s["data"][p], tab, s["iu"][p], s["iv"][p], s["coff"][p], width, grid, g)
            vis.append(_degrid64(grid, tab, s["iu"][p], s["iv"][p], s["coff"][p], width, g))
            grids.append(grid)
            at += n
        return [torch.cat(vis)] + grids
    if op == "track":
        tab = _stored(s["tab"], case["form"], s["scale"])
        width = torch.from_numpy(s["s_size"]).cuda()[s["wp"].long()]
        gridding = case["way"] == "grid"
        out = torch.zeros(s["g"] ** 2 if gridding else s["n"], dtype=torch.complex128, device="cuda")
        grid = None if gridding else s["grid"].to(torch.complex128)
        for k in sorted(set(s["s_size"].tolist())):
            m = (width == k).nonzero().view(-1)
            if m.numel() and gridding:
                _grid64(s["data"][m], tab, s["iu"][m], s["iv"][m], s["co"][m], k, out, s["g"])
            elif m.numel():
                out[m] = _degrid64(grid, tab, s["iu"][m], s["iv"][m], s["co"][m], k, s["g"])
        return out
    if op == "hogbom":
        model, residual = _clean64(s["dirty"], case["width"], s["psf"], case["psf"], case["iters"], 1e-5)
        return {"model": model, "residual": residual}
    if op == "fft":
        if case["way"] == "round":
            return _image64(_spectrum64(s["model"], case["g"]), case["g"], case["g"] ** -2.0)
        x = torch.fft.fftshift(s["source"].to(torch.complex128).view(case["g"], case["g"]))
        x = torch.fft.fft2(x) if case["way"] == "forward" else torch.fft.ifft2(x, norm="forward")
        return torch.fft.fftshift(x).reshape(-1)
    g, tab, width = case["g"], _stored(s["tab"], case["form"], s["scale"]), 2 * s["support"] + 1
    iu, iv, coff = s["iu"], s["iv"], s["coff"]
    grid = torch.zeros(g * g, dtype=torch.complex128, device="cuda")
    _grid64(s["vis"], tab, iu, iv, coff, width, grid, g)
    dirty = _image64(grid, g, s["norm"])
    model, residual = _clean64(dirty, g, s["psf"], g, case["iters"], 0.0)
    pred = _degrid64(_spectrum64(model, g), tab, iu, iv, coff, width, g)
    return {"dirty": dirty, "model": model, "residual": residual, "pred": pred}
