"""The work a user of this framework has it do, as measurable cases.

An imaging program plans an observation once and then grids residual visibilities, images the w
layers, correlates the dirty image with the PSF, runs coordinate descent on the result and
degrids the model, over and over.  Each case is one of these steps (or a small call that chains
them) through the public entry points, at sizes from the repository's own workloads (256^2,
3072^2, the batched mixes), its tests (odd grids, subgrids of 16 to 48) and its options (the
FP32 default, BF16x3 and FP16x3 tensor-core modes, wide fields, host and device arrays).

``listed()`` gives the fixed cases, ``draw(rng)`` one more of the same ranges, ``prepare`` the
inputs and plans a program has in hand, ``run`` one pass, ``work`` what a pass cannot do without
and ``exact`` the pass's results in 64 bits from plain torch.
"""
from __future__ import annotations

import functools
import importlib
import math

import numpy as np
import torch

import __graft_entry__ as entry

pkg = entry.load_package()
synth = importlib.import_module(entry.PKG_NAME + ".synth")

C = 299792458.0
MODES = {"fp32": pkg.MODE_FP32, "bf16x3": pkg.MODE_TC_BF16X3, "fp16x3": pkg.MODE_TC_FP16X3}


# ---------------------------------------------------------------- cases

def _obs(op, mode, n, ants, nt, nch, *, s=32, w=8, cell=1.5, diameter=8000.0, f_lo=1.2e9, f_hi=1.5e9):
    """A gridding case: grid size n, subgrid size s, w layers, and the observation's sizes."""
    return dict(op=op, mode=mode, n=n, ants=ants, nt=nt, nch=nch, s=s, kernel=8, w=w, cell=cell, diameter=diameter,
                f_lo=f_lo, f_hi=f_hi)


def listed():
    return [
        # the headline workload: all residual visibilities of a 64-antenna observation onto 3072^2
        dict(name="grid bf16x3 3072", **_obs("grid", "bf16x3", 3072, 64, 2000, 16)),
        # ... and the model back to visibilities, once per major cycle
        dict(name="degrid bf16x3 3072", **_obs("degrid", "bf16x3", 3072, 64, 2000, 16)),
        # the mode a plan has unless the program asks for another, on a 40-antenna observation
        dict(name="grid fp32 3072", **_obs("grid", "fp32", 3072, 40, 2000, 16)),
        # the same mode the other way, on ragged sizes and a smaller subgrid
        dict(name="degrid fp32 2047 s24", **_obs("degrid", "fp32", 2047, 40, 1501, 11, s=24)),
        # the FP16 mode on a wide field (second-order w term), odd grid, small subgrid
        dict(name="grid fp16x3 wide 1025 s16", **_obs("grid", "fp16x3", 1025, 36, 777, 5, s=16, w=4, cell=20.0,
                                                      diameter=1100.0, f_lo=1.0e9, f_hi=1.1e9)),
        # a snapshot of a small array, one whole residual step: launches and latency count
        dict(name="step bf16x3 256 small", **_obs("step", "bf16x3", 256, 10, 120, 4, w=4, cell=5.0, diameter=2000.0,
                                                  f_lo=1.0e9, f_hi=1.1e9)),
        # the 256^2 workload's dirty image from host arrays, as a program that calls the C# members does
        dict(name="dirty image fp32 256 host", **_obs("dirty_host", "fp32", 256, 30, 1440, 8, w=4, cell=5.0,
                                                      diameter=2000.0, f_lo=1.0e9, f_hi=1.1e9)),
        # model image to model visibilities on host arrays, of a 1024^2 field
        dict(name="predict bf16x3 1024 host", **_obs("predict_host", "bf16x3", 1024, 24, 400, 16)),
        # many small problems in one launch per stage, replayed from a graph
        dict(name="batch bf16x3 12 small", op="batch", mode="bf16x3", count=12, n_lo=512, n_hi=1024, ants_lo=16,
             ants_hi=32, nt_lo=200, nt_hi=500, nch_lo=4, nch_hi=16, s=32, w=8, layout=4),
        # w layers to the dirty image, once per major cycle
        dict(name="image 3072", op="image", n=3072, w=8),
        # dirty image to the gradient map: the padded correlation with the cut PSF
        dict(name="correlate 3072", op="correlate", n=3072, psf=384),
        # the coordinate descent on that map, which most of a reconstruction's time goes into
        dict(name="deconvolve 3072", op="deconvolve", n=3072, psf=384, iters=1000),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["grid", "grid", "grid", "degrid", "degrid", "degrid", "step", "dirty_host", "predict_host", "batch",
                     "image", "correlate", "deconvolve"])
    if op == "batch":
        return dict(op=op, mode=rng.choice(["fp32", "bf16x3", "bf16x3", "fp16x3"]), count=rng.randint(2, 14), n_lo=256,
                    n_hi=_log_int(rng, 300, 1024), ants_lo=8, ants_hi=rng.randint(12, 24), nt_lo=60,
                    nt_hi=rng.randint(100, 500), nch_lo=1, nch_hi=rng.randint(4, 16), s=rng.choice([16, 24, 32, 32]),
                    w=rng.randint(2, 8), layout=rng.randint(0, 1 << 20))
    if op == "image":
        return dict(op=op, n=_log_int(rng, 256, 3072), w=rng.randint(1, 8))
    if op in ("correlate", "deconvolve"):
        n = _log_int(rng, 256, 3072)
        p = max(16, 2 * (n // (2 * rng.choice([4, 8, 8]))))
        return dict(op=op, n=n, psf=p) if op == "correlate" else dict(op=op, n=n, psf=p, iters=rng.randint(100, 1000))
    mode = rng.choice(["fp32", "fp32", "bf16x3", "bf16x3", "fp16x3"])
    host = op.endswith("_host")
    n = _log_int(rng, 256, 1024 if host else 512 if op == "step" else 3072)
    s = rng.choice([16, 24, 32, 32, 32, 48] if mode == "fp32" else [16, 24, 32, 32, 32])
    f_lo = rng.choice([1.0e9, 1.2e9])
    f_hi = f_lo * rng.choice([1.02, 1.1, 1.25])
    cell = math.exp(rng.uniform(math.log(1.0), math.log(20.0)))
    # the longest baseline reaches 0.2 to 0.32 of the grid's width (half of it is the limit)
    diameter = rng.uniform(0.2, 0.32) / synth.cell_rad(cell) * C / f_hi
    most = 2.0e6 if op == "step" or host else 1.2e7 if mode == "fp32" else 4.0e7
    while True:
        ants, nt, nch = _log_int(rng, 6, 64), _log_int(rng, 60, 2000), _log_int(rng, 1, 32)
        if ants * (ants - 1) // 2 * nt * nch <= most:
            break
    return _obs(op, mode, n, ants, nt, nch, s=s, w=rng.randint(1, 8), cell=round(cell, 3), diameter=round(diameter, 1),
                f_lo=f_lo, f_hi=round(f_hi, 1))


# ---------------------------------------------------------------- geometry and inputs

@functools.lru_cache(maxsize=32)
def _geometry(key):
    """uvw [nbl][nt][3], channel frequencies and gridding constants: the array and its tracks."""
    c = dict(key)
    rng = np.random.default_rng([c.get("layout", 0), c["ants"], c["nt"], c["nch"], c["n"]])
    uvw = synth.earth_rotation_uvw(synth.antennas_log_radial(rng, c["ants"], c["diameter"]), -30.7215, -70.0, c["nt"],
                                   10.0)
    freq = np.linspace(c["f_lo"], c["f_hi"], c["nch"])
    return uvw, freq, dict(vis_count=uvw.shape[0] * c["nt"] * c["nch"], grid_size=c["n"], subgrid_size=c["s"],
                           kernel_size=c["kernel"], max_timesteps=1024,
                           scale_arcsec=float(np.float32(synth.cell_rad(c["cell"]))), wlayer_count=c["w"],
                           # a hair above max |w| / layers: one channel's largest w has a layer too
                           wstep=synth.wstep_for(uvw, freq, c["w"]) * (1 + 1e-6))


_GEOMETRY_KEYS = ("n", "ants", "nt", "nch", "s", "kernel", "w", "cell", "diameter", "f_lo", "f_hi", "layout")


def _geom(case):
    return _geometry(tuple((k, case[k]) for k in _GEOMETRY_KEYS if k in case))


def _problems(case):
    """The imaging problems of a batch case: their sizes come from its layout number."""
    rng = np.random.default_rng([case["layout"], case["count"]])
    pick = lambda k: int(rng.integers(case[k + "_lo"], case[k + "_hi"] + 1))  # noqa: E731
    return [dict(_obs("grid", case["mode"], pick("n"), pick("ants"), pick("nt"), pick("nch"), s=case["s"], w=case["w"]),
                 layout=case["layout"] + i) for i in range(case["count"])]


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _generator(seed, dev):
    return torch.Generator(device=dev).manual_seed(int(seed))


def _sky(case, seed):
    """A few point sources in the inner half of the field: directions and fluxes."""
    rng = np.random.default_rng([seed, case["n"]])
    cell, n = synth.cell_rad(case["cell"]), case["n"]
    xy = rng.uniform(-0.25 * n, 0.25 * n, (3, 2)) * cell
    return xy, np.array([1.0, 0.5, 0.2]) * rng.uniform(0.8, 1.2, 3)


def _visibilities(case, seed):
    """Point sources plus noise, complex64 [nbl][nt][nch]."""
    uvw, freq, _ = _geom(case)
    dev = _device()
    lm, flux = _sky(case, seed)
    dirs = torch.tensor(np.concatenate([lm, np.sqrt(1.0 - (lm ** 2).sum(1, keepdims=True)) - 1.0], 1), device=dev)
    f = torch.tensor(freq / C, device=dev)
    g = _generator(seed, dev)
    rows = torch.from_numpy(uvw.reshape(-1, 3)).to(dev)
    vis = torch.randn((rows.shape[0], len(freq), 2), generator=g, device=dev, dtype=torch.float32).mul_(0.1)
    vis = torch.view_as_complex(vis)
    step = max(1, (1 << 23) // len(freq))
    for a in range(0, rows.shape[0], step):
        path = rows[a:a + step] @ dirs.T
        for s in range(len(flux)):
            turns = path[:, s, None] * f
            ph = ((turns - torch.round(turns)) * (-2 * math.pi)).float()
            vis[a:a + step] += torch.polar(torch.full_like(ph, float(flux[s])), ph)
    return vis.reshape(uvw.shape[0], case["nt"], case["nch"])


def _model_image(n, seed):
    """A sky model: sparse points and a broad Gaussian, float32 [n][n]."""
    dev = _device()
    g = _generator(seed + 17, dev)
    img = torch.zeros(n * n, device=dev)
    at = torch.randint(0, n * n, (max(4, n // 8),), generator=g, device=dev)
    img[at] = torch.rand(len(at), generator=g, device=dev) + 0.05
    ax = torch.arange(n, device=dev, dtype=torch.float32) - n / 2
    y0, x0 = ((torch.rand(2, generator=g, device=dev) - 0.5) * n / 4).tolist()
    blob = torch.exp(-((ax - y0) / 12) ** 2)[:, None] * torch.exp(-((ax - x0) / 9) ** 2)[None]
    return img.reshape(n, n) + 0.01 * blob


def _model_grid(n, seed):
    """The forward transform of the (shifted) sky model: what DeGridW takes, complex64 [n][n]."""
    return torch.fft.fft2(torch.fft.ifftshift(_model_image(n, seed))).to(torch.complex64).contiguous()


def _psf(p, seed):
    """A cut PSF: a narrow beam on sidelobes that fall off, symmetric, float32 [p][p]."""
    dev = _device()
    g = _generator(seed + 29, dev)
    ax = torch.arange(p, device=dev, dtype=torch.float64) - p // 2
    r2 = ax[:, None] ** 2 + ax[None] ** 2
    lobes = torch.randn((p, p), generator=g, device=dev, dtype=torch.float64)
    lobes = 0.5 * (lobes + torch.roll(lobes.flip(0, 1), (1, 1), (0, 1)) if p % 2 == 0 else lobes + lobes.flip(0, 1))
    return (torch.exp(-r2 / 3.0) + 0.02 * lobes / (1 + r2 / 64.0).sqrt() * (r2 > 0)).float()


def _convolve(img, ker):
    """Linear convolution with a centred kernel, same size, 64 bits."""
    n, p = img.shape[0], ker.shape[0]
    m = n + p
    f = torch.fft.rfft2(img.double(), (m, m)) * torch.fft.rfft2(ker.double(), (m, m))
    return torch.fft.irfft2(f, (m, m))[p // 2:p // 2 + n, p // 2:p // 2 + n]


@functools.lru_cache(maxsize=1)
def _stream():
    """The one stream an imaging program keeps its gridding on."""
    return torch.cuda.Stream()


def _plan(case):
    uvw, freq, consts = _geom(case)
    c = pkg.GriddingConstants.from_dict(consts)
    part = pkg.Partitioner.CreatePartition(c, uvw, freq)
    part.plan.set_mode(MODES[case["mode"]])
    part.plan.set_stream(_stream().cuda_stream)
    return c, part


def prepare(case, seed):
    op, dev = case["op"], _device()
    st = dict(case=case)
    if op == "image":
        n, w = case["n"], case["w"]
        # a w stack as gridding leaves it: its energy in the inner uv plane (the corners after FFT.Shift)
        ax = torch.fft.ifftshift(torch.arange(n, device=dev, dtype=torch.float32) - n // 2) / (0.15 * n)
        env = torch.exp(-ax ** 2)
        z = torch.randn((w, n, n, 2), generator=_generator(seed, dev), device=dev)
        st["layers"] = torch.view_as_complex(z).mul_(env[:, None]).mul_(env)
        st["image"] = torch.empty((n, n), device=dev)
        uvw, freq = np.zeros((1, 1, 3)), np.array([1.2e9])
        c = pkg.GriddingConstants(1000, n, 32, 8, 1024, synth.cell_rad(1.5), w, 0.0)
        st["part"] = pkg.Partitioner.CreatePartition(c, uvw, freq)
        st["part"].plan.set_stream(_stream().cuda_stream)
        return st
    if op in ("correlate", "deconvolve"):
        n, p = case["n"], case["psf"]
        psf = _psf(p, seed)
        sky = _model_image(n, seed)
        dirty = _convolve(sky, psf)
        dirty += 0.01 * torch.randn((n, n), generator=_generator(seed + 5, dev), device=dev)
        whole = pkg.Rectangle(0, 0, n, n)
        if op == "correlate":
            st["dirty"] = dirty.float().contiguous()
            st["map"] = torch.empty((n, n), device=dev)
            st["conv"] = pkg.PaddedConvolver.correlation(psf.cpu().numpy(), whole)
        else:
            st["map0"] = _convolve(dirty, psf.flip(0, 1)).float().contiguous()
            st["x"], st["map"] = torch.empty((n, n), device=dev), torch.empty((n, n), device=dev)
            st["cd"] = pkg.FastSerialCD(whole, psf.cpu().numpy())
            st["lambda"] = 0.05 * float(st["cd"].MaxLipschitz)
        return st
    if op == "batch":
        probs = _problems(case)
        st["plans"] = [_plan(p) for p in probs]
        st["vis"] = [_visibilities(p, seed + i) for i, p in enumerate(probs)]
        st["grids"] = [_model_grid(p["n"], seed + i) for i, p in enumerate(probs)]
        st["layers"] = [torch.empty((p["w"], p["n"], p["n"]), dtype=torch.complex64, device=dev) for p in probs]
        st["out"] = [torch.empty_like(v) for v in st["vis"]]
        ptr = lambda k: [t.data_ptr() for t in st[k]]  # noqa: E731
        torch.cuda.synchronize()
        st["batch"] = pkg.Batch([p.plan for _, p in st["plans"]], ptr("vis"), ptr("layers"), ptr("grids"), ptr("out"))
        st["batch"].capture_graph()
        st["batch"].synchronize()
        return st
    n, w = case["n"], case["w"]
    uvw, st["freq"], _ = _geom(case)
    st["uvw"] = uvw
    st["c"], st["part"] = _plan(case)
    if op in ("grid", "step", "dirty_host"):
        st["vis"] = _visibilities(case, seed)
    if op in ("degrid", "step"):
        st["grid"] = _model_grid(n, seed)
        st["vis_out"] = torch.empty((uvw.shape[0], case["nt"], case["nch"]), dtype=torch.complex64, device=dev)
    if op in ("grid", "step"):
        st["layers"] = torch.empty((w, n, n), dtype=torch.complex64, device=dev)
    if op == "step":
        st["image"] = torch.empty((n, n), device=dev)
    if op == "dirty_host":
        st["vis"] = st["vis"].cpu().numpy().astype(np.complex128)
        st["layers"] = np.empty((w, n, n), np.complex128)
    if op == "predict_host":
        st["model"] = _model_image(n, seed).cpu().numpy()
        st["vis_out"] = np.empty((uvw.shape[0], case["nt"], case["nch"]), np.complex128)
    return st


def run(st):
    case = st["case"]
    op = case["op"]
    if op == "image":
        st["part"].plan.wstack_image_device(st["layers"].data_ptr(), st["image"].data_ptr())
        return st["image"]
    if op == "correlate":
        st["conv"].convolve_device(st["dirty"].data_ptr(), case["n"], st["map"].data_ptr())
        return st["map"]
    if op == "deconvolve":
        st["x"].zero_()
        st["map"].copy_(st["map0"])
        torch.cuda.current_stream().synchronize()  # the deconvolver works on a stream of its own
        r = st["cd"].deconvolve_device(st["x"].data_ptr(), st["map"].data_ptr(), st["lambda"], 0.2, case["iters"], 1e-5)
        return [st["x"], st["map"], r.IterationCount, int(r.Converged)]
    if op == "batch":
        st["batch"].run()
        return [st["layers"], st["out"]]
    c, part = st["c"], st["part"]
    plan = part.plan
    if op == "grid":
        plan.grid_w_device(st["vis"].data_ptr(), st["layers"].data_ptr())
        return st["layers"]
    if op == "degrid":
        plan.degrid_w_device(st["grid"].data_ptr(), st["vis_out"].data_ptr())
        return st["vis_out"]
    if op == "step":
        plan.grid_w_device(st["vis"].data_ptr(), st["layers"].data_ptr())
        plan.wstack_image_device(st["layers"].data_ptr(), st["image"].data_ptr())
        plan.degrid_w_device(st["grid"].data_ptr(), st["vis_out"].data_ptr())
        return [st["layers"], st["image"], st["vis_out"]]
    if op == "dirty_host":
        layers = pkg.IDG.GridW(c, part, st["vis"], st["uvw"], st["freq"], out=st["layers"])
        return [layers, pkg.FFT.WStackIFFTFloat(layers, c.VisibilitiesCount)]
    grid = pkg.FFT.Forward(st["model"])
    return pkg.IDG.DeGridW(c, part, grid, st["uvw"], st["freq"], out=st["vis_out"])


# ---------------------------------------------------------------- what a pass cannot do without

def work(case):
    op = case["op"]
    if op == "batch":
        parts = [work(dict(p, op=o)) for p in _problems(case) for o in ("grid", "degrid")]
        return {k: sum(w[k] for w in parts) for k in ("bytes", "flops")}
    n = case["n"]
    nn = n * n
    if op == "image":
        return dict(bytes=8 * nn * case["w"] + 4 * nn, flops=5 * nn * math.log2(nn))
    if op == "correlate":
        m = (n + case["psf"]) ** 2  # two real transforms of the padded size
        return dict(bytes=8 * nn + 8 * m, flops=5 * m * math.log2(m))
    if op == "deconvolve":
        win = min(n, 2 * case["psf"]) ** 2  # the update of PSF^2's window, each iteration
        return dict(bytes=16 * nn, flops=2.0 * win * case["iters"])
    subs = _partition(case)
    nvis, s = int(subs[:, 2].sum()) * case["nch"], case["s"]
    total = case["ants"] * (case["ants"] - 1) // 2 * case["nt"] * case["nch"]
    flops = 8.0 * s * s * nvis + len(subs) * 10 * s * s * math.log2(s)
    wide = 2 if op.endswith("_host") else 1
    grid = dict(bytes=wide * 8 * (nvis + nn * case["w"]), flops=flops)
    degrid = dict(bytes=wide * 8 * (nn + total), flops=flops)
    if op == "grid":
        return grid
    if op == "degrid":
        return degrid
    image = dict(bytes=4 * nn, flops=5 * nn * math.log2(nn))
    parts = {"step": (grid, image, degrid), "dirty_host": (grid, image), "predict_host": (image, degrid)}[op]
    return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}


# ---------------------------------------------------------------- 64-bit results

@functools.lru_cache(maxsize=32)
def _partition_of(key):
    """The subgrids (baseline, first time, times, u, v, w layer): the greedy partition of each
    baseline's track into boxes of at most subgrid - kernel pixels and 1024 times, all baselines at once."""
    uvw, freq, k = _geometry(key)
    nbl, nt, _ = uvw.shape
    size = float(np.float32(k["scale_arcsec"]) * np.float32(k["grid_size"]))
    f0, f1 = freq[0] / C, freq[-1] / C
    pts = [uvw[..., :2] * size * f for f in (f0, f1)]
    wl = uvw[..., 2] * f0
    wi = np.floor(wl / k["wstep"]).astype(np.int64) if k["wstep"] else np.zeros((nbl, nt), np.int64)
    lo, hi = np.full((nbl, 2), np.inf), np.full((nbl, 2), -np.inf)
    wb, time, count = np.zeros(nbl, np.int64), np.zeros(nbl, np.int64), np.zeros(nbl, np.int64)
    found = []
    shift = k["grid_size"] // 2 - k["subgrid_size"] // 2

    def close(b):
        c = np.rint((hi[b] + lo[b]) / 2).astype(np.int64) + shift
        found.append(np.stack([b, time[b] - count[b], count[b], c[:, 0], c[:, 1], wb[b]], 1))
        lo[b], hi[b], count[b] = np.inf, -np.inf, 0

    while True:
        b = np.nonzero(time < nt)[0]
        if not len(b):
            break
        ok = np.ones(len(b), bool)
        for p in pts:  # the first channel's point, then the last one's; a box keeps what it took in
            q, new = p[b, time[b]], np.isinf(lo[b, 0])
            nlo, nhi = np.minimum(lo[b], q), np.maximum(hi[b], q)
            ok &= (new | (wb[b] == wi[b, time[b]])) & ((nhi - nlo).max(1) + k["kernel_size"] < k["subgrid_size"])
            g = b[ok]
            lo[g], hi[g], wb[g] = nlo[ok], nhi[ok], wi[g, time[g]]
        g = b[ok]
        count[g] += 1
        time[g] += 1
        done = g[(count[g] == k["max_timesteps"]) | (time[g] == nt)]
        if len(done):
            close(done)
        bad = b[~ok]
        drop = bad[count[bad] == 0]
        if len(drop):
            lo[drop], hi[drop] = np.inf, -np.inf
            time[drop] += 1
        cut = bad[count[bad] > 0]
        if len(cut):
            close(cut)
    subs = np.concatenate(found) if found else np.zeros((0, 6), np.int64)
    return subs[np.lexsort((subs[:, 1], subs[:, 0]))]


def _partition(case):
    return _partition_of(tuple((k, case[k]) for k in _GEOMETRY_KEYS if k in case))


def _tables(case):
    """l [S] and n [S][S] of the subgrid pixels, as the method defines them: single precision."""
    s = case["s"]
    _, _, k = _geom(case)
    img = np.float32(k["scale_arcsec"]) * np.float32(case["n"])
    l = ((np.arange(s) - s // 2).astype(np.float32) + np.float32(0.5)) * img / np.float32(s)
    t = l[None, :] * l[None, :] + l[:, None] * l[:, None]
    n = t / (t.astype(np.float64) + np.sqrt(1.0 - t.astype(np.float64))).astype(np.float32)
    return l, n, float(img)


def _groups(case):
    """The subgrids in groups of about equal length: (subgrid rows, flat sample index, mask, du, dv, dw)."""
    subs = _partition(case)
    uvw, freq, _ = _geom(case)
    dev = _device()
    _, _, img = _tables(case)
    k = torch.tensor(2 * math.pi * freq / C, device=dev)
    flat = torch.from_numpy(uvw.reshape(-1, 3)).to(dev)
    order = np.argsort(-subs[:, 2], kind="stable")
    most = (1 << 20) // case["s"] * 16
    a = 0
    while a < len(order):
        length = int(subs[order[a], 2]) * case["nch"]
        rows = order[a:a + max(1, most // length)]
        a += len(rows)
        sub = torch.from_numpy(subs[rows]).to(dev)
        t = torch.arange(int(subs[rows[0], 2]), device=dev)
        mask = (t[None] < sub[:, 2:3])
        row = torch.where(mask, sub[:, 0:1] * case["nt"] + sub[:, 1:2] + t[None], 0)
        p = flat[row][:, :, None, :] * k[None, None, :, None]
        off = (sub[:, 3:5] + case["s"] // 2 - case["n"] // 2).double() * (2 * math.pi / img)
        idx = row[:, :, None] * case["nch"] + torch.arange(case["nch"], device=dev)
        full = (len(rows), -1)
        mask = mask[:, :, None].expand(-1, -1, case["nch"]).reshape(full)
        yield (sub, idx.reshape(full), mask, off[:, 0:1] - p[..., 0].reshape(full), off[:, 1:2] - p[..., 1].reshape(full),
               -p[..., 2].reshape(full))


def _factors(case):
    """n = f(x) + f(y) + r(y, x) on the subgrid, and l."""
    l, n, _ = _tables(case)
    n = torch.from_numpy(n.astype(np.float64)).to(_device())
    mid = case["s"] // 2
    f = n[mid] - n[mid, mid] / 2
    return torch.from_numpy(l.astype(np.float64)).to(_device()), f, n - f[:, None] - f[None, :]


def _expi(x):
    return torch.polar(torch.ones_like(x), x)


def _phasor(s):
    i = torch.arange(s, device=_device(), dtype=torch.float64)
    return _expi(math.pi * (i[:, None] + i[None, :] - s) / s)


def _shift_matrix(a):
    """FFT.Shift: the quadrants of the leading even part swap."""
    n2 = a.shape[-1] // 2
    b = a.clone()
    m = 2 * n2
    b[..., :m, :m] = torch.roll(a[..., :m, :m], (n2, n2), (-2, -1))
    return b


def _exact_layers(case, vis):
    s, n = case["s"], case["n"]
    l, f, r = _factors(case)
    out = torch.zeros((case["w"], n, n), dtype=torch.complex128, device=_device())
    half = (torch.arange(s, device=_device()) + s // 2) % s
    for sub, idx, mask, du, dv, dw in _groups(case):
        v = torch.where(mask, vis.reshape(-1)[idx].to(torch.complex128), 0)
        a = _expi(du[..., None] * l + dw[..., None] * f) * v[..., None]
        b = _expi(dv[..., None] * l + dw[..., None] * f).transpose(1, 2)
        eps, fac, j = float((dw.abs() * mask).max() * r.abs().max()), 1.0, 0
        pix = torch.zeros((len(sub), s, s), dtype=torch.complex128, device=_device())
        while fac > 1e-12:  # exp(i dw r) in powers of dw r
            pix += (1j * r) ** j / math.factorial(j) * torch.bmm(b, a)
            a, j = a * dw[..., None], j + 1
            fac *= eps / j
        img = torch.fft.ifft2(pix[:, half][:, :, half])[:, half][:, :, half] * _phasor(s)
        y, x, w = sub[:, 4], sub[:, 3], sub[:, 5]
        neg = w < 0
        img = torch.where(neg[:, None, None], img.flip(1, 2).conj(), img)
        x, y = torch.where(neg, n - x - s + 1, x), torch.where(neg, n - y - s + 1, y)
        w = torch.where(neg, -w - 1, w)
        keep = (x >= 1) & (x < n - s) & (y >= 1) & (y < n - s)
        x, y, w, img = x[keep], y[keep], w[keep], img[keep]
        i = torch.arange(s, device=_device())
        at = (w[:, None, None] * n + y[:, None, None] + i[:, None]) * n + x[:, None, None] + i
        flat = torch.view_as_real(out).reshape(-1, 2)
        flat.index_add_(0, at.reshape(-1), torch.view_as_real(img.contiguous()).reshape(-1, 2))
    return _shift_matrix(out)


def _exact_visibilities(case, grid):
    s, n = case["s"], case["n"]
    l, f, r = _factors(case)
    uvw, freq, _ = _geom(case)
    out = torch.zeros(uvw.shape[0] * case["nt"] * case["nch"], dtype=torch.complex128, device=_device())
    src = _shift_matrix(grid.to(torch.complex128)).reshape(-1)
    i = torch.arange(s, device=_device())
    half = (i + s // 2) % s
    for sub, idx, mask, du, dv, dw in _groups(case):
        x, y, neg = sub[:, 3, None, None], sub[:, 4, None, None], (sub[:, 5] < 0)[:, None, None]
        inside = (x >= 1) & (x < n - s) & (y >= 1) & (y < n - s)
        row = torch.where(neg, n - y - i[:, None], y + i[:, None])
        col = torch.where(neg, n - x - i, x + i)
        val = src[torch.where(inside, row * n + col, 0)]
        val = torch.where(neg, val.conj(), val) * _phasor(s).conj() * inside
        pix = torch.fft.fft2(val[:, half][:, :, half])[:, half][:, :, half]
        a = _expi(-(du[..., None] * l + dw[..., None] * f))
        b = _expi(-(dv[..., None] * l + dw[..., None] * f))
        eps, fac, j = float((dw.abs() * mask).max() * r.abs().max()), 1.0, 0
        vis = torch.zeros_like(du, dtype=torch.complex128)
        while fac > 1e-12:
            t = torch.bmm(a, ((-1j * r) ** j / math.factorial(j) * pix).transpose(1, 2))
            vis += dw ** j * (t * b).sum(-1)
            j += 1
            fac *= eps / j
        out[idx[mask]] = vis[mask] / (s * s)
    return out.reshape(uvw.shape[0], case["nt"], case["nch"])


def _exact_image(layers, vis_count, shift):
    img = torch.fft.ifft2(layers.sum(0).to(torch.complex128)).real * (layers.shape[-1] ** 2 / vis_count)
    return _shift_matrix(img) if shift else img


def exact(case, seed):
    op = case["op"]
    if op == "deconvolve":
        return None  # the sequence is defined in single precision; there is no 64-bit value of it
    if op == "image":
        return _exact_image(prepare(case, seed)["layers"].to(torch.complex128), 1000, True)
    if op == "correlate":
        n, p = case["n"], case["psf"]
        st = prepare(case, seed)
        img, psf = st["dirty"].double(), _psf(p, seed).double()
        m = n + p
        pad = torch.zeros((m, m), dtype=torch.float64, device=img.device)
        pad[n // 2 + 1:n // 2 + 1 + p, n // 2 + 1:n // 2 + 1 + p] = psf.flip(0, 1)
        box = torch.zeros_like(pad)
        box[p // 2:p // 2 + n, p // 2:p // 2 + n] = img
        full = torch.fft.ifft2(torch.fft.fft2(box) * torch.fft.fft2(_shift_matrix(pad))).real
        return full[p // 2:p // 2 + n, p // 2:p // 2 + n]
    if op == "batch":
        probs = _problems(case)
        return [[_exact_layers(p, _visibilities(p, seed + i)) for i, p in enumerate(probs)],
                [_exact_visibilities(p, _model_grid(p["n"], seed + i)) for i, p in enumerate(probs)]]
    if op in ("grid", "step", "dirty_host"):
        layers = _exact_layers(case, _visibilities(case, seed))
        if op == "grid":
            return layers
        image = _exact_image(layers, _geom(case)[2]["vis_count"], op == "step")
        if op == "dirty_host":
            return [layers, image]
        return [layers, image, _exact_visibilities(case, _model_grid(case["n"], seed))]
    if op == "degrid":
        return _exact_visibilities(case, _model_grid(case["n"], seed))
    # the model's transform takes the place of the single-precision one
    return _exact_visibilities(case, torch.fft.fft2(_model_image(case["n"], seed).double()))
