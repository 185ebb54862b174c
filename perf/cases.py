"""Performance cases of the imaging path, run through the package's public calls.

A case is a dict of plain values.  Its "path" names what is called:

  gridder    ops.gridder, batched: visibilities -> image-domain subgrids
  degridder  ops.degridder, batched: subgrids -> predicted visibilities
  grid       ops.grid_visibilities: gridder, subgrid FFT and adder in one step
  degrid     ops.degrid_visibilities: splitter, subgrid FFT and degridder
  cycle      one captured imaging cycle of an ops.Plan: zero the grid, grid, degrid
  adder      ops.TileBins.add into a cleared grid (the reproducible adder)
  image      ops.grid_fft: uv-grid to corrected image, out of place
  host       ops.imaging_cycle on page-locked host buffers

Geometries ("plan"): "even" cuts every baseline into subgrids of equal length
over all channels (10 km array, 150-160 MHz); "split" plans long baselines
(100 km, 100-200 MHz) with channel and time splitting, so subgrids have ragged
channel ranges and lengths; "uneven" has subgrids of 16 to 256 timesteps on
groups of 8 to 64 channels.  All arrays are single precision, which is the only
type of this path; all A-terms are near-identity and differ per station.
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "ska-spc-tender-benchmarks_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from idg_gb300 import datasets, ops  # noqa: E402

DEV = "cuda"
C_LIGHT = 299792458.0


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # A first look at a few seconds of a small array (8 stations, 64 s, 28 subgrids):
        # the smallest call, where launches and one subgrid's latency count.
        dict(name="gridder_28", path="gridder", plan="even", S=32, G=512, stations=8, steps=64, T=64, C=16),
        dict(name="degridder_28", path="degridder", plan="even", S=32, G=512, stations=8, steps=64, T=64, C=16),
        # The benchmark observation's subgrids (S = 32, 128 steps x 16 channels), a chunk of
        # them: what a host-driven pipeline hands to each kernel at a time.
        dict(name="gridder_4416", path="gridder", plan="even", S=32, G=4096, stations=24, steps=2048, T=128, C=16),
        dict(name="degridder_4416", path="degridder", plan="even", S=32, G=4096, stations=24, steps=2048, T=128, C=16),
        # Long baselines over a wide band on large subgrids: ragged channel ranges and lengths.
        dict(name="gridder_split64", path="gridder", plan="split", S=64, G=8192, stations=8, steps=512, T=128, C=64),
        dict(name="degridder_split32", path="degridder", plan="split", S=32, G=8192, stations=10, steps=512, T=128, C=64),
        # Subgrids of very different lengths, whole gridding and degridding steps on a
        # resident grid, at the two subgrid sizes that are no power of two.
        dict(name="grid_uneven24", path="grid", plan="uneven", S=24, G=1024, subgrids=2500, C=64),
        dict(name="degrid_uneven48", path="degrid", plan="uneven", S=48, G=1024, subgrids=1500, C=64),
        # The imaging loop: one cycle of a resident plan, replayed as a graph.
        dict(name="cycle_8128", path="cycle", plan="even", S=32, G=2048, stations=128, steps=128, T=128, C=16),
        # The reproducible adder alone, after a gridding step elsewhere.
        dict(name="adder_9180", path="adder", plan="even", S=32, G=2048, stations=136, steps=32, T=32, C=1),
        # The dirty image of a finished uv-grid.
        dict(name="image_4096", path="image", G=4096),
        # One cycle from and to host memory, copies included.
        dict(name="host_2016", path="host", plan="even", S=32, G=2048, stations=64, steps=64, T=64, C=16),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges."""
    path = rng.choice(["gridder", "degridder", "gridder", "degridder", "grid", "degrid", "cycle", "adder", "image", "host"])
    if path == "image":
        G = rng.choice([256, 512, 1024, 2048, 4096])
        return dict(path=path, G=G, planes=rng.randint(1, 3) if G < 4096 else 1)
    plan = rng.choice(["even", "even", "split", "uneven"]) if path in ("gridder", "degridder", "grid", "degrid") else "even"
    S = rng.choice([16, 24, 32, 32, 48, 64])
    case = dict(path=path, plan=plan, S=S)
    if plan == "uneven":
        case.update(G=rng.choice([1024, 2048]), subgrids=_log(rng, 30, 2000 if S <= 32 else 800), C=64)
    elif plan == "split":
        case.update(G=8192, stations=rng.randint(4, 9 if S <= 32 else 7), steps=rng.randint(100, 500),
                    T=rng.randint(32, 128), C=rng.randint(24, 64))
    else:
        # up to about the listed 4416 subgrids of 2048 visibilities at S = 32
        T, C = _log(rng, 5, 256), 1 if path == "adder" else _log(rng, 1, 48)
        per = T * C * S * S
        n = _log(rng, 28, max(40, min(8000, int(8e9 / per))))
        stations = max(4, min(100, int(math.sqrt(2 * n))))
        times = max(1, round(n / (stations * (stations - 1) / 2)))
        case.update(G=rng.choice([1024, 2048]), stations=stations, steps=T * times, T=T, C=C)
    if path in ("gridder", "degridder") and rng.random() < 0.3:
        case["w_step"] = 100.0  # w-stacking: the plan's planes enter the phases
    return case


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _uneven(case, seed):
    """Subgrids of 16-256 timesteps and 8-64 channels with rows of their own."""
    rng = np.random.default_rng(seed)
    n, S, G, C, ns, img = case["subgrids"], case["S"], case["G"], case["C"], 64, 0.05
    st = datasets.stations_in_disk(ns, 5000.0, rng)
    freqs = np.linspace(150e6, 160e6, C)
    # the same set of lengths for every seed (the arrays keep their shapes), in another order
    T = rng.permutation(np.exp(np.log(16) + (np.arange(n) + 0.5) / n * np.log(257 / 16)).astype(np.int64))
    s1 = rng.integers(0, ns - 1, n)
    s2 = s1 + 1 + (rng.random(n) * (ns - 1 - s1)).astype(np.int64)
    glen = rng.choice([8, 16, 32, 64], n)
    c0 = (rng.random(n) * (C // glen)).astype(np.int64) * glen
    start = np.concatenate([[0], np.cumsum(T)[:-1]])
    of = np.repeat(np.arange(n), T)
    H = (rng.uniform(-4, 4, n) * 3600)[of] + (np.arange(T.sum()) - start[of])
    H = H * datasets.EARTH_ROTATION_RATE
    lat = dec = np.deg2rad(-30.0)
    enu = (st[s2] - st[s1])[of]
    X, Y, Z = -np.sin(lat) * enu[:, 1], enu[:, 0], np.cos(lat) * enu[:, 1]
    u = np.sin(H) * X + np.cos(H) * Y
    v = -np.sin(dec) * np.cos(H) * X + np.sin(dec) * np.sin(H) * Y + np.cos(dec) * Z
    w = np.cos(dec) * np.cos(H) * X - np.cos(dec) * np.sin(H) * Y + np.sin(dec) * Z
    uvw = np.stack([u, v, w], 1).astype(np.float32)
    md = np.zeros(n, datasets.METADATA_DTYPE)
    md["time_offset"], md["nr_timesteps"], md["station1"], md["station2"] = start, T, s1, s2
    for k, name in ((0, "x"), (1, "y")):
        a = uvw[:, k].astype(np.float64) * img / C_LIGHT
        lo, hi = np.minimum.reduceat(a, start), np.maximum.reduceat(a, start)
        fa, fb = freqs[c0], freqs[c0 + glen - 1]
        mid = 0.5 * (np.minimum(lo * fa, lo * fb) + np.maximum(hi * fa, hi * fb))
        md[name] = np.floor(mid + G / 2 - S / 2 + 0.5)
    return md, np.stack([c0, c0 + glen], 1).astype(np.int32), uvw, freqs, ns, 1


def _inputs(case, seed):
    """The arrays of a case on the GPU, and its plan on the host."""
    S, G, C = case["S"], case["G"], case["C"]
    w_step, W = float(case.get("w_step", 0.0)), 1
    if case["plan"] == "uneven":
        md, ext, uvw, freqs, ns, slots = _uneven(case, seed)
    else:
        split = case["plan"] == "split"
        o = datasets.ObservationSpec(
            nstations=case["stations"], disk_radius_m=50000.0 if split else 5000.0, ntimesteps=case["steps"],
            timesteps_per_subgrid=case["T"], nchannels=C, f_start=100e6 if split else 150e6,
            f_end=200e6 if split else 160e6, subgrid_size=S, grid_size=G, image_size=0.05, w_step=w_step,
            aterm_interval=256, nr_w_planes=8,
            # how many subgrids a split plan has follows from its geometry: that one keeps its stations
            seed=case["stations"] if split else seed % (1 << 31))
        ob = datasets.make_observation(o, split=split)
        md, uvw, freqs, ns, slots = ob.metadata, ob.uvw, ob.frequencies, case["stations"], o.n_aterm_slots
        ext = ob.ext.view(np.int32).reshape(-1, 2) if split else None
        if w_step and not split:
            w = uvw[md["time_offset"] + md["nr_timesteps"] // 2, 2] * freqs.mean() / C_LIGHT
            md["z"] = np.floor(w / w_step)
    k = (2 * np.pi * freqs / C_LIGHT).astype(np.float32)
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)

    def normal(*shape):
        return torch.view_as_complex(torch.randn(*shape, 2, generator=g, device=DEV))

    eye = torch.tensor([1, 0, 0, 1], dtype=torch.complex64, device=DEV)
    return dict(
        spec=ops.GridSpec(G, S, C, ns, slots, W, 0.05, w_step), md_host=md, ext_host=ext,
        md=ops.metadata_tensor(md, DEV), ext=None if ext is None else torch.from_numpy(ext.copy()).to(DEV),
        uvw_host=uvw, uvw=torch.from_numpy(uvw).to(DEV), k_host=k, k=torch.from_numpy(k).to(DEV),
        taper_host=datasets.pswf_taper(S), taper=torch.from_numpy(datasets.pswf_taper(S)).to(DEV),
        aterms=eye + 0.05 * normal(slots, ns, S, S, 4), normal=normal)


def _image_inputs(case, seed):
    G, W = case["G"], case.get("planes", 1)
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    grid = torch.view_as_complex(torch.randn(W, 4, G, G, 2, generator=g, device=DEV))
    x = torch.linspace(-1, 1, G, device=DEV)
    return grid, (1.0 / (1.0 - 0.5 * x * x)).contiguous()


def _visibilities(d):
    return d["normal"](d["uvw"].shape[0], d["spec"].nr_channels, 4)


def _subgrids(d):
    S = d["spec"].subgrid_size
    return d["normal"](d["md"].shape[0], 4, S, S)


def _grid(d):
    G = d["spec"].grid_size
    return d["normal"](1, 4, G, G)


def prepare(case, seed):
    path = case["path"]
    if path == "image":
        grid, corr = _image_inputs(case, seed)
        G = case["G"]
        return dict(path=path, spec=ops.GridSpec(G, 32, 1, 1, nr_w_planes=grid.shape[0], image_size=0.05), grid=grid,
                    corr=corr, image=torch.empty_like(grid))
    d = _inputs(case, seed)
    s = dict(d, path=path)
    spec, rows, C = d["spec"], d["uvw"].shape[0], d["spec"].nr_channels
    S, G, N = spec.subgrid_size, spec.grid_size, d["md"].shape[0]

    def empty(*shape):
        return torch.empty(shape, dtype=torch.complex64, device=DEV)

    if path in ("gridder", "grid", "cycle", "host"):
        s["vis"] = _visibilities(d)
    if path in ("degridder", "degrid", "cycle"):
        s["out"] = torch.zeros((rows, C, 4), dtype=torch.complex64, device=DEV)
    if path in ("gridder", "grid", "degrid"):
        s["subgrids"] = empty(N, 4, S, S)
    if path in ("degridder", "adder"):
        s["subgrids"] = _subgrids(d)
    if path == "degrid":
        s["grid"] = _grid(d)
    if path in ("grid", "cycle", "adder"):
        s["grid"] = torch.zeros((1, 4, G, G), dtype=torch.complex64, device=DEV)
    if path == "adder":
        s["bins"] = ops.TileBins(spec, d["md_host"])
    if path == "cycle":
        s["plan"] = ops.Plan(spec, d["md_host"], rows)
        s["plan"].capture_cycle(d["uvw"], d["k"], s["vis"], d["taper"], d["aterms"], s["grid"], s["out"])
    if path == "host":
        s["vis_host"] = s.pop("vis").cpu().pin_memory()
        s["aterms_host"] = d["aterms"].cpu().pin_memory()
        s["out_host"] = torch.zeros((rows, C, 4), dtype=torch.complex64).pin_memory()
        s["grid_host"] = torch.zeros((1, 4, G, G), dtype=torch.complex64).pin_memory()
    return s


def run(s):
    path = s["path"]
    if path == "image":
        s["image"].copy_(s["grid"])
        return ops.grid_fft(s["spec"], s["image"], -1, s["corr"])
    common = (s["spec"], s["md"], s["uvw"], s["k"])
    if path == "gridder":
        return ops.gridder(*common, s["vis"], s["taper"], s["aterms"], s["subgrids"], variant=ops.VARIANT_BATCHED,
                           ext=s["ext"])
    if path == "degridder":
        return ops.degridder(*common, s["out"], s["taper"], s["aterms"], s["subgrids"], variant=ops.VARIANT_BATCHED,
                             ext=s["ext"])
    if path == "grid":
        s["grid"].zero_()
        return ops.grid_visibilities(*common, s["vis"], s["taper"], s["aterms"], s["subgrids"], s["grid"], ext=s["ext"])
    if path == "degrid":
        return ops.degrid_visibilities(*common, s["out"], s["taper"], s["aterms"], s["subgrids"], s["grid"],
                                       ext=s["ext"])
    if path == "cycle":
        s["plan"].launch_cycle()
        return dict(grid=s["grid"], vis=s["out"])
    if path == "adder":
        s["grid"].zero_()
        return s["bins"].add(s["subgrids"], s["grid"])
    ops.imaging_cycle(s["spec"], s["md_host"], s["uvw_host"], s["k_host"], s["vis_host"], s["taper_host"],
                      s["aterms_host"], s["out_host"], s["grid_host"], chunk_subgrids=-1)
    return dict(grid=s["grid_host"], vis=s["out_host"])


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
def _sizes(case):
    """(subgrids, rows, visibilities) of a case, without making its arrays."""
    if case["plan"] == "even":
        per = case["steps"] // case["T"]
        n = case["stations"] * (case["stations"] - 1) // 2
        return n * per, n * case["steps"], n * per * case["T"] * case["C"]
    if case["plan"] == "uneven":
        n = case["subgrids"]
        rows = n * 240 / math.log(257 / 16)  # mean length of a log-uniform draw
        return n, rows, rows * 30
    n = case["stations"] * (case["stations"] - 1) // 2
    rows = n * case["steps"]
    return 3 * n * max(1, case["steps"] // case["T"]), rows, rows * case["C"]


def work(case):
    path = case["path"]
    if path == "image":
        G, W = case["G"], case.get("planes", 1)
        return {"bytes": 2 * W * 4 * G * G * 8 + 4 * G, "flops": W * 4 * 5 * G * G * 2 * math.log2(G)}
    n, rows, nvis = _sizes(case)
    S, G = case["S"], case["G"]
    sub, vis, grid = 32 * S * S * n, 32 * nvis + 12 * rows, 32 * G * G
    # gridding and degridding: four complex multiply-adds per pixel and visibility
    mac, fft = 32 * nvis * S * S, n * 4 * 5 * S * S * 2 * math.log2(S)
    total = {
        "gridder": (vis + sub, mac), "degridder": (vis + sub, mac),
        "grid": (vis + grid, mac + fft), "degrid": (vis + grid, mac + fft),
        "cycle": (2 * vis + grid, 2 * (mac + fft)), "host": (2 * vis + grid, 2 * (mac + fft)),
        "adder": (sub + grid, 2 * 4 * S * S * n),
    }[path]
    return {"bytes": int(total[0] + 36 * n), "flops": int(total[1])}


# ---------------------------------------------------------------------------
# The same outputs in 64 bits
# ---------------------------------------------------------------------------
def _phase_terms(d, i):
    """(pixels x visibilities) phases of subgrid i, its rows and channels."""
    sp, m = d["spec"], d["md_host"][i]
    S, G, img = sp.subgrid_size, sp.grid_size, float(np.float32(sp.image_size))
    ax = (torch.arange(S, device=DEV, dtype=torch.float64) + 0.5 - S / 2) * (img / S)
    l, mm = ax.repeat(S), ax.repeat_interleave(S)
    r2 = l * l + mm * mm
    n = r2 / (1 + torch.sqrt(1 - r2))
    rows = slice(int(m["time_offset"]), int(m["time_offset"]) + int(m["nr_timesteps"]))
    c0, c1 = (0, sp.nr_channels) if d["ext_host"] is None else (int(v) for v in d["ext_host"][i])
    uvw, k = d["uvw"][rows].double(), d["k"][c0:c1].double()
    step = 2 * math.pi / img
    off = ((int(m["x"]) + S / 2 - G / 2) * step * l + (int(m["y"]) + S / 2 - G / 2) * step * mm
           + 2 * math.pi * float(np.float32(sp.w_step)) * (int(m["z"]) + 0.5) * n)
    q = torch.stack([l, mm, n]).T @ uvw.T
    return (off[:, None, None] - q[:, :, None] * k).reshape(S * S, -1), rows, slice(c0, c1)


def _jones(d, i):
    m = d["md_host"][i]
    S = d["spec"].subgrid_size
    a = d["aterms"][int(m["aterm_index"])].to(torch.complex128)
    return (a[int(m["station1"])].reshape(S * S, 2, 2), a[int(m["station2"])].reshape(S * S, 2, 2))


def _exact_gridder(d, vis, tapered):
    S, N = d["spec"].subgrid_size, d["md_host"].shape[0]
    out = torch.empty((N, 4, S, S), dtype=torch.complex128, device=DEV)
    taper = d["taper"].double().reshape(-1) if tapered else 1.0
    for i in range(N):
        phase, rows, chans = _phase_terms(d, i)
        v = torch.view_as_real(vis[rows, chans].reshape(-1, 4)).double().reshape(-1, 8)
        c, s = phase.cos() @ v, phase.sin() @ v
        px = torch.complex(c[:, 0::2] - s[:, 1::2], c[:, 1::2] + s[:, 0::2]).reshape(-1, 2, 2)
        a1, a2 = _jones(d, i)
        px = a1.mH @ px @ a2
        out[i] = (px.reshape(-1, 4).T * taper).reshape(4, S, S)
    return out


def _exact_degridder(d, sub, tapered):
    S, N = d["spec"].subgrid_size, d["md_host"].shape[0]
    out = torch.zeros((d["uvw"].shape[0], d["spec"].nr_channels, 4), dtype=torch.complex128, device=DEV)
    taper = d["taper"].double().reshape(-1) if tapered else 1.0
    for i in range(N):
        phase, rows, chans = _phase_terms(d, i)
        px = (sub[i].to(torch.complex128).reshape(4, -1) * taper).T.reshape(-1, 2, 2)
        a1, a2 = _jones(d, i)
        px = torch.view_as_real((a1 @ px @ a2.mH).reshape(-1, 4)).reshape(-1, 8)
        c, s = phase.cos().T @ px, phase.sin().T @ px
        v = torch.complex(c[:, 0::2] + s[:, 1::2], c[:, 1::2] - s[:, 0::2])
        out[rows, chans] = v.reshape(rows.stop - rows.start, -1, 4)
    return out


def _subgrid_dft(S):
    j = torch.arange(S, device=DEV, dtype=torch.float64) - S / 2
    return torch.polar(torch.ones((S, S), device=DEV, dtype=torch.float64), 2 * math.pi / S * j[:, None] * (j + 0.5))


def _cells(d, i):
    """The part of subgrid i inside the grid: (grid y, grid x, subgrid y, subgrid x) slices."""
    S, G = d["spec"].subgrid_size, d["spec"].grid_size
    x, y = int(d["md_host"][i]["x"]), int(d["md_host"][i]["y"])
    gx, gy = (max(0, x), min(G, x + S)), (max(0, y), min(G, y + S))
    return slice(*gy), slice(*gx), slice(gy[0] - y, gy[1] - y), slice(gx[0] - x, gx[1] - x)


def _exact_add(d, sub):
    G = d["spec"].grid_size
    grid = torch.zeros((1, 4, G, G), dtype=torch.complex128, device=DEV)
    for i in range(sub.shape[0]):
        gy, gx, sy, sx = _cells(d, i)
        grid[0, :, gy, gx] += sub[i, :, sy, sx]
    return grid


def _exact_grid_step(d, vis):
    e = _subgrid_dft(d["spec"].subgrid_size)
    sub = _exact_gridder(d, vis, False) * d["taper"].double()
    return _exact_add(d, e @ sub @ e.T)


def _exact_degrid_step(d, grid):
    S = d["spec"].subgrid_size
    sub = torch.zeros((d["md_host"].shape[0], 4, S, S), dtype=torch.complex128, device=DEV)
    for i in range(sub.shape[0]):
        gy, gx, sy, sx = _cells(d, i)
        sub[i, :, sy, sx] = grid[0, :, gy, gx]
    e = _subgrid_dft(S)
    return _exact_degridder(d, (e.mH @ sub @ e.conj()) * d["taper"].double(), False)


def exact(case, seed):
    path = case["path"]
    if path == "image":
        grid, corr = _image_inputs(case, seed)
        G = case["G"]
        out = torch.empty(grid.shape, dtype=torch.complex128, device=DEV)
        c = corr.double()
        for w in range(grid.shape[0]):
            for p in range(4):  # centre cell G/2 is the origin of both domains
                a = torch.fft.ifftshift(grid[w, p].to(torch.complex128))
                out[w, p] = torch.fft.fftshift(torch.fft.fft2(a)) * c[:, None] * c[None, :]
        return out
    if path != "adder" and _sizes(case)[2] * case["S"] ** 2 > 2.5e10:
        return None
    d = _inputs(case, seed)
    if path == "gridder":
        return _exact_gridder(d, _visibilities(d), True)
    if path == "degridder":
        return _exact_degridder(d, _subgrids(d), True)
    if path == "grid":
        return _exact_grid_step(d, _visibilities(d))
    if path == "degrid":
        return _exact_degrid_step(d, _grid(d))
    if path == "adder":
        return _exact_add(d, _subgrids(d).to(torch.complex128))
    grid = _exact_grid_step(d, _visibilities(d))
    return dict(grid=grid, vis=_exact_degrid_step(d, grid))
