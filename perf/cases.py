"""Workloads for timing the framework through its public entry points: the
Python mirror (peakpatch_b200.Context) and, where the arrays live on the GPU,
the C ABI of include/ppb.h that the mirror loads.

A case is a dict of plain values whose "kind" names the entry point:

  noise   ppb_noise_threefry         white noise on an n^3 grid
  fields  ppb_generate_fields        delta, 1LPT, 2LPT (and Laplacian) of a tile
  peaks   ppb_peak_find_tile         filter bank + peak search of one field
  shells  ppb_analyse_peaks_lim      radial-shell collapse of a batch of peaks
  tile    Context.run_tile_into      one tile, records to device memory
  split   Context.run_multitile_split_arrays   multi-resolution tiles
  chain   Context.run_multitile_arrays + merge_catalog   a lightcone and its catalogue
  table   Context.make_table         a collapse table
  serve   Context.submit / wait      a burst of mixed requests

Peak lists and catalogues are returned as the caller's whole buffers (zero
beyond the count) with their counts.  One context (the package's default one) serves every case, as a program that
links the library keeps one; the P(k) and collapse tables stay installed.
The cell is 2 Mpc/h and the P(k) table Eisenstein-Hu (sigma8 0.808) unless a
case says otherwise.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "peakpatch.jl_b200"))

import peakpatch_b200 as pp  # noqa: E402
from peakpatch_b200 import powerspec  # noqa: E402

OMB, OMV, H = 0.049, 0.685, 0.674
OM = 0.315


def listed():
    return [
        # white noise of a small box: the smallest call, launch latency
        {"name": "noise_64", "kind": "noise", "n": 64},
        # the fields of the example configuration's 142^3 tile (2 x 71: not a smooth size)
        {"name": "fields_142", "kind": "fields", "n": 142, "ilpt": 2, "shear": 0, "cell": 200.0 / 142},
        # the fields of the benchmark tile, Laplacian included
        {"name": "fields_384", "kind": "fields", "n": 384, "ilpt": 2, "shear": 1, "cell": 2.0},
        # a filter bank with the k^2-weighted twin on a caller's field
        {"name": "peaks_192", "kind": "peaks", "n": 192, "nbuff": 16, "nfilt": 20, "ws": 1, "shear": 1, "cell": 2.0},
        # a batch of peaks of all radii on a caller's fields (a catalogue's re-analysis)
        {"name": "shells_256", "kind": "shells", "n": 256, "npk": 200000, "nhunt": 24, "rmed": 6.0, "shear": 1,
         "plain": 0},
        # the small tile of a served stream or a parameter scan
        {"name": "tile_128", "kind": "tile", "n": 128, "nbuff": 16, "nfilt": 20, "rmax": 30.0, "ws": 1, "shear": 1,
         "ilpt": 2, "ievol": 0, "rmax2rs": 0.0, "cell": 2.0},
        # the example configuration: 142^3, Gaussian filters, 11-field records, capped shell lists
        {"name": "tile_142", "kind": "tile", "n": 142, "nbuff": 4, "nfilt": 16, "rmax": 32.0, "ws": 0, "shear": 0,
         "ilpt": 2, "ievol": 0, "rmax2rs": 1.0, "cell": 200.0 / 142},
        # the benchmark tile
        {"name": "tile_384", "kind": "tile", "n": 384, "nbuff": 32, "nfilt": 20, "rmax": 30.0, "ws": 1, "shear": 1,
         "ilpt": 2, "ievol": 0, "rmax2rs": 0.0, "cell": 2.0},
        # the multi-resolution sweep's middle size, 8 tiles
        {"name": "split_192", "kind": "split", "n": 192, "nbuff": 8, "ntile": 2, "cell": 226.67 / 68 * 368 / 192,
         "ilpt": 2, "shear": 0},
        # a lightcone of four tiles, then the merged catalogue
        {"name": "chain_192", "kind": "chain", "n": 192, "nbuff": 16, "ntile": 2, "tiles": 4, "shear": 1, "cell": 2.0},
        # the reference's collapse table size
        {"name": "table_50", "kind": "table", "nx": 50, "ny": 20, "nz": 20},
        # requests of mixed sizes arriving at once
        {"name": "serve_8", "kind": "serve", "requests": 8, "nmax": 256},
    ]


def draw(rng):
    def size(lo, hi, even=False):
        v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
        if rng.random() < 0.4:   # grids are usually multiples of 16
            v = max(lo, 16 * round(v / 16))
        return v + (v & 1) if even else v

    kind = rng.choice(["noise", "fields", "peaks", "shells", "tile", "tile", "tile", "split", "chain", "table",
                       "serve"])
    cell = round(rng.uniform(1.2, 2.4), 3)
    if kind == "noise":
        return {"kind": kind, "n": size(32, 320)}
    if kind == "fields":
        return {"kind": kind, "n": size(48, 384), "ilpt": rng.choice([1, 2, 2]), "shear": rng.randint(0, 1),
                "cell": cell}
    if kind == "peaks":
        n = size(64, 256)
        return {"kind": kind, "n": n, "nbuff": rng.randint(4, n // 8), "nfilt": rng.randint(4, 20),
                "ws": rng.choice([0, 1, 1, 3]), "shear": rng.randint(0, 1), "cell": cell}
    if kind == "shells":
        return {"kind": kind, "n": size(96, 256), "npk": int(math.exp(rng.uniform(math.log(500), math.log(200000)))),
                "nhunt": rng.randint(8, 24), "rmed": round(rng.uniform(3.0, 6.0), 2), "shear": rng.randint(0, 1),
                "plain": int(rng.random() < 0.15)}
    if kind == "tile":
        n = size(64, 360)
        return {"kind": kind, "n": n, "nbuff": rng.randint(max(4, n // 24), n // 8), "nfilt": rng.randint(4, 20),
                "rmax": round(rng.uniform(10.0, 30.0), 2), "ws": rng.choice([0, 1, 1]), "shear": rng.randint(0, 1),
                "ilpt": rng.choice([1, 2, 2]), "ievol": int(rng.random() < 0.3), "rmax2rs": rng.choice([0.0, 0.0, 1.0]),
                "cell": cell}
    if kind == "split":
        return {"kind": kind, "n": 16 * rng.randint(5, 12), "nbuff": 8, "ntile": 2,
                "cell": round(rng.uniform(4.0, 6.4), 3), "ilpt": rng.choice([1, 2]), "shear": rng.randint(0, 1)}
    if kind == "chain":
        n = size(80, 192, even=True)
        return {"kind": kind, "n": n, "nbuff": rng.randint(8, n // 10 + 2), "ntile": 2, "tiles": rng.randint(2, 4),
                "shear": rng.randint(0, 1), "cell": cell}
    if kind == "table":
        return {"kind": kind, "nx": rng.randint(10, 50), "ny": rng.randint(6, 20), "nz": rng.randint(6, 20)}
    return {"kind": kind, "requests": rng.randint(3, 8), "nmax": rng.choice([128, 192, 256])}


# --------------------------------------------------------------------------
# what a program holds before the call
# --------------------------------------------------------------------------
_ready = {}


def _context():
    """The package's default context with the resident tables installed."""
    if not _ready:
        ctx = pp.default_context()
        k, pk = powerspec.eh_table()
        ctx.set_pk_table(k, pk)
        tab = pp.read_homeltab(os.path.join(ROOT, "tests", "golden", "HomelTab_julia.dat"))
        ctx.set_collapse_table(tab)
        _ready.update(ctx=ctx, k=k, pk=pk, tab=tab)
    return _ready["ctx"]


def _bank(nfilt, rmax=30.0, rmin=1.5):
    """Log-spaced filter radii (Mpc/h), the benchmark's bank for 20 of 1.5 to 30."""
    return [float(rmin * (rmax / rmin) ** (i / (nfilt - 1))) for i in range(nfilt)]


def _config(c, **more):
    d = dict(Omx=OM - OMB, OmB=OMB, Omvac=OMV, h=H, n=c["n"], boxsize=c["cell"] * c["n"], nbuff=c.get("nbuff", 4),
             z_out=0.0, z_max=0.0, ievol=c.get("ievol", 0), ilpt=c.get("ilpt", 2), ioutshear=c["shear"],
             wsmooth=c.get("ws", 1), rmax2rs=c.get("rmax2rs", 0.0))
    if d["ievol"]:   # an observer at the box corner
        edge = -0.5 * d["boxsize"]
        d.update(z_max=1.2, cenx=edge, ceny=edge, cenz=edge)
    d.update(more)
    return pp.PipelineConfig(**d)


def _kgrid(n, box, dtype=torch.float64):
    f = torch.fft.fftfreq(n, 1.0 / n, device="cuda", dtype=dtype) * (2 * math.pi / box)
    r = torch.arange(n // 2 + 1, device="cuda", dtype=dtype) * (2 * math.pi / box)
    return r[None, None, :], f[None, :, None], f[:, None, None]


def _gaussian_field(n, cell, seed, slope=None, sigma=None):
    """A Gaussian field on the GPU: the resident P(k), or A k^slope of unit-cell rms sigma."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    w = torch.fft.rfftn(torch.randn(n, n, n, generator=g, device="cuda", dtype=torch.float32))
    kx, ky, kz = _kgrid(n, n * cell, torch.float32)
    k = torch.sqrt(kx * kx + ky * ky + kz * kz)
    k[0, 0, 0] = 1.0
    if slope is not None:
        amp = k ** (slope / 2)
    else:
        lk, lp = np.log(_ready["k"]), np.log(_ready["pk"])
        x = (torch.log(k) - float(lk[0])) / float(lk[1] - lk[0])   # the table is log-spaced
        i = x.long().clamp(0, len(lk) - 2)
        t = torch.from_numpy(lp).float().cuda()
        amp = torch.exp(0.5 * (t[i] + (x - i) * (t[i + 1] - t[i]))) * (2 * math.pi / cell) ** 1.5
    amp[0, 0, 0] = 0.0
    dk = w * amp
    d = torch.fft.irfftn(dk, s=(n, n, n))
    if sigma is not None:
        s = sigma / d.square().mean().sqrt()
        dk, d = dk * s, d * s
    return d.contiguous(), dk


def _catalogue(cells, shear):
    return torch.zeros((cells // 30 + 1024, 33 if shear else 11), device="cuda")


def prepare(case, seed):
    ctx = _context()
    c, kind = case, case["kind"]
    s = {"ctx": ctx, "c": c, "kind": kind, "seed": seed}
    if kind == "noise":
        s["out"] = torch.empty((c["n"],) * 3, device="cuda")
    elif kind == "fields":
        n = c["n"]
        s["p"] = ctx._params(_config(c), seed, False)
        s["delta"] = torch.empty((n, n, n), device="cuda")
        s["psi"] = torch.empty((3, n, n, n), device="cuda")
        s["psi2"] = torch.empty((3, n, n, n), device="cuda") if c["ilpt"] == 2 else None
        s["lapd"] = torch.empty((n, n, n), device="cuda") if c["shear"] else None
    elif kind == "peaks":
        n = c["n"]
        s["delta"] = _gaussian_field(n, c["cell"], seed)[0]
        s["Rf"] = np.array(_bank(c["nfilt"])[::-1])   # largest first
        s["fc"] = np.full(c["nfilt"], 1.686)
        s["mask"] = torch.zeros((n, n, n), dtype=torch.int8, device="cuda")
        cap = s["cap"] = max(1, n ** 3 // 30)
        for k in ("i", "j", "k", "filter"):
            s[k] = torch.zeros(cap, dtype=torch.int32, device="cuda")
        s["ipp"] = torch.zeros(cap, dtype=torch.int64, device="cuda")
        for k in ("x", "y", "z", "R"):
            s[k] = torch.zeros(cap, dtype=torch.float64, device="cuda")
        for k in ("FcRf", "d2Rf"):
            s[k] = torch.zeros(cap, device="cuda")
    elif kind == "shells":
        n, npk, cell = c["n"], c["npk"], 2.0
        s["delta"], dk = _gaussian_field(n, cell, seed, slope=-2.5, sigma=1.0)
        kx, ky, kz = _kgrid(n, n * cell, torch.float32)
        k2 = kx * kx + ky * ky + kz * kz
        k2[0, 0, 0] = 1.0
        s["psi"] = torch.stack([torch.fft.irfftn(1j * q / k2 * dk, s=(n, n, n)) for q in (kx, ky, kz)])
        # a second-order field of the right size and correlation length
        src = torch.fft.rfftn(0.5 * s["delta"] ** 2)
        s["psi2"] = torch.stack([torch.fft.irfftn(-1j * q / k2 * src * torch.exp(-2 * k2), s=(n, n, n))
                                 for q in (kx, ky, kz)])
        s["lapd"] = torch.fft.irfftn(k2 * dk, s=(n, n, n)).contiguous() if c["shear"] else None
        g = torch.Generator(device="cuda").manual_seed(seed + 1)
        s["ipp"] = torch.randint(1, n ** 3 + 1, (npk,), generator=g, device="cuda")
        rmax = float(c["nhunt"])
        r = torch.exp(math.log(c["rmed"]) + 0.5 * torch.randn(npk, generator=g, device="cuda", dtype=torch.float64))
        r = r.clamp(2.0, rmax)
        s["Rf"] = r * cell
        s["ir2"] = torch.floor((1.75 * r) ** 2).clamp(max=math.floor((40.0 / cell - 1) ** 2)).long()
        s["lim"] = torch.floor(r * r).int()
        s["Z"] = torch.ones(npk, dtype=torch.float64, device="cuda")
        s["fc"] = torch.full((npk,), 1.686, dtype=torch.float64, device="cuda")
        s["out"] = torch.empty((npk, 31), dtype=torch.float64, device="cuda")
    elif kind == "tile":
        s["cfg"] = _config(c)
        s["Rf"] = _bank(c["nfilt"], c["rmax"])
        s["rec"] = _catalogue(c["n"] ** 3, c["shear"])
    elif kind == "split":
        s["cfg"] = _config(c)
        s["Rf"] = [8.0, 5.0, 3.0]
        s["p"] = ctx._params(s["cfg"], seed, False)
        s["rec"] = _catalogue(((c["n"] - 2 * c["nbuff"]) * c["ntile"]) ** 3, c["shear"])
    elif kind == "chain":
        ncore = (c["n"] - 2 * c["nbuff"]) * c["ntile"]
        edge = -ncore * c["cell"] / 2
        s["cfg"] = _config(c, ievol=1, z_max=4.6, cenx=edge, ceny=edge, cenz=edge)
        s["Rf"] = _bank(20)
        s["tiles"] = np.array([(1, 1, 1), (2, 1, 1), (1, 2, 1), (2, 2, 1)][:c["tiles"]], np.int32)
        s["p"] = ctx._params(s["cfg"], seed, False)
        s["rec"] = _catalogue(c["tiles"] * (c["n"] - 2 * c["nbuff"]) ** 3, c["shear"])
        s["merged"] = torch.zeros_like(s["rec"])
    elif kind == "table":
        s["tp"] = pp.CollapseTableParams(Nx=c["nx"], Ny=c["ny"], Nz=c["nz"])
        s["Om"] = 0.30 + 0.02 * ((seed * 2654435761) % 1000003) / 1000003.0
    elif kind == "serve":
        r = np.random.default_rng(seed)
        sizes = [n for n in (128, 192, 256) if n <= c["nmax"]]
        s["req"], s["rec"] = [], []
        for q in range(c["requests"]):
            n = sizes[q % len(sizes)]
            t = {"n": n, "nbuff": n // 12, "cell": 2.0, "shear": 1, "ievol": q % 2}
            s["req"].append((_config(t), int(r.integers(1 << 30)), float(r.uniform(0.75, 0.85) / 0.808) ** 2))
            s["rec"].append(_catalogue(n ** 3, 1))
        s["Rf"] = _bank(20)
    return s


def _ptr(t):
    return None if t is None else ctypes.c_void_p(t.data_ptr())


def _halo_buf(rec):
    return pp._HaloBuf(records=rec.data_ptr(), capacity=rec.shape[0])


def _radii(Rf):
    a = np.ascontiguousarray(Rf, dtype=np.float64)
    return a.ctypes.data_as(ctypes.c_void_p), len(a)


def run(s):
    ctx, c, kind = s["ctx"], s["c"], s["kind"]
    L = ctx.L
    if kind == "noise":
        ctx._check(L.ppb_noise_threefry(ctx.h, _ptr(s["out"]), c["n"], s["seed"]))
        return s["out"]
    if kind == "fields":
        ctx._check(L.ppb_generate_fields(ctx.h, ctypes.byref(s["p"]), _ptr(s["delta"]), _ptr(s["psi"]),
                                         _ptr(s["psi2"]), _ptr(s["lapd"])))
        return {k: s[k] for k in ("delta", "psi", "psi2", "lapd")}
    if kind == "peaks":
        s["mask"].zero_()
        torch.cuda.current_stream().synchronize()   # the library runs on its own stream
        m, rf, fc = ctypes.c_int64(), s["Rf"], s["fc"]
        half = 0.5 * c["cell"] * c["n"]
        ctx._check(L.ppb_peak_find_tile(
            ctx.h, _ptr(s["delta"]), c["n"], rf.ctypes.data_as(ctypes.c_void_p), fc.ctypes.data_as(ctypes.c_void_p),
            len(rf), _ptr(s["mask"]), half, half, half, c["cell"], c["nbuff"], c["ws"], c["shear"], s["cap"],
            *[_ptr(s[k]) for k in ("i", "j", "k", "ipp", "x", "y", "z", "FcRf", "R", "d2Rf", "filter")],
            ctypes.byref(m)))
        out = {k: s[k] for k in ("i", "j", "k", "ipp", "x", "y", "z", "FcRf", "R", "d2Rf", "filter", "mask")}
        out["npeaks"] = m.value
        return out
    if kind == "shells":
        psi, psi2 = s["psi"], s["psi2"]
        ctx._check(L.ppb_analyse_peaks_lim(
            ctx.h, _ptr(s["delta"]), _ptr(psi[0]), _ptr(psi[1]), _ptr(psi[2]), _ptr(psi2[0]), _ptr(psi2[1]),
            _ptr(psi2[2]), _ptr(s["lapd"]), c["n"], c["nhunt"], c["npk"], _ptr(s["ipp"]), _ptr(s["Rf"]),
            _ptr(s["ir2"]), _ptr(s["Z"]), _ptr(s["fc"]), _ptr(s["lim"]), 2.0, c["plain"], _ptr(s["out"])))
        return s["out"]
    if kind == "tile":
        rec = s["rec"]
        count, rmax, npk, _ = ctx.run_tile_into(s["cfg"], s["seed"], s["Rf"], rec.data_ptr(), rec.shape[0])
        return {"records": rec, "count": count, "RTHLmax": rmax, "npeaks": npk}
    if kind == "split":
        hb = _halo_buf(s["rec"])
        ctx._check(L.ppb_run_multitile_split(ctx.h, ctypes.byref(s["p"]), *_radii(s["Rf"]), c["ntile"], 0, 0, None, 0,
                                             ctypes.byref(hb)))
        return {"records": s["rec"], "count": hb.count, "RTHLmax": hb.RTHLmax, "npeaks": hb.npeaks}
    if kind == "chain":
        hb, m, tiles = _halo_buf(s["rec"]), ctypes.c_int64(), s["tiles"]
        ctx._check(L.ppb_run_multitile(ctx.h, ctypes.byref(s["p"]), *_radii(s["Rf"]), c["ntile"],
                                       tiles.ctypes.data_as(ctypes.c_void_p), len(tiles), ctypes.byref(hb)))
        ctx._check(L.ppb_merge_catalog(ctx.h, _ptr(s["rec"]), hb.count, hb.nfields, _ptr(s["merged"]),
                                       ctypes.byref(m)))
        return {"records": s["rec"], "count": hb.count, "merged": s["merged"], "kept": m.value, "npeaks": hb.npeaks}
    if kind == "table":
        return ctx.make_table(s["Om"], 0.0493, 1.0 - s["Om"], 0.6735, s["tp"])
    tickets = [ctx.submit(cfg, seed, s["Rf"], pk_scale=a) for cfg, seed, a in s["req"]]
    counts = []
    for t, rec in zip(tickets, s["rec"]):
        hb = _halo_buf(rec)
        ctx._check(L.ppb_wait(ctx.h, t, -1, ctypes.byref(hb)))
        counts.append(hb.count)
    return {"records": s["rec"], "counts": counts}


# --------------------------------------------------------------------------
# what a pass cannot do without
# --------------------------------------------------------------------------
def _fft_flops(n):
    return 2.5 * n ** 3 * math.log2(n ** 3)   # one real transform


def _tile_work(n, nfilt, shear, ilpt, peaks=True, shells=True):
    N = n ** 3
    bytes_, tr = 4.0 * N * (4 + (3 if ilpt == 2 else 0) + shear), 6 + (10 if ilpt == 2 else 0) + shear
    flops = 150.0 * N
    if peaks:
        tr += nfilt * (1 + shear)
    if shells:   # about a peak per 65 cells, 950 cells visited each, 22 sums per visit; 0.63 of them halos
        flops += N / 65 * 950 * 22 * 2
        bytes_ += N / 65 * 0.63 * 4 * (33 if shear else 11)
    return bytes_, flops + tr * _fft_flops(n)


def work(case):
    c, kind = case, case["kind"]
    n = c.get("n", 0)
    N = float(n) ** 3
    if kind == "noise":
        return {"bytes": 4 * N, "flops": 100 * N}
    if kind == "fields":
        b, f = _tile_work(n, 0, c["shear"], c["ilpt"], peaks=False, shells=False)
        return {"bytes": b, "flops": f}
    if kind == "peaks":
        return {"bytes": 4 * N + 2 * N + N / 65 * 60, "flops": _fft_flops(n) * (1 + c["nfilt"] * (1 + c["shear"]))}
    if kind == "shells":
        return {"bytes": 4 * N * (7 + c["shear"]) + c["npk"] * (44.0 + 31 * 8),
                "flops": c["npk"] * 4.19 * c["rmed"] ** 3 * math.exp(1.1) * 44}
    if kind == "tile":
        b, f = _tile_work(n, c["nfilt"], c["shear"], c["ilpt"])
        return {"bytes": b, "flops": f}
    if kind == "split":
        t = c["ntile"] ** 3
        b, f = _tile_work(n, 3, c["shear"], c["ilpt"])
        return {"bytes": t * b, "flops": t * (f + 5 * _fft_flops(2 * n) / 2)}
    if kind == "chain":
        b, f = _tile_work(c["ntile"] * (n - 2 * c["nbuff"]) + 2 * c["nbuff"], 20, c["shear"], 2, shells=False)
        tb, tf = _tile_work(n, 0, c["shear"], 2, peaks=False)
        return {"bytes": b + c["tiles"] * tb, "flops": f + c["tiles"] * tf}
    if kind == "table":
        nodes = c["nx"] * c["ny"] * c["nz"]
        return {"bytes": 8.0 * nodes, "flops": nodes * 700 * 4 * 600.0}   # about 700 RK4 steps, two Carlson RD each
    b = f = 0.0
    sizes = [m for m in (128, 192, 256) if m <= c["nmax"]]
    for q in range(c["requests"]):
        tb, tf = _tile_work(sizes[q % len(sizes)], 20, 1, 2)
        b, f = b + tb, f + tf
    return {"bytes": b, "flops": f}


# --------------------------------------------------------------------------
# the same in 64 bits
# --------------------------------------------------------------------------
def _threefry(seed, count):
    """Threefry-2x64-20 of counters (0 .. count - 1, 0) under the key (seed, 0), as int64 bit patterns."""
    def i64(v):
        v &= 2 ** 64 - 1
        return v - 2 ** 64 if v >= 2 ** 63 else v
    ks = [i64(seed), 0, i64(0x1BD11BDAA9FC1A22 ^ seed)]
    a = torch.arange(count, device="cuda", dtype=torch.int64) + ks[0]
    b = torch.full((count,), ks[1], device="cuda", dtype=torch.int64)
    rot = (16, 42, 12, 31, 16, 32, 24, 21)
    for r in range(20):
        a = a + b
        q = rot[r % 8]
        b = ((b << q) | ((b >> (64 - q)) & ((1 << q) - 1))) ^ a
        if r % 4 == 3:
            t = r // 4 + 1
            a = a + ks[t % 3]
            b = b + i64(ks[(t + 1) % 3] + t)
    return a, b


def _noise64(n, seed):
    """fill_noise_threefry: Box-Muller pairs in cell order, rounded to single as the grid stores them."""
    N = n ** 3
    a, b = _threefry(seed, (N + 1) // 2)
    u = (((a >> 11) & (2 ** 53 - 1)).double() + 1) * 2.0 ** -53
    v = (((b >> 11) & (2 ** 53 - 1)).double() + 1) * 2.0 ** -53
    r = torch.sqrt(-2 * torch.log(u))
    g = torch.stack([r * torch.cos(2 * math.pi * v), r * torch.sin(2 * math.pi * v)], dim=1)
    return g.reshape(-1)[:N].reshape(n, n, n)


def _fields64(case, seed):
    n, box = case["n"], case["cell"] * case["n"]
    kx, ky, kz = _kgrid(n, box)
    k2 = kx * kx + ky * ky + kz * kz
    k = torch.sqrt(k2)
    k[0, 0, 0] = 1.0
    lk, lp = (torch.from_numpy(np.log(_ready[q])).cuda() for q in ("k", "pk"))
    x = torch.log(k).reshape(-1)
    i = (torch.searchsorted(lk, x, right=True) - 1).clamp(0, len(lk) - 2)
    P = torch.exp(torch.lerp(lp[i], lp[i + 1], (x - lk[i]) / (lk[i + 1] - lk[i]))).reshape(k.shape)
    amp = torch.sqrt(P * (2 * math.pi / box) ** 3 * float(n) ** 3)
    amp[0, 0, 0] = 0.0
    del x, i, P, k

    def back(f):   # the real transform keeps the Hermitian part of the kx = 0 and Nyquist planes
        for q in ([0, n // 2] if n % 2 == 0 else [0]):
            f[:, :, q] = 0.5 * (f[:, :, q] + f[:, :, q].flip(0, 1).roll((1, 1), (0, 1)).conj())
        return torch.fft.irfftn(f, s=(n, n, n))

    delta = back(torch.fft.rfftn(_noise64(n, seed).float().double()) * amp)
    dk = torch.fft.rfftn(delta)
    k2[0, 0, 0] = 1.0
    odd_ok = torch.ones(n, n, n // 2 + 1, device="cuda", dtype=torch.bool)   # odd kernels: index n // 2 zeroed
    odd_ok[:, :, n // 2] = False
    odd_ok[:, n // 2, :] = False
    odd_ok[n // 2, :, :] = False
    out = {"delta": delta, "psi": torch.stack([back(1j * q / k2 * dk * odd_ok) for q in (kx, ky, kz)])}
    if case["ilpt"] == 2:
        ax = (kx, ky, kz)
        phi = {(a, b): back(-ax[a] * ax[b] / k2 * dk) for a, b in ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))}
        src = (phi[0, 0] * phi[1, 1] - phi[0, 1] ** 2 + phi[0, 0] * phi[2, 2] - phi[0, 2] ** 2 +
               phi[1, 1] * phi[2, 2] - phi[1, 2] ** 2)
        sk = torch.fft.rfftn(src)
        out["psi2"] = torch.stack([back(-1j * q / k2 * sk * odd_ok) for q in ax])
    if case["shear"]:
        k2[0, 0, 0] = 0.0
        out["lapd"] = back(k2 * dk) / float(n) ** 3
    return out


def _peaks64(case, seed):
    """The filter loop in 64 bits: window, inverse transform, 3^3 maxima above fcrit, mask carried."""
    n, nb, cell = case["n"], case["nbuff"], case["cell"]
    delta = _gaussian_field(n, cell, seed)[0].double()
    dk = torch.fft.rfftn(delta)
    kx, ky, kz = _kgrid(n, n * cell)
    k = torch.sqrt(kx * kx + ky * ky + kz * kz)
    k[0, 0, 0] = 1.0

    def window(R, ws):
        x = k * R
        if ws == 1:
            w = 3 * (torch.sin(x) - x * torch.cos(x)) / x ** 3
        else:
            w = torch.exp(-x * x / 8) * (k * k if ws == 3 else 1.0)
        w[0, 0, 0] = 1.0
        return w

    mask = torch.zeros(n, n, n, dtype=torch.bool, device="cuda")
    inner = torch.zeros_like(mask)
    inner[nb:n - nb, nb:n - nb, nb:n - nb] = True
    cols = {q: [] for q in ("x", "y", "z", "FcRf", "R", "d2Rf")}
    for R in _bank(case["nfilt"])[::-1]:
        d = torch.fft.irfftn(dk * window(R, case["ws"]), s=(n, n, n))
        m = torch.nn.functional.max_pool3d(d[None, None], 3, 1, 1)[0, 0]
        pk = inner & ~mask & (d >= m) & (d >= 1.686)
        mask |= pk
        at = pk.nonzero()   # (k, j, i) in scan order
        for q, col in (("x", 2), ("y", 1), ("z", 0)):
            cols[q].append(0.5 * cell * n + cell * (at[:, col].double() + 1 - 0.5 * (n + 1)))
        cols["FcRf"].append(d[pk])
        cols["R"].append(torch.full_like(d[pk], R))
        lap = torch.fft.irfftn(dk * window(R, 3), s=(n, n, n))[pk] if case["shear"] else torch.zeros_like(d[pk])
        cols["d2Rf"].append(lap)
    cap, found = max(1, n ** 3 // 30), sum(len(v) for v in cols["x"])
    out = {q: torch.cat(v + [torch.zeros(cap - found, dtype=torch.float64, device="cuda")]) for q, v in cols.items()}
    return out


def exact(case, seed):
    """64-bit values where a pass computes fields or samples of fields; the
    collapse analysis, catalogues and tables are decisions and long
    integrations with no short 64-bit form."""
    if case["kind"] not in ("noise", "fields", "peaks"):
        return None
    _context()
    if case["kind"] == "noise":
        return _noise64(case["n"], seed)
    if case["kind"] == "fields":
        return _fields64(case, seed)
    return _peaks64(case, seed)
