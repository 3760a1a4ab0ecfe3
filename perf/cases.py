"""What the performance of this library is measured on: calls that its users make.

A case is one kind of call through the Python binding of the C ABI (``bsar``):

  image      pulses -> image.  ``data`` says where the pulses are before the call:
             "host_raw" / "host_compressed": host arrays; the call uploads the scene, images
             and releases it (a program that images each acquisition once); "resident": a
             scene on the device that is pulse-compressed again and imaged into device memory
             (a program that keeps acquisitions on the GPU)
  serve      a burst of image requests through the continuous-batching server
  slant      the path solver for one voxel over all pulses (the per-voxel function of the
             reference's imager, called through the C++ shims)
  crossings  a batch of refraction points
  correlate  the batched matched filter on host arrays

``exact`` recomputes each of them in 64 bits with plain torch operations.
"""
import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "c-_bistatic_sar_b200"))

import bsar  # noqa: E402

C_LIGHT = 3e8
DEV = "cuda"
F64 = torch.float64


# ---------------------------------------------------------------------------- the cases
def _scene(name, n, dz, nodes, pulses, samples, **kw):
    """An image case on the small scene's signal (kw: the fields that differ)."""
    c = {"name": name, "kind": "image", "nx": n[0], "ny": n[1], "nz": n[2], "dxy": 0.04, "dz": dz,
         "dem_n": nodes[0], "dem_d": nodes[1], "dem": "fbm", "sigma": 0.3, "beta": 2.0, "eps_r": 6.0, "pulses": pulses,
         "samples": samples, "bandwidth": 800e6, "fs": 1.92e9, "scatterers": 20, "snr_db": 15.0, "data": "resident",
         "solver": "newton", "legs": "per_pulse", "precision": "mixed"}
    c.update(kw)
    return c


_SMALL = dict(dem="plane", sigma=0.03, eps_r=4.0, bandwidth=500e6, fs=1.2e9, scatterers=3, snr_db=20.0)


def listed():
    return [
        # the reference's own call, once per voxel: both crossings of 256 pulses, grid search
        {"name": "slant-voxel", "kind": "slant", "dem_n": 64, "dem_d": 0.5, "dem": "plane", "sigma": 0.03, "beta": 2.0,
         "eps_r": 4.0, "pulses": 256, "solver": "grid"},
        # refraction points of many (antenna, voxel) pairs: accuracy studies, ray displays
        {"name": "crossings", "kind": "crossings", "dem_n": 256, "dem_d": 0.25, "dem": "fbm", "sigma": 0.3, "beta": 2.0,
         "eps_r": 6.0, "points": 65536, "solver": "newton", "precision": "fp64"},
        # the simulator's matched filter over an acquisition, host arrays in and out
        {"name": "correlate", "kind": "correlate", "batch": 256, "samples": 4096, "reference": 1201},
        # the reference's program as it stands: compressed pulses from the host, upsampling,
        # grid search and mean legs in FP64 (the defaults of backproject)
        _scene("image-reference", (41, 41, 21), 0.08, (64, 0.5), 256, 4096, data="host_compressed", solver="grid",
               legs="mean", precision="fp64", **_SMALL),
        # the small scene through the fast form, host to host: a latency-sensitive user
        _scene("image-small", (41, 41, 21), 0.08, (64, 0.5), 256, 4096, data="host_raw", **_SMALL),
        # one depth slice of an acquisition with FP16 samples: a quick look
        _scene("slice-fp16", (161, 161, 1), 0.02, (256, 0.25), 1024, 8192, dxy=0.02, scatterers=50,
               precision="mixed_fp16"),
        # odd sizes and a DEM spacing between the usual ones (17 x 17 node scans)
        _scene("image-odd", (97, 83, 11), 0.03, (201, 0.2), 701, 2048, dxy=0.03),
        # the FP64 form on the rough DEM: the image the fast forms are checked against
        _scene("image-fp64", (81, 77, 13), 0.02, (256, 0.25), 512, 8192, dxy=0.02, precision="fp64"),
        # the medium scene (161 x 161 x 81 voxels, 1024 pulses of 8192 samples)
        _scene("image-medium", (161, 161, 81), 0.02, (256, 0.25), 1024, 8192, dxy=0.02, scatterers=50),
        # a slab of the large scene: 0.125 m DEM (25 x 25 node scans), 2048 pulses of 16384
        _scene("image-large", (256, 256, 8), 0.02, (1024, 0.125), 2048, 16384, dxy=0.02, sigma=0.5, beta=2.2, eps_r=5.0,
               bandwidth=1e9, fs=2.4e9, scatterers=200, snr_db=10.0),
        # a burst of uneven requests: grids of 21 to 81 voxels a side, 128 to 1024 pulses,
        # four DEMs, echoes synthesised at admission
        {"name": "serve-burst", "kind": "serve", "requests": 16, "mix": 4, "side_max": 81, "pulses_max": 1024,
         "log2_min": 11, "log2_max": 13},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed ranges.  Image cases stay below the medium scene."""
    kind = rng.choice(["slant", "crossings", "correlate", "image", "image", "image", "image", "serve"])
    rough = {"dem": "fbm", "sigma": round(rng.uniform(0.1, 0.5), 3), "beta": round(rng.uniform(1.9, 2.3), 2),
             "eps_r": round(rng.uniform(3.0, 9.0), 2)}
    smooth = {"dem": "plane", "sigma": round(rng.uniform(0.01, 0.05), 3), "beta": 2.0,
              "eps_r": round(rng.uniform(3.0, 9.0), 2)}
    if kind == "slant":
        return {"kind": kind, "dem_n": rng.randint(40, 128), "dem_d": round(rng.uniform(0.25, 0.6), 3), **smooth,
                "pulses": _log(rng, 64, 2048), "solver": rng.choice(["grid", "newton"])}
    if kind == "crossings":
        solver = rng.choice(["grid", "newton", "newton"])
        return {"kind": kind, "dem_n": rng.randint(150, 400), "dem_d": round(rng.uniform(0.125, 0.5), 3), **rough,
                "points": _log(rng, 500, 100000), "solver": solver,
                "precision": "fp64" if solver == "grid" else rng.choice(["fp64", "mixed"])}
    if kind == "correlate":
        s = _log(rng, 700, 8000)
        return {"kind": kind, "batch": _log(rng, 1, 400), "samples": s, "reference": rng.randint(200, s)}
    if kind == "serve":
        return {"kind": kind, "requests": rng.randint(4, 16), "mix": rng.randint(10, 10 ** 6),
                "side_max": rng.randint(40, 81), "pulses_max": rng.randint(300, 1024), "log2_min": 11, "log2_max": 13}
    form = rng.choice(["mixed", "mixed", "mixed", "mixed_fp16", "fp64", "reference"])
    # voxel-pulses by form, so that a pass stays well below a second
    budget = {"mixed": 6e7, "mixed_fp16": 6e7, "fp64": 3e7, "reference": 6e6}[form]
    work = math.exp(rng.uniform(math.log(budget / 60), math.log(budget)))
    pulses = _log(rng, 100, 1400)
    voxels = work / pulses
    flat = rng.uniform(0.05, 1.0)                       # nz / nx
    side = max(3.0, (voxels / flat) ** (1 / 3))
    nz = max(1, round(flat * side))
    nx = max(3, round(side * rng.uniform(0.8, 1.25)))
    ny = max(3, round(voxels / (nx * nz)))
    if rng.random() < 0.3:
        dem, d = smooth, round(rng.uniform(0.3, 0.6), 3)
    else:
        dem, d = rough, rng.choice([0.25, 0.25, round(rng.uniform(0.12, 0.5), 3)])
    log2 = rng.randint(11, 13)
    return _scene("", (nx, ny, nz), round(rng.uniform(0.01, 0.08), 3), (max(64, int(50 / d)), d), pulses, 1 << log2,
                  dxy=round(rng.uniform(0.01, 0.06), 3), scatterers=rng.randint(3, 40),
                  data=rng.choice(["resident", "host_raw", "host_compressed"]),
                  solver="grid" if form == "reference" else "newton",
                  legs=rng.choice(["mean", "per_pulse"]) if form == "reference" else "per_pulse",
                  precision="fp64" if form == "reference" else form, **dem)


# ------------------------------------------------------------------ inputs, from the seed
def _dem(case, rng):
    """Axes centred 20 m downrange and heights: independent roughness, or an fBm surface."""
    n, d = case["dem_n"], case["dem_d"]
    k = (np.arange(n) - (n - 1) / 2.0) * d
    if case["dem"] == "plane":
        return 20.0 + k, k.copy(), rng.normal(0.0, case["sigma"], (n, n))
    f = np.fft.fftfreq(n)
    r = np.hypot(f[None, :], f[:, None])
    r[0, 0] = 1.0
    amp = r ** (-case["beta"] / 2.0)
    amp[0, 0] = 0.0
    z = np.real(np.fft.ifft2(amp * rng.normal(size=(n, n)) * np.exp(2j * np.pi * rng.uniform(size=(n, n)))))
    z -= z.mean()
    return 20.0 + k, k.copy(), np.ascontiguousarray(z * (case["sigma"] / z.std()))


def _tracks(n, rng):
    """Archimedean spirals at 30 m (three turns, 15 m to 0), receiver 5 m beside."""
    s = np.arange(n) / max(n - 1, 1)
    th = 2.0 * np.pi * (3.0 * s + rng.uniform())
    tx = np.stack([15.0 * (1 - s) * np.cos(th), 15.0 * (1 - s) * np.sin(th), np.full(n, 30.0)], axis=1)
    return np.ascontiguousarray(tx), tx + np.array([5.0, 0.0, 0.0])


def _axes(case):
    def line(c, n, d):
        return c + (np.arange(n) - (n - 1) / 2.0) * d
    return line(20.0, case["nx"], case["dxy"]), line(0.0, case["ny"], case["dxy"]), line(-5.0, case["nz"], case["dz"])


def _targets(case, axes, rng):
    ix = [rng.integers(0, len(a), case["scatterers"]) for a in axes]
    amp = np.exp(rng.uniform(math.log(0.1), 0.0, case["scatterers"]))
    return np.stack([a[i] for a, i in zip(axes, ix)], axis=1), amp


def _signal(case):
    f0, f1 = -case["bandwidth"] / 2, case["bandwidth"] / 2
    return dict(upsample=4, n1=1.0, n2=math.sqrt(case["eps_r"]), c=C_LIGHT, fc=1e9, fs=case["fs"], chirp_f0=f0,
                chirp_f1=f1, chirp_T=1e-6)


def _inputs(case, seed):
    rng = np.random.default_rng([seed, 1])
    dem = _dem(case, rng)
    tx, rx = _tracks(case["pulses"], rng)
    axes = _axes(case)
    pos, amp = _targets(case, axes, rng)
    return dem, tx, rx, axes, pos, amp


def _t(a):
    return torch.as_tensor(np.ascontiguousarray(a), device=DEV)


def _echoes(case, dem, tx, rx, pos, amp, seed, snr_db):
    """Raw echoes (pulses, samples): a delayed chirp per scatterer, and noise."""
    sig = _signal(case)
    fs, f0, k = sig["fs"], sig["chirp_f0"], (sig["chirp_f1"] - sig["chirp_f0"]) / sig["chirp_T"]
    nc = int(sig["chirp_T"] * fs) + 1
    half, ns, n_p = nc // 2, case["samples"], len(tx)
    tau = _two_way(dem, _t(tx), _t(rx), _t(pos), sig["n2"]) / C_LIGHT           # (pulses, scatterers)
    raw = torch.zeros((n_p, ns, 2), dtype=F64, device=DEV)
    off = torch.arange(nc + 2, device=DEV)
    for s in range(len(amp)):
        t0 = tau[:, s:s + 1]
        n = torch.floor(t0 * fs).long() - half + off
        t = n / fs - t0 + half / fs
        ok = (t >= 0) & (t <= (nc - 1) / fs) & (n >= 0) & (n < ns)
        cyc = f0 * t + 0.5 * k * t * t - 1e9 * t0
        e = torch.polar(amp[s] * ok.to(F64), 2 * math.pi * (cyc - torch.round(cyc)))
        raw.scatter_add_(1, n.clamp(0, ns - 1)[:, :, None].expand(-1, -1, 2), torch.view_as_real(e))
    if math.isfinite(snr_db):
        g = torch.Generator(device=DEV).manual_seed(seed + 77)
        raw += torch.randn(raw.shape, dtype=F64, device=DEV, generator=g) * math.sqrt(nc / 10 ** (snr_db / 10) / 2)
    return torch.view_as_complex(raw)


def _pulses(case, dem, tx, rx, pos, amp, seed):
    raw = _echoes(case, dem, tx, rx, pos, amp, seed, case["snr_db"])
    return _compress(raw, _signal(case)) if case["data"] == "host_compressed" else raw


def _requests(case, seed):
    """The burst's requests: sizes from the case, contents from the seed."""
    sizes = np.random.default_rng(case["mix"])
    dems = []
    for k in range(4):
        spec = {"dem_n": 256, "dem_d": 0.25, "dem": "fbm", "sigma": float(sizes.uniform(0.1, 0.5)), "beta": 2.0,
                "eps_r": float(sizes.uniform(3.0, 9.0))}
        dems.append((spec, _dem(spec, np.random.default_rng([seed, 2, k]))))
    reqs = []
    for i in range(case["requests"]):
        side = int(round(math.exp(sizes.uniform(math.log(21), math.log(case["side_max"])))))
        c = {"nx": side, "ny": side, "nz": (side + 1) // 2, "dxy": 0.02, "dz": 0.02, "bandwidth": 800e6, "fs": 1.92e9,
             "pulses": int(round(math.exp(sizes.uniform(math.log(128), math.log(case["pulses_max"]))))),
             "samples": 1 << int(sizes.integers(case["log2_min"], case["log2_max"] + 1)),
             "scatterers": int(sizes.integers(5, 51)), "precision": "mixed", "solver": "newton", "legs": "per_pulse"}
        spec, dem = dems[int(sizes.integers(0, 4))]
        c.update(spec)
        rng = np.random.default_rng([seed, 3, i])
        tx, rx = _tracks(c["pulses"], rng)
        axes = _axes(c)
        reqs.append((c, dem, tx, rx, axes, *_targets(c, axes, rng)))
    return reqs


# ----------------------------------------------------------------------------- the calls
_ctx = None
_server = None


def _context():
    global _ctx
    if _ctx is None:
        _ctx = bsar.Context(0)
    return _ctx


def _serving():
    global _server
    if _server is None:
        _server = bsar.Server(_context(), max_inflight=64)
    return _server


class _Resident:
    """A scene on the device, released with the object."""

    def __init__(self, ctx, sid):
        self.ctx, self.sid = ctx, sid

    def __del__(self):
        try:
            self.ctx.scene_release(self.sid)
        except Exception:
            pass


def prepare(case, seed):
    ctx = _context()
    kind = case["kind"]
    if kind == "serve":
        return {"case": case, "server": _serving(),
                "requests": [(bsar.DemArrays(*r[1]), r) for r in _requests(case, seed)]}
    rng = np.random.default_rng([seed, 1])
    if kind == "correlate":
        g = torch.Generator(device=DEV).manual_seed(seed)
        s = torch.randn((case["batch"], case["samples"], 2), dtype=F64, device=DEV, generator=g)
        return {"case": case, "ctx": ctx, "signal": torch.view_as_complex(s).cpu().numpy(),
                "reference": _chirp(case["reference"])}
    if kind == "slant":
        dem = _dem(case, rng)
        tx, rx = _tracks(case["pulses"], rng)
        return {"case": case, "ctx": ctx, "dem": bsar.DemArrays(*dem), "tx": tx, "rx": rx, "P": _voxel(rng),
                "raw": (dem, tx, rx)}
    if kind == "crossings":
        dem = _dem(case, rng)
        a, b = _pairs(case, rng)
        return {"case": case, "ctx": ctx, "dem": bsar.DemArrays(*dem), "a": a, "b": b}
    dem, tx, rx, axes, pos, amp = _inputs(case, seed)
    data = _pulses(case, dem, tx, rx, pos, amp, seed).cpu().numpy()
    st = {"case": case, "ctx": ctx, "dem": bsar.DemArrays(*dem), "tx": tx, "rx": rx, "axes": axes}
    if case["data"] == "resident":
        st["scene"] = _Resident(ctx, ctx.scene_upload(st["dem"], tx, rx, data, **_signal(case)))
        st["image"] = torch.empty((case["nx"], case["ny"], case["nz"]), dtype=torch.complex128, device=DEV)
    else:
        st["data"] = data
    return st


def _chirp(n):
    t = np.arange(n) / n
    return np.exp(1j * np.pi * 0.4 * n * (t - 0.5) ** 2)


def _voxel(rng):
    return np.array([20.0 + rng.uniform(-1, 1), rng.uniform(-1, 1), -5.0 + rng.uniform(-1, 1)])


def _pairs(case, rng):
    n = case["points"]
    tx, _ = _tracks(1024, rng)
    return tx[rng.integers(0, len(tx), n)], np.stack([_voxel(rng) for _ in range(min(n, 512))])[rng.integers(0, min(n, 512), n)]


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "serve":
        srv = st["server"]
        ids = [srv.submit(dem, tx, rx, *axes, n_samples=c["samples"], scat_pos=pos, scat_amp=amp, precision="mixed",
                          **_signal(c)) for dem, (c, _, tx, rx, axes, pos, amp) in st["requests"]]
        return [srv.wait(i)[0] for i in ids]
    ctx = st["ctx"]
    if kind == "correlate":
        return ctx.fft_correlate(st["signal"], st["reference"])
    n2 = math.sqrt(case["eps_r"])
    if kind == "slant":
        ranges, ida, volta, _ = ctx.slant_range_fermat(st["dem"], st["tx"], st["rx"], st["P"], 1.0, n2,
                                                       solver=case["solver"])
        return ranges, ida, volta
    if kind == "crossings":
        return ctx.refraction_points(st["dem"], st["a"], st["b"], 1.0, n2, solver=case["solver"],
                                     precision=case["precision"])
    how = dict(solver=case["solver"], legs=case["legs"], precision=case["precision"])
    if case["data"] == "resident":
        sid = st["scene"].sid
        ctx.scene_compress(sid, case["precision"])
        ctx.backproject_device(sid, *st["axes"], st["image"].data_ptr(), **how)
        return st["image"]
    sid = ctx.scene_upload(st["dem"], st["tx"], st["rx"], st["data"],
                           kind="compressed" if case["data"] == "host_compressed" else "raw", **_signal(case))
    try:
        return ctx.backproject(sid, *st["axes"], **how)
    finally:
        ctx.scene_release(sid)


# ------------------------------------------------------------------- work and tolerances
# Operations one solve cannot do without, by solver: the flat-interface start (4 steps of
# 25), the nine nodes around the crossing ranked (17 each), three Newton steps on one facet
# (80) and the final one (80); the grid search's points are its result's definition: 709
# heights and two-leg paths of 40.
_SOLVE = {"newton": 100 + 9 * 17 + 3 * 80 + 80, "grid": 709 * 40}


def _image_work(c, host):
    vp = c["nx"] * c["ny"] * c["nz"] * c["pulses"]
    s = c["samples"] * c["pulses"]
    flops = vp * (2 * _SOLVE[c["solver"]] + 40)
    if c.get("data") != "host_compressed":
        flops += s * (10 * math.log2(c["samples"]) + 6)
    if c["legs"] == "mean":
        flops += vp * c["pulses"] * 2 * 9
    return {"bytes": (16 * s if host else 0) + 16 * vp // c["pulses"] + 8 * c["dem_n"] ** 2 + 48 * c["pulses"],
            "flops": flops}


def work(case):
    kind = case["kind"]
    if kind == "image":
        return _image_work(case, True)
    if kind == "serve":
        w = [_image_work(r[0], False) for r in _requests(case, 0)]
        return {k: sum(x[k] for x in w) for k in ("bytes", "flops")}
    if kind == "correlate":
        n = 1 << (max(case["samples"], case["reference"]) - 1).bit_length()
        return {"bytes": 16 * (case["batch"] * (case["samples"] + max(case["samples"], case["reference"])) +
                               case["reference"]),
                "flops": case["batch"] * n * (10 * math.log2(n) + 6)}
    solves = 2 * case["pulses"] if kind == "slant" else case["points"]
    return {"bytes": 8 * case["dem_n"] ** 2 + (128 if kind == "slant" else 72) * solves,
            "flops": solves * _SOLVE[case["solver"]]}


def tolerance(case):
    """About four times what was measured against ``exact``.  FP64: 2.4e-13 (the carrier phase
    turns 300 times, so the last bit of a path is about 1e-13 of a turn), widened for longer
    paths.  Mixed forms: 1e-5 to 4.2e-5 (FP32 delays, samples and sums).  Mixed crossing
    points: 1e-10, but a point moves by millimetres where the path is flat along it."""
    if case["kind"] == "serve" or case.get("precision", "fp64") != "fp64":
        return {"rel": 2e-6 if case["kind"] == "crossings" else 2e-4}
    return {"rel": 1e-11}


# ------------------------------------------------------------- the same in 64 bits, torch
def _elevation(dem, x, y):
    """Bilinear height as the reference looks it up: an axis value that no interval holds
    takes the first node with weight clamp(x - v[0], 0, 1)."""
    def axis(v, q):
        n = len(v)
        i = torch.searchsorted(v[1:].contiguous(), q.contiguous(), right=False)
        ok = i < n - 1
        i = i.clamp(max=n - 2)
        ok &= (q >= v[i]) & (q <= v[i + 1])
        i0 = torch.where(ok, i, 0)
        i1 = torch.where(ok, i + 1, 0)
        d = v[i1] - v[i0]
        d = torch.where(d == 0, torch.ones_like(d), d)
        return i0, i1, ((q - v[i0]) / d).clamp(0.0, 1.0)
    xv, yv, z = dem
    i0, i1, u = axis(xv, x)
    j0, j1, v = axis(yv, y)
    w = z[j0, i0] * (1 - u) * (1 - v) + z[j0, i1] * u * (1 - v) + z[j1, i0] * (1 - u) * v + z[j1, i1] * u * v
    return torch.where((i0 == i1) & (j0 == j1), z[j0, i0], w)


def _facet(dem, i, j, A, B, na, nb, u, v):
    """Position, path and one projected Newton step on facet (i, j) at (u, v)."""
    xv, yv, z = dem
    dx, dy = xv[i + 1] - xv[i], yv[j + 1] - yv[j]
    b, c = z[j, i + 1] - z[j, i], z[j + 1, i] - z[j, i]
    e = z[j + 1, i + 1] - z[j, i + 1] - z[j + 1, i] + z[j, i]
    X = torch.stack([xv[i] + u * dx, yv[j] + v * dy, z[j, i] + b * u + c * v + e * u * v], 1)
    r1, r2 = X - A, X - B
    q1, q2 = (r1 * r1).sum(1), (r2 * r2).sum(1)
    path = na * q1.sqrt() + nb * q2.sqrt()
    zx, zy, zxy = (b + e * v) / dx, (c + e * u) / dy, e / (dx * dy)
    g1, g2 = na / q1.sqrt(), nb / q2.sqrt()
    p1, p2 = r1[:, 0] + r1[:, 2] * zx, r2[:, 0] + r2[:, 2] * zx
    s1, s2 = r1[:, 1] + r1[:, 2] * zy, r2[:, 1] + r2[:, 2] * zy
    gx, gy = g1 * p1 + g2 * p2, g1 * s1 + g2 * s2
    hxx = g1 * (1 + zx * zx - p1 * p1 / q1) + g2 * (1 + zx * zx - p2 * p2 / q2)
    hyy = g1 * (1 + zy * zy - s1 * s1 / q1) + g2 * (1 + zy * zy - s2 * s2 / q2)
    hxy = g1 * (zx * zy - p1 * s1 / q1) + g2 * (zx * zy - p2 * s2 / q2) + (g1 * r1[:, 2] + g2 * r2[:, 2]) * zxy
    au = ((u <= 0) & (gx > 0)) | ((u >= 1) & (gx < 0))
    av = ((v <= 0) & (gy > 0)) | ((v >= 1) & (gy < 0))
    det, gs = hxx * hyy - hxy * hxy, g1 + g2
    ok = (det > 0) & (hxx > 0)
    det = torch.where(ok, det, torch.ones_like(det))
    su = torch.where(ok, -(hyy * gx - hxy * gy) / det, -gx / gs)
    sv = torch.where(ok, -(hxx * gy - hxy * gx) / det, -gy / gs)
    su = torch.where(av, -gx / torch.where(hxx > 0, hxx, gs), su)
    sv = torch.where(au, -gy / torch.where(hyy > 0, hyy, gs), sv)
    zero = torch.zeros_like(su)
    su, sv = torch.where(au, zero, su), torch.where(av, zero, sv)
    return X, path, (u + su / dx).clamp(0, 1), (v + sv / dy).clamp(0, 1)


def _newton(dem, A, B, na, nb, radius=1.5):
    """Crossing of the path A (index na) -> B (index nb): flat-interface start, best node
    within `radius`, Newton steps on the facets around it."""
    xv, yv, z = dem
    nx, ny = len(xv), len(yv)
    dx, dy = float(xv[-1] - xv[0]) / (nx - 1), float(yv[-1] - yv[0]) / (ny - 1)
    W = max(1, math.ceil(radius / min(dx, dy) - 1e-9))
    U, L, nu, nl = (A, B, na, nb) if nb >= na else (B, A, nb, na)
    h0 = _elevation(dem, L[:, 0], L[:, 1])
    h = L[:, :2] - U[:, :2]
    D = h.norm(dim=1)
    ha, hb = (U[:, 2] - h0).abs(), (L[:, 2] - h0).abs()
    s = D * ha / (ha + hb + 1e-30)
    for _ in range(4):
        q1, q2 = (s * s + ha * ha).sqrt(), ((D - s) ** 2 + hb * hb).sqrt()
        g = nu * s / q1 - nl * (D - s) / q2
        gp = nu * ha * ha / q1 ** 3 + nl * hb * hb / q2 ** 3
        s = torch.minimum((s - g / gp).clamp(min=0.0), D)
    f = torch.where(D >= 1e-9, s / D, torch.ones_like(D))[:, None]
    start = U[:, :2] + h * f
    i_s = torch.floor((start[:, 0] - xv[0]) / dx + 0.5).clamp(0, nx - 1).long()
    j_s = torch.floor((start[:, 1] - yv[0]) / dy + 0.5).clamp(0, ny - 1).long()
    best = torch.full_like(D, math.inf)
    bi, bj = i_s.clone(), j_s.clone()
    for di in range(-W, W + 1):
        i = i_s + di
        ic = i.clamp(0, nx - 1)
        x = xv[ic]
        xa, xb = (x - A[:, 0]) ** 2, (x - B[:, 0]) ** 2
        for dj in range(-W, W + 1):
            j = j_s + dj
            jc = j.clamp(0, ny - 1)
            y, zz = yv[jc], z[jc, ic]
            p = na * (xa + (y - A[:, 1]) ** 2 + (zz - A[:, 2]) ** 2).sqrt()
            p += nb * (xb + (y - B[:, 1]) ** 2 + (zz - B[:, 2]) ** 2).sqrt()
            m = (p < best) & (i == ic) & (j == jc)
            best = torch.where(m, p, best)
            bi, bj = torch.where(m, i, bi), torch.where(m, j, bj)
    bfi, bfj = bi.clamp(max=nx - 2), bj.clamp(max=ny - 2)
    bu, bv = (bi - bfi).to(F64), (bj - bfj).to(F64)
    best = torch.full_like(D, math.inf)
    for k in range(4):
        fi, fj = bi - 1 + (k >> 1), bj - 1 + (k & 1)
        ok = (fi >= 0) & (fj >= 0) & (fi <= nx - 2) & (fj <= ny - 2)
        fi, fj = fi.clamp(0, nx - 2), fj.clamp(0, ny - 2)
        u, v = (bi - fi).to(F64), (bj - fj).to(F64)
        for _ in range(3):
            _, _, u, v = _facet(dem, fi, fj, A, B, na, nb, u, v)
        p = _facet(dem, fi, fj, A, B, na, nb, u, v)[1]
        m = ok & (p < best)
        best = torch.where(m, p, best)
        bu, bv = torch.where(m, u, bu), torch.where(m, v, bv)
        bfi, bfj = torch.where(m, fi, bfi), torch.where(m, fj, bfj)
    _, _, bu, bv = _facet(dem, bfi, bfj, A, B, na, nb, bu, bv)
    return _facet(dem, bfi, bfj, A, B, na, nb, bu, bv)[0]


def _grid_search(dem, A, B, na, nb):
    """The reference's five-level search: 15 x 15, then 11 x 11 points around the best."""
    bx, by = (A[:, 0] + B[:, 0]) / 2, (A[:, 1] + B[:, 1]) / 2
    R = ((B[:, 0] - A[:, 0]) ** 2 + (B[:, 1] - A[:, 1]) ** 2).sqrt().clamp(min=500.0)
    best = torch.full_like(bx, 1e9)
    for level in range(5):
        G = 15 if level == 0 else 11
        x0, x1, y0, y1 = bx - R, bx + R, by - R, by + R
        for i in range(G):
            px = x0 + i * (x1 - x0) / (G - 1)
            for j in range(G):
                py = y0 + j * (y1 - y0) / (G - 1)
                pz = _elevation(dem, px, py)
                d1 = ((px - A[:, 0]) ** 2 + (py - A[:, 1]) ** 2 + (pz - A[:, 2]) ** 2).sqrt()
                d2 = ((B[:, 0] - px) ** 2 + (B[:, 1] - py) ** 2 + (B[:, 2] - pz) ** 2).sqrt()
                p = na * d1 + nb * d2
                m = p < best
                best = torch.where(m, p, best)
                bx, by = torch.where(m, px, bx), torch.where(m, py, by)
        R = R / (5.0 if level == 0 else 3.0)
    return torch.stack([bx, by, _elevation(dem, bx, by)], 1)


def _solve(solver, dem, A, B, na, nb):
    dem = [d if isinstance(d, torch.Tensor) else _t(d) for d in dem]
    step, out = 1 << 21, []
    for k in range(0, len(A), step):
        a, b = A[k:k + step], B[k:k + step]
        out.append(_newton(dem, a, b, na, nb) if solver == "newton" else _grid_search(dem, a, b, na, nb))
    return torch.cat(out)


def _legs(solver, dem, tx, rx, P, n2):
    """Crossings of both legs of every (row of P, pulse): (points * pulses, 3) each."""
    n = len(tx)
    p = P.repeat_interleave(n, 0)
    t, r = tx.repeat(len(P), 1), rx.repeat(len(P), 1)
    return t, r, p, _solve(solver, dem, t, p, 1.0, n2), _solve(solver, dem, p, r, n2, 1.0)


def _two_way(dem, tx, rx, P, n2):
    t, r, p, a, b = _legs("newton", dem, tx, rx, P, n2)
    L = (t - a).norm(dim=1) + n2 * (p - a).norm(dim=1) + n2 * (p - b).norm(dim=1) + (r - b).norm(dim=1)
    return L.reshape(len(P), len(tx)).T


def _compress(raw, sig):
    """Circular correlation with the chirp, its centre at lag 0."""
    n = raw.shape[1]
    nc = int(sig["chirp_T"] * sig["fs"]) + 1
    t = torch.arange(nc, dtype=F64, device=DEV) / sig["fs"]
    k = (sig["chirp_f1"] - sig["chirp_f0"]) / sig["chirp_T"]
    ch = torch.polar(torch.ones_like(t), 2 * math.pi * (sig["chirp_f0"] * t + (k / 2) * t * t))
    ref = torch.zeros(n, dtype=torch.complex128, device=DEV)
    ref[: nc - nc // 2] = ch[nc // 2:]
    ref[n - nc // 2:] = ch[: nc // 2]
    return torch.fft.ifft(torch.fft.fft(raw) * torch.fft.fft(ref).conj())


def _upsample(x, factor):
    """Hermite interpolation with backward and forward differences as the end slopes."""
    n = x.shape[1]
    pos = torch.arange(n * factor, dtype=F64, device=DEV) / factor
    i = pos.long()
    t = torch.where(i >= n - 1, torch.ones_like(pos), pos - i)
    i = i.clamp(max=n - 2)
    p0, p1 = x[:, i], x[:, i + 1]
    a = (p0 - x[:, (i - 1).clamp(min=0)]) * (i > 0)
    b = (x[:, (i + 2).clamp(max=n - 1)] - p1) * (i < n - 2)
    t2, t3 = t * t, t * t * t
    return (2 * t3 - 3 * t2 + 1) * p0 + (3 * t2 - 2 * t3) * p1 + (t3 - 2 * t2 + t) * a + (t3 - t2) * b


def _image(case, dem, tx, rx, axes, pulses):
    sig = _signal(case)
    n2, fs = sig["n2"], sig["fs"] * sig["upsample"]
    up = _upsample(pulses, sig["upsample"])
    nr, n_p = up.shape[1], len(tx)
    dem, tx, rx = [_t(d) for d in dem], _t(tx), _t(rx)
    gx, gy, gz = (_t(a) for a in axes)
    P = torch.stack(torch.meshgrid(gx, gy, gz, indexing="ij"), -1).reshape(-1, 3)
    img = []
    step = max(1, (1 << 21) // n_p)
    row = torch.arange(n_p, device=DEV)[None, :]
    for k in range(0, len(P), step):
        V = P[k:k + step]
        t, r, p, a, b = _legs(case["solver"], dem, tx, rx, V, n2)
        if case["legs"] == "mean":
            ra = sum((a - tx[q]).norm(dim=1) for q in range(n_p)) / n_p
            rb = sum((b - rx[q]).norm(dim=1) for q in range(n_p)) / n_p
        else:
            ra, rb = (t - a).norm(dim=1), (r - b).norm(dim=1)
        L = (ra + n2 * (p - a).norm(dim=1) + n2 * (p - b).norm(dim=1) + rb).reshape(len(V), n_p)
        pos = L / C_LIGHT * fs
        lo = torch.floor(pos)
        q = pos - lo
        ok = (pos >= 0) & (pos <= nr - 1)
        i = lo.long().clamp(0, nr - 1)
        s = (1 - q) * up[row, i] + q * up[row, (i + 1).clamp(max=nr - 1)]
        cyc = L * 1e9 / C_LIGHT
        ph = 2 * math.pi * (cyc - torch.round(cyc))
        img.append((s * torch.polar(ok.to(F64), ph)).sum(1))
    return torch.cat(img).reshape(case["nx"], case["ny"], case["nz"])


def _cost(c):
    """Points ranked by the 64-bit image."""
    W = math.ceil(1.5 / c["dem_d"] - 1e-9)
    return c["nx"] * c["ny"] * c["nz"] * c["pulses"] * (709 if c["solver"] == "grid" else (2 * W + 1) ** 2)


def exact(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng([seed, 1])
    if kind == "serve":
        reqs, out, spent = _requests(case, seed), [], 0.0
        for c, dem, tx, rx, axes, pos, amp in reqs:
            spent += _cost(c)
            if spent > 1.2e10:
                out.append(None)
                continue
            raw = _echoes(c, dem, tx, rx, pos, amp, seed, math.inf)
            out.append(_image(c, dem, tx, rx, axes, _compress(raw, _signal(c))))
        return out
    if kind == "correlate":
        g = torch.Generator(device=DEV).manual_seed(seed)
        s = torch.view_as_complex(torch.randn((case["batch"], case["samples"], 2), dtype=F64, device=DEV, generator=g))
        n = max(case["samples"], case["reference"])
        m = 1 << (n - 1).bit_length()
        return torch.fft.ifft(torch.fft.fft(s, m) * torch.fft.fft(_t(_chirp(case["reference"])), m).conj())[:, :n]
    if kind in ("slant", "crossings"):
        dem = _dem(case, rng)
        n2 = math.sqrt(case["eps_r"])
        if kind == "crossings":
            a, b = _pairs(case, rng)
            return _solve(case["solver"], dem, _t(a), _t(b), 1.0, n2)
        tx, rx = _tracks(case["pulses"], rng)
        t, r, p, a, b = _legs(case["solver"], dem, _t(tx), _t(rx), _t(_voxel(rng))[None], n2)
        return torch.stack([(t - a).norm(dim=1), (p - a).norm(dim=1), (r - b).norm(dim=1), (p - b).norm(dim=1)]), a, b
    if _cost(case) > 2.5e10:
        return None
    dem, tx, rx, axes, pos, amp = _inputs(case, seed)
    data = _pulses(case, dem, tx, rx, pos, amp, seed)
    if case["data"] != "host_compressed":
        data = _compress(data, _signal(case))
    return _image(case, dem, tx, rx, axes, data)
