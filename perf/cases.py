"""The work that a program using this package has it do, as timed cases.

listed() gives the cases, draw() more of the same ranges; prepare() makes what
a program holds before the call (raw spectra on the device, a context with its
geometry, stitch plans, a network), run() is one pass through the public entry
points, work() the bytes and operations a pass cannot do without, exact() the
result in float64 by plain torch and numpy.

Raw spectra are the package's seeded spectrum model (uint16 counts, 2048
samples a line, 25 apodisation lines); the CNN's weights are random.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from oct_recon_af_v1_gb300 import estimation, geometry, learned, reconstruct, spectral, stitching, synthetic
from oct_recon_af_v1_gb300._lib import U16, Context

N, HALF, APOD = 2048, 1024, 25
BETA_PX = 1e-5                       # dispersion of the spectrum model (rad/px^2)
SIGMA = 80.0                         # focus sigma (px)
SINC_TAPS = 10                       # source samples of an output of the sinc5 band


def listed():
    return [
        # one B-scan while the user aims the scanner: latency and launches
        {"name": "preview", "kind": "magnitude", "bscans": 1, "ascans": 500},
        # a whole tile to dB with its range, as a preview or single-tile scan is shown
        {"name": "tile_db", "kind": "db", "bscans": 50, "ascans": 500, "z0": 0, "depth": 1000},
        # the autofocus of a scan stored with A-scan binning: odd line counts,
        # float32 spectra made on the device, x-median depth profiles
        {"name": "focus_binned", "kind": "focus", "bscans": 9, "ascans": 333, "binning": 2},
        # the main use: frames of one y-row of a 2 x 3-depth tiled volume, stitched to dB planes
        {"name": "volume", "kind": "volume", "frames": 54, "ascans": 1000, "tiles_x": 2, "depths": 3},
        # the row interface (batches of one tile at a time) with the optical-path correction
        {"name": "row_opc", "kind": "row", "frames": 7, "ascans": 411, "depths": 2, "batch": 3},
        # many tiles of uneven size in one call
        {"name": "tiles_uneven", "kind": "tiles", "tiles": 12, "bscans": 12, "ascans": 1200, "depth": 1500, "mix": 3},
        # the form that is accurate against float64 at tensor-core speed
        {"name": "precision", "kind": "precision", "bscans": 30, "ascans": 1000},
        # the float64 form, used to check a scan's reconstruction
        {"name": "float64", "kind": "float64", "bscans": 6, "ascans": 500},
        # the coarse grid of the dispersion search
        {"name": "search", "kind": "search", "bscans": 10, "ascans": 500, "betas": 41},
        # one finished plane to its TIFF codes (both quantisations) and packed rows
        {"name": "tiff_plane", "kind": "plane", "rows": 1767, "cols": 1900},
        # the learned estimator on new B-scans: probe images and the network
        {"name": "learned_predict", "kind": "predict", "bscans": 100, "ascans": 500},
        # a training step of the learned estimator: forward, gradients, Adam
        {"name": "learned_train", "kind": "train", "batch": 128},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(["magnitude", "db", "focus", "volume", "row", "tiles", "precision", "float64", "search",
                       "plane", "predict", "train"])
    if kind == "magnitude":
        return {"kind": kind, "bscans": _log(rng, 1, 60), "ascans": _log(rng, 200, 1200)}
    if kind == "db":
        z0 = rng.randint(0, 80)
        return {"kind": kind, "bscans": _log(rng, 1, 60), "ascans": _log(rng, 200, 1200), "z0": z0,
                "depth": rng.randint(400, HALF - z0)}
    if kind == "focus":
        return {"kind": kind, "bscans": _log(rng, 1, 20), "ascans": _log(rng, 150, 800), "binning": rng.randint(2, 4)}
    if kind == "volume":
        return {"kind": kind, "frames": _log(rng, 3, 50), "ascans": rng.randint(300, 1000), "tiles_x": rng.randint(1, 2),
                "depths": rng.randint(1, 3)}
    if kind == "row":
        return {"kind": kind, "frames": _log(rng, 2, 24), "ascans": rng.randint(200, 800), "depths": rng.randint(1, 3),
                "batch": rng.randint(2, 9)}
    if kind == "tiles":
        return {"kind": kind, "tiles": _log(rng, 2, 24), "bscans": _log(rng, 3, 14), "ascans": rng.randint(300, 1200),
                "depth": rng.randint(400, 1400), "mix": rng.randint(0, 1 << 20)}
    if kind == "precision":
        return {"kind": kind, "bscans": _log(rng, 1, 60), "ascans": _log(rng, 200, 1200)}
    if kind == "float64":
        return {"kind": kind, "bscans": _log(rng, 1, 12), "ascans": _log(rng, 150, 800)}
    if kind == "search":
        return {"kind": kind, "bscans": _log(rng, 1, 16), "ascans": rng.randint(200, 600), "betas": rng.randint(9, 41)}
    if kind == "plane":
        return {"kind": kind, "rows": rng.randint(400, 1800), "cols": rng.randint(300, 2000)}
    if kind == "predict":
        return {"kind": kind, "bscans": _log(rng, 1, 100), "ascans": rng.randint(260, 600)}
    return {"kind": kind, "batch": _log(rng, 8, 128)}


# ------------------------------------------------------------------ inputs
def _spectra(bscans, lines, seed, **kw):
    """uint16 spectra (bscans, 25 + lines, 2048) on the device."""
    t = synthetic.generate(bscans, lines, APOD, seed=seed, device="cuda", precision="float32", **kw)
    return synthetic.u16_bits(t).view(torch.uint16)


def _scan_geometry():
    return geometry.build_spectral_geometry(synthetic.lambda_nm(), synthetic.beta_ref_from_px(BETA_PX), 1.33)


def _layout(case):
    """Lateral centres, depths (mm) and focus pixels of a tiled scan at 1 um pixels."""
    nx = case["ascans"]
    half = 0.45e-3 * nx                                        # 10 % lateral overlap
    xc = np.array([-half, half]) if case.get("tiles_x", 1) == 2 else np.array([0.0])
    zd = np.array([0.0, 0.15, 0.30])[:case["depths"]]
    focus = 400.0 + np.array([11.0, -7.5, 22.25])[:case["depths"]]
    return xc, zd, focus


def _tile_sizes(case):
    """(B-scans, A-scans, first output row, output rows) of every tile: U[1/2, 1] of the largest."""
    r = random.Random(case["mix"])
    out = []
    for _ in range(case["tiles"]):
        b, x, z = (r.randint((m + 1) // 2, m) for m in (case["bscans"], case["ascans"], case["depth"]))
        out.append((b, x, r.randint(0, 20), z))
    return out


def _tile_crop_mm(out_z, z0, rows):
    z0 = min(z0, len(out_z) - 1)
    return out_z[z0] - 1e-9, out_z[min(z0 + rows, len(out_z)) - 1] + 1e-9


OPC_POLY = (0.004, -0.003, 1.5e-5, -1.0e-5, 4.0e-6)             # um over the tile's x / y (um)


def prepare(case, seed):
    kind, seed = case["kind"], int(seed) % (1 << 30)
    st = {"kind": kind, "case": case}
    if kind in ("magnitude", "db", "precision", "float64"):
        st["raw"] = _spectra(case["bscans"], case["ascans"], seed)
        st["proc"] = spectral.SpectralProcessor(_scan_geometry(), APOD)
    elif kind == "focus":
        st["raw"] = _spectra(case["bscans"], case["ascans"] * case["binning"], seed)
        st["proc"] = spectral.SpectralProcessor(_scan_geometry(), APOD, ascan_binning=case["binning"])
    elif kind in ("volume", "row"):
        xc, zd, focus = _layout(case)
        sg = _scan_geometry()
        ctx = Context(0)
        ctx.set_geometry(sg.sinc_idx, sg.sinc_w, sg.window)
        F, nx = case["frames"], case["ascans"]
        lay = stitching.ScanLayout(xc, np.array([0.0]), zd, nx, F, nx * 1e-3, F * 1e-3)
        tg = stitching.tiled_geometry(lay, sg.z_um, focus, 1.0)
        oc = None
        if kind == "row":
            oc = stitching.OpticalPathCorrection.build(OPC_POLY, tg.tile_x_mm, tg.tile_y_mm, tg.tile_z_mm)
        st["tiles"], st["raws"] = [], []
        for xi, x in enumerate(xc):
            for zi, z in enumerate(zd):
                s = stitching.TileStitcher.build(tg, x, z, focus[zi], SIGMA)
                s.upload(ctx, oc)
                st["tiles"].append(s)
                st["raws"].append(_spectra(F, nx, seed * 8 + 3 * xi + zi))
        st["ctx"], st["nz"], st["nx"] = ctx, len(tg.out_z_mm), len(tg.out_x_mm)
        if kind == "row":
            st["row"] = reconstruct.RowReconstructor(ctx, APOD, st["nz"], st["nx"], case["batch"])
        else:
            st["planes"] = torch.empty((F, st["nz"], st["nx"]), device="cuda")
    elif kind == "tiles":
        sg = _scan_geometry()
        ctx = Context(0)
        ctx.set_geometry(sg.sinc_idx, sg.sinc_w, sg.window)
        st["ctx"], st["tiles"] = ctx, []
        for k, (b, nx, z0, rows) in enumerate(_tile_sizes(case)):
            lay = stitching.ScanLayout(np.array([0.0]), np.array([0.0]), np.array([0.0]), nx, b, nx * 1e-3, b * 1e-3)
            full = stitching.tiled_geometry(lay, sg.z_um, [np.nan], 1.0)
            tg = stitching.tiled_geometry(lay, sg.z_um, [np.nan], 1.0, _tile_crop_mm(full.out_z_mm, z0, rows))
            plan = stitching.TileStitcher.build(tg, 0.0, 0.0, np.nan, SIGMA).upload(ctx)
            db = torch.empty((b, nx, len(tg.out_z_mm)), device="cuda")
            st["tiles"].append((_spectra(b, nx, seed * 32 + k), APOD, plan, db))
    elif kind == "search":
        st["raw"] = _spectra(case["bscans"], case["ascans"], seed)
        st["betas"] = np.linspace(-1.0, 1.0, case["betas"]) * learned.beta_scale()
        st["scorer"] = estimation.DispersionScorer(synthetic.lambda_nm(), st["raw"], "top_percentile", APOD, rep=1)
    elif kind == "plane":
        st["ctx"] = Context(0)
        st["db"] = _db_plane(case, seed)
        st["clim"] = (-20.0, 55.0)
        fin = st["db"][torch.isfinite(st["db"])]
        st["plane_clim"] = (float(fin.min()), float(fin.max()))
        st["codes"] = torch.empty(st["db"].shape, dtype=torch.uint16, device="cuda")
        st["strips"], st["used"] = np.zeros(st["db"].numel() * 9 // 4, np.uint8), 0
    elif kind == "predict":
        st["maker"] = learned.ImageMaker(synthetic.lambda_nm(), APOD)
        st["net"] = learned.BetaFocusNet(Context(0), seed=seed)
        st["raw"] = _bscans_of_dispersions(case["bscans"], case["ascans"], seed)
        st["images"] = torch.empty((case["bscans"], 3, learned.IMG, learned.IMG), device="cuda")
    else:
        st["net"] = learned.BetaFocusNet(Context(0), seed=seed, train_tensor_cores=True)
        st["x"], st["y"] = _training_batch(case, seed)
    torch.cuda.synchronize()
    return st


def _db_plane(case, seed):
    """A stitched plane: speckle over a depth profile, NaN where no tile reaches."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    r, c = case["rows"], case["cols"]
    z = torch.arange(r, device="cuda", dtype=torch.float32)[:, None] / r
    db = 30.0 * torch.exp(-((z - 0.35) / 0.2) ** 2) + 10.0 * torch.log10(
        (-torch.log(torch.rand((r, c), generator=g, device="cuda").clamp_min(1e-30))).clamp_min(1e-12))
    edge = r // 12 + torch.arange(c, device="cuda")[None, :] * r // (40 * c)
    return torch.where(torch.arange(r, device="cuda")[:, None] < edge, torch.nan, db)


def _bscans_of_dispersions(bscans, ascans, seed):
    r = np.random.default_rng(seed)
    return _spectra(bscans, ascans, seed, beta_px=r.uniform(-5e-5, 5e-5, bscans), focus_px=r.uniform(100, 900, bscans),
                    chunk=50)


def _training_batch(case, seed):
    """Probe images of B-scans and the network's targets."""
    n = case["batch"]
    maker = learned.ImageMaker(synthetic.lambda_nm(), APOD)
    x = maker.images(_bscans_of_dispersions(n, 130, seed))
    torch.cuda.synchronize()
    maker.close()
    r = np.random.default_rng(seed)
    y = learned.targets(r.uniform(-1, 1, n) * learned.beta_scale(), r.uniform(100, 900, n))
    return x, torch.tensor(y, device="cuda")


# ------------------------------------------------------------------ one pass
def run(st):
    kind, case = st["kind"], st["case"]
    if kind == "magnitude":
        return {"magnitude": st["proc"].magnitude(st["raw"])}
    if kind == "db":
        # the range that the call gives beside the planes is their own smallest
        # and largest value, and is in them
        planes, _ = st["proc"].db(st["raw"], case["z0"], case["depth"])
        return {"db": planes}
    if kind == "focus":
        mag = st["proc"].magnitude(st["raw"])
        return {"magnitude": mag, "profile": st["proc"].ctx.xmedian(mag)}
    if kind == "volume":
        st["ctx"].frames_process([t.plan for t in st["tiles"]], st["raws"], APOD, 0, st["nz"], st["nx"],
                                 stitching.min_weight_threshold(np.float32), out=st["planes"])
        return {"db": st["planes"]}
    if kind == "row":
        tiles = [reconstruct.RowTile(t, lambda fr, r=r: r[int(fr[0]):int(fr[-1]) + 1])
                 for t, r in zip(st["tiles"], st["raws"])]
        out = torch.empty((case["frames"], st["nz"], st["nx"]), device="cuda")
        return {"db": st["row"].process_row(tiles, np.arange(case["frames"]), out)}
    if kind == "tiles":
        st["ctx"].batch_process(st["tiles"], stitching.min_weight_threshold(np.float32))
        return {"db": [t[3] for t in st["tiles"]]}
    if kind in ("precision", "float64"):
        raw, ctx = st["raw"], st["proc"].ctx
        out = torch.empty((raw.shape[0], raw.shape[1] - APOD, HALF), device="cuda")
        form = ctx.magnitude_precision if kind == "precision" else ctx.magnitude_exact
        return {"magnitude": form(raw, APOD, out)}
    if kind == "search":
        return {"scores": st["scorer"].scores_grid(st["betas"])}
    if kind == "plane":
        codes = st["ctx"].quantise_double(st["db"], st["plane_clim"], st["clim"], st["codes"])
        packed, sizes = st["ctx"].packbits(codes)
        strips = st["strips"]                                  # the file's buffer
        strips[:len(packed)] = np.frombuffer(packed, np.uint8)
        strips[len(packed):st["used"]] = 0
        st["used"] = len(packed)
        return {"codes": codes, "strips": strips, "sizes": sizes}
    if kind == "predict":
        images = st["maker"].images(st["raw"], out=st["images"])
        return {"images": images, "prediction": st["net"].predict(images)}
    net = st["net"]
    net.train_step(st["x"], st["y"], 1e-5)
    return {"gradients": net.grads, "prediction": net._buffers(case["batch"])["out"]}


# ------------------------------------------------------------------ bytes and operations
FFT = 5 * N * 11                                              # operations of one transform
LINEARISE = 2 * SINC_TAPS * N + 4 * N                         # background and band of one A-scan


def _conv_flops():
    """Multiply-adds of the network's layers for one image, twice."""
    f, h, cin = 0, 256, 3
    for _ in range(4):
        f += 2 * 9 * cin * 32 * h * h
        cin, h = 32, h // 2
    return f + 2 * 32 * 16 * 16 * 64


def work(case):
    kind = case["kind"]
    b, x = case.get("bscans", 0), case.get("ascans", 0)
    raw = b * (x + APOD) * N * 2
    per = LINEARISE + 2 * N + FFT + 3 * HALF
    if kind in ("magnitude", "precision", "float64"):
        return {"bytes": raw + b * x * HALF * 4, "flops": b * x * per}
    if kind == "db":
        return {"bytes": raw + b * x * case["depth"] * 4, "flops": b * x * per}
    if kind == "focus":
        return {"bytes": b * (x * case["binning"] + APOD) * N * 2 + b * x * HALF * 4 + b * HALF * 8,
                "flops": b * x * (per + case["binning"] * N)}
    if kind in ("volume", "row"):
        nt, F = case.get("tiles_x", 1) * case["depths"], case["frames"]
        n_z = 1426 + 150 * (case["depths"] - 1)               # 1 um rows of the tiles' depth range
        n_x = x if case.get("tiles_x", 1) == 1 else x + int(0.9 * x)
        return {"bytes": nt * F * (x + APOD) * N * 2 + F * n_z * n_x * 4,
                "flops": nt * F * x * per + nt * F * x * 1426 * 16}
    if kind == "tiles":
        s = _tile_sizes(case)
        return {"bytes": sum(b * (x + APOD) * N * 2 + b * x * min(z, 1426) * 4 for b, x, _, z in s),
                "flops": sum(b * x * (per + 10 * z) for b, x, _, z in s)}
    if kind == "search":
        n = case["betas"]
        return {"bytes": b * x * N * 4 + n * b * 8, "flops": n * b * x * (2 * N + FFT + 4 * HALF)}
    if kind == "plane":
        n = case["rows"] * case["cols"]
        return {"bytes": n * (4 + 2 + 2 + 2), "flops": 10 * n}
    if kind == "predict":
        img = 3 * 256 * 256 * 4
        return {"bytes": raw + b * img, "flops": b * (x * (LINEARISE + 3 * (2 * N + FFT)) + _conv_flops())}
    n, acts, h = case["batch"], 3 * 256 * 256, 256
    for _ in range(4):
        acts += 2 * 32 * h * h + 2 * 32 * (h // 2) ** 2       # pre-activations and pooled, forward and gradient
        h //= 2
    return {"bytes": n * acts * 4, "flops": 3 * n * _conv_flops()}


# ------------------------------------------------------------------ float64 results
def _f64_geometry(beta_px):
    """The banded sinc operator (2048 x 2048), the window (complex) and the depth axis (um), from their definitions."""
    lam = synthetic.lambda_nm()
    k = 2 * np.pi / lam
    k_lin = np.linspace(k.max(), k.min(), N)
    at = (k_lin - k_lin.min()) / (k_lin.max() - k_lin.min()) * (N - 1)
    src = (k - k.min()) / (k.max() - k.min()) * (N - 1)
    d = at[:, None] - src[None, :]
    band = np.where(np.abs(d) < 5, np.sinc(d), 0.0)
    hann = 0.5 * (1 - np.cos(2 * np.pi * np.arange(N) / (N - 1)))
    hann /= np.sqrt(np.mean(hann ** 2))
    dk2 = (k_lin - k_lin.mean()) ** 2
    beta = beta_px / ((k.max() - k.min()) / (N - 1)) ** 2
    lo, hi = 2 * np.pi / k_lin[0] / 1e3, 2 * np.pi / k_lin[-1] / 1e3
    z = np.linspace(0.0, 0.5 * (0.5 * (lo + hi)) ** 2 / abs(hi - lo) / 1.33 * N / 2, HALF)
    return band, hann, dk2, hann * np.exp(-1j * beta * dk2), z


def _f64_lines(raw, band):
    """Background-free, k-linearised lines of raw B-scans (B, 25 + nX, N) in float64."""
    raw = raw.to(torch.int32).double() if raw.dtype == torch.uint16 else raw.double()
    d = raw[:, APOD:] - raw[:, :APOD].mean(1, keepdim=True)
    m = d.mean(-1, keepdim=True)
    return (d - m) @ torch.as_tensor(band, device=raw.device).T + m


def _f64_magnitude(raw, geo):
    w = torch.as_tensor(geo[3], device=raw.device)
    return torch.cat([torch.fft.ifft(_f64_lines(r, geo[0]) * w).abs()[..., :HALF] for r in raw.split(8)])


def _f64_taps(src, dst):
    """Left node, fraction and validity of linear interpolation from src to dst (0 outside)."""
    src = np.array(src, float)
    src[0] -= 1e-10
    src[-1] += 1e-10
    j = np.clip(np.searchsorted(src, dst, side="right") - 1, 0, len(src) - 2)
    t = (dst - src[j]) / (src[j + 1] - src[j])
    t = np.where(np.abs(t) < 1e-9, 0.0, np.where(np.abs(1 - t) < 1e-9, 1.0, t))
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    return (torch.as_tensor(j, device=dev), torch.as_tensor(t, device=dev),
            torch.as_tensor((dst >= src[0]) & (dst <= src[-1]), device=dev))


def _f64_apply(v, taps):
    """Interpolate along the last axis."""
    j, t, ok = taps
    return torch.where(ok, v[..., j] * (1 - t) + v[..., j + 1] * t, 0.0)


def _colon(a, d, b):
    return a + d * np.arange(int(np.floor((b - a) / d + 1e-10)) + 1)


def _f64_stitched(case, raws, geo):
    """Focus-weighted planes of a tiled scan: sum of tiles over sum of weights, in dB."""
    F, nx = case["frames"], case["ascans"]
    xc, zd, focus = _layout(case)
    tile_x = (nx * 1e-3 * np.linspace(-0.5, 0.5, nx + 1))[:-1]
    tile_y = (F * 1e-3 * np.linspace(-0.5, 0.5, F + 1))[:-1]
    tile_z = geo[4] / 1e3
    tile_z = tile_z - tile_z[int(np.round(focus[0])) - 1]
    dx, dz = tile_x[1] - tile_x[0], tile_z[1] - tile_z[0]
    out_x = tile_x if len(xc) == 1 else _colon(xc.min() + tile_x[0], dx, xc.max() + tile_x[-1] + dx / 2)
    cover = _colon(zd.min() + tile_z[0], dz, zd.max() + tile_z[-1] + dz / 2)
    cover = dz * (np.arange(len(cover)) - int(np.argmin(np.abs(cover))))
    out_z = _colon(cover[0], 1e-3, cover.max())
    rows = torch.arange(HALF, device="cuda")
    valid, at = torch.ones((F, nx, HALF), dtype=torch.bool, device="cuda"), None
    if case["kind"] == "row":
        X, Y = np.meshgrid(tile_x * 1e3, tile_y * 1e3)
        p = OPC_POLY
        shift = (p[0] * X + p[1] * Y + p[2] * X ** 2 + p[3] * Y ** 2 + p[4] * X * Y) / (dz * 1e3)
        q = torch.as_tensor(shift, device="cuda")[..., None] + rows
        valid = (q >= 0) & (q <= HALF - 1)
        at = (torch.as_tensor(np.floor(shift + 0.5), device="cuda").long()[..., None] + rows).clamp(0, HALF - 1)
    num = den = 0.0
    floor = math.exp(-4.5)
    for k, raw in enumerate(raws):
        xi, zi = divmod(k, len(zd))
        mag = _f64_magnitude(raw, geo)
        if at is not None:
            mag = mag.gather(-1, at)
        wz = torch.exp(-((rows + 1 - focus[zi]) ** 2) / (2 * SIGMA) ** 2) + floor
        w = torch.where(valid, wz, 0.0)
        tz = _f64_taps(tile_z + zd[zi] - tile_z[int(np.round(focus[zi])) - 1], out_z)
        tx = _f64_taps(tile_x + xc[xi], out_x)
        num = num + _f64_apply(_f64_apply(mag * w, tz).transpose(1, 2), tx)
        den = den + _f64_apply(_f64_apply(w.double(), tz).transpose(1, 2), tx)
        del mag, w
    den = torch.where(den < floor * (1 - 8 * 2.0 ** -23), torch.nan, den)
    return 20 * torch.log10(num / den)


def _f64_images(raw, geo, probes):
    """Standardised probe images (B, probes, 256, 256)."""
    hann, dk2 = torch.as_tensor(geo[1], device="cuda"), torch.as_tensor(geo[2], device="cuda")
    out = []
    for r in raw.split(8):
        x = _f64_lines(r, geo[0]) * hann
        img = [torch.nn.functional.adaptive_avg_pool2d(
            torch.fft.ifft(x * torch.exp(-1j * b * dk2)).abs()[..., :learned.Z_KEEP].transpose(1, 2),
            (learned.IMG, learned.IMG)) for b in probes]
        v = 20 * torch.log10(torch.stack(img, 1))
        out.append((v - v.mean((1, 2, 3), keepdim=True)) / v.std((1, 2, 3), keepdim=True, correction=0))
    return torch.cat(out)


def _f64_network(net, x):
    """The network's predictions from float64 copies of its weights, and these."""
    p = [t.double().requires_grad_() for t in net.params]
    fn = torch.nn.functional
    for i in range(4):
        x = fn.avg_pool2d(fn.relu(fn.conv2d(x, p[2 * i], p[2 * i + 1], padding=1)), 2)
    h = fn.relu(x.flatten(1) @ p[8].T + p[9])
    return h @ p[10].T + p[11], p


def exact(case, seed):
    kind, seed = case["kind"], int(seed) % (1 << 30)
    geo = _f64_geometry(BETA_PX)
    if kind in ("magnitude", "db", "precision", "float64"):
        mag = _f64_magnitude(_spectra(case["bscans"], case["ascans"], seed), geo)
        if kind == "db":
            return {"db": 20 * torch.log10(mag[..., case["z0"]:case["z0"] + case["depth"]])}
        return {"magnitude": mag}
    if kind == "focus":
        n = case["binning"]
        raw = _spectra(case["bscans"], case["ascans"] * n, seed).to(torch.int32).double()
        scan = raw[:, APOD:]
        first = max(1, n // 2) - 1 - ((n + 1) // 2 - 1)        # first line of the first bin
        cols = first + n * torch.arange(case["ascans"], device="cuda")[:, None] + torch.arange(n, device="cuda")
        lines = torch.where(((cols >= 0) & (cols < scan.shape[1]))[..., None],
                            scan[:, cols.clamp(0, scan.shape[1] - 1)], 0.0).mean(2)
        mag = _f64_magnitude(torch.cat([raw[:, :APOD], lines], 1), geo)
        return {"magnitude": mag, "profile": torch.quantile(mag, 0.5, dim=1)}
    if kind in ("volume", "row"):
        raws = [_spectra(case["frames"], case["ascans"], seed * 8 + 3 * xi + zi)
                for xi in range(case.get("tiles_x", 1)) for zi in range(case["depths"])]
        return {"db": _f64_stitched(case, raws, geo)}
    if kind == "tiles":
        tz = geo[4] / 1e3
        full = _colon(tz[0], 1e-3, (tz[1] - tz[0]) * (HALF - 1))
        db = []
        for k, (b, nx, z0, rows) in enumerate(_tile_sizes(case)):
            lo, hi = _tile_crop_mm(full, z0, rows)
            mag = _f64_magnitude(_spectra(b, nx, seed * 32 + k), geo)
            db.append(20 * torch.log10(_f64_apply(mag, _f64_taps(tz, full[(full >= lo) & (full <= hi)]))))
        return {"db": db}
    if kind == "search":
        raw = _spectra(case["bscans"], case["ascans"], seed)
        x = _f64_lines(raw, geo[0]) * torch.as_tensor(geo[1], device="cuda")
        dk2 = torch.as_tensor(geo[2], device="cuda")
        top = max(1, int(case["ascans"] * (HALF - estimation.Z_MIN_PIX) * estimation.TOP_FRACTION))
        scores = []
        for b in np.linspace(-1.0, 1.0, case["betas"]) * learned.beta_scale():
            a = torch.fft.ifft(x * torch.exp(-1j * b * dk2)).abs()[..., estimation.Z_MIN_PIX:HALF].flatten(1)
            scores.append(torch.log((a ** 2).topk(top, dim=1).values.mean(1)))
        return {"scores": torch.stack(scores)}
    if kind == "predict":
        images = _f64_images(_bscans_of_dispersions(case["bscans"], case["ascans"], seed), geo,
                             learned.probe_betas())
        with torch.no_grad():
            net = learned.BetaFocusNet(Context(0), seed=seed)
            pred = torch.cat([_f64_network(net, v)[0] for v in images.split(10)])
        return {"images": images, "prediction": pred}
    if kind == "train":
        x, y = _training_batch(case, seed)
        net = learned.BetaFocusNet(Context(0), seed=seed)
        n, grads, preds = case["batch"], None, []
        for i in range(0, n, 8):
            pred, p = _f64_network(net, x[i:i + 8].double())
            g = torch.autograd.grad(((pred - y[i:i + 8].double()) ** 2).sum() / (2 * n), p)
            grads = g if grads is None else [a + b for a, b in zip(grads, g)]
            preds.append(pred.detach())
        return {"gradients": [g.detach() for g in grads], "prediction": torch.cat(preds)}
    return None                                               # codes and bytes: whole numbers
