"""Kernels at the sizes where their tiling can go wrong (remainders of warps
and blocks, the smallest and the largest of a range), against plain NumPy."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bscans,rep,nx", [(1, 1, 1), (1, 1, 5), (2, 2, 3), (1, 3, 7), (2, 1, 1000)])
def test_transform_of_loaded_lines(gpu_ctx, bscans, rep, nx):
    """|ifft(line * phase)| of every loaded line and beta, averaged over the
    repeats.  Tolerance: float32 transform of 11 radix-2 layers, each rounding
    within 2^-24 of the line's largest magnitude (a few ulps in all): 1e-6."""
    from oct_recon_af_v1_gb300 import estimation as E
    from oct_recon_af_v1_gb300 import geometry as G
    from oct_recon_af_v1_gb300 import synthetic
    lam = synthetic.lambda_nm()
    sg = G.build_spectral_geometry(lam, 0.0, 1.33)
    dk2 = G.dispersion_dk2(sg)
    gpu_ctx.set_geometry(sg.sinc_idx, sg.sinc_w, np.ones(2048, np.complex128))
    gpu_ctx.disp_set_dk2(dk2)
    raw = synthetic.generate_numpy(bscans * rep, nx, 25, seed=5)
    gpu_ctx.disp_load(raw, 25, bscans, rep, E.hann_rms(2048))
    lines = gpu_ctx.disp_lines().astype(np.float64).reshape(bscans, rep, nx, 2048)
    betas = [0.0, 2.5e7]
    mag = np.empty((2, bscans, nx, 1024), np.float32)
    gpu_ctx.disp_eval(betas, 0, bscans, 0, mag=mag)
    for got, beta in zip(mag, betas):
        phase = np.exp(-1j * beta * dk2).astype(np.complex64).astype(np.complex128)
        ref = np.abs(np.fft.ifft(lines * phase)[..., :1024]).mean(1)
        assert np.abs(got - ref).max() < 1e-6 * ref.max()


@pytest.mark.parametrize("bscans,nx,betas,z_min", [(1, 1, 1, 20), (1, 3, 1, 0), (1, 37, 2, 21), (2, 130, 3, 1000),
                                                   (1, 900, 1, 20), (40, 9, 13, 20)])
def test_top_percentile_of_returned_magnitudes(gpu_ctx, bscans, nx, betas, z_min):
    """The score is the log of the mean of the k largest squared magnitudes:
    against the magnitudes the same call returns (in a buffer aligned to one
    float only), for clusters of 1 to 8 blocks, all elements equal included
    (k of them tie).  Both sides sum float64 values of the same float32 squares:
    1e-12."""
    torch = pytest.importorskip("torch")
    from oct_recon_af_v1_gb300 import estimation as E
    from oct_recon_af_v1_gb300 import geometry as G
    from oct_recon_af_v1_gb300 import synthetic
    sg = G.build_spectral_geometry(synthetic.lambda_nm(), 0.0, 1.33)
    gpu_ctx.set_geometry(sg.sinc_idx, sg.sinc_w, np.ones(2048, np.complex128))
    gpu_ctx.disp_set_dk2(G.dispersion_dk2(sg))
    raw = synthetic.generate_numpy(bscans, nx, 25, seed=6)
    if nx == 9:
        raw[:, 25:] = raw[:, 25:26]                     # identical A-scans: every value repeats nine times
    gpu_ctx.disp_load(raw, 25, bscans, 1, E.hann_rms(2048))
    n = nx * (1024 - z_min)
    buf = torch.empty(betas * bscans * nx * 1024 + 1, dtype=torch.float32, device="cuda")
    mag = buf[1:].view(betas, bscans, nx, 1024)
    for k in (1, max(1, n // 100), n):
        got = gpu_ctx.disp_eval(np.linspace(-2e7, 2e7, betas), 0, bscans, 1, k, z_min, mag=mag)
        sq = np.sort((mag * mag).cpu().numpy()[..., z_min:].reshape(betas, bscans, n).astype(np.float64))[..., n - k:]
        np.testing.assert_allclose(got, np.log(sq.mean(-1)), rtol=1e-12, atol=1e-12)


@pytest.mark.parametrize("rows,cols", [(1, 1), (3, 2), (5, 63), (4, 64), (2, 65), (130, 129), (1030, 7), (3, 5001)])
def test_packbits_rows(gpu_ctx, rows, cols):
    """Packets around the 128-byte limit, runs that end at a packet's or a
    row's end, more rows than one scan block: the oracle's bytes exactly."""
    from oracle import numerics as O
    rng = np.random.default_rng(rows * 7919 + cols)
    img = rng.integers(0, 65536, size=(rows, cols)).astype(np.uint16)
    for r in range(rows):
        x = 0
        while x < cols:                                    # literals and runs of every length, byte runs of two kinds
            n = int(rng.integers(1, 140))
            v = rng.integers(0, 4)
            if v < 2:
                img[r, x:x + n] = (0, 0x4141, 0x0041, 0xffff)[int(rng.integers(0, 4))]
            x += n
    packed, sizes = gpu_ctx.packbits(img)
    ref = [O.packbits_encode_row(img[r].astype("<u2").tobytes()) for r in range(rows)]
    assert [int(s) for s in sizes] == [len(b) for b in ref]
    assert packed == b"".join(ref)


@pytest.mark.parametrize("rows,cols", [(1030, 130), (33, 2000), (3000, 7), (1, 33000)])
def test_packbits_rows_put_together_on_the_device(gpu_ctx, rows, cols):
    """The same for images whose rows are gathered on the device (more than 64 KB)."""
    test_packbits_rows(gpu_ctx, rows, cols)


@pytest.mark.parametrize("nx,nz", [(1, 1), (2, 17), (31, 16), (32, 5), (33, 40), (256, 20), (257, 20), (512, 9),
                                   (1024, 33), (1025, 9), (4096, 3)])
def test_x_profiles_equal_numpy(gpu_ctx, nx, nz):
    """Median, nanmedian and mean over x at the edges of the kernel's register
    forms: ties, negative values, infinities and NaN, odd and even counts.
    The medians are exact; a float64 mean of up to 4096 values: 1e-12."""
    rng = np.random.default_rng(nx * 31 + nz)
    mag = rng.normal(size=(2, nx, nz)).astype(np.float32)
    mag[0] = np.round(mag[0])                                   # many ties, both zeros
    np.testing.assert_array_equal(gpu_ctx.xmedian(mag), np.median(mag.astype(np.float64), axis=1))
    np.testing.assert_allclose(gpu_ctx.xmean(mag), mag.astype(np.float64).mean(1), rtol=1e-12, atol=1e-12)
    mag[1, rng.integers(0, nx, nx // 3), rng.integers(0, nz, nx // 3)] = np.nan
    mag[0, nx // 2, 0] = np.inf
    mag[1, 0, nz - 1] = -np.inf
    mag[1, :, nz // 2] = np.nan
    with np.errstate(all="ignore"):
        import warnings
        warnings.simplefilter("ignore", RuntimeWarning)
        np.testing.assert_array_equal(gpu_ctx.xmedian(mag), np.median(mag.astype(np.float64), axis=1))
        np.testing.assert_array_equal(gpu_ctx.xmedian(mag, ignore_nan=True),
                                      np.nanmedian(mag.astype(np.float64), axis=1))


@pytest.mark.parametrize("nx", [1, 2, 31, 32, 33, 257, 513])
def test_x_profiles_of_many_columns(gpu_ctx, nx):
    """The same where the columns fill the GPU sixteen to a block (a ragged last one)."""
    test_x_profiles_equal_numpy(gpu_ctx, nx, 1305)


@pytest.mark.parametrize("nx,nz", [(1, 3), (33, 20), (1025, 9)])
def test_x_mean_with_infinities_and_nan(gpu_ctx, nx, nz):
    """NaN is left out, an infinity is not: numpy.nanmean's values (1e-12, as
    above), infinite columns, opposite infinities and columns of NaN included."""
    rng = np.random.default_rng(nx)
    mag = rng.normal(size=(3, nx, nz)).astype(np.float32)
    mag[0, rng.integers(0, nx, nx // 3), rng.integers(0, nz, nx // 3)] = np.nan
    mag[0, nx // 2, 0] = np.inf
    mag[1, 0, nz - 1] = -np.inf
    mag[1, :, 1] = np.nan
    mag[2, 0, 2], mag[2, -1, 2] = np.inf, -np.inf
    with np.errstate(all="ignore"):
        import warnings
        warnings.simplefilter("ignore", RuntimeWarning)
        np.testing.assert_allclose(gpu_ctx.xmean(mag), np.nanmean(mag.astype(np.float64), axis=1), rtol=1e-12,
                                   atol=1e-12)


@pytest.mark.parametrize("dtype", [np.uint16, np.int16, np.float32])
@pytest.mark.parametrize("bscans,nx", [(1, 1), (1, 2), (3, 1), (2, 7), (1, 305), (5, 123)])
def test_lines_and_magnitudes_of_ragged_batches(gpu_ctx, dtype, bscans, nx):
    """Fewer A-scans than blocks, odd counts, B-scans of one A-scan, signed and
    negative counts: the linearised spectra and magnitudes against the oracle's
    float32 restatement.  Tolerance 2e-6 of the largest value: about ten
    float32 roundings in the band sum, eleven layers of the transform."""
    from oracle import numerics as O
    from oct_recon_af_v1_gb300 import geometry as G
    from oct_recon_af_v1_gb300 import synthetic
    lam, beta = synthetic.lambda_nm(), synthetic.beta_ref_from_px(1e-5)
    sg = G.build_spectral_geometry(lam, beta, 1.33)
    gpu_ctx.set_geometry(sg.sinc_idx, sg.sinc_w, sg.window)
    raw = synthetic.generate_numpy(bscans, nx, 25, seed=bscans * 1000 + nx)
    if dtype == np.int16:
        raw = (raw.astype(np.int32) - 9000).astype(np.int16)
    raw = raw.astype(dtype)
    og = O.spectral_geometry(lam, beta, 1.33)
    ref = O.magnitude_numba(raw, og, 25)
    assert np.abs(gpu_ctx.magnitude(raw, 25) - ref).max() < 2e-6 * np.abs(ref).max()
    spec = O.fused_pre_fft_numba(raw, 25, og.sinc_idx.T, og.sinc_w.T.astype(np.float32),
                                 og.window.astype(np.complex64))
    assert np.abs(gpu_ctx.fused_pre_fft(raw, 25) - spec).max() < 2e-6 * np.abs(spec).max()


@pytest.mark.parametrize("dtype", [np.uint16, np.int16, np.float32])
@pytest.mark.parametrize("apod", [9, 10, 127, 128, 144, 145, 1024, 1057])
def test_apodisation_mean_of_many_lines(gpu_ctx, dtype, apod):
    """Line counts around the batches in flight and where they grow: with equal
    scan lines of zero the linearised spectrum is minus the mean's, exactly that
    of a call with the mean as its one float32 line."""
    from oct_recon_af_v1_gb300 import geometry as G
    from oct_recon_af_v1_gb300 import synthetic
    sg = G.build_spectral_geometry(synthetic.lambda_nm(), 0.0, 1.33)
    gpu_ctx.set_geometry(sg.sinc_idx, sg.sinc_w, sg.window)
    rng = np.random.default_rng(apod)
    raw = np.zeros((3, apod + 2, 2048), dtype)
    raw[:, :apod] = rng.integers(0, 30000, (3, apod, 2048))
    mean = np.zeros((3, 3, 2048), np.float32)
    mean[:, 0] = raw[:, :apod].astype(np.float64).sum(1) / apod
    np.testing.assert_array_equal(gpu_ctx.fused_pre_fft(raw, apod), gpu_ctx.fused_pre_fft(mean, 1))


@pytest.mark.parametrize("dtype", [np.uint16, np.float32])
@pytest.mark.parametrize("span_nm,bscans,nx", [(300.0, 2, 7), (600.0, 1, 1), (600.0, 3, 305), (800.0, 1, 154), (800.0, 5, 61)])
def test_lines_of_wide_windows(gpu_ctx, dtype, span_nm, bscans, nx):
    """Spectrometers whose four neighbouring outputs read up to 18, 22 and 26
    source samples: magnitudes against the oracle's float32 restatement (4e-6 of
    the largest: a band of up to twenty products and the transform's eleven
    layers), the scorer's lines exactly (the plain line times the float64 window,
    rounded once)."""
    from oracle import numerics as O
    from oct_recon_af_v1_gb300 import estimation as E
    from oct_recon_af_v1_gb300 import geometry as G
    from oct_recon_af_v1_gb300 import synthetic
    lam = np.linspace(1300 - span_nm / 2, 1300 + span_nm / 2, 2048)
    sg, og = G.build_spectral_geometry(lam, 0.0, 1.33), O.spectral_geometry(lam, 0.0, 1.33)
    gpu_ctx.set_geometry(sg.sinc_idx, sg.sinc_w, sg.window)
    raw = synthetic.generate_numpy(bscans, nx, 25, seed=nx).astype(dtype)
    ref = O.magnitude_numba(raw, og, 25)
    assert np.abs(gpu_ctx.magnitude(raw, 25) - ref).max() < 4e-6 * np.abs(ref).max()
    gpu_ctx.set_geometry(sg.sinc_idx, sg.sinc_w, np.ones(2048, np.complex128))
    line = gpu_ctx.fused_pre_fft(raw, 25).real.astype(np.float64)
    gpu_ctx.disp_load(raw, 25, bscans, 1, E.hann_rms(2048))
    np.testing.assert_array_equal(gpu_ctx.disp_lines(), (line * E.hann_rms(2048)).astype(np.float32))


def test_batched_tiles_equal_single_tiles_across_passes(gpu_ctx):
    """Tiles of uneven size (an empty one, B-scans shorter than a group of
    four, one B-scan longer than the smallest pass) in one call against one
    call a tile: the same bits and the same running range."""
    torch = pytest.importorskip("torch")
    from oct_recon_af_v1_gb300 import _lib
    from oct_recon_af_v1_gb300 import geometry as G
    from oct_recon_af_v1_gb300 import stitching as S
    from oct_recon_af_v1_gb300 import synthetic
    ctx = _lib.Context(0)
    try:
        sg = G.build_spectral_geometry(synthetic.lambda_nm(), 0.0, 1.33)
        ctx.set_geometry(sg.sinc_idx, sg.sinc_w, sg.window)
        tiles = []
        for k, (b, nx, rows) in enumerate(((2, 3, 50), (0, 9, 40), (1, 3801, 33), (3, 130, 257), (1, 5, 700))):
            lay = S.ScanLayout(np.array([0.0]), np.array([0.0]), np.array([0.0]), nx, max(b, 1), nx * 1e-3,
                                max(b, 1) * 1e-3)
            z = S.tiled_geometry(lay, sg.z_um, [np.nan], 1.0).out_z_mm
            tg = S.tiled_geometry(lay, sg.z_um, [np.nan], 1.0, (z[10] - 1e-9, z[9 + rows] + 1e-9))
            plan = S.TileStitcher.build(tg, 0.0, 0.0, np.nan, 80.0).upload(ctx)
            raw = torch.from_numpy(synthetic.generate_numpy(max(b, 1), nx, 25, seed=k).view(np.int16)).cuda()[:b]
            tiles.append((raw.contiguous(), 25, plan, torch.empty((b, nx, len(tg.out_z_mm)), device="cuda")))
        if tiles[1][3].data_ptr() == 0:                     # an empty tile still has a place in memory
            tiles[1] = (tiles[0][0][:0], 25, tiles[1][2], torch.empty(16, device="cuda")[:0].view(0, 9, 0))
        args = [t for t in tiles if t[0].data_ptr() and t[3].data_ptr()]
        thr = S.min_weight_threshold(np.float32)
        ctx.clim_reset()
        ctx.batch_process(args, thr)
        together, clim = [t[3].clone() for t in args], ctx.clim_get()
        ctx.clim_reset()
        for t in args:
            t[3].fill_(0)
            ctx.batch_process([t], thr)
        assert ctx.clim_get() == clim
        for t, ref in zip(args, together):
            assert torch.isfinite(ref).all()
            assert torch.equal(t[3], ref)
    finally:
        ctx.close()


@pytest.mark.parametrize("pass_lines", [64, 101, 1000, 1266, 3797, 3800])
def test_batched_tiles_do_not_depend_on_the_pass(pass_lines):
    """Passes that end at a B-scan's start, inside a B-scan longer than a pass,
    at and among its last four A-scans, against one pass for everything: the same
    bits and range.  The lateral operator blends neighbours wherever a group of
    four allows it."""
    torch = pytest.importorskip("torch")
    from oct_recon_af_v1_gb300 import _lib
    from oct_recon_af_v1_gb300 import geometry as G
    from oct_recon_af_v1_gb300 import stitching as S
    from oct_recon_af_v1_gb300 import synthetic
    ctx = _lib.Context(0)
    try:
        ctx.follow_torch_stream()
        sg = G.build_spectral_geometry(synthetic.lambda_nm(), 0.0, 1.33)
        ctx.set_geometry(sg.sinc_idx, sg.sinc_w, sg.window)
        tiles = []
        for k, (b, nx, rows) in enumerate(((2, 3, 50), (1, 3801, 33), (3, 130, 257), (1, 64, 9), (2, 1003, 20))):
            lay = S.ScanLayout(np.array([0.0]), np.array([0.0]), np.array([0.0]), nx, b, nx * 1e-3, b * 1e-3)
            z = S.tiled_geometry(lay, sg.z_um, [np.nan], 1.0).out_z_mm
            tg = S.tiled_geometry(lay, sg.z_um, [np.nan], 1.0, (z[10] - 1e-9, z[9 + rows] + 1e-9))
            st = S.TileStitcher.build(tg, 0.0, 0.0, np.nan, 80.0)
            assert st.c0 == 0 and st.c1 == nx
            for x in range(0, nx - 8, 2):
                st.WxT[x:x + 2, x:x + 2] = ((0.75, 0.25), (0.25, 0.75))
            raw = torch.from_numpy(synthetic.generate_numpy(b, nx, 25, seed=k).view(np.int16)).cuda()
            tiles.append((raw, 25, st.upload(ctx), torch.empty((b, nx, len(tg.out_z_mm)), device="cuda")))
        thr = S.min_weight_threshold(np.float32)

        def run():
            ctx.clim_reset()
            for t in tiles:
                t[3].fill_(7.0)
            ctx.batch_process(tiles, thr)
            return [t[3].clone() for t in tiles], ctx.clim_get()
        whole, clim = run()
        ctx.set_pass_lines(pass_lines)
        parts, clim2 = run()
        assert clim2 == clim
        assert all(torch.isfinite(w).all() and torch.equal(w, p) for w, p in zip(whole, parts))
        small, raw = torch.empty((2, 1003, 1024), device="cuda"), tiles[4][0]       # and the magnitudes
        ctx.magnitude(raw, 25, small, raw_dtype=0)
        ctx.set_pass_lines()
        assert torch.equal(small, ctx.magnitude(raw, 25, torch.empty_like(small), raw_dtype=0))
        for bad in (-1, 63, 91_201):
            assert ctx.lib.octgb_set_pass_lines(ctx.h, bad) == _lib.ERR_ARG
    finally:
        ctx.close()


@pytest.mark.parametrize("nx,frames,tiles_x,depths,fraction", [(7, 1, 1, 1, 0.0), (33, 2, 2, 3, 0.0), (64, 3, 2, 2, 0.5),
                                                               (301, 2, 2, 3, 0.3), (1000, 1, 2, 3, 0.0)])
def test_stitched_frames_against_oracle_and_row_interface(gpu_ctx, nx, frames, tiles_x, depths, fraction):
    """Blocks where columns take one A-scan of a tile, two (tiles a fraction of
    a pixel apart, the widened end columns), tiles that miss a block, ragged
    last blocks, every block height: the oracle's planes from the same
    magnitudes, the row interface bit for bit, and the range of the planes.
    Tolerance: a ratio of sums of at most 12 products, each rounded a few
    times (2e-6 relative, 2e-5 dB), and dB values up to 100 to an ulp."""
    torch = pytest.importorskip("torch")
    from oracle import numerics as O
    from oct_recon_af_v1_gb300 import geometry as G
    from oct_recon_af_v1_gb300 import reconstruct as R
    from oct_recon_af_v1_gb300 import stitching as S
    from oct_recon_af_v1_gb300 import synthetic
    sg = G.build_spectral_geometry(synthetic.lambda_nm(), 0.0, 1.33)
    gpu_ctx.set_geometry(sg.sinc_idx, sg.sinc_w, sg.window)
    xc = np.array([0.0, (nx - max(1, nx // 10) + fraction) * 1e-3])[:tiles_x]
    zd = np.array([0.0, 0.15, 0.3])[:depths]
    focus = np.array([411.0, 392.5, 422.25])[:depths]
    lay = S.ScanLayout(xc, np.array([0.0]), zd, nx, frames, nx * 1e-3, frames * 1e-3)
    tg = S.tiled_geometry(lay, sg.z_um, focus, 1.0)
    desc = O.ScanDesc(xc, np.array([0.0]), zd, nx, frames, nx * 1e-3, frames * 1e-3)
    og = O.tiled_geometry(desc, sg.z_um, focus, 1.0)
    nz, nxo = len(tg.out_z_mm), len(tg.out_x_mm)
    num, den = np.zeros((frames, nz, nxo), np.float32), np.zeros((frames, nz, nxo), np.float32)
    ids, raws, stitchers = [], [], []
    for xi in range(tiles_x):
        for zi in range(depths):
            st = S.TileStitcher.build(tg, xc[xi], zd[zi], focus[zi], 80.0)
            ids.append(st.upload(gpu_ctx))
            stitchers.append(st)
            raw = torch.from_numpy(synthetic.generate_numpy(frames, nx, 25, seed=9 * xi + zi).view(np.int16)).cuda()
            raws.append(raw)
            mag = torch.empty((frames, nx, 1024), device="cuda")
            gpu_ctx.magnitude(raw, 25, mag, raw_dtype=0)
            gpu_ctx.synchronize()
            o = O.Stitcher(og, xc[xi], zd[zi], focus[zi], 80.0)
            a, b = o.contribute(mag.cpu().numpy())
            num[:, :, o.c0:o.c1] += a
            den[:, :, o.c0:o.c1] += b
    ref = O.finalise(num, den)
    thr = S.min_weight_threshold(np.float32)
    row = R.RowReconstructor(gpu_ctx, 25, nz, nxo, 2)
    out = torch.empty((frames, nz, nxo), device="cuda")
    row.process_row([R.RowTile(t, lambda fr, r=r: r[int(fr[0]):int(fr[-1]) + 1].view(torch.uint16))
                     for t, r in zip(stitchers, raws)], np.arange(frames), out)
    gpu_ctx.synchronize()
    rows_db = out.cpu().numpy()
    try:
        for height in (32, 64, 128):
            gpu_ctx.set_stitch_rows(height)
            gpu_ctx.clim_reset()
            planes = torch.full((frames, nz, nxo), 7.0, device="cuda")
            _, mm = gpu_ctx.frames_process(ids, raws, 25, 0, nz, nxo, thr, out=planes, plane_minmax=True, raw_dtype=0)
            db = planes.cpu().numpy()
            np.testing.assert_array_equal(db, rows_db)
            assert np.array_equal(np.isnan(db), np.isnan(ref))
            fin = np.isfinite(ref)
            assert np.abs(db[fin] - ref[fin]).max() < 4e-5
            for f in range(frames):
                assert (mm[f] == [db[f][np.isfinite(db[f])].min(), db[f][np.isfinite(db[f])].max()]).all()
            assert gpu_ctx.clim_get() == (db[fin].min(), db[fin].max())
    finally:
        gpu_ctx.set_stitch_rows(64)


@pytest.mark.parametrize("dtype", [np.uint16, np.int16])
@pytest.mark.parametrize("bscans,nx,apod", [(1, 1, 1), (3, 5, 25), (1, 200, 255), (2, 130, 256), (1, 40, 700)])
def test_precision_lines_of_integer_raws(gpu_ctx, dtype, bscans, nx, apod):
    """The exact background on either side of the count up to which its sums
    are float32 integers, full-range counts included: the linearised lines
    against float64.  Tolerance: one rounding of d - m and about eleven of the
    band (2^-24 each of sums up to ~3 times the largest value): 2e-6."""
    from oracle import numerics as O
    from oct_recon_af_v1_gb300 import geometry as G
    from oct_recon_af_v1_gb300 import synthetic
    lam = synthetic.lambda_nm()
    sg = G.build_spectral_geometry(lam, 0.0, 1.33)
    gpu_ctx.set_geometry(sg.sinc_idx, sg.sinc_w, np.ones(2048, np.complex128))
    raw = synthetic.generate_numpy(bscans, nx, apod, seed=nx)
    raw[0, -1, ::3] = 65535                                   # the ends of the range beside ordinary counts
    raw[0, 0, ::5] = 65535
    raw = (raw.astype(np.int64) - (32768 if dtype == np.int16 else 0)).astype(dtype)
    x64 = O.linearise_numpy(raw, O.spectral_geometry(lam, 0.0, 1.33), apod, np.float64)
    got = gpu_ctx.linearise_precision(raw, apod)
    assert np.abs(got - x64).max() < 2e-6 * np.abs(x64).max()


@pytest.mark.parametrize("dtype", [np.uint16, np.int16])
@pytest.mark.parametrize("bscans,nx,apod", [(1, 1, 1), (1, 6, 700), (2, 3, 255), (1, 9, 3)])
def test_float64_form_at_the_ends_of_the_range(gpu_ctx, dtype, bscans, nx, apod):
    """Full-range counts, many apodisation lines, a constant spectrum (all its
    magnitudes zero): the float32 rounding of float64's magnitudes but for the
    pairs' ~1e-12 of the line's largest."""
    from oracle import numerics as O
    from oct_recon_af_v1_gb300 import geometry as G
    from oct_recon_af_v1_gb300 import synthetic
    lam, beta = synthetic.lambda_nm(), synthetic.beta_ref_from_px(1e-5)
    sg = G.build_spectral_geometry(lam, beta, 1.33)
    gpu_ctx.set_geometry(sg.sinc_idx, sg.sinc_w, sg.window)
    raw = synthetic.generate_numpy(bscans, nx, apod, seed=nx + apod)
    raw[0, apod, ::3] = 65535
    raw = (raw.astype(np.int64) - (32768 if dtype == np.int16 else 0)).astype(dtype)
    if nx == 9:
        raw[:, :apod] = raw[:, apod:apod + 1]
        raw[:, -2:] = raw[:, apod:apod + 1]               # equal to the apodisation lines
    ref = O.magnitude_numpy(raw, O.spectral_geometry(lam, beta, 1.33), apod, np.float64)
    got = gpu_ctx.magnitude_exact(raw, apod).astype(np.float64)
    assert (np.abs(got - ref) <= 2.0 ** -24 * np.abs(ref) + 1e-12 * np.abs(ref).max(-1, keepdims=True)).all()
    if nx == 9:
        assert (got[:, -2:] == 0).all()


def _offset(torch, a, shift):
    """a on the device, its first element `shift` floats past a 16-byte boundary."""
    buf = torch.empty(a.size + shift, device="cuda")
    v = buf[shift:].reshape(a.shape)
    v.copy_(torch.from_numpy(a))
    return v


@pytest.mark.parametrize("n,cin,cout,h,w,pool,shift", [
    (1, 3, 32, 5, 640, 0, 0), (2, 9, 32, 7, 384, 0, 1), (1, 32, 128, 6, 1152, 1, 0), (1, 8, 32, 2, 256, 1, 3),
    (1, 17, 32, 64, 2, 0, 0), (3, 16, 32, 33, 128, 0, 2), (1, 7, 96, 1, 256, 0, 0), (30, 24, 64, 32, 8, 0, 0),
    (200, 3, 32, 10, 128, 1, 0)])
def test_conv_bands(gpu_ctx, n, cin, cout, h, w, pool, shift):
    """Bands at the ends of an image, column segments of wide rows, rows off
    16-byte boundaries, one row or two columns: against the float64 convolution
    of the FP16-rounded operands.  Tolerance: float32 accumulation of 9 cin
    products, 1e-5 of the largest value per square root of their number."""
    torch = pytest.importorskip("torch")
    from oracle import cnn as C
    from oct_recon_af_v1_gb300.learned import _p
    rng = np.random.default_rng(h * w + cin)
    x = rng.standard_normal((n, cin, h, w)).astype(np.float32)
    wt = (rng.standard_normal((cout, cin, 3, 3)) * 0.3).astype(np.float32)
    b = rng.standard_normal(cout).astype(np.float32)
    keep = [0, n // 2, n - 1]                                  # images compared
    r16 = lambda a: a.astype(np.float16).astype(np.float64)
    ref = C.conv3x3(r16(x[keep]), r16(wt), b.astype(np.float64))
    tol = 1e-5 * np.abs(ref).max() * np.sqrt(9 * cin)
    if pool:
        ref = np.maximum(ref, 0).reshape(3, cout, h // 2, 2, w // 2, 2).mean(axis=(3, 5))
    xd, wd, bd = _offset(torch, x, shift), torch.tensor(wt, device="cuda"), torch.tensor(b, device="cuda")
    y = torch.full((n,) + ref.shape[1:], float("nan"), device="cuda")
    torch.cuda.synchronize()
    f = gpu_ctx.lib.octgb_cnn_conv3x3_relu_pool_tc if pool else gpu_ctx.lib.octgb_cnn_conv3x3_tc
    gpu_ctx._check(f(gpu_ctx.h, _p(xd), _p(wd), _p(bd), _p(y), n, cin, cout, h, w))
    gpu_ctx.synchronize()
    assert torch.isfinite(y).all()
    np.testing.assert_allclose(y[keep].cpu().numpy(), ref, rtol=0, atol=tol)


@pytest.mark.parametrize("n,cin,cout,h,w,shift", [(1, 3, 32, 7, 640, 0), (2, 16, 40, 5, 701, 0), (1, 48, 128, 3, 130, 0),
                                                  (2, 1, 9, 1, 260, 1), (3, 33, 8, 31, 128, 2), (200, 8, 16, 5, 4, 0),
                                                  (1, 5, 1, 300, 1, 0), (90, 32, 32, 9, 64, 0)])
def test_weight_gradient_bands(gpu_ctx, n, cin, cout, h, w, shift):
    """The same for the weight and bias gradients: against the float64 sums of
    the BF16-rounded operands' products (dw) and of dy (db).  Tolerance: float32
    accumulation, 1e-4 of the sum of the terms' magnitudes."""
    torch = pytest.importorskip("torch")
    from oct_recon_af_v1_gb300.learned import _p
    rng = np.random.default_rng(h * w + cin)
    x = torch.tensor(rng.standard_normal((n, cin, h, w)), dtype=torch.float32)
    dy = torch.tensor(rng.standard_normal((n, cout, h, w)), dtype=torch.float32)
    xb, db16 = x.bfloat16().double(), dy.bfloat16().double()
    grad = lambda a, g: torch.nn.grad.conv2d_weight(a, (cout, cin, 3, 3), g, padding=1).numpy()
    ref, mag = grad(xb, db16), grad(xb.abs(), db16.abs())
    xd, dyd = _offset(torch, x.numpy(), shift), _offset(torch, dy.numpy(), shift)
    wd = torch.zeros((cout, cin, 3, 3), device="cuda")
    dw, db = torch.full_like(wd, float("nan")), torch.full((cout,), float("nan"), device="cuda")
    torch.cuda.synchronize()
    gpu_ctx._check(gpu_ctx.lib.octgb_cnn_conv3x3_bwd_tc(gpu_ctx.h, _p(xd), _p(wd), _p(dyd), None, _p(dw), _p(db), None,
                                                        n, cin, cout, h, w))
    gpu_ctx.synchronize()
    assert (np.abs(dw.cpu().numpy() - ref) <= 1e-4 * mag).all()
    assert (np.abs(db.cpu().double().numpy() - dy.double().sum((0, 2, 3)).numpy())
            <= 1e-4 * dy.double().abs().sum((0, 2, 3)).numpy()).all()


@pytest.mark.parametrize("n,cin,cout,h,w", [(304, 3, 8, 146, 3), (400, 9, 16, 141, 3), (152, 1, 1, 292, 3),
                                            (304, 4, 8, 93, 7), (304, 2, 9, 200, 1)])
def test_weight_gradient_of_narrow_images(gpu_ctx, n, cin, cout, h, w):
    """Images a few pixels wide, enough of them that a band holds as many rows
    as its staging takes: the comparison and tolerance of the test above."""
    test_weight_gradient_bands(gpu_ctx, n, cin, cout, h, w, 0)


@pytest.mark.parametrize("n,cin,cout,h,w,shift", [(1, 3, 32, 6, 640, 0), (2, 16, 40, 2, 264, 1), (3, 33, 9, 10, 128, 0),
                                                  (90, 5, 1, 8, 8, 0), (1, 48, 128, 4, 136, 0), (130, 3, 32, 14, 128, 2)])
def test_weight_gradient_through_pool(gpu_ctx, n, cin, cout, h, w, shift):
    """dy = y > 0 ? dp / 4 : 0 formed inside the kernel: the same comparison
    and tolerance as test_weight_gradient_bands (x alone off 16-byte boundaries)."""
    torch = pytest.importorskip("torch")
    from oct_recon_af_v1_gb300.learned import _p
    rng = np.random.default_rng(h * w + cin)
    x = torch.tensor(rng.standard_normal((n, cin, h, w)), dtype=torch.float32)
    y = torch.tensor(rng.standard_normal((n, cout, h, w)), dtype=torch.float32)
    y[:, :, ::3, ::5] = 0.0
    dp = torch.tensor(rng.standard_normal((n, cout, h // 2, w // 2)), dtype=torch.float32)
    dy = torch.where(y > 0, 0.25 * dp.repeat_interleave(2, 2).repeat_interleave(2, 3), 0.0)
    xb, dyb = x.bfloat16().double(), dy.bfloat16().double()
    grad = lambda a, g: torch.nn.grad.conv2d_weight(a, (cout, cin, 3, 3), g, padding=1).numpy()
    ref, mag = grad(xb, dyb), grad(xb.abs(), dyb.abs())
    xd, yd, dpd = _offset(torch, x.numpy(), shift), y.cuda(), dp.cuda()
    dw, db = torch.full((cout, cin, 3, 3), float("nan"), device="cuda"), torch.full((cout,), float("nan"), device="cuda")
    torch.cuda.synchronize()
    gpu_ctx._check(gpu_ctx.lib.octgb_cnn_conv3x3_pool_bwd_tc(gpu_ctx.h, _p(xd), _p(dw), _p(yd), _p(dpd), None, _p(dw),
                                                             _p(db), None, n, cin, cout, h, w))
    gpu_ctx.synchronize()
    assert (np.abs(dw.cpu().numpy() - ref) <= 1e-4 * mag).all()
    assert (np.abs(db.cpu().double().numpy() - dy.double().sum((0, 2, 3)).numpy())
            <= 1e-4 * dy.double().abs().sum((0, 2, 3)).numpy()).all()


@pytest.mark.parametrize("n,cin,cout,h,w,shift", [(3, 32, 32, 5, 128, 1), (2, 9, 96, 7, 256, 2), (160, 17, 32, 16, 16, 3),
                                                  (2, 24, 128, 4, 384, 1)])
def test_rows_off_boundaries_equal_aligned_rows(gpu_ctx, n, cin, cout, h, w, shift):
    """Forward, weight and data gradients read rows off 16-byte boundaries from
    memory: the bits of aligned rows (the same products in the same order), but
    for the bias gradient's order of sums (1e-5 of its terms' magnitudes)."""
    torch = pytest.importorskip("torch")
    from oct_recon_af_v1_gb300.learned import _p
    rng = np.random.default_rng(h * w + cin)
    x, dy = (rng.standard_normal((n, c, h, w)).astype(np.float32) for c in (cin, cout))
    wt = torch.tensor(rng.standard_normal((cout, cin, 3, 3)), dtype=torch.float32, device="cuda")
    L, c, out = gpu_ctx.lib, gpu_ctx, []
    for k in (0, shift):
        xd, dyd = _offset(torch, x, k), _offset(torch, dy, k)
        y, dx = torch.full_like(dyd, float("nan")), torch.full_like(xd, float("nan"))
        dw, db, scratch = torch.empty_like(wt), torch.empty(cout, device="cuda"), torch.empty_like(wt)
        torch.cuda.synchronize()
        c._check(L.octgb_cnn_conv3x3_tc(c.h, _p(xd), _p(wt), None, _p(y), n, cin, cout, h, w))
        c._check(L.octgb_cnn_conv3x3_bwd_tc(c.h, _p(xd), _p(wt), _p(dyd), _p(dx), _p(dw), _p(db), _p(scratch), n, cin,
                                            cout, h, w))
        c.synchronize()
        assert all(torch.isfinite(t).all() for t in (y, dx, dw, db))
        out.append((y.contiguous(), dx.contiguous(), dw, db))
    assert all(torch.equal(a, b) for a, b in zip(out[0][:3], out[1][:3]))
    bound = 1e-5 * torch.tensor(np.abs(dy).sum((0, 2, 3)), device="cuda")
    assert ((out[0][3] - out[1][3]).abs() <= bound).all()


@pytest.mark.parametrize("n,cin,cout,h,w", [(1, 3, 32, 2, 128), (2, 32, 64, 6, 384), (1, 9, 128, 4, 256)])
def test_conv_with_pool_beside_pre_activations(gpu_ctx, n, cin, cout, h, w):
    """The one kernel's two outputs equal the two kernels' exactly (the same
    sums in the same order)."""
    torch = pytest.importorskip("torch")
    from oct_recon_af_v1_gb300.learned import _p
    rng = np.random.default_rng(w + cin)
    x, wt, b = (torch.tensor(rng.standard_normal(s), dtype=torch.float32, device="cuda")
                for s in ((n, cin, h, w), (cout, cin, 3, 3), (cout,)))
    y, y2 = (torch.full((n, cout, h, w), float("nan"), device="cuda") for _ in range(2))
    p, p2 = (torch.full((n, cout, h // 2, w // 2), float("nan"), device="cuda") for _ in range(2))
    torch.cuda.synchronize()
    L, c = gpu_ctx.lib, gpu_ctx
    c._check(L.octgb_cnn_conv3x3_tc(c.h, _p(x), _p(wt), _p(b), _p(y), n, cin, cout, h, w))
    c._check(L.octgb_cnn_relu_pool(c.h, _p(y), _p(p), n * cout, h, w))
    c._check(L.octgb_cnn_conv3x3_keep_relu_pool_tc(c.h, _p(x), _p(wt), _p(b), _p(y2), _p(p2), n, cin, cout, h, w))
    c.synchronize()
    assert torch.isfinite(y).all() and torch.equal(y, y2) and torch.equal(p, p2)


@pytest.mark.parametrize("n,cin,cout,h,w", [(2, 32, 32, 128, 128), (3, 32, 32, 64, 64), (130, 32, 9, 32, 32),
                                            (1, 32, 17, 2, 128), (2, 32, 3, 16, 8)])
def test_data_gradient_through_pool(gpu_ctx, n, cin, cout, h, w):
    """dx equals, bit for bit, that of the two kernels that put dy in memory
    (the same products in the same order)."""
    torch = pytest.importorskip("torch")
    from oct_recon_af_v1_gb300.learned import _p
    rng = np.random.default_rng(w + cin)
    x, wt, y, dp = (torch.tensor(rng.standard_normal(s), dtype=torch.float32, device="cuda")
                    for s in ((n, cin, h, w), (cout, cin, 3, 3), (n, cout, h, w), (n, cout, h // 2, w // 2)))
    dy, (dx, dx2) = torch.empty_like(y), (torch.full((n, cin, h, w), float("nan"), device="cuda") for _ in range(2))
    dw, db, scratch = torch.empty_like(wt), torch.empty(cout, device="cuda"), torch.empty(wt.numel(), device="cuda")
    torch.cuda.synchronize()
    L, c = gpu_ctx.lib, gpu_ctx
    c._check(L.octgb_cnn_relu_pool_bwd(c.h, _p(dp), _p(y), _p(dy), n * cout, h, w))
    c._check(L.octgb_cnn_conv3x3_bwd_tc(c.h, _p(x), _p(wt), _p(dy), _p(dx), _p(dw), _p(db), _p(scratch), n, cin, cout,
                                        h, w))
    c._check(L.octgb_cnn_conv3x3_pool_bwd_tc(c.h, _p(x), _p(wt), _p(y), _p(dp), _p(dx2), _p(dw), _p(db), _p(scratch), n,
                                             cin, cout, h, w))
    c.synchronize()
    assert torch.isfinite(dx).all() and torch.equal(dx, dx2)


def test_adam_list(gpu_ctx):
    """Tensors of uneven sizes, more than one launch takes, equal those stepped one at a time."""
    torch = pytest.importorskip("torch")
    import ctypes
    from oct_recon_af_v1_gb300.learned import _p
    sizes = [1, 255, 257, 400_000] + [3] * 13
    rng = np.random.default_rng(3)
    one = [[torch.tensor(np.abs(rng.standard_normal(n)), dtype=torch.float32, device="cuda") for n in sizes]
           for _ in range(4)]
    many = [[t.clone() for t in ts] for ts in one]
    torch.cuda.synchronize()
    for p, g, m, v in zip(*one):
        gpu_ctx._check(gpu_ctx.lib.octgb_cnn_adam(gpu_ctx.h, _p(p), _p(g), _p(m), _p(v), p.numel(), 1e-3, 0.9, 0.999,
                                                  1e-8, 3))
    n = len(sizes)
    lists = [(ctypes.c_void_p * n)(*(t.data_ptr() for t in ts)) for ts in many]
    gpu_ctx._check(gpu_ctx.lib.octgb_cnn_adam_list(gpu_ctx.h, n, *lists, (ctypes.c_int64 * n)(*sizes), 1e-3, 0.9, 0.999,
                                                   1e-8, 3))
    gpu_ctx.synchronize()
    assert all(torch.equal(a, b) for x, y in zip(one, many) for a, b in zip(x, y))


@pytest.mark.parametrize("n", [24 * 12 * 152 - 1, 24 * 12 * 152, 24 * 12 * 152 + 12 * 152 + 5])
def test_transform_with_lines_in_shared_memory(gpu_ctx, n):
    """From 24 A-scans a warp on the transform takes its lines from shared
    memory: every A-scan equals, bit for bit, its magnitudes in a call of few
    A-scans (the same operations), on either side of the rule."""
    torch = pytest.importorskip("torch")
    from oct_recon_af_v1_gb300 import geometry as G
    from oct_recon_af_v1_gb300 import synthetic
    sg = G.build_spectral_geometry(synthetic.lambda_nm(), 0.0, 1.33)
    gpu_ctx.set_geometry(sg.sinc_idx, sg.sinc_w, sg.window)
    raw = torch.randint(0, 65536, (1, n + 1, 2048), generator=torch.Generator().manual_seed(1)).to(torch.uint16).cuda()
    mag = torch.full((1, n, 1024), float("nan"), device="cuda")
    torch.cuda.synchronize()
    gpu_ctx.magnitude(raw, 1, mag, raw_dtype=0)
    small = torch.empty((1, 500, 1024), device="cuda")
    for lo in (0, n // 2, n - 500):
        part = torch.cat([raw[:, :1], raw[:, 1 + lo:501 + lo]], 1).contiguous()
        torch.cuda.synchronize()
        gpu_ctx.magnitude(part, 1, small, raw_dtype=0)
        gpu_ctx.synchronize()
        assert torch.equal(mag[:, lo:lo + 500], small)
    assert torch.isfinite(mag).all()


def test_captured_gradients_after_larger_ones():
    """A graph over a weight gradient replays after a call that needs more room
    for its partial sums (the float32 form's bias gradient likewise)."""
    torch = pytest.importorskip("torch")
    from oct_recon_af_v1_gb300 import _lib
    from oct_recon_af_v1_gb300.learned import _p
    ctx = _lib.Context(0)
    try:
        stream = torch.cuda.Stream()
        ctx.set_stream(stream.cuda_stream)
        g = torch.Generator(device="cuda").manual_seed(4)

        def buffers(n, h):
            x, dy, w = (torch.randn(s, device="cuda", generator=g) for s in ((n, 8, h, h), (n, 32, h, h), (32, 8, 3, 3)))
            return x, w, dy, torch.empty_like(w), torch.empty(32, device="cuda")

        def run(f, b):
            x, w, dy, dw, db = b
            ctx._check(f(ctx.h, _p(x), _p(w), _p(dy), None, _p(dw), _p(db), None, x.shape[0], 8, 32, x.shape[2], x.shape[3]))
        small, large = buffers(1, 16), buffers(300, 32)
        torch.cuda.synchronize()
        for f in (ctx.lib.octgb_cnn_conv3x3_bwd_tc, ctx.lib.octgb_cnn_conv3x3_bwd):
            run(f, small)
            ctx.synchronize()
            ref = [t.clone() for t in small[3:]]
            torch.cuda.synchronize()
            ctx.graph_begin()
            run(f, small)
            gid = ctx.graph_end()
            run(f, large)
            ctx.synchronize()
            fill = torch.empty(1 << 24, device="cuda").fill_(3.0)       # what was freed is in use again
            for t in small[3:]:
                t.zero_()
            torch.cuda.synchronize()
            ctx.graph_launch(gid)
            ctx.synchronize()
            assert (fill == 3.0).all()
            for t, r in zip(small[3:], ref):
                assert (t - r).abs().max() <= 1e-5 * r.abs().max()
    finally:
        ctx.close()
