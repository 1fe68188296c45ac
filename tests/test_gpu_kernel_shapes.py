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
