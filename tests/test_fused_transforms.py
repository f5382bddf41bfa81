"""The fused transforms (k_fft.cu) against the plain path's separate cuFFT
transforms and, for the tile-local 2LPT and Laplacian, the oracle.

Tolerance: both sides are single-precision transforms of the same delta_k.
One transform's rounding is about 3e-7 rms of the field (log2 n^3 butterfly
roundings of 6e-8); psi2 passes through three in a row and a product, and
1/k^2 weights the few largest modes, so 1e-5 rms and 1e-4 of the field's
maximum bound the difference of the two sides."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# every factor of the register transforms, the smallest and
# largest size, sizes with more and with fewer threads than 16 per column
SIZES = [64, 80, 96, 112, 128, 144, 160, 176, 192, 208, 224, 240, 256, 272, 288, 304, 320, 336, 352, 368, 384, 448, 512,
         74, 142]   # not multiples of 16: cuFFT with phi_33 from the trace


def _close(a, b, name):
    b = b.astype(np.float64)
    d = a - b
    rms = np.sqrt(np.mean(b * b))
    assert np.sqrt(np.mean(d * d)) <= 1e-5 * rms, (name, np.sqrt(np.mean(d * d)) / rms)
    assert np.abs(d).max() <= 1e-4 * np.abs(b).max(), name


@pytest.mark.parametrize("n", SIZES)
def test_fused_psi2_and_laplacian_match_plain(ctx, eh_pk, n):
    import ctypes

    import peakpatch_b200 as pp
    ctx.set_pk_table(*eh_pk)
    cfg = pp.PipelineConfig(n=n, boxsize=2.0 * n, nbuff=4, ilpt=2, ioutshear=1)
    out = []
    for plain in (False, True):
        p = ctx._params(cfg, 11, plain)
        psi2 = np.empty((3, n, n, n), np.float32)
        lap = np.empty((n, n, n), np.float32)
        ctx._check(ctx.L.ppb_generate_fields(ctx.h, ctypes.byref(p), None, None, psi2.ctypes.data, lap.ctypes.data))
        out.append((psi2, lap))
    for c in range(3):
        _close(out[0][0][c], out[1][0][c], f"psi2[{c}]")
    _close(out[0][1], out[1][1], "lapd")


@pytest.mark.parametrize("n", [64, 112, 176])
def test_tile_local_2lpt_and_laplacian_match_oracle(ctx, ora, n):
    rng = np.random.default_rng(n)
    k = np.fft.fftfreq(n)
    kr = np.fft.rfftfreq(n)
    kk = np.sqrt(k[:, None, None] ** 2 + k[None, :, None] ** 2 + kr[None, None, :] ** 2)
    d = np.fft.irfftn(np.fft.rfftn(rng.standard_normal((n, n, n))) * np.exp(-30 * kk ** 2), s=(n, n, n), axes=(0, 1, 2)) + 0.01
    d = d.astype(np.float32)
    ref2, refl = ora.tile_2lpt_laplacian(d, n, 2.0 * n)
    got2 = ctx.compute_2lpt_gpu(d, n, 2.0 * n)
    for c in range(3):
        _close(got2[c], np.asarray(ref2[c]), f"psi2[{c}]")
    _close(ctx.compute_laplacian_gpu(d, n, 2.0 * n), np.asarray(refl), "lapd")


@pytest.mark.parametrize("n,cell,ws", [(64, 1.0, 1), (80, 2.0, 0), (112, 2.0, 3), (144, 1.3, 1), (176, 2.0, 1), (142, 2.0, 1)])
def test_twin_at_peaks_matches_oracle(ctx, ora, n, cell, ws):
    """d2Rf from the pruned twin (large radii) and the whole one (small radii)."""
    rng = np.random.default_rng(7 * n)
    k = 2 * np.pi * np.fft.fftfreq(n, cell)
    kr = 2 * np.pi * np.fft.rfftfreq(n, cell)
    kk = np.sqrt(k[:, None, None] ** 2 + k[None, :, None] ** 2 + kr[None, None, :] ** 2)
    kk[0, 0, 0] = 1.0
    dk = np.fft.rfftn(rng.standard_normal((n, n, n))) * kk ** -1.0
    dk[0, 0, 0] = 0.0
    d = np.fft.irfftn(dk, s=(n, n, n), axes=(0, 1, 2))
    d = (d * (2.5 / d.std())).astype(np.float32)
    radii = [14.0, 9.0, 6.0, 3.0, 1.6]
    mask = np.zeros((n, n, n), np.int8)
    peaks, rf, fc, d2, _ = ctx.peak_find_tile(d, radii, [0.8] * 5, mask, 0.0, 0.0, 0.0, cell, 5, ws, 1)
    dk64 = np.fft.rfftn(d.astype(np.float64))
    kk[0, 0, 0] = 0.0
    for R in radii:
        w = np.exp(-(kk * R) ** 2 / 8) * kk ** 2
        w[0, 0, 0] = 1.0
        t = np.fft.irfftn(dk64 * w, s=(n, n, n), axes=(0, 1, 2))
        m = rf == R
        if not m.any():   # W_3 alone passes no large-radius peak above 0.8
            assert ws == 3
            continue
        ref = t[peaks["k"][m] - 1, peaks["j"][m] - 1, peaks["i"][m] - 1]
        assert np.abs(d2[m] - ref).max() <= 4e-6 * np.abs(t).max(), R
