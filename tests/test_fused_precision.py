"""The tile-local 2LPT by the fused transforms is no further from 64 bits than
separate single-precision cuFFT transforms whose factors are formed in FP64
and rounded with the product (torch), on fields of the resident P(k).  Its
source cancels at low k, so roundings that are the same in every transform
show there; the mean over three fields is compared, since a single field's
error varies by a few percent."""
import ctypes
import math

import pytest

pytestmark = pytest.mark.gpu

import peakpatch_b200 as pp

CELL = 2.0


def _separate(d, real):
    """psi2 of MultiResolution.jl:804-831 with transforms in the precision of `real`, factors in FP64."""
    import torch
    n = d.shape[0]
    cplx = torch.complex64 if real == torch.float32 else torch.complex128
    f = torch.fft.fftfreq(n, 1.0 / n, device="cuda", dtype=torch.float64) * (2 * math.pi / (n * CELL))
    r = torch.arange(n // 2 + 1, device="cuda", dtype=torch.float64) * (2 * math.pi / (n * CELL))
    ax = (r[None, None, :], f[None, :, None], f[:, None, None])
    k2 = ax[0] ** 2 + ax[1] ** 2 + ax[2] ** 2
    inv = 1.0 / k2.clamp(min=1e-300)
    inv[0, 0, 0] = 0.0
    inv[:, :, n // 2] = 0.0
    inv[:, n // 2, :] = 0.0
    inv[n // 2, :, :] = 0.0

    def back(spec, factor):
        return torch.fft.irfftn((spec.to(torch.complex128) * factor).to(cplx), s=(n, n, n))

    d = d.to(real)
    dk = torch.fft.rfftn(d)
    src = 0.5 * d * d
    for a in range(3):
        for b in range(a, 3):
            phi = back(dk, -ax[a] * ax[b] * inv)
            src = src - phi * phi * (0.5 if a == b else 1.0)
    sk = torch.fft.rfftn(src)
    return torch.stack([back(sk, -1j * q * inv) for q in ax])


@pytest.mark.parametrize("n", [64, 80, 96, 112, 144, 176, 208])
def test_tile_local_2lpt_error(ctx, eh_pk, n):
    import torch
    ctx.set_pk_table(*eh_pk)
    cfg = pp.PipelineConfig(n=n, boxsize=CELL * n, nbuff=4, ilpt=1, ioutshear=0)
    ours = theirs = 0.0
    for seed in (1, 2, 3):
        p = ctx._params(cfg, seed, False)
        d = torch.empty((n, n, n), device="cuda")
        psi2 = torch.empty((3, n, n, n), device="cuda")
        torch.cuda.synchronize()
        ctx._check(ctx.L.ppb_generate_fields(ctx.h, ctypes.byref(p), d.data_ptr(), None, None, None))
        ctx._check(ctx.L.ppb_compute_2lpt(ctx.h, d.data_ptr(), n, ctypes.c_double(CELL * n), psi2.data_ptr()))
        exact = _separate(d, torch.float64)
        ours += (psi2.double() - exact).square().mean().sqrt().item() / exact.square().mean().sqrt().item()
        theirs += (_separate(d, torch.float32).double() - exact).square().mean().sqrt().item() / \
            exact.square().mean().sqrt().item()
    print(n, ours / 3, theirs / 3)
    assert ours <= theirs, (n, ours / 3, theirs / 3)
