"""Spectra past the range of the starburst's 32-bit lookups: a side of 2^22 texels or more, a plane of 2^31 or
more. The spectrum is s + t in normalised coordinates, which bilinear lookups reproduce at any size, so the image
equals that of a 64 x 64 spectrum, also with jitter and rotation (the noise depends on the pixel alone); the bound
is that of the other comparisons (FP32 rounding of positions and sums)."""
from __future__ import annotations

import ctypes

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip('torch')

from realflare_gb300._abi import StarburstArgs, check, lib  # noqa: E402
from realflare_gb300.constants import light_spectrum  # noqa: E402


def image(width, height, blur, rotation):
    s = ((torch.arange(width, device='cuda', dtype=torch.float64) + 0.5) / width).float()
    t = ((torch.arange(height, device='cuda', dtype=torch.float64) + 0.5) / height).float()
    spectrum = s[None, :] + t[:, None]
    a = StarburstArgs()
    a.width, a.height, a.spectrum_width, a.spectrum_height, a.spectrum_count = 41, 33, width, height, 1
    a.samples, a.blur, a.rotation, a.rotation_weight = 5, blur, rotation, 1.5
    a.vignetting[0] = a.vignetting[1] = float('nan')
    a.intensity = 1.0
    a.scale[0] = a.scale[1] = 2.5  # every lookup inside the spectrum
    a.lambda_first, a.lambda_step = 560.0, 1.0
    out = torch.empty((33, 41, 4), device='cuda')
    light = torch.from_numpy(light_spectrum()).cuda()
    check(lib().rf_starburst(spectrum.data_ptr(), light.data_ptr(), ctypes.byref(a), out.data_ptr(),
                             int(torch.cuda.current_stream().cuda_stream)), 'rf_starburst')
    torch.cuda.synchronize()
    return out.double()


@pytest.mark.parametrize('width,height', [((1 << 22) - 1, 64), (1 << 22, 64), (5_000_000, 64), (64, 5_000_000),
                                          (46341, 46341)])
@pytest.mark.parametrize('blur,rotation', [(0.0, 0.0), (0.05, 0.0), (0.05, 0.2)])
def test_wide_spectrum(width, height, blur, rotation):
    if torch.cuda.mem_get_info()[0] < 16 * width * height:
        pytest.skip('not enough device memory')
    got, want = image(width, height, blur, rotation), image(64, 64, blur, rotation)
    assert want.abs().sum() > 0
    assert (got - want).norm() <= 1e-5 * want.norm()
