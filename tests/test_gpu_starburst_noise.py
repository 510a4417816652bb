"""The starburst's kernels with jitter and with rotation. A radius or an angle of 1e-30 moves no position, so each noisy
kernel then gives the image of the one without (within a rounding or two of each pixel: 1e-6). With a radius and an
angle that count, the hash amplifies the sine's rounding, so single samples differ from the oracle's and 8 x 8
boxes agree, within the bound of the other such comparison."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip('torch')

from helpers import rel_l2  # noqa: E402
from test_gpu_diffraction import aperture_image, starburst_args, stream  # noqa: E402

from realflare_gb300._abi import check, lib  # noqa: E402
from realflare_gb300.constants import light_spectrum  # noqa: E402


def image(a, spectrum):
    out = torch.empty((a.height, a.width, 4), device='cuda')
    spec, light = torch.from_numpy(spectrum).cuda(), torch.from_numpy(light_spectrum()).cuda()
    check(lib().rf_starburst(spec.data_ptr(), light.data_ptr(), ctypes.byref(a), out.data_ptr(), stream()), 'starburst')
    torch.cuda.synchronize()
    return out.cpu().numpy()


# one and two pixels a thread without noise; one table chunk and more; several spectra
@pytest.mark.parametrize('size,samples,spectra', [((61, 47), 7, 1), ((61, 47), 300, 3), ((640, 401), 9, 1)])
@pytest.mark.parametrize('blur,rotation', [(1e-30, 0.0), (0.0, 1e-30), (1e-30, 1e-30)])
def test_noise_of_no_effect(size, samples, spectra, blur, rotation):
    spectrum = np.random.default_rng(3).uniform(0.5, 1.5, (spectra, 37, 24)).astype(np.float32)

    def args(blur, rotation):
        a = starburst_args(*size, 24, 37, samples=samples, blur=blur, rotation=rotation, weight=1.5)
        a.spectrum_count, a.lambda_first, a.lambda_step = spectra, 390.0, 150.0
        return a

    want = image(args(0.0, 0.0), spectrum)
    assert np.abs(want).sum() > 0
    assert rel_l2(image(args(blur, rotation), spectrum), want) < 1e-6


@pytest.mark.parametrize('blur,rotation,weight', [(0.02, 0.0, 1.0), (0.0, 0.2, 1.0), (0.0, 0.2, 1.5), (0.02, 0.2, 2.0)])
def test_noise_matches_oracle(blur, rotation, weight):
    from oracle.oracle import Oracle, fft_power_spectrum

    oracle = Oracle('f32')
    spectrum = fft_power_spectrum(aperture_image(oracle, 64), 560e-6, 1000.0).astype(np.float32)
    a = starburst_args(96, 64, 64, 64, samples=256, blur=blur, rotation=rotation, weight=weight)
    want, got = oracle.starburst(spectrum, light_spectrum(), a), image(a, spectrum)

    def boxes(x):
        return x[..., :3].reshape(8, 8, 12, 8, 3).mean(axis=(1, 3))

    assert rel_l2(boxes(got), boxes(want)) < 3e-2
    assert abs(got[..., :3].sum() / want[..., :3].sum() - 1) < 1e-2
