"""The starburst compositor at the sizes where its variants and lookups meet: images on both sides of
the size from which a thread takes two pixels (200,000 pixels), ragged against its 16-pixel blocks,
spectra down to one texel and one row, positions far outside the spectrum, more samples than one
table chunk (256). Deterministic settings (no jitter, no rotation) against the oracle; the bound is
that of the other such comparison (FP32 rounding of positions and sums)."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip('torch')

from helpers import rel_l2  # noqa: E402

from realflare_gb300._abi import StarburstArgs, check, lib  # noqa: E402
from realflare_gb300.constants import light_spectrum  # noqa: E402


@pytest.mark.parametrize('size,spectrum,samples,scale', [
    ((17, 33), (1, 1), 5, 1.0), ((33, 16), (1, 9), 257, 1.0), ((50, 47), (31, 1), 3, 0.25),
    ((447, 447), (24, 33), 9, 1.0), ((449, 450), (24, 33), 9, 1.0), ((801, 251), (64, 48), 9, 0.01),
])
def test_starburst_sizes_match_oracle(size, spectrum, samples, scale):
    from oracle.oracle import Oracle

    (w, h), (sw, sh) = size, spectrum
    spec = np.random.default_rng(3).uniform(0.5, 1.5, (sh, sw)).astype(np.float32)
    a = StarburstArgs()
    a.width, a.height, a.spectrum_width, a.spectrum_height, a.spectrum_count = w, h, sw, sh, 1
    a.samples, a.blur, a.rotation, a.rotation_weight = samples, 0.0, 0.0, 1.0
    a.vignetting[0] = a.vignetting[1] = float('nan')
    a.intensity = 1.0
    a.offset[0], a.offset[1] = 0.1, -0.05
    a.scale[0], a.scale[1] = scale, scale
    a.lambda_first, a.lambda_step = 560.0, 1.0
    want = Oracle('f32').starburst(spec, light_spectrum(), a)
    img = torch.empty((h, w, 4), device='cuda')
    spec_d, light_d = torch.from_numpy(spec).cuda(), torch.from_numpy(light_spectrum()).cuda()
    check(lib().rf_starburst(spec_d.data_ptr(), light_d.data_ptr(), ctypes.byref(a), img.data_ptr(),
                             int(torch.cuda.current_stream().cuda_stream)), 'rf_starburst')
    torch.cuda.synchronize()
    got = img.cpu().numpy()
    assert np.isfinite(got).all() and np.abs(want[..., :3]).sum() > 0
    assert rel_l2(got, want) < 1e-5
