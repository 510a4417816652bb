"""The colour matrix of every pixel is evaluated as in double: each output lies within half a float's last place and the
double form's own rounding (three products, two sums: 2^-51 of the terms) of the exact value, also where the terms
cancel to their last bits, at extreme magnitudes, and for infinities. One starburst sample with unit weights hands
(X, Y, Z) to the matrix unchanged."""
from __future__ import annotations

import ctypes
import math
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip('torch')

from realflare_gb300._abi import StarburstArgs, check, lib  # noqa: E402
from realflare_gb300.constants import light_spectrum  # noqa: E402

MATRIX = ((1.6410233797, -0.3248032942, -0.2364246952), (-0.6636628587, 1.6153315917, 0.0167563477),
          (0.0117218943, -0.0082844420, 0.9883948585))


def ap1(values):
    """Images of one starburst per (X, Y, Z): the light's first texel enters with weight 1 / 4, the intensity is 4."""
    a = StarburstArgs()
    a.width = a.height = 2
    a.spectrum_width = a.spectrum_height = 8
    a.spectrum_count = a.samples = 1
    a.vignetting[0] = a.vignetting[1] = float('nan')
    a.rotation_weight, a.intensity = 1.0, 4.0
    a.scale[0] = a.scale[1] = 8.0
    a.lambda_first, a.lambda_step = 560.0, 1.0
    spectrum = torch.ones((8, 8), device='cuda')
    lights = torch.zeros((len(values), *light_spectrum().shape), device='cuda')
    lights.view(len(values), -1, 4)[:, 0, :3] = torch.from_numpy(np.asarray(values, np.float32)).cuda()
    out = torch.empty((len(values), 2, 2, 4), device='cuda')
    stream = int(torch.cuda.current_stream().cuda_stream)
    for light, image in zip(lights, out):
        check(lib().rf_starburst(spectrum.data_ptr(), light.data_ptr(), ctypes.byref(a), image.data_ptr(), stream),
              'rf_starburst')
    torch.cuda.synchronize()
    assert (out == out[:, :1, :1]).all() or not torch.isfinite(out).all()
    return out[:, 0, 0].cpu().numpy()


def cancelling(row, n, rng):
    """(X, Y, Z) whose output `row` cancels to the last bits of its terms."""
    c = MATRIX[row]
    k = int(np.argmax(np.abs(c)))
    v = rng.uniform(0.25, 4.0, (n, 3)).astype(np.float32)
    others = sum(c[i] * v[:, i].astype(np.float64) for i in range(3) if i != k)
    v[:, k] = (-others / c[k]).astype(np.float32)
    return v


def test_as_accurate_as_double():
    rng = np.random.default_rng(12)
    values = [cancelling(row, 60, rng) for row in range(3)]
    values.append(rng.uniform(0, 1, (100, 3)).astype(np.float32))
    values.append((2.0 ** rng.uniform(-100, 100, (100, 3))).astype(np.float32))
    values = np.concatenate([*values, np.zeros((1, 3), np.float32)])
    got = ap1(values)
    for v, g in zip(values, got):
        for c, out in zip(MATRIX, g):
            terms = [Fraction(float(x)) * Fraction(k) for x, k in zip(v, c)]
            exact = sum(terms)
            last_place = Fraction(float(np.spacing(np.float32(max(abs(float(exact)), 2.0 ** -126)))))
            assert abs(Fraction(float(out)) - exact) <= last_place / 2 + sum(map(abs, terms)) / 2 ** 51


def test_infinities():
    inf = math.inf
    got = ap1([(inf, 1.0, 1.0), (inf, inf, 1.0), (3e38, 3e38, 0.0)])
    assert got[0][0] == inf and got[0][1] == -inf and got[0][2] == inf
    assert math.isnan(got[1][0])
    # the second output's sum is a float although one of its terms is not
    assert got[2][0] == inf
    assert float(got[2][1]) == pytest.approx(3e38 * (MATRIX[1][0] + MATRIX[1][1]), rel=1e-6)
