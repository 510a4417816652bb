"""Row lengths at the edges of the FFT's forms: the shortest direct transform (8), every remainder of
the radix-8 steps up to the longest row (4096), several rows per block with a ragged last block,
and the lengths below 8 and odd ones that take the chirp-z form. Against numpy in FP64; the bounds
are those of the other lengths (a few roundings per step; the chirp-z form goes through three
transforms)."""
from __future__ import annotations

import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip('torch')

from helpers import rel_l2  # noqa: E402

from realflare_gb300._abi import check, lib  # noqa: E402


@pytest.mark.parametrize('shape', [(2, 3), (4, 2), (8, 8), (1031, 8), (9, 16), (33, 32), (130, 64), (1024, 515),
                                   (2048, 257), (4096, 5), (6, 2048)])
@pytest.mark.parametrize('direction', [-1, 1])
def test_fft_lengths_match_numpy(shape, direction):
    h, w = shape
    x = np.random.default_rng(2).standard_normal((2, h, w, 2)).astype(np.float32)
    data = torch.from_numpy(x.copy()).cuda()
    scratch = torch.empty_like(data)
    check(lib().rf_fft2(data.data_ptr(), scratch.data_ptr(), 2, w, h, direction, 1.0 / math.sqrt(h * w),
                        int(torch.cuda.current_stream().cuda_stream)), 'rf_fft2')
    torch.cuda.synchronize()
    z = x[..., 0].astype(np.complex128) + 1j * x[..., 1]
    want = (np.fft.fftn if direction < 0 else np.fft.ifftn)(z, axes=(1, 2), norm='ortho')
    got = data.cpu().numpy()
    direct = all(n >= 8 and n & (n - 1) == 0 for n in shape)
    assert rel_l2(got, np.stack([want.real, want.imag], -1)) < (2e-6 if direct else 1e-5)
