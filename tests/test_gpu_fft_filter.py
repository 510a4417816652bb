"""Chirp-z rows on both sides of the rule that gives the filter threads of its own: rows of the shortest and longest
lengths with them (a warp to 512 threads), in as many blocks as the SMs hold at once and in more. Against numpy in FP64;
the bound is that of the other chirp-z lengths."""
from __future__ import annotations

import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip('torch')

from helpers import rel_l2  # noqa: E402

from realflare_gb300._abi import check, lib  # noqa: E402


# (width, height, batch): lengths 65 to 127 take 32 threads a row, 1025 to 2047 take 512, above 2048 all 1024
@pytest.mark.parametrize('width,height,batch', [(65, 3, 1), (127, 67, 1), (129, 5, 3), (100, 100, 40), (513, 9, 1),
                                                (300, 77, 1), (300, 77, 30), (1025, 3, 1), (2047, 150, 1),
                                                (2047, 160, 2), (2049, 6, 1)])
@pytest.mark.parametrize('direction', [-1, 1])
def test_chirp_z(width, height, batch, direction):
    rng = np.random.default_rng(width + batch)
    shape = (batch, height, width)
    x = (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(np.complex64)
    data = torch.from_numpy(x.view(np.float32).copy()).cuda()
    scratch = torch.empty_like(data)
    check(lib().rf_fft2(data.data_ptr(), scratch.data_ptr(), batch, width, height, direction,
                        1.0 / math.sqrt(width * height), int(torch.cuda.current_stream().cuda_stream)), 'rf_fft2')
    torch.cuda.synchronize()
    got = data.cpu().numpy().view(np.complex64)
    want = (np.fft.fftn if direction < 0 else np.fft.ifftn)(x.astype(np.complex128), axes=(1, 2), norm='ortho')
    assert rel_l2(got.view(np.float32), want.astype(np.complex64).view(np.float32)) < 1e-5
