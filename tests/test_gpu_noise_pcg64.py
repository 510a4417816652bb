"""The device's PCG64 noise against numpy's generator, bit for bit."""

import numpy as np
import pytest
import torch

from realflare_gb300._abi import check, lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('seed', [0, 1, 20240607])
@pytest.mark.parametrize('count', [1, 2, 7, 8, 9, 2047, 2048, 2055, 333 * 217, 1 << 20])
def test_equal_to_numpy(count, seed):
    g = np.random.PCG64(seed).state['state']
    word = (1 << 64) - 1
    out = torch.full((count + 8,), -1.0, device='cuda')
    check(lib().rf_noise_pcg64(g['state'] >> 64, g['state'] & word, g['inc'] >> 64, g['inc'] & word, out.data_ptr(),
                               count, torch.cuda.current_stream().cuda_stream), 'rf_noise_pcg64')
    want = np.random.Generator(np.random.PCG64(seed)).random(count, dtype=np.float32)
    got = out.cpu().numpy()
    assert np.array_equal(got[:count], want)
    assert (got[count:] == -1.0).all()
