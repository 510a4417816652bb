"""The transforms' butterflies are the plain radix-2 decimation in time, operation for operation: the same
bits from a straightforward evaluation of it in FP32 (fused multiply-adds through exact 64-bit products)."""

import numpy as np
import pytest
import torch

from realflare_gb300._abi import check, lib
from realflare_gb300.device import stream_handle

pytestmark = pytest.mark.gpu


def fma(a, b, c):
    # the product is exact in 64 bits; one rounding of the sum to 64 bits and one to 32
    return (a.astype(np.float64) * b.astype(np.float64) + c.astype(np.float64)).astype(np.float32)


def rows(x, table):
    """Radix-2 decimation in time along the last axis; table[k] = exp(-+2 pi i k / n)."""
    n = x.shape[-1]
    log_n = n.bit_length() - 1
    rev = [int(format(i, f'0{log_n}b')[::-1], 2) for i in range(n)]
    re, im = x.real[..., rev].astype(np.float32), x.imag[..., rev].astype(np.float32)
    for s in range(1, log_n + 1):
        half = 1 << (s - 1)
        w = table[:n // 2:n >> s]
        re, im = re.reshape(*x.shape[:-1], -1, 2 * half), im.reshape(*x.shape[:-1], -1, 2 * half)
        ar, ai, br, bi = re[..., :half], im[..., :half], re[..., half:], im[..., half:]
        wr, wi = np.broadcast_to(w.real, br.shape), np.broadcast_to(w.imag, br.shape)
        vr, vi = fma(br, wr, -(bi * wi)), fma(bi, wr, br * wi)
        re, im = np.concatenate([ar + vr, ar - vr], -1), np.concatenate([ai + vi, ai - vi], -1)
        re, im = re.reshape(x.shape), im.reshape(x.shape)
    return re + 1j * im


@pytest.mark.parametrize('width, height, direction', [(8, 8, -1), (16, 32, 1), (64, 8, -1), (128, 256, -1), (512, 16, 1)])
def test_radix_2(width, height, direction):
    g = torch.Generator(device='cuda').manual_seed(width + height)
    x = torch.randn((height, width, 2), generator=g, device='cuda')
    data, scratch = x.clone(), torch.empty_like(x)
    check(lib().rf_fft2(data.data_ptr(), scratch.data_ptr(), 1, width, height, direction, 1.0, stream_handle()), 'rf_fft2')

    def table(n):
        # a row transform of a unit impulse at 1 gives the kernel's own twiddles
        e = torch.zeros((8, n, 2), device='cuda')
        e[0, 1, 0] = 1.0
        s = torch.empty_like(e)
        check(lib().rf_fft2(e.data_ptr(), s.data_ptr(), 1, n, 8, direction, 1.0, stream_handle()), 'rf_fft2')
        return torch.view_as_complex(e[0]).cpu().numpy()

    host = torch.view_as_complex(x).cpu().numpy()
    want = rows(np.ascontiguousarray(rows(host, table(width)).T), table(height)).T
    got = torch.view_as_complex(data).cpu().numpy()
    # (the sum's rounding to 64 bits can move a tie: allow one unit in the last place in a few elements)
    differ = (got.real != want.real) | (got.imag != want.imag)
    assert differ.mean() < 1e-3
    assert np.abs(got - want).max() <= 2e-6 * np.abs(want).max()
