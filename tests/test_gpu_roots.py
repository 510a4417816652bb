"""The short square roots and reciprocals of the traces (rf_common.cuh, rf_trace_core.cuh, rf_trace_accurate.cu) against
CUDA's correctly rounded operations: in FP32 for every operand of two binades and samples of the range, in double
for random operands, squares and their neighbours, and mantissas near all zeros and all ones. The kernels under test
are compiled here, with the units' own flags."""
from __future__ import annotations

import ctypes
import subprocess

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip('torch')

SOURCE = r'''
#include "rf_api.cu"
#include "rf_trace_accurate.cu"
namespace rf {
__global__ void k_roots_f32(unsigned long long* wrong) {
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    auto compare = [&](float x, int k) {
        if (__float_as_uint(sqrt_rn(x)) != __float_as_uint(__fsqrt_rn(x))) atomicAdd(wrong + k, 1ull);
        if (fabsf(x) <= 0x1p100f && __float_as_uint(rcp_rn(x)) != __float_as_uint(__frcp_rn(x))) atomicAdd(wrong + 2 + k, 1ull);
    };
    compare(__uint_as_float(0x3f800000u + (i & 0xffffffu)), 0);  // every float in [1, 4)
    const unsigned exponent = 127 - 100 + (i >> 3) % 201;         // samples of [2^-100, 2^101)
    compare(__uint_as_float(exponent << 23 | (i * 2654435761u >> 9)), 1);
}
__device__ unsigned long long mix(unsigned long long x) {
    x ^= x >> 33, x *= 0xff51afd7ed558ccdull, x ^= x >> 33, x *= 0xc4ceb9fe1a85ec53ull;
    return x ^ x >> 33;
}
__global__ void k_roots_f64(unsigned long long* wrong) {
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    const unsigned long long r = mix(i + 1), mantissa = (1ull << 52) - 1;
    auto compare = [&](double x, int k) {
        double y;
        const double s = sqrt_rn_d(x, y), want = __dsqrt_rn(x);
        if (__double_as_longlong(s) != __double_as_longlong(want)) atomicAdd(wrong + k, 1ull);
        if (__double_as_longlong(rcp_root(s, y)) != __double_as_longlong(__drcp_rn(want))) atomicAdd(wrong + 4 + k, 1ull);
    };
    const unsigned long long exponent = (1023ull - 60 + (r >> 52) % 121) << 52;
    compare(__longlong_as_double(exponent | (r & mantissa)), 0);
    const double s = __longlong_as_double(1023ull << 52 | (mix(r) & mantissa));
    compare(__longlong_as_double(__double_as_longlong(s * s) + (int)(i % 5) - 2), 1);  // about a square
    const unsigned long long edge = (i & 1) ? mantissa - (r & 1023) : (r & 1023);
    compare(__longlong_as_double(exponent | edge), 2);
    // roots with mantissas near all ones
    const double q = __longlong_as_double((1023ull - 30 + (i >> 9) % 61) << 52 | (mantissa - (i >> 3) % 64));
    compare(__longlong_as_double(__double_as_longlong(q * q) + (int)(i % 8) - 4), 3);
}
}
extern "C" int run(unsigned long long* wrong) {
    rf::k_roots_f32<<<1 << 16, 256>>>(wrong);
    rf::k_roots_f64<<<1 << 18, 256>>>(wrong + 4);
    return (int)cudaDeviceSynchronize();
}
'''


def test_roots_are_correctly_rounded(tmp_path):
    from realflare_gb300 import build

    source, library = tmp_path / 'roots.cu', tmp_path / 'roots.so'
    source.write_text(SOURCE)
    assert '-fmad=false' in build.UNITS['rf_trace_accurate.cu']
    subprocess.check_call([build.nvcc(), *build.ARCH, '-O3', '-std=c++17', *build.UNITS['rf_trace_accurate.cu'],
                           '-Xcompiler', '-fPIC,-ffp-contract=off', '-I', build.CSRC, '-shared', '-o', str(library),
                           str(source), '-lcudart'])
    wrong = torch.zeros((12,), dtype=torch.int64, device='cuda')
    torch.cuda.synchronize()
    assert ctypes.CDLL(str(library)).run(ctypes.c_void_p(wrong.data_ptr())) == 0
    assert wrong.tolist() == [0] * 12
