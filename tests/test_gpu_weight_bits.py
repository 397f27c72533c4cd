"""The one-formula TSC and PCS weights of deposit.cuh against both formulas of each weight
with CUDA's division, bit for bit, at every float32 coordinate, and its division by six at
every numerator that the weights form (0, and 2^-69 to 8)."""
import ctypes
import subprocess

import pytest

pytestmark = pytest.mark.gpu

SOURCE = r'''
#include <cuda_runtime.h>
#include "common.cuh"
#include "deposit.cuh"
using namespace pyl;

__device__ bool same(float a, float b)
{
    return __float_as_uint(a) == __float_as_uint(b) || (a != a && b != b);
}

template <int MAS>
__device__ float both(float s)                          // s: distance to the cell's centre
{
    if (MAS == PYL_MAS_TSC) {
        if (s < 0.5f) return __fsub_rn(0.75f, __fmul_rn(s, s));
        const float t = __fsub_rn(1.5f, s);
        return s < 1.5f ? __fmul_rn(__fmul_rn(0.5f, t), t) : 0.0f;
    }
    if (s < 1.0f) {
        const float a = __fmul_rn(__fmul_rn(6.0f, s), s), b = __fmul_rn(__fmul_rn(__fmul_rn(3.0f, s), s), s);
        return __fdiv_rn(__fadd_rn(__fsub_rn(4.0f, a), b), 6.0f);
    }
    const float t = __fsub_rn(2.0f, s);
    return s < 2.0f ? __fdiv_rn(__fmul_rn(__fmul_rn(t, t), t), 6.0f) : 0.0f;
}

template <int MAS>
__global__ void weights(unsigned long long *bad)
{
    unsigned long long n = 0;
    for (unsigned long long i = blockIdx.x * blockDim.x + threadIdx.x; i < 1ull << 32; i += gridDim.x * blockDim.x) {
        const float x = __uint_as_float((unsigned)i);
        float c[MAS];
        const int f = axis_weights<MAS>(x, 1.0f, c);
        const float fl = floorf(x), frac = __fsub_rn(x, fl);
        const bool up = MAS == PYL_MAS_TSC && frac >= 0.5f;
        const float low = __fsub_rn(up ? __fadd_rn(fl, 1.0f) : fl, 2.0f);
        n += f != __float2int_rz(fl) - 1 + (up ? 1 : 0);
        for (int j = 0; j < MAS; j++) n += !same(c[j], both<MAS>(fabsf(__fsub_rn(__fadd_rn(low, (float)(j + 1)), x))));
    }
    if (n) atomicAdd(bad, n);
}

__global__ void sixths(unsigned long long *bad)
{
    unsigned long long n = 0;
    const unsigned lo = __float_as_uint(ldexpf(1.0f, -69)), hi = __float_as_uint(8.0f);
    for (unsigned i = lo + blockIdx.x * blockDim.x + threadIdx.x; i <= hi; i += gridDim.x * blockDim.x)
        n += !same(sixth(__uint_as_float(i)), __fdiv_rn(__uint_as_float(i), 6.0f));
    if (blockIdx.x == 0 && threadIdx.x == 0) n += !same(sixth(0.0f), 0.0f);
    if (n) atomicAdd(bad, n);
}

extern "C" long long mismatches(int which)
{
    unsigned long long *bad, host = 0;
    if (cudaMalloc(&bad, 8) != cudaSuccess) return -1;
    cudaMemset(bad, 0, 8);
    if (which == 3) weights<PYL_MAS_TSC><<<1024, 256>>>(bad);
    else if (which == 4) weights<PYL_MAS_PCS><<<1024, 256>>>(bad);
    else sixths<<<1024, 256>>>(bad);
    const cudaError_t e = cudaMemcpy(&host, bad, 8, cudaMemcpyDeviceToHost);
    cudaFree(bad);
    return e == cudaSuccess ? (long long)host : -1;
}
'''


@pytest.fixture(scope='module')
def probe(tmp_path_factory):
    import pylians_gb300.build as b
    d = tmp_path_factory.mktemp('weights')
    src, lib = d / 'weights.cu', d / 'weights.so'
    src.write_text(SOURCE)
    r = subprocess.run([b.nvcc()] + b.ARCH + ['-O3', '-std=c++17', '-Xcompiler', '-fPIC', '-shared', '--expt-relaxed-constexpr',
                        '-I' + b.CSRC, '-I' + b.ROOT + '/include', str(src), '-o', str(lib)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    f = ctypes.CDLL(str(lib)).mismatches
    f.restype = ctypes.c_longlong
    return f


@pytest.mark.parametrize('mas', [3, 4])
def test_weights_equal_both_formulas(probe, mas):
    assert probe(mas) == 0


def test_sixth_equals_the_division(probe):
    assert probe(6) == 0
