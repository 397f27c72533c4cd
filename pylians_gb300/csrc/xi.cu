// Correlation function of a grid (Pk_library.Xi, Pk_library.pyx:2035-2150):
//   pyl_xi_power: every stored mode of the R2C output becomes
//                 (|delta_k * W(k)^-1|^2, 0), the MAS factor rounded to float as
//                 the reference's MAS_factor (:2073-2083);
//   (C2R of that, unnormalised, by the caller)
//   pyl_xi_bin:   over all dims^3 separations r = (rx, ry, rz) (signed like
//                 frequencies): bin int(|r|), sums of xi, xi (3 mu^2 - 1)/2,
//                 xi (35 mu^4 - 30 mu^2 + 3)/8, |r| and counts (:2101-2136).
#include <cuda_runtime.h>

#include <algorithm>

#include "pk_rows.cuh"

namespace pyl {
namespace {

// Float64 MAS factors C(k), k = 0..dims/2 (C(-k) = C(k)), built once per CTA: a
// float64 sine per mode and axis took 1.5 ms on a 256^3 grid (fp64 runs at a 64th of
// the fp32 rate here).
__device__ __forceinline__ void corr_table(double *corr, const PkDims &d, int p)
{
    for (int k = threadIdx.x; k < d.nz; k += blockDim.x) corr[k] = mas_corr_d(k, d.dims, p);
    __syncthreads();
}

// A warp takes the four sign rows (+-kx, +-ky) of a representative: one float64
// product and rounding of the factor per kz serves their modes.
__global__ void __launch_bounds__(512) xi_power_kernel(float2 *dk, PkDims d, int p)
{
    extern __shared__ double corr[];
    corr_table(corr, d, p);
    const int G = sym_groups(d.dims), lane = threadIdx.x & 31;
    const int nwarp = (int)(gridDim.x * (blockDim.x >> 5));
    for (int rep = (int)(blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)); rep < G * G; rep += nwarp) {
        const int xr = rep / G, yr = rep % G;
        const SignRows R = sign_rows<false>(xr, yr, d, nullptr);
        const double cxy = corr[xr] * corr[yr];
        for (int kz = lane; kz < d.nz; kz += 32) {
            const float mf = (float)(cxy * corr[kz]);
            float2 v[4];
#pragma unroll
            for (int r = 0; r < 4; r++)
                if ((R.used >> r) & 1u) v[r] = dk[R.off[r] + kz];
#pragma unroll
            for (int r = 0; r < 4; r++) {
                if (!((R.used >> r) & 1u)) continue;
                const float re = __fmul_rn(v[r].x, mf), im = __fmul_rn(v[r].y, mf);
                dk[R.off[r] + kz] = make_float2(__fadd_rn(__fmul_rn(re, re), __fmul_rn(im, im)), 0.0f);
            }
        }
    }
}

// sums: X[nb3][3] | R[nb3] | N[nb3] (float64)
//
// A thread walks a row (rx, ry) along rz and adds to its CTA's float32 sums when the bin
// changes; the CTAs' sums meet in float64.  The order and the widths of these additions
// are part of the result: bins of few separations (the smallest and, in the corners of the
// cube, the largest |r|) show them.  Adding the eight separations (+-rx, +-ry, +-rz) in
// float32 first, in a kernel that took 0.05 ms for the 0.62 of this one at 256^3, lost the
// smaller ones of different x planes, which meet in float64 here, and moved xi of 512^3 by
// 1e-9 where two runs of this order differ by 2e-10.  Bound by the float32 shared-memory
// additions (compare and swap): rows staged through shared memory took no less.
__global__ void __launch_bounds__(256) xi_bin_kernel(const float *__restrict__ xi, PkDims d, int axis,
                                                     double *__restrict__ sums)
{
    extern __shared__ float acc[];                      // [nb3][3]
    const int dims = d.dims, nb = d.nb3;
    for (int i = threadIdx.x; i < 3 * nb; i += blockDim.x) acc[i] = 0.0f;
    __syncthreads();
    const long long rows = (long long)dims * dims;
    for (long long row = (long long)blockIdx.x * blockDim.x + threadIdx.x; row < rows;
         row += (long long)gridDim.x * blockDim.x) {
        const int rx = freq_of((int)(row / dims), dims), ry = freq_of((int)(row % dims), dims);
        const float *g = xi + row * dims;
        int cur = -1;
        float s0 = 0.0f, s2 = 0.0f, s4 = 0.0f;
        for (int zz = 0; zz < dims; zz++) {
            const int rz = freq_of(zz, dims);
            const int n2 = rx * rx + ry * ry + rz * rz;
            const int bin = isqrt_exact(n2);
            const int par = axis == 0 ? rx : (axis == 1 ? ry : rz);
            const float mu2 = n2 ? (float)((double)(par * par) / (double)n2) : 0.0f;
            const float v = __ldg(g + zz);
            if (bin != cur) {
                if (cur >= 0) {
                    atomicAdd(acc + 3 * cur, s0);
                    atomicAdd(acc + 3 * cur + 1, s2);
                    atomicAdd(acc + 3 * cur + 2, s4);
                }
                cur = bin;
                s0 = s2 = s4 = 0.0f;
            }
            s0 += v;
            s2 += v * (0.5f * (3.0f * mu2 - 1.0f));
            s4 += v * (0.125f * ((35.0f * mu2 - 30.0f) * mu2 + 3.0f));
        }
        if (cur >= 0) {
            atomicAdd(acc + 3 * cur, s0);
            atomicAdd(acc + 3 * cur + 1, s2);
            atomicAdd(acc + 3 * cur + 2, s4);
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 3 * nb; i += blockDim.x)
        if (acc[i] != 0.0f) atomicAdd(sums + i, (double)acc[i]);
}


// Data-independent sums: R[bin] = sum |r|, N[bin] = count, over all dims^3 separations.
// |r| and its bin are the same for (+-rx, +-ry, +-rz) and for rx and ry exchanged: a warp
// takes a representative (|rx|, |ry|) with ry >= rx, its lanes a run of rz each, one
// float64 root for up to sixteen separations.  A root for each separation took 1.45 ms at
// 256^3, this 0.04 ms (512^3: 0.24 ms).
constexpr int XI_WARPS = 8;
__global__ void __launch_bounds__(32 * XI_WARPS) xi_geometry_kernel(PkDims d, double *__restrict__ sums)
{
    extern __shared__ __align__(16) double xsm[];
    const int dims = d.dims, nb = d.nb3;
    double *R = xsm;
    unsigned *N = (unsigned *)(xsm + nb);
    for (int i = threadIdx.x; i < nb; i += blockDim.x) {
        R[i] = 0.0;
        N[i] = 0u;
    }
    __syncthreads();
    const int G = sym_groups(dims), lane = threadIdx.x & 31, run = (d.nz + 31) / 32;
    const int nwarp = (int)(gridDim.x * XI_WARPS);
    for (int rep = (int)(blockIdx.x * XI_WARPS + (threadIdx.x >> 5)); rep < G * G; rep += nwarp) {
        const int xr = rep / G, yr = rep % G;
        if (yr < xr) continue;
        const int rows = ((xr == 0 || 2 * xr == dims) ? 1 : 2) * ((yr == 0 || 2 * yr == dims) ? 1 : 2) * (yr > xr ? 2 : 1);
        const int kb = lane * run, ke = min(d.nz, kb + run);
        if (kb >= ke) continue;
        int n2 = xr * xr + yr * yr + kb * kb, bin = isqrt_exact(n2);
        unsigned c = 0;
        double len = 0.0;
        for (int z = kb; z < ke; z++) {
            const unsigned m = (unsigned)(rows * (z != 0 && 2 * z != dims ? 2 : 1));
            c += m;
            len += (double)m * sqrt((double)n2);
            n2 += 2 * z + 1;
            const bool next = (bin + 1) * (bin + 1) <= n2;
            if (next || z + 1 == ke) {
                atomicAdd(N + bin, c);
                atomicAdd(R + bin, len);
                c = 0u;
                len = 0.0;
                bin += next ? 1 : 0;
            }
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < nb; i += blockDim.x) {
        if (N[i] == 0u) continue;
        atomicAdd(sums + 3 * nb + i, R[i]);
        atomicAdd(sums + 4 * nb + i, (double)N[i]);
    }
}

// correct_MAS's mode loop (Pk_library.pyx:1776-1794): every stored mode but the
// redundant half of the kz = 0 and kz = N/2 planes (:1789-1792) is multiplied by
// the float-rounded MAS factor.
__global__ void __launch_bounds__(512) correct_mas_kernel(float2 *dk, PkDims d, int p)
{
    extern __shared__ double corr[];
    corr_table(corr, d, p);
    const bool even = (d.dims & 1) == 0;
    const int G = sym_groups(d.dims), lane = threadIdx.x & 31;
    const int nwarp = (int)(gridDim.x * (blockDim.x >> 5));
    for (int rep = (int)(blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)); rep < G * G; rep += nwarp) {
        const int xr = rep / G, yr = rep % G;
        const SignRows R = sign_rows<false>(xr, yr, d, nullptr);
        const double cxy = corr[xr] * corr[yr];
        for (int kz = lane; kz < d.nz; kz += 32) {
            const float mf = (float)(cxy * corr[kz]);
            const unsigned skip = kz == 0 ? R.skip0 : ((even && kz == d.middle) ? R.skipm : 0u);
            const unsigned take = R.used & ~skip;
            float2 v[4];
#pragma unroll
            for (int r = 0; r < 4; r++)
                if ((take >> r) & 1u) v[r] = dk[R.off[r] + kz];
#pragma unroll
            for (int r = 0; r < 4; r++)
                if ((take >> r) & 1u) dk[R.off[r] + kz] = make_float2(__fmul_rn(v[r].x, mf), __fmul_rn(v[r].y, mf));
        }
    }
}

// The reference's half-corrected kz = 0 and kz = N/2 planes are not Hermitian; its
// C2R (FFTW through pyFFTW, or any C2R that transforms x and y before z) uses
// their Hermitian part (P(k) + conj P(-k)) / 2.  Writing that part explicitly
// makes cuFFT's C2R give the same field whatever its internal order.  One thread
// per (k, -k) pair of a plane (the pair's lower flat index does the work).
__global__ void __launch_bounds__(256) hermitian_planes_kernel(float2 *dk, PkDims d)
{
    const int dims = d.dims;
    const long long plane = (long long)dims * dims;
    const int nplanes = (dims & 1) ? 1 : 2;
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < nplanes * plane; t += stride) {
        const int kz = t < plane ? 0 : d.middle;
        const long long j = t % plane;
        const int kxx = (int)(j / dims), kyy = (int)(j % dims);
        const int mxx = kxx ? dims - kxx : 0, myy = kyy ? dims - kyy : 0;
        const long long jm = (long long)mxx * dims + myy;
        if (jm < j) continue;
        float2 *a = dk + j * d.nz + kz, *b = dk + jm * d.nz + kz;
        const float2 va = *a, vb = *b;
        const float re = 0.5f * (va.x + vb.x), im = 0.5f * (va.y - vb.y);
        *a = make_float2(re, im);
        *b = make_float2(re, -im);
    }
}

inline unsigned blocks_of(long long n)
{
    long long b = (n + 255) / 256;
    const long long cap = (long long)num_sms() * 8;
    return (unsigned)(b < 1 ? 1 : (b > cap ? cap : b));
}

// Two 512-thread CTAs per SM, a warp per representative: each builds its table once.
inline unsigned rep_blocks(const PkDims &d)
{
    const long long reps = (long long)sym_groups(d.dims) * sym_groups(d.dims);
    const long long b = (reps + 15) / 16, cap = 2LL * num_sms();
    return (unsigned)(b < cap ? b : cap);
}

}  // namespace
}  // namespace pyl

using namespace pyl;

extern "C" int64_t pyl_xi_sums_len(int dims) { return dims < 2 ? 0 : 5LL * pk_dims(dims).nb3; }

extern "C" int pyl_correct_mas(void *dk, int dims, int mas_p, void *stream)
{
    PYL_CHECK_ARG(dk != nullptr && dims >= 2 && dims <= 8192, "bad arguments");
    PYL_CHECK_ARG(mas_p >= 0 && mas_p <= 4, "MAS exponent must be 0..4");
    const PkDims d = pk_dims(dims);
    cudaStream_t st = (cudaStream_t)stream;
    const size_t smem = sizeof(double) * d.nz;
    correct_mas_kernel<<<rep_blocks(d), 512, smem, st>>>((float2 *)dk, d, mas_p);
    PYL_LAUNCH_CHECK();
    hermitian_planes_kernel<<<blocks_of(2LL * dims * dims), 256, 0, st>>>((float2 *)dk, d);
    PYL_LAUNCH_CHECK();
    return PYL_OK;
}

extern "C" int pyl_xi_power(void *dk, int dims, int mas_p, void *stream)
{
    PYL_CHECK_ARG(dk != nullptr && dims >= 2 && dims <= 8192, "bad arguments");
    PYL_CHECK_ARG(mas_p >= 0 && mas_p <= 4, "MAS exponent must be 0..4");
    const PkDims d = pk_dims(dims);
    xi_power_kernel<<<rep_blocks(d), 512, sizeof(double) * d.nz, (cudaStream_t)stream>>>((float2 *)dk, d, mas_p);
    PYL_LAUNCH_CHECK();
    return PYL_OK;
}

extern "C" int pyl_xi_bin(const float *xi_grid, int dims, int axis, double *sums, void *stream)
{
    PYL_CHECK_ARG(xi_grid != nullptr && sums != nullptr && dims >= 2 && dims <= 8192, "bad arguments");
    PYL_CHECK_ARG(axis >= 0 && axis <= 2, "axis must be 0, 1 or 2");
    const PkDims d = pk_dims(dims);
    cudaStream_t st = (cudaStream_t)stream;
    PYL_CUDA(cudaMemsetAsync(sums, 0, sizeof(double) * 5 * d.nb3, st));
    const size_t smem = sizeof(float) * 3 * d.nb3;
    PYL_CHECK_ARG(smem <= 48 * 1024, "grid too large for the shared-memory bins");
    xi_bin_kernel<<<blocks_of((long long)dims * dims), 256, smem, st>>>(xi_grid, d, axis, sums);
    PYL_LAUNCH_CHECK();
    const long long reps = (long long)sym_groups(dims) * sym_groups(dims);
    const size_t gsm = 12 * (size_t)d.nb3;
    const long long b = std::min((reps + 2 * XI_WARPS - 1) / (2 * XI_WARPS), 4LL * num_sms());
    xi_geometry_kernel<<<(unsigned)b, 32 * XI_WARPS, gsm, st>>>(d, sums);
    PYL_LAUNCH_CHECK();
    return PYL_OK;
}
