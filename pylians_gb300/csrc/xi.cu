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

// sums: X[nb3][3] | R[nb3] | N[nb3] (float64).
//
// |r|, its bin and every Legendre weight are the same for the eight separations
// (+-rx, +-ry, +-rz): a warp adds the (up to eight) values per rz from coalesced reads
// of the four sign rows and their mirrored halves into shared memory, and each lane
// walks its run of rz (an odd number of them: distinct banks), adding to the CTA's
// shared sums only when the bin changes (bins below `core`: counts and R alone,
// xi_row_kernel has their values).  One thread per row, 4 bytes at a time and
// 1 KB apart, took 0.62 ms for 256^3, and float64 roots of every separation for R
// another 1.45 ms; this kernel takes 0.05 ms (0.30 ms for 512^3).  Counts are exact in float32: the CTAs
// share a bin's 4 pi r^2 separations, far below 2^24 each.  R adds |r| in float64 over
// ry >= rx only, twice off the diagonal.
struct XiRun {
    int segments, run;
};

inline XiRun xi_run(int nz)
{
    XiRun x;
    x.segments = (nz + 32 * 9 - 1) / (32 * 9);
    x.run = ((nz + 32 * x.segments - 1) / (32 * x.segments)) | 1;
    return x;
}

constexpr int XI_WARPS = 8;
constexpr int XI_CORE = 32;              // bins that xi_row_kernel sums on large grids
constexpr int XI_ROWS_BELOW = 256;       // grids whose every bin it sums

inline size_t xi_smem(const PkDims &d, const XiRun &x)
{
    return (size_t)d.nb3 * (sizeof(double) + 4 * sizeof(float)) + sizeof(float) * XI_WARPS * 32 * x.run;
}

// |r| to float64 from the float32 square root and one Newton correction: relative
// error below 2^-47 of each term (n2 < 2^24 is exact in float32).
__device__ __forceinline__ double length_of(int n2)
{
    if (n2 == 0) return 0.0;
    const float f = (float)n2, s = sqrtf(f);
    const float e = __fmaf_rn(-s, s, f);                 // exact residual
    return (double)s + (double)__fdividef(e, 2.0f * s);
}

__global__ void __launch_bounds__(32 * XI_WARPS) xi_bin_kernel(const float *__restrict__ xi, PkDims d, int axis,
                                                               XiRun x, int core, double *__restrict__ sums)
{
    extern __shared__ __align__(16) double xsm[];
    const int dims = d.dims, nb = d.nb3;
    double *R = xsm;
    float *acc = (float *)(xsm + nb);                    // [nb3][4]: l = 0, 2, 4, count
    float *stage = acc + 4 * nb + (threadIdx.x >> 5) * 32 * x.run;
    for (int i = threadIdx.x; i < nb; i += blockDim.x) {
        R[i] = 0.0;
        acc[4 * i] = acc[4 * i + 1] = acc[4 * i + 2] = acc[4 * i + 3] = 0.0f;
    }
    __syncthreads();
    const int G = sym_groups(dims), lane = threadIdx.x & 31;
    const int nwarp = (int)(gridDim.x * XI_WARPS), slots = 32 * x.run;
    for (int rep = (int)(blockIdx.x * XI_WARPS + (threadIdx.x >> 5)); rep < G * G; rep += nwarp) {
        const int xr = rep / G, yr = rep % G;
        const int nx = (xr == 0 || 2 * xr == dims) ? 1 : 2, ny = (yr == 0 || 2 * yr == dims) ? 1 : 2;
        const int rows = nx * ny, rho2 = xr * xr + yr * yr;
        long long off[4];
#pragma unroll
        for (int r = 0; r < 4; r++) {
            const int ix = ((r & 1) && nx == 2) ? dims - xr : xr, iy = ((r & 2) && ny == 2) ? dims - yr : yr;
            off[r] = ((long long)ix * dims + iy) * dims;
        }
        const unsigned used = 1u | (nx == 2 ? 2u : 0u) | (ny == 2 ? 4u : 0u) | (rows == 4 ? 8u : 0u);
        for (int sgm = 0; sgm < x.segments; sgm++) {
            const int k0 = sgm * slots, k1 = min(d.nz, k0 + slots);
            for (int z = k0 + lane; core < nb && z < k1; z += 32) {
                const bool two = z != 0 && 2 * z != dims;
                float a[4], b[4];
#pragma unroll
                for (int r = 0; r < 4; r++) {
                    a[r] = (used >> r) & 1u ? __ldg(xi + off[r] + z) : 0.0f;
                    b[r] = two && ((used >> r) & 1u) ? __ldg(xi + off[r] + dims - z) : 0.0f;
                }
                stage[z - k0] = ((a[0] + b[0]) + (a[1] + b[1])) + ((a[2] + b[2]) + (a[3] + b[3]));
            }
            __syncwarp();
            const int kb = k0 + lane * x.run, ke = min(k1, kb + x.run);
            if (kb < ke) {
                int n2 = rho2 + kb * kb;
                int bin = isqrt_exact(n2);
                float s0 = 0.0f, s2 = 0.0f, s4 = 0.0f, c = 0.0f;
                double len = 0.0;
                const int par2 = axis == 0 ? xr * xr : yr * yr;
                const float wl = yr > xr ? 2.0f : 1.0f;
                for (int z = kb; z < ke; z++) {
                    // correctly rounded, as the float64 quotient rounded to float32 is
                    // (both operands are integers below 2^24)
                    const float mu2 = n2 ? __fdiv_rn((float)(axis == 2 ? z * z : par2), (float)n2) : 0.0f;
                    const float v = stage[z - k0];
                    const float m = (float)(rows * (z != 0 && 2 * z != dims ? 2 : 1));
                    if (bin >= core) {
                        s0 += v;
                        s2 += v * (0.5f * (3.0f * mu2 - 1.0f));
                        s4 += v * (0.125f * ((35.0f * mu2 - 30.0f) * mu2 + 3.0f));
                    }
                    c += m;
                    if (yr >= xr) len += (double)(wl * m) * length_of(n2);
                    n2 += 2 * z + 1;
                    const bool next = (bin + 1) * (bin + 1) <= n2;
                    if (next || z + 1 == ke) {
                        atomicAdd(acc + 4 * bin, s0);
                        atomicAdd(acc + 4 * bin + 1, s2);
                        atomicAdd(acc + 4 * bin + 2, s4);
                        atomicAdd(acc + 4 * bin + 3, c);
                        if (len != 0.0) atomicAdd(R + bin, len);
                        s0 = s2 = s4 = c = 0.0f;
                        len = 0.0;
                        bin += next ? 1 : 0;
                    }
                }
            }
            __syncwarp();
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < nb; i += blockDim.x) {
        if (acc[4 * i + 3] == 0.0f) continue;
#pragma unroll
        for (int l = 0; l < 3; l++) atomicAdd(sums + 3 * i + l, (double)acc[4 * i + l]);
        if (R[i] != 0.0) atomicAdd(sums + 3 * nb + i, R[i]);
        atomicAdd(sums + 4 * nb + i, (double)acc[4 * i + 3]);
    }
}

// The sums of the bins below `core`: XI_CORE of them, or every bin of grids below
// XI_ROWS_BELOW, where they hold few separations each.  There the order of the float32
// additions shows in xi (1e-8 of the largest multipole; the larger bins of larger grids
// average it away), and the sums keep one order: a thread walks a row (rx, ry) along rz
// in step with the other rows of its CTA and adds to the CTA's sums when its bin
// changes.  Bound by the latency of a step, about 1.5 us: 0.09 ms for |rz| < XI_CORE of
// the CTAs with rows of the core at 256^3; below that size whole rows take less than
// 0.6 ms (0.53 ms at 200^3, where xi_bin_kernel would add the values in 0.03 ms).
__global__ void __launch_bounds__(256) xi_row_kernel(const float *__restrict__ xi, PkDims d, int axis, int core,
                                                     double *__restrict__ sums)
{
    extern __shared__ float acc[];                      // [nb3][3]; bins from `core` up are scratch
    const int dims = d.dims, nb = d.nb3;
    const long long rows = (long long)dims * dims;
    bool any = false;
    for (long long row = (long long)blockIdx.x * blockDim.x + threadIdx.x; row < rows;
         row += (long long)gridDim.x * blockDim.x) {
        const int rx = freq_of((int)(row / dims), dims), ry = freq_of((int)(row % dims), dims);
        any |= rx * rx + ry * ry < core * core;
    }
    if (!__syncthreads_or(any)) return;
    for (int i = threadIdx.x; i < 3 * nb; i += blockDim.x) acc[i] = 0.0f;
    __syncthreads();
    // rz = 0 .. up, then -down .. -1; with larger bins between them, a new run
    const int up = min(core - 1, dims / 2), down = min(core - 1, (dims - 1) / 2);
    const bool gap = up + 1 < dims - down;
    for (long long row = (long long)blockIdx.x * blockDim.x + threadIdx.x; row < rows;
         row += (long long)gridDim.x * blockDim.x) {
        const int rx = freq_of((int)(row / dims), dims), ry = freq_of((int)(row % dims), dims);
        const float *g = xi + row * dims;
        int cur = -1;
        float s0 = 0.0f, s2 = 0.0f, s4 = 0.0f;
        for (int zz = 0; zz < dims; zz++) {
            if (gap && zz == up + 1) zz = dims - down;
            const int rz = freq_of(zz, dims);
            const int n2 = rx * rx + ry * ry + rz * rz;
            const int bin = isqrt_exact(n2);
            const int par = axis == 0 ? rx : (axis == 1 ? ry : rz);
            const float mu2 = n2 ? (float)((double)(par * par) / (double)n2) : 0.0f;
            const float v = __ldg(g + zz);
            if (bin != cur || (gap && zz == dims - down)) {
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
    for (int i = threadIdx.x; i < 3 * min(core, nb); i += blockDim.x)
        if (acc[i] != 0.0f) atomicAdd(sums + i, (double)acc[i]);
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
    PYL_CHECK_ARG(sizeof(float) * 3 * d.nb3 <= 48 * 1024, "grid too large for the shared-memory bins");
    const XiRun x = xi_run(d.nz);
    const size_t smem = xi_smem(d, x);
    PYL_CUDA(ensure_smem(xi_bin_kernel, smem));
    // one wave of resident CTAs, at least two representatives a warp
    const long long reps = (long long)sym_groups(dims) * sym_groups(dims);
    const long long per_sm = std::max<long long>(1, std::min<long long>(6, (long long)(227 * 1024 / (smem + 1024))));
    const long long b = std::min((reps + 2 * XI_WARPS - 1) / (2 * XI_WARPS), per_sm * num_sms());
    const int core = dims < XI_ROWS_BELOW ? d.nb3 : XI_CORE;
    xi_bin_kernel<<<(unsigned)b, 32 * XI_WARPS, smem, st>>>(xi_grid, d, axis, x, core, sums);
    PYL_LAUNCH_CHECK();
    xi_row_kernel<<<blocks_of((long long)dims * dims), 256, sizeof(float) * 3 * d.nb3, st>>>(xi_grid, d, axis, core, sums);
    PYL_LAUNCH_CHECK();
    return PYL_OK;
}
