// The four sign rows of a representative (|kx|, |ky|), for the kernels over modes (or
// separations) whose bins and weights depend on kx^2, ky^2 and kz only: the rows
// (+-kx, +-ky) share them at every kz.  The representatives are 0..dims/2 on each axis;
// 0 and dims/2 have no partner.
#pragma once
#include "pk_common.cuh"

namespace pyl {
namespace {

__host__ __device__ inline int sym_groups(int dims) { return dims / 2 + 1; }

struct SignRows {
    long long off[4];       // row r = (y sign << 1) | x sign
    float2 pxy[4];          // interlacing phase exp(i pi (kx + ky) / dims) of each row
    unsigned skip0, skipm;  // rows whose kz = 0 / kz = dims/2 modes the Hermitian skip drops
    unsigned used;          // rows that exist (a representative without partner repeats row 0)
};

template <bool INTER>
__device__ __forceinline__ SignRows sign_rows(int xr, int yr, const PkDims &d, const float2 *ph)
{
    const int dims = d.dims;
    const bool even = (dims & 1) == 0;
    const int nx = (xr == 0 || 2 * xr == dims) ? 1 : 2, ny = (yr == 0 || 2 * yr == dims) ? 1 : 2;
    SignRows R;
    R.skip0 = R.skipm = 0u;
    R.used = 1u | (nx == 2 ? 2u : 0u) | (ny == 2 ? 4u : 0u) | (nx == 2 && ny == 2 ? 8u : 0u);
#pragma unroll
    for (int r = 0; r < 4; r++) {
        const int kxx = ((r & 1) && nx == 2) ? dims - xr : xr;     // in range for every r
        const int kyy = ((r & 2) && ny == 2) ? dims - yr : yr;
        R.off[r] = ((long long)kxx * dims + kyy) * d.nz;
        const int kx = freq_of(kxx, dims), ky = freq_of(kyy, dims);
        R.pxy[r] = make_float2(1.0f, 0.0f);
        if (INTER) {
            const float2 px = ph[kxx], py = ph[kyy];
            R.pxy[r] = make_float2(px.x * py.x - px.y * py.y, px.x * py.y + px.y * py.x);
        }
        if (hermitian_skip(kx, ky, 0, d)) R.skip0 |= 1u << r;
        if (even && hermitian_skip(kx, ky, d.middle, d)) R.skipm |= 1u << r;
    }
    return R;
}

}  // namespace
}  // namespace pyl
