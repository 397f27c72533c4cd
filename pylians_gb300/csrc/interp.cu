// Neighbours of the mass assignment on the particle side:
//   * CIC interpolation of a grid at particle positions (MAS_library.pyx:558-599),
//     the gather dual of the CIC scatter;
//   * redshift-space positions s = x + v (1+z)/H(z) along one axis with the
//     periodic wrap of redshift_space_library.pyx:29-43.
// One thread per particle, grid-stride loops; positions are read as float32
// [n][3] rows exactly as the reference's typed memoryviews hold them.
#include <algorithm>
#include <string>

#include <cuda_runtime.h>

#include "common.cuh"

namespace pyl {
namespace {

// Interpolated density at p(0), p(1), p(2): the sum of the eight corner values times d/u weights, added
// in the reference's order: (d,d,d), (d,d,u), (d,u,d), (d,u,u), (u,d,d), (u,d,u), (u,u,d),
// (u,u,u); each term density * w0 * w1 * w2 left to right.  (One 16-byte load for both
// values along z measured slower, 322 -> 354 us at 256^3: the lanes' loads, not their
// number of sectors, bound it.)
template <typename P>
__device__ __forceinline__ float cic_value(const float *__restrict__ g, int dims, float inv, P p)
{
    float u[3], dd[3];
    long long id[3], iu[3];
    const long long D = dims;
#pragma unroll
    for (int a = 0; a < 3; a++) {
        const float dist = __fmul_rn(p(a), inv);
        const float t = truncf(dist);
        u[a] = __fsub_rn(dist, t);
        dd[a] = __fsub_rn(1.0f, u[a]);
        const int k = wrap_index(__float2int_rz(t), dims);
        id[a] = k;
        iu[a] = k + 1 == dims ? 0 : k + 1;
    }
    const float w0[2] = {dd[0], u[0]}, w1[2] = {dd[1], u[1]}, w2[2] = {dd[2], u[2]};
    const long long c0[2] = {id[0], iu[0]}, c1[2] = {id[1], iu[1]}, c2[2] = {id[2], iu[2]};
    float acc = 0.0f;
#pragma unroll
    for (int l = 0; l < 2; l++)
#pragma unroll
        for (int m = 0; m < 2; m++)
#pragma unroll
            for (int q = 0; q < 2; q++) {
                const float v = __ldg(g + (c0[l] * D + c1[m]) * D + c2[q]);
                const float term = __fmul_rn(__fmul_rn(__fmul_rn(v, w0[l]), w1[m]), w2[q]);
                acc = (l | m | q) ? __fadd_rn(acc, term) : term;
            }
    return acc;
}

__device__ __forceinline__ float cic_at(const float *__restrict__ g, int dims, float inv, const float *__restrict__ q)
{
    return cic_value(g, dims, inv, [&](int a) { return __ldg(q + a); });
}

// Four particles a thread, a grid's width apart: CTAs that start in order keep ordered
// particles together in L2, where a resident grid of threads drifts apart, and a CTA for
// every 256 particles costs more than they do (256^3 particles, resident / 4 / 1 each, us:
// lattice, x slowest, on 256^3 115, 113, 130, on 320^3 120, 117, 135, on 512^3 145, 141, 151;
// z slowest on 400^3 545, 455, 450, on 512^3 1382, 1286, 1219; no order on 512^3 1230, 1221, 1208).
constexpr int IP_PER_THREAD = 4;

__device__ __forceinline__ void interp_direct(const float *__restrict__ g, int dims, float inv,
                                              const float *__restrict__ pos, long long n, float *__restrict__ den,
                                              unsigned ctas)
{
    const long long stride = (long long)ctas * blockDim.x;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
        den[i] = cic_at(g, dims, inv, pos + 3 * i);
}

__global__ void __launch_bounds__(256) cic_interp_kernel(const float *__restrict__ g, int dims, float inv,
                                                         const float *__restrict__ pos, long long n,
                                                         float *__restrict__ den)
{
    interp_direct(g, dims, inv, pos, n, den, gridDim.x);
}

// ---- interpolation by slabs ----------------------------------------------------------
// Particles in no order read a grid larger than L2 from DRAM, some 100 bytes for each of
// a particle's 4 rows.  Instead:
//   1. interp_split_kernel sorts tiles of IT particles by slab of x (IS_BYTES of the grid
//      each) and writes them with their places;
//   2. interp_slab_kernel takes slab after slab, the particles of all tiles, from L2;
//   3. interp_place_kernel puts each tile's values back into the particles' order.
// Whether the particles are in no order, over more of the grid than stays in L2, is read off
// a sample (interp_scattered); else the second kernel interpolates them as
// cic_interp_kernel does and the others have nothing to do.  The same bits either way: every value comes from cic_value.
// 256^3 particles in no order on 512^3: 1250 -> 449 us (split 102, slabs 311, places 27).  The
// slabs' kernel is bound by the random loads in L1 and L2 (87 and 78 % of their throughput;
// 8 loads of 12 wavefronts, 94 million sectors); a grid that fits L2 takes as long (322 at
// 256^3).  Values written straight to their places instead of by 3.: 494 + 107 us.
constexpr int IT = 4096, IT_THREADS = 512, IT_PER = IT / IT_THREADS;
constexpr int IS_MAX = IT_THREADS;                          // slabs
constexpr long long IS_BYTES = 16ll << 20;
constexpr long long INTERP_PASS = 1ll << 25;                // particles of one pass (18 bytes each)

struct Slabs {
    int planes, count;        // grid planes of a slab, slabs
};

inline Slabs interp_slabs(int dims)
{
    const long long plane = 4ll * dims * dims;
    const int planes = (int)std::max<long long>(std::max<long long>(1, IS_BYTES / plane), (dims + IS_MAX - 1) / IS_MAX);
    return Slabs{planes, (dims + planes - 1) / planes};
}

struct InterpWs {
    float *rec, *val;         // positions by tile and slab, their values
    unsigned short *place;    // their places in the tile
    unsigned *scattered;      // written by interp_split_kernel
    unsigned *start;          // [slab][tile] first record of the slab in the tile; row `count`: the tile's records
    size_t bytes;
};

inline InterpWs interp_layout(void *base, long long n, int dims)
{
    const size_t tiles = (size_t)((std::min<long long>(n, INTERP_PASS) + IT - 1) / IT);
    char *b = (char *)base;
    InterpWs w;
    w.rec = (float *)b;
    w.val = (float *)(b + tiles * IT * 12);
    w.place = (unsigned short *)(b + tiles * IT * 16);
    w.scattered = (unsigned *)(b + tiles * IT * 18);
    w.start = w.scattered + 4;
    w.bytes = tiles * IT * 18 + 16 + sizeof(unsigned) * tiles * (interp_slabs(dims).count + 1);
    return w;
}

constexpr size_t INTERP_SMEM = (size_t)IT * 14 + sizeof(unsigned) * IS_MAX;

// True where IT consecutive particles lie, as a rule, in more than half of the slabs that
// as many particles in no order would, and all of them in a part of the grid of more than
// INTERP_PART bytes: 64 of each of 16 tiles, one tile a warp, at hashed places (a lattice's
// rows have a period); the part is the share of 8^3 cells of the box that hold particles,
// by how many of them hold one of 512.  (256^3 particles in one octant, direct
// and by slabs: 400^3 302 and 442 us, 450^3 308 and 441, 512^3 609 and 439.)  Every CTA comes
// to the same answer.
constexpr float INTERP_PART = 56.0f * (1 << 20);

__device__ bool interp_scattered(const float *__restrict__ pos, long long n, int dims, float inv, Slabs sl)
{
    __shared__ unsigned seen[IT_THREADS / 32][IS_MAX / 32], boxes[16];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned span = (unsigned)min((long long)IT, n);
    const float *tile = pos + 3 * ((n - span) / (IT_THREADS / 32) * warp);
    unsigned at[2];
#pragma unroll
    for (int j = 0; j < 2; j++) {
        at[j] = (threadIdx.x * 2 + j) * 2654435769u >> 20;                      // below IT
        if (span < IT) at[j] %= span;
    }
    const float x[2] = {__ldg(tile + 3 * at[0]), __ldg(tile + 3 * at[1])};
    const float y = __ldg(tile + 3 * at[0] + 1), z = __ldg(tile + 3 * at[0] + 2);
    if (lane < IS_MAX / 32) seen[warp][lane] = 0;
    if (threadIdx.x < 16) boxes[threadIdx.x] = 0;
    __syncthreads();
    auto cell = [&](float p) { return (unsigned)wrap_index(__float2int_rz(truncf(__fmul_rn(p, inv))), dims); };
    auto eighth = [&](unsigned k) { return min(7u, (unsigned)(k * (8.0f / dims))); };
    const unsigned k[2] = {cell(x[0]), cell(x[1])};
#pragma unroll
    for (int j = 0; j < 2; j++) {
        const unsigned b = k[j] / (unsigned)sl.planes;
        atomicOr(&seen[warp][b / 32], 1u << (b % 32));
    }
    const unsigned box = (8 * eighth(k[0]) + eighth(cell(y))) * 8 + eighth(cell(z));
    atomicOr(&boxes[box / 32], 1u << (box % 32));
    __syncwarp();
    const int used = __reduce_add_sync(~0u, lane < IS_MAX / 32 ? __popc(seen[warp][lane]) : 0);
    const float fresh = sl.count * (1.0f - __expf(-64.0f / sl.count));
    const bool mixed = __syncthreads_count(2 * used > fresh) > IT_THREADS / 2;
    int held = 0;
#pragma unroll
    for (int i = 0; i < 16; i++) held += __popc(boxes[i]);
    float boxed = (float)held;                               // of them, m (1 - exp(-512 / m)) hold one
#pragma unroll
    for (int i = 0; i < 3; i++) boxed = held / (1.0f - __expf(-512.0f / boxed));
    return mixed && boxed * (4.0f / 512.0f) * dims * dims * dims > INTERP_PART;
}

__global__ void __launch_bounds__(IT_THREADS, 3) interp_split_kernel(const float *__restrict__ pos, long long n,
                                                                     int dims, float inv, int tiles, Slabs sl, InterpWs ws)
{
    extern __shared__ float4 smem[];
    float *rec = (float *)smem;
    unsigned short *place = (unsigned short *)(rec + 3 * IT);
    unsigned *cnt = (unsigned *)(place + IT);
    __shared__ unsigned wsum[IT_THREADS / 32];
    const int t = threadIdx.x;
    const bool scattered = interp_scattered(pos, n, dims, inv, sl);
    if (blockIdx.x == 0 && t == 0) *ws.scattered = scattered;
    if (!scattered) return;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const long long base = (long long)tile * IT;
        const int m = (int)min((long long)IT, n - base);
        cnt[t] = 0;
        __syncthreads();
        float p[IT_PER][3];
        unsigned key[IT_PER];
#pragma unroll
        for (int j = 0; j < IT_PER; j++) {
            const int i = t + j * IT_THREADS;
            if (i < m) {
#pragma unroll
                for (int a = 0; a < 3; a++) p[j][a] = __ldg(pos + 3 * (base + i) + a);
            }
        }
#pragma unroll
        for (int j = 0; j < IT_PER; j++)
            if (t + j * IT_THREADS < m) {
                const unsigned b =
                    (unsigned)wrap_index(__float2int_rz(truncf(__fmul_rn(p[j][0], inv))), dims) / (unsigned)sl.planes;
                key[j] = b * IT + atomicAdd(cnt + b, 1u);
            }
        __syncthreads();
        const unsigned c = cnt[t];
        unsigned s = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned v = __shfl_up_sync(~0u, s, o);
            if ((t & 31) >= o) s += v;
        }
        if ((t & 31) == 31) wsum[t >> 5] = s;
        __syncthreads();
        s -= c;
        for (int w = 0; w < (t >> 5); w++) s += wsum[w];
        cnt[t] = s;
        if (t < sl.count) ws.start[(long long)t * tiles + tile] = s;
        if (t == 0) ws.start[(long long)sl.count * tiles + tile] = m;
        __syncthreads();
#pragma unroll
        for (int j = 0; j < IT_PER; j++)
            if (t + j * IT_THREADS < m) {
                const unsigned at = cnt[key[j] / IT] + key[j] % IT;
#pragma unroll
                for (int a = 0; a < 3; a++) rec[3 * at + a] = p[j][a];
                place[at] = (unsigned short)(t + j * IT_THREADS);
            }
        __syncthreads();
        float4 *out = (float4 *)(ws.rec + 3 * base);        // the tile's places past m stay unread
        for (int i = t; i < 3 * IT / 4; i += IT_THREADS) __stcs(out + i, smem[i]);
        uint4 *outp = (uint4 *)(ws.place + base);
        for (int i = t; i < IT / 8; i += IT_THREADS) __stcs(outp + i, ((const uint4 *)place)[i]);
        __syncthreads();
    }
}

// `width` lanes (a power of two) to each (slab, tile) run, in the order of the CTAs' start
// (a resident grid with a stride drifts apart over the slabs: 590 us for 310).
__global__ void __launch_bounds__(256) interp_slab_kernel(const float *__restrict__ g, int dims, float inv,
                                                          const float *__restrict__ pos, long long n, Slabs sl, int tiles,
                                                          int width, unsigned direct_ctas, InterpWs ws, float *__restrict__ den)
{
    const long long first = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (!*ws.scattered) {
        if (blockIdx.x < direct_ctas) interp_direct(g, dims, inv, pos, n, den, direct_ctas);
        return;
    }
    const long long job = first / width;
    if (job >= (long long)sl.count * tiles) return;
    const unsigned b = ws.start[job], e = ws.start[job + tiles];
    const long long base = job % tiles * IT;
    for (unsigned s = b + threadIdx.x % width; s < e; s += width) {
        const float *r = ws.rec + 3 * (base + s);
        const float p[3] = {__ldcs(r), __ldcs(r + 1), __ldcs(r + 2)};
        __stcs(ws.val + base + s, cic_value(g, dims, inv, [&](int a) { return p[a]; }));
    }
}

__global__ void __launch_bounds__(IT_THREADS) interp_place_kernel(InterpWs ws, int slabs, int tiles, float *__restrict__ den)
{
    __shared__ float v[IT];
    if (!*ws.scattered) return;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const long long base = (long long)tile * IT;
        const int m = (int)ws.start[(long long)slabs * tiles + tile];
        for (int i = threadIdx.x; i < m; i += IT_THREADS) v[__ldcs(ws.place + base + i)] = __ldcs(ws.val + base + i);
        __syncthreads();
        for (int i = threadIdx.x; i < m; i += IT_THREADS) den[base + i] = v[i];
        __syncthreads();
    }
}

__global__ void __launch_bounds__(256) rsd_kernel(float *__restrict__ pos, const float *__restrict__ vel,
                                                  long long n, float box, float factor, int axis)
{
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        float p = __fadd_rn(pos[3 * i + axis], __fmul_rn(__ldg(vel + 3 * i + axis), factor));
        if (p > box || p < 0.0f) p = fmodf(__fadd_rn(p, box), box);
        pos[3 * i + axis] = p;
    }
}

inline unsigned blocks_of(long long n)
{
    long long b = (n + 255) / 256;
    const long long cap = (long long)num_sms() * 16;
    return (unsigned)(b < 1 ? 1 : (b > cap ? cap : b));
}

// CTAs of interp_direct: IP_PER_THREAD particles a thread, fewer where that leaves SMs idle.
inline unsigned direct_blocks(long long n)
{
    const long long per_cta = 256 * IP_PER_THREAD;
    return std::max(blocks_of(n), (unsigned)std::min((n + per_cta - 1) / per_cta, 1ll << 30));
}

}  // namespace
}  // namespace pyl

using namespace pyl;

// Slabs and direct, 256^3 particles in no order / sorted by z (us): 320^3 449, 578 / -, 450; 400^3
// 442, 960 / 484, 573; 512^3 446, 1221 / 589, 1163; 640^3 478, 1429 / 602, 1440.  Ordered particles pay
// the sample and two empty kernels, 9 to 13 us of 137 (256^3, lattice on 400^3) or of 87 (204^3).
constexpr long long INTERP_MIN_BYTES = 240ll << 20;
constexpr long long INTERP_MIN_N = 1ll << 23;

extern "C" size_t pyl_cic_interp_workspace_size(int dims, int64_t n)
{
    if (dims <= 0 || dims > 65536 || n < INTERP_MIN_N || 4ll * dims * dims * dims < INTERP_MIN_BYTES) return 0;
    return interp_layout(nullptr, n, dims).bytes;
}

extern "C" int pyl_cic_interp_slabs(const float *grid, int dims, float box_size, const float *pos, int64_t n,
                                    float *out, void *workspace, size_t workspace_bytes, void *stream)
{
    PYL_CHECK_ARG(dims > 0 && dims <= 65536, "dims out of range");
    PYL_CHECK_ARG(n >= 0, "negative particle count");
    PYL_CHECK_ARG(n == 0 || (grid != nullptr && pos != nullptr && out != nullptr), "null pointer");
    PYL_CHECK_ARG(box_size > 0.0f && isfinite(box_size), "BoxSize must be positive and finite");
    if (n == 0) return PYL_OK;
    const InterpWs ws = interp_layout(workspace, n, dims);
    if (workspace == nullptr || ((uintptr_t)workspace & 15) != 0 || workspace_bytes < ws.bytes) {
        set_error("pyl_cic_interp_slabs: needs " + std::to_string(ws.bytes) + " workspace bytes, 16-byte aligned");
        return PYL_ERR_WORKSPACE;
    }
    const cudaStream_t st = (cudaStream_t)stream;
    const float inv = (float)dims / box_size;             // MAS_library.pyx:575
    const Slabs sl = interp_slabs(dims);
    int width = 32;                                       // half of an average run or less
    while (width > 1 && width * sl.count > IT) width /= 2;
    PYL_CUDA(ensure_smem(interp_split_kernel, INTERP_SMEM));
    for (long long done = 0; done < n; done += INTERP_PASS) {
        const long long len = std::min<long long>(n - done, INTERP_PASS);
        const int tiles = (int)((len + IT - 1) / IT);
        interp_split_kernel<<<std::min(tiles, 3 * num_sms()), IT_THREADS, INTERP_SMEM, st>>>(pos + 3 * done, len, dims, inv,
                                                                                             tiles, sl, ws);
        PYL_LAUNCH_CHECK();
        const long long threads = (long long)sl.count * tiles * width;
        const unsigned direct = direct_blocks(len);
        interp_slab_kernel<<<std::max((unsigned)((threads + 255) / 256), direct), 256, 0, st>>>(
            grid, dims, inv, pos + 3 * done, len, sl, tiles, width, direct, ws, out + done);
        PYL_LAUNCH_CHECK();
        interp_place_kernel<<<std::min(tiles, 4 * num_sms()), IT_THREADS, 0, st>>>(ws, sl.count, tiles, out + done);
        PYL_LAUNCH_CHECK();
    }
    return PYL_OK;
}

extern "C" int pyl_cic_interp(const float *grid, int dims, float box_size, const float *pos, int64_t n,
                              float *out, void *stream)
{
    PYL_CHECK_ARG(dims > 0 && dims <= 65536, "dims out of range");
    PYL_CHECK_ARG(n >= 0, "negative particle count");
    PYL_CHECK_ARG(n == 0 || (grid != nullptr && pos != nullptr && out != nullptr), "null pointer");
    PYL_CHECK_ARG(box_size > 0.0f && isfinite(box_size), "BoxSize must be positive and finite");
    if (n == 0) return PYL_OK;
    const float inv = (float)dims / box_size;             // MAS_library.pyx:575
    cic_interp_kernel<<<direct_blocks(n), 256, 0, (cudaStream_t)stream>>>(grid, dims, inv, pos, n, out);
    PYL_LAUNCH_CHECK();
    return PYL_OK;
}

extern "C" int pyl_pos_redshift_space(float *pos, const float *vel, int64_t n, float box_size, float hubble,
                                      float redshift, int axis, void *stream)
{
    PYL_CHECK_ARG(n >= 0, "negative particle count");
    PYL_CHECK_ARG(n == 0 || (pos != nullptr && vel != nullptr), "null pointer");
    PYL_CHECK_ARG(axis >= 0 && axis <= 2, "axis must be 0, 1 or 2");
    PYL_CHECK_ARG(box_size > 0.0f && isfinite(box_size), "BoxSize must be positive and finite");
    PYL_CHECK_ARG(hubble != 0.0f, "Hubble must be non-zero");
    if (n == 0) return PYL_OK;
    // factor = (1.0 + redshift) / Hubble in double, kept as float (redshift_space_library.pyx:36)
    const float factor = (float)((1.0 + (double)redshift) / (double)hubble);
    rsd_kernel<<<blocks_of(n), 256, 0, (cudaStream_t)stream>>>(pos, vel, n, box_size, factor, axis);
    PYL_LAUNCH_CHECK();
    return PYL_OK;
}
