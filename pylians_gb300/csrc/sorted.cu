// SORTED strategy of pyl_ma / pyl_ma_overdensity: a deterministic mass
// assignment built from a sort by cell key and a per-cell segmented reduction.
//
//   1. every particle's base cell (the first cell of its support on each axis, wrapped;
//      MAS_library.pyx:123-545 index arithmetic) gives a 32-bit key (ix*dims + iy)*dims + iz.
//   2. stable LSD radix sort by key, 8-bit digits, of the particles themselves: per-tile
//      digit histograms, one exclusive scan over [digit][tile], and a scatter that
//      ranks each tile's records stably (warp ballots + per-warp digit counts) and
//      writes them in digit order, coalesced.  Equal keys keep increasing particle index.
//   3. a table of where each column (ix, iy) and every SD_Z cells along it start.
//   4. the sums of crowded cells, a warp or CTA each.
//   5. deposit (sd_deposit_kernel): a thread walks a base column (ix, iy) along z and
//      keeps the S^3 sums that its particles add to, S output layers of S x S columns,
//      in registers; at every z the layer that no later particle reaches is exchanged
//      through shared memory and each output cell adds its S^2 base columns' values.
//      The interlaced grid runs all steps again on the shifted positions (its own sort).
//      No atomics: every cell's sum has one fixed order (base columns by (l, m), within a
//      column by z and index, in crowded cells by lane), so the grid is bit-reproducible whatever the
//      launch configuration; NGP adds each cell's particles in index order onto the
//      grid's value, exactly the serial reference loop.
// Limits: dims^3 <= 2^32 (dims <= 1625) and fewer than 2^32 particles.
#include <cuda_runtime.h>

#include <string>

#include "common.cuh"
#include "deposit.cuh"
#include "sorted.cuh"

namespace pyl {
namespace {

constexpr int RS_THREADS = 512;
constexpr int RS_ITEMS = 8;
constexpr int RS_TILE = RS_THREADS * RS_ITEMS;       // 4096 records per tile
constexpr int RS_WARPS = RS_THREADS / 32;
constexpr int SCAN_THREADS = 1024;
constexpr int SCAN_ITEMS = 4;
constexpr int SCAN_BLOCK = SCAN_THREADS * SCAN_ITEMS;  // 4096 entries per scan block

template <int MAS>
__device__ __forceinline__ int sd_first(float p, float inv)
{
    const float dist = __fmul_rn(p, inv);
    if (MAS == PYL_MAS_CIC) return __float2int_rz(dist);
    const float fl = floorf(dist);
    const float frac = __fsub_rn(dist, fl);
    const int fi = __float2int_rz(fl);
    if (MAS == PYL_MAS_NGP) {
        int k = fi + (frac >= 0.5f ? 1 : 0);
        if (dist < -0.5f && frac != 0.5f) k += 1;
        return k;
    }
    if (MAS == PYL_MAS_TSC) return fi - 1 + (frac >= 0.5f ? 1 : 0);
    return fi - 1;
}

// ---- 1. records and keys ------------------------------------------------------
// A record is (x, y, z, weight), or without weights (x, y, z, key's bits): the key then
// needs no second computation.  The first pass forms them from the caller's arrays, on
// positions p + halfcell for the half-cell-shifted grid (SHIFT: the float32 sum the other
// strategies form for the interlaced grid).
struct RsSource {
    const float *pos, *w;
    const float4 *rec;
    float inv, halfcell;
    int dims;
};

template <int MAS>
__device__ __forceinline__ int sd_cell(float p, float inv, int dims)
{
    return wrap_index(sd_first<MAS>(p, inv), dims);
}

template <int MAS>
__device__ __forceinline__ unsigned sd_key(const float4 &r, float inv, int dims)
{
    const unsigned d = (unsigned)dims;
    return ((unsigned)sd_cell<MAS>(r.x, inv, dims) * d + (unsigned)sd_cell<MAS>(r.y, inv, dims)) * d +
           (unsigned)sd_cell<MAS>(r.z, inv, dims);
}

template <int MAS, bool FIRST, bool SHIFT, bool WEIGHTED>
__device__ __forceinline__ float4 rs_record(const RsSource &s, long long i, unsigned &key)
{
    float4 r;
    if (FIRST) {
        r = make_float4(__ldg(s.pos + 3 * i), __ldg(s.pos + 3 * i + 1), __ldg(s.pos + 3 * i + 2),
                        WEIGHTED ? __ldg(s.w + i) : 0.0f);
        if (SHIFT) {
            r.x = __fadd_rn(r.x, s.halfcell);
            r.y = __fadd_rn(r.y, s.halfcell);
            r.z = __fadd_rn(r.z, s.halfcell);
        }
    } else {
        r = __ldg(s.rec + i);
    }
    key = FIRST || WEIGHTED ? sd_key<MAS>(r, s.inv, s.dims) : __float_as_uint(r.w);
    if (FIRST && !WEIGHTED) r.w = __uint_as_float(key);
    return r;
}

// ---- 2. radix sort ----------------------------------------------------------
// Per-tile histogram of one digit, stored digit-major: hist[digit * tiles + tile].
template <int MAS, bool FIRST, bool SHIFT, bool WEIGHTED>
__global__ void __launch_bounds__(RS_THREADS) rs_hist_kernel(RsSource src, long long n, int shift, unsigned tiles,
                                                             unsigned *__restrict__ hist)
{
    __shared__ unsigned h[256];
    if (threadIdx.x < 256) h[threadIdx.x] = 0u;
    __syncthreads();
    const long long base = (long long)blockIdx.x * RS_TILE;
#pragma unroll 4
    for (int r = 0; r < RS_ITEMS; r++) {
        const long long i = base + r * RS_THREADS + threadIdx.x;
        if (i < n) {
            unsigned key;
            rs_record<MAS, FIRST, SHIFT, WEIGHTED>(src, i, key);
            atomicAdd(&h[(key >> shift) & 255u], 1u);
        }
    }
    __syncthreads();
    if (threadIdx.x < 256) hist[(long long)threadIdx.x * tiles + blockIdx.x] = h[threadIdx.x];
}

// Exclusive scan of a block of SCAN_THREADS values (one per thread); returns the
// block total through *total.
__device__ __forceinline__ unsigned block_excl_scan(unsigned v, unsigned *warp_sums, unsigned *total)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    unsigned x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_sums[warp] = x;
    __syncthreads();
    if (warp == 0) {
        unsigned s = lane < nw ? warp_sums[lane] : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned y = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += y;
        }
        if (lane < nw) warp_sums[lane] = s;
    }
    __syncthreads();
    const unsigned prefix = (warp ? warp_sums[warp - 1] : 0u) + x - v;
    if (total) *total = warp_sums[nw - 1];
    __syncthreads();
    return prefix;
}

// Scan phase 1: sum of each SCAN_BLOCK slice.
__global__ void __launch_bounds__(SCAN_THREADS) scan_reduce_kernel(const unsigned *__restrict__ a, long long n,
                                                                   unsigned *__restrict__ partial)
{
    __shared__ unsigned ws[32];
    const long long base = (long long)blockIdx.x * SCAN_BLOCK;
    unsigned s = 0u;
#pragma unroll
    for (int r = 0; r < SCAN_ITEMS; r++) {
        const long long i = base + r * SCAN_THREADS + threadIdx.x;
        if (i < n) s += a[i];
    }
    unsigned tot;
    block_excl_scan(s, ws, &tot);
    if (threadIdx.x == 0) partial[blockIdx.x] = tot;
}

// Scan phase 2: exclusive scan of the partial sums by one block.
__global__ void __launch_bounds__(SCAN_THREADS) scan_partials_kernel(unsigned *__restrict__ partial, long long m)
{
    __shared__ unsigned ws[32];
    __shared__ unsigned carry;
    if (threadIdx.x == 0) carry = 0u;
    __syncthreads();
    for (long long b = 0; b < m; b += SCAN_THREADS) {
        const long long i = b + threadIdx.x;
        const unsigned v = i < m ? partial[i] : 0u;
        unsigned tot;
        const unsigned ex = block_excl_scan(v, ws, &tot);
        if (i < m) partial[i] = carry + ex;
        __syncthreads();
        if (threadIdx.x == 0) carry += tot;
        __syncthreads();
    }
}

// Scan phase 3: exclusive scan of each slice in place, offset by its partial.
__global__ void __launch_bounds__(SCAN_THREADS) scan_apply_kernel(unsigned *__restrict__ a, long long n,
                                                                  const unsigned *__restrict__ partial)
{
    __shared__ unsigned ws[32];
    const long long base = (long long)blockIdx.x * SCAN_BLOCK + (long long)threadIdx.x * SCAN_ITEMS;
    unsigned v[SCAN_ITEMS];
    unsigned s = 0u;
#pragma unroll
    for (int r = 0; r < SCAN_ITEMS; r++) {
        v[r] = base + r < n ? a[base + r] : 0u;
        s += v[r];
    }
    unsigned run = partial[blockIdx.x] + block_excl_scan(s, ws, nullptr);
#pragma unroll
    for (int r = 0; r < SCAN_ITEMS; r++) {
        if (base + r < n) a[base + r] = run;
        run += v[r];
    }
}

// Stable scatter of one tile by one digit.  Warp w holds the tile's elements
// w*256 .. w*256+255 (round r, lane l: element w*256 + r*32 + l), so the order
// (warp, round, lane) is the tile's order.  Each warp ranks its elements with
// its own digit counters (no block barrier), one block scan turns the tile's digit counts
// into each digit's first slot and each warp's first slot within it, and the records go
// from shared memory to global in digit order, coalesced.
// Moves the records, not (key, index) pairs: at 256^3 particles a pass of pairs took 193 us
// (two CTAs per SM of 16 records a thread in registers, a match_any per 32) and the positions'
// gather at the end 294; a pass of records takes 135 us, the first, which forms the keys,
// 195, at 536 and 470 MB: bound by latency at 32 warps per SM, half of them at barriers.
struct RsSmem {
    float4 rec[RS_TILE];
    unsigned short place[RS_TILE];           // element in each slot
    unsigned char digit[RS_TILE];            // its digit
    unsigned short wc[RS_WARPS][256];        // a warp's count of each digit, then its first slot
    unsigned start[256];                     // first slot of each digit
    unsigned gbase[256];                     // global position of the digit's first element
    unsigned ws[32];
};

template <int MAS, bool FIRST, bool SHIFT, bool WEIGHTED>
__global__ void __launch_bounds__(RS_THREADS, 2) rs_scatter_kernel(RsSource src, long long n, int shift, unsigned tiles,
                                                                   const unsigned *__restrict__ goff,
                                                                   float4 *__restrict__ out)
{
    extern __shared__ float4 rs_raw[];
    RsSmem &sm = *reinterpret_cast<RsSmem *>(rs_raw);
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const long long tile0 = (long long)blockIdx.x * RS_TILE;
    const int base = warp * RS_ITEMS * 32 + lane;            // the thread's elements: base + 32 r
    const int cnt = (int)min((long long)RS_TILE, n - tile0);
    for (int i = lane; i < 256; i += 32) sm.wc[warp][i] = 0;
    unsigned dg[RS_ITEMS], rk[RS_ITEMS];
#pragma unroll
    for (int r = 0; r < RS_ITEMS; r++) {
        const int i = base + r * 32;
        dg[r] = 256u;
        if (i < cnt) {
            unsigned key;
            sm.rec[i] = rs_record<MAS, FIRST, SHIFT, WEIGHTED>(src, tile0 + i, key);
            dg[r] = (key >> shift) & 255u;
        }
    }
    __syncwarp();
    const unsigned lt = (1u << lane) - 1u;
#pragma unroll
    for (int r = 0; r < RS_ITEMS; r++) {
        const unsigned d = dg[r];
        unsigned peers = __ballot_sync(0xffffffffu, d < 256u);   // lanes past the end matter to none before it
#pragma unroll
        for (int b = 0; b < 8; b++) {
            const bool one = (d >> b) & 1u;
            const unsigned v = __ballot_sync(0xffffffffu, one);
            peers &= one ? v : ~v;
        }
        const unsigned lrank = __popc(peers & lt);
        const unsigned before = d < 256u ? sm.wc[warp][d] : 0u;
        __syncwarp();
        if (lrank == 0u && d < 256u) sm.wc[warp][d] = (unsigned short)(before + __popc(peers));
        __syncwarp();
        rk[r] = before + lrank;
    }
    __syncthreads();
    // thread t < 256 = digit t: the tile's count, its first slot, each warp's first slot
    unsigned c = 0u;
    if (t < 256)
#pragma unroll
        for (int w = 0; w < RS_WARPS; w++) c += sm.wc[w][t];
    const unsigned s0 = block_excl_scan(c, sm.ws, nullptr);
    if (t < 256) {
        sm.start[t] = s0;
        sm.gbase[t] = goff[(long long)t * tiles + blockIdx.x];
        unsigned run = s0;
#pragma unroll
        for (int w = 0; w < RS_WARPS; w++) {
            const unsigned v = sm.wc[w][t];
            sm.wc[w][t] = (unsigned short)run;
            run += v;
        }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < RS_ITEMS; r++) {
        if (dg[r] < 256u) {
            const unsigned slot = sm.wc[warp][dg[r]] + rk[r];
            sm.place[slot] = (unsigned short)(base + r * 32);
            sm.digit[slot] = (unsigned char)dg[r];
        }
    }
    __syncthreads();
    for (int p = t; p < cnt; p += RS_THREADS) {
        const unsigned d = sm.digit[p];
        out[sm.gbase[d] + ((unsigned)p - sm.start[d])] = sm.rec[sm.place[p]];
    }
}

// ---- 3. column starts ----------------------------------------------------------
constexpr int SD_Z = 8;           // cells along z of a segment

// start[t] = first sorted particle with key >= (t / nseg) * dims + (t % nseg) * SD_Z, for
// t = 0 .. dims^2 * nseg (the last entry: n).  A particle's thread writes the entries after
// the previous particle's segment, up to its own; where these are more than SD_GAP (an
// empty part of the box), it lists them in pieces for sd_gap_kernel instead.  16.8 million
// particles in one octant of 512^3: 27.9 ms with the longest gap in one thread, 0.1 so.  A
// binary search per entry takes 204 us for the 82 of uniform particles at 512^3.
constexpr long long SD_GAP = 256, SD_PIECE = 16384;

struct SdGap {
    unsigned first, len, value, reserved;
};

// The most pieces that all gaps make: one for each gap, each more than SD_GAP entries, and
// one for each full SD_PIECE.
inline long long sd_max_gaps(long long entries) { return entries / SD_GAP + entries / SD_PIECE + 1; }

template <int MAS, bool WEIGHTED>
__global__ void __launch_bounds__(256) sd_start_kernel(RsSource src, long long n, unsigned nseg, long long entries,
                                                       unsigned *__restrict__ start, unsigned *n_gaps,
                                                       SdGap *__restrict__ gaps)
{
    const long long stride = (long long)gridDim.x * blockDim.x;
    const unsigned dims = (unsigned)src.dims;
    for (long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x; j <= n; j += stride) {
        unsigned a = 0, b = 0;
        if (j > 0) rs_record<MAS, false, false, WEIGHTED>(src, j - 1, a);
        if (j < n) rs_record<MAS, false, false, WEIGHTED>(src, j, b);
        long long t = j == 0 ? 0 : (long long)(a / dims) * nseg + a % dims / SD_Z + 1;
        const long long e = j == n ? entries : (long long)(b / dims) * nseg + b % dims / SD_Z;
        if (e - t >= SD_GAP) {
            const long long len = e - t + 1, pieces = (len + SD_PIECE - 1) / SD_PIECE;
            SdGap *g = gaps + atomicAdd(n_gaps, (unsigned)pieces);
            for (long long i = 0; i < pieces; i++)
                g[i] = SdGap{(unsigned)(t + i * SD_PIECE), (unsigned)min(SD_PIECE, len - i * SD_PIECE), (unsigned)j, 0u};
        } else {
            for (; t <= e; t++) start[t] = (unsigned)j;
        }
    }
}

__global__ void __launch_bounds__(256) sd_gap_kernel(const unsigned *__restrict__ n_gaps, const SdGap *__restrict__ gaps,
                                                     unsigned *__restrict__ start)
{
    for (unsigned i = blockIdx.x; i < *n_gaps; i += gridDim.x) {
        const SdGap g = gaps[i];
        for (unsigned t = threadIdx.x; t < g.len; t += blockDim.x) start[g.first + t] = g.value;
    }
}

// ---- 4. crowded cells ----------------------------------------------------------
// A thread of the deposit walks its column one particle at a time.  A cell with a whole
// block (SD_BLOCK records from a multiple of it on) is summed by a warp, or past SD_BIG
// particles by a CTA, beforehand: the S^3 sums of all its particles but the first
// SD_SERIAL, which the walk takes as it finds the cell.  A lane adds every 32nd (256th)
// particle, the lanes and warps are added in a fixed order.  16.8 million particles in 343
// cells of 128^3, CIC: 149 ms with all of them walked, 0.9 ms so.  Uniform particles have no
// such cells and pay the look at every 64th record, 1 % (256^3: 10 us).
constexpr long long SD_BLOCK = 64;
constexpr unsigned SD_SERIAL = 8, SD_BIG = 8192, SD_NONE = 0xffffffffu;

struct SdCrowd {
    unsigned *at;             // by the cell's first whole block: its index in list, else SD_NONE
    unsigned *count;          // cells in list
    uint2 *list;              // records [x, y) of the cell that its sums hold
    float *sums;              // S^3 a cell, [l][m][q]
};

// In the 16 n bytes that the sort leaves unused; none (at null) for fewer than SD_BLOCK.
inline SdCrowd sd_crowd_layout(float4 *spare, long long n)
{
    const long long blocks = n / SD_BLOCK;
    if (!blocks) return SdCrowd{nullptr, nullptr, nullptr, nullptr};
    SdCrowd c;
    c.list = (uint2 *)spare;
    c.sums = (float *)(c.list + blocks);
    c.at = (unsigned *)(c.sums + 64 * blocks);
    c.count = c.at + blocks + 2;
    return c;
}

template <int MAS, bool WEIGHTED>
__global__ void __launch_bounds__(256) sd_crowd_find_kernel(RsSource src, long long n, SdCrowd crowd)
{
    const long long slots = n / SD_BLOCK + 2, stride = (long long)gridDim.x * blockDim.x;
    auto key_of = [&](long long i) {
        unsigned k;
        rs_record<MAS, false, false, WEIGHTED>(src, i, k);
        return k;
    };
    for (long long b = (long long)blockIdx.x * blockDim.x + threadIdx.x; b < slots; b += stride) {
        const long long i = b * SD_BLOCK;
        unsigned at = SD_NONE;
        if (i + SD_BLOCK <= n) {
            const unsigned k = key_of(i);
            if (k == key_of(i + SD_BLOCK - 1) && (b == 0 || k != key_of(i - SD_BLOCK))) {
                long long lo = b == 0 ? 0 : i - SD_BLOCK + 1, hi = i;          // the cell's first particle
                while (lo < hi) {
                    const long long mid = (lo + hi) >> 1;
                    if (key_of(mid) < k) lo = mid + 1; else hi = mid;
                }
                long long end = i + SD_BLOCK, top = n;                          // past its last
                while (end < top) {
                    const long long mid = (end + top) >> 1;
                    if (key_of(mid) <= k) end = mid + 1; else top = mid;
                }
                at = atomicAdd(crowd.count, 1u);
                crowd.list[at] = make_uint2((unsigned)lo + SD_SERIAL, (unsigned)end);
            }
        }
        crowd.at[b] = at;
    }
}

template <int MAS, bool WEIGHTED>
__global__ void __launch_bounds__(256) sd_crowd_sum_kernel(const float4 *__restrict__ spos, float inv, SdCrowd crowd)
{
    constexpr int S = MAS, S3 = S * S * S, WARPS = 8;
    __shared__ float part[WARPS][S3];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned cells = *crowd.count;
    // sums of the records first, first + step, ... below end, added over the warp: lane v % 32
    // has value v in out(v, sum)
    auto warp_sums = [&](unsigned first, unsigned end, unsigned step, auto out) {
        float acc[S3];
#pragma unroll
        for (int v = 0; v < S3; v++) acc[v] = 0.0f;
        for (unsigned long long i = first; i < end; i += step) {
            const float4 r = __ldg(spos + i);
            float cx[S], cy[S], cz[S];
            axis_weights<MAS>(r.x, inv, cx);
            axis_weights<MAS>(r.y, inv, cy);
            axis_weights<MAS>(r.z, inv, cz);
#pragma unroll
            for (int l = 0; l < S; l++)
#pragma unroll
                for (int m = 0; m < S; m++) {
                    float c = __fmul_rn(cx[l], cy[m]);
                    if (WEIGHTED) c = __fmul_rn(c, r.w);
#pragma unroll
                    for (int q = 0; q < S; q++) acc[(l * S + m) * S + q] = __fmaf_rn(c, cz[q], acc[(l * S + m) * S + q]);
                }
        }
#pragma unroll
        for (int v = 0; v < S3; v++) {
            float x = acc[v];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) x = __fadd_rn(x, __shfl_xor_sync(0xffffffffu, x, o));
            if (lane == (v & 31)) out(v, x);
        }
    };
    for (unsigned i = blockIdx.x * WARPS + warp; i < cells; i += gridDim.x * WARPS) {
        const uint2 r = crowd.list[i];
        float *to = crowd.sums + (size_t)i * S3;
        if (r.y - r.x <= SD_BIG) warp_sums(r.x + lane, r.y, 32u, [&](int v, float x) { to[v] = x; });
    }
    for (unsigned i = blockIdx.x; i < cells; i += gridDim.x) {
        const uint2 r = crowd.list[i];
        if (r.y - r.x <= SD_BIG) continue;
        warp_sums(r.x + threadIdx.x, r.y, 32u * WARPS, [&](int v, float x) { part[warp][v] = x; });
        __syncthreads();
        if (threadIdx.x < S3) {
            float x = 0.0f;
            for (int w = 0; w < WARPS; w++) x = __fadd_rn(x, part[w][threadIdx.x]);
            crowd.sums[(size_t)i * S3 + threadIdx.x] = x;
        }
        __syncthreads();
    }
}

// ---- 5. deposit --------------------------------------------------------------------
// A CTA of 16 x 32 threads takes the base columns (X0 - (S-1) + tx, Y0 - (S-1) + ty) and
// `zs` output layers; its output cells are those whose S x S base columns are all its
// own.  Thread (tx, ty) walks its column's particles from base layer z0 - (S-1) on: at
// base layer z they add to the output layers z .. z + S-1 of the S x S columns from it,
// acc[l][m][q] (q turns with z: the loop is unrolled by S).  After layer z its S^2 sums
// are complete and go to shared memory; every few layers (ZB) the CTA meets, and output cell
// (tx, ty) adds those of the columns (tx - l, ty - m).  Outputs are written 8 layers at a
// time, whole sectors.  Two particles ahead are in flight.
// Bound by instructions of half-empty warps (at one particle per cell the fullest of a
// warp's 32 cells holds 3.9: 13 lanes in use, 60 % of issue slots, 30 warps per SM):
// 256^3 TSC of 256^3 particles 0.81 ms; 1.89 ms for a gather that visited S^3 base cells
// for each output cell.  More base layers between meetings leave one CTA per SM (1.26 ms).
constexpr int SDX = 16, SDY = 32;
constexpr int SD_CTA_LAYERS = 32;

template <int MAS>
struct SdShape {
    static constexpr int S = MAS, NT = SDX * SDY, FL = 8, PAD = 4;
    static constexpr int ZB = S == 2 ? 8 : S;               // base layers between two meetings (S divides it)
    static constexpr size_t SMEM = sizeof(float) * (ZB * S * S * NT + FL * (NT + PAD));
};

template <int MAS, bool WEIGHTED, bool CROWD>
__device__ __forceinline__ void sd_walk(const float4 *__restrict__ spos, const unsigned *__restrict__ start, int dims,
                                        int nseg, int zs, float inv, float *__restrict__ out, float scale_h,
                                        const float *__restrict__ scale_d, int fold, const SdCrowd &crowd)
{
    using SH = SdShape<MAS>;
    constexpr int S = SH::S, NT = SH::NT, H = S - 1, FL = SH::FL, PAD = SH::PAD, ZB = SH::ZB;
    extern __shared__ float sd_sm[];
    float *ex = sd_sm;                                       // [ZB][S * S][NT]
    float *res = sd_sm + ZB * S * S * NT;                    // [FL][NT + PAD]
    const int ty = threadIdx.x, tx = threadIdx.y, tid = tx * SDY + ty;
    const int X0 = blockIdx.z * (SDX - H), Y0 = blockIdx.y * (SDY - H);
    const int z0 = blockIdx.x * zs, z1 = min(dims, z0 + zs);
    const int bx = wrap_index(X0 - H + tx, dims), by = wrap_index(Y0 - H + ty, dims);
    const unsigned col = (unsigned)bx * (unsigned)dims + (unsigned)by;
    const float scale = scale_d ? *scale_d : scale_h;
    // first sorted particle of this column at or past layer z
    auto first_from = [&](int z) {
        const unsigned *t = start + (long long)col * nseg + z / SD_Z;
        unsigned lo = t[0], hi = t[1];
        while (lo < hi) {
            const unsigned mid = lo + (hi - lo) / 2;
            if (sd_cell<MAS>(__ldg(spos + mid).z, inv, dims) < z) lo = mid + 1; else hi = mid;
        }
        return lo;
    };
    const unsigned col_end = start[(long long)(col + 1) * nseg];
    const int X = X0 + tx - H, Y = Y0 + ty - H;             // output column (tx, ty >= H)
    const bool live = tx >= H && ty >= H && X < dims && Y < dims;
    float acc[S][S][S];
#pragma unroll
    for (int l = 0; l < S; l++)
#pragma unroll
        for (int m = 0; m < S; m++)
#pragma unroll
            for (int q = 0; q < S; q++) acc[l][m][q] = 0.0f;

    // particles j, j + 1 of the column; layer: base layer of the first (-1: none left)
    unsigned j = 0;
    float4 p = make_float4(0.0f, 0.0f, 0.0f, 0.0f), p2 = p;
    int layer = -1;
    auto layer_of = [&]() { return j < col_end ? sd_cell<MAS>(p.z, inv, dims) : -1; };
    const int layers = z1 - z0 + H;
    for (int k0 = 0; k0 < layers; k0 += ZB) {                // base layers z0 - H + k0 ..
#pragma unroll 1
        for (int g = 0; g < ZB; g += S) {
#pragma unroll
            for (int u = 0; u < S; u++) {
                const int k = k0 + g + u;
                if (k >= layers) break;
                const int zb = wrap_index(z0 - H + k, dims);
                if (k == 0 || zb == 0) {
                    j = first_from(zb);
                    if (j < col_end) p = __ldg(spos + j);
                    if (j + 1 < col_end) p2 = __ldg(spos + j + 1);
                    layer = layer_of();
                }
                // the cell's first SD_SERIAL particles, its sums if it is crowded, the others
                unsigned stop = CROWD && col_end - j > SD_SERIAL ? j + SD_SERIAL : col_end;
                for (;;) {
                    while (layer == zb) {
                        const float4 r = p;
                        p = p2;
                        j++;
                        if (j + 1 < col_end) p2 = __ldg(spos + j + 1);
                        layer = j < stop ? sd_cell<MAS>(p.z, inv, dims) : -1;
                        float cx[S], cy[S], cz[S];
                        axis_weights<MAS>(r.x, inv, cx);
                        axis_weights<MAS>(r.y, inv, cy);
                        axis_weights<MAS>(r.z, inv, cz);
#pragma unroll
                        for (int l = 0; l < S; l++)
#pragma unroll
                            for (int m = 0; m < S; m++) {
                                float c = __fmul_rn(cx[l], cy[m]);
                                if (WEIGHTED) c = __fmul_rn(c, r.w);
#pragma unroll
                                for (int q = 0; q < S; q++) acc[l][m][(u + q) % S] = __fmaf_rn(c, cz[q], acc[l][m][(u + q) % S]);
                            }
                    }
                    if (!CROWD || j != stop || stop == col_end) break;
                    const unsigned first = j - SD_SERIAL;
                    const unsigned at = crowd.at[first / (unsigned)SD_BLOCK + (first % (unsigned)SD_BLOCK != 0u)];
                    const uint2 rest = at != SD_NONE ? crowd.list[at] : make_uint2(0u, 0u);
                    if (rest.x == j) {                       // else the block is another cell's
                        const float *c = crowd.sums + (size_t)at * (S * S * S);
#pragma unroll
                        for (int l = 0; l < S; l++)
#pragma unroll
                            for (int m = 0; m < S; m++)
#pragma unroll
                                for (int q = 0; q < S; q++)
                                    acc[l][m][(u + q) % S] = __fadd_rn(acc[l][m][(u + q) % S], __ldg(c + (l * S + m) * S + q));
                        j = rest.y;
                        if (j < col_end) p = __ldg(spos + j);
                        if (j + 1 < col_end) p2 = __ldg(spos + j + 1);
                    }
                    stop = col_end;
                    layer = layer_of();
                }
                // the layer is complete: its sums out, its place free for layer k + S
                float *e = ex + (g + u) * S * S * NT + tid;
#pragma unroll
                for (int l = 0; l < S; l++)
#pragma unroll
                    for (int m = 0; m < S; m++) {
                        e[(l * S + m) * NT] = acc[l][m][u];
                        acc[l][m][u] = 0.0f;
                    }
            }
        }
        __syncthreads();
        // output layers z0 + k - H of the base layers k since the last meeting; eight of
        // them, or the last ones, are written together
        for (int u = 0; u < ZB; u++) {
            const int zi = k0 + u - H;
            if (zi < 0 || k0 + u >= layers) continue;
            if (live) {
                float v = 0.0f;
                const float *f = ex + u * S * S * NT + tid;
#pragma unroll
                for (int l = 0; l < S; l++)
#pragma unroll
                    for (int m = 0; m < S; m++) v = __fadd_rn(v, f[(l * S + m) * NT - l * SDY - m]);
                res[(zi % FL) * (NT + PAD) + tid] = v;
            }
            if (zi % FL == FL - 1 || z0 + zi + 1 == z1) {    // uniform
                __syncthreads();
                const int zf = zi - zi % FL;
                for (int i = tid; i < NT * FL; i += NT) {
                    const int row = i / FL, dz = i % FL, rx = row / SDY, ry = row % SDY;
                    const int ox = X0 + rx - H, oy = Y0 + ry - H;
                    if (rx < H || ry < H || ox >= dims || oy >= dims || zf + dz > zi) continue;
                    const float v = res[dz * (NT + PAD) + row];
                    float *c = out + ((long long)ox * dims + oy) * dims + z0 + zf + dz;
                    if (fold) *c = __fadd_rn(*c, v);
                    else if (v != 0.0f) *c = __fadd_rn(*c, __fmul_rn(v, scale));
                }
                __syncthreads();
            }
        }
        __syncthreads();                                     // ex is read
    }
}

// Both in one kernel: the look for crowded cells is 2 to 5 % of the uniform deposit.
template <int MAS, bool WEIGHTED>
__global__ void __launch_bounds__(SDX * SDY, MAS == PYL_MAS_PCS ? 1 : 2) sd_deposit_kernel(
    const float4 *__restrict__ spos, const unsigned *__restrict__ start, int dims, int nseg, int zs, float inv,
    float *__restrict__ out, float scale_h, const float *__restrict__ scale_d, int fold, const SdCrowd crowd)
{
    if (crowd.count && *crowd.count)
        sd_walk<MAS, WEIGHTED, true>(spos, start, dims, nseg, zs, inv, out, scale_h, scale_d, fold, crowd);
    else
        sd_walk<MAS, WEIGHTED, false>(spos, start, dims, nseg, zs, inv, out, scale_h, scale_d, fold, crowd);
}

// NGP: a thread per cell finds its particles in the column's segment (cell = key) and
// adds them in index order onto the grid's value (fold), as the serial loop does.  In
// segments of more than 64 particles the end of the cell's is searched too, and their
// number added at once while the sum is a whole number that float32 holds: with a read of
// every particle to find the end, 16.8 million of them in 343 cells of 128^3 took 28.2 ms
// in all for 0.8 (masses: 29.0 for 3.5).
template <bool WEIGHTED>
__global__ void __launch_bounds__(256) sd_ngp_kernel(const float4 *__restrict__ spos, const unsigned *__restrict__ start,
                                                     int dims, int nseg, float inv, long long cells,
                                                     float *__restrict__ out, float scale_h,
                                                     const float *__restrict__ scale_d, int fold)
{
    const long long stride = (long long)gridDim.x * blockDim.x;
    const float scale = scale_d ? *scale_d : scale_h;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < cells; i += stride) {
        const unsigned key = (unsigned)i;
        const int z = (int)(key % (unsigned)dims);
        const unsigned *t = start + (long long)(key / (unsigned)dims) * nseg + z / SD_Z;
        unsigned lo = t[0], hi = t[1];
        const unsigned end = hi;
        auto cell = [&](unsigned j) { return sd_cell<PYL_MAS_NGP>(__ldg(spos + j).z, inv, dims); };
        while (lo < hi) {
            const unsigned mid = lo + (hi - lo) / 2;
            if (cell(mid) < z) lo = mid + 1; else hi = mid;
        }
        if (lo >= end || cell(lo) != z) continue;
        float v = fold ? out[i] : 0.0f;
        if (end - lo > 64u) {                                // a crowded segment
            unsigned stop = lo;
            for (unsigned top = end; stop < top;) {
                const unsigned mid = stop + (top - stop) / 2;
                if (cell(mid) <= z) stop = mid + 1; else top = mid;
            }
            if (WEIGHTED) {
#pragma unroll 32
                for (; lo < stop; lo++) v = __fadd_rn(v, __ldg(&spos[lo].w));
            } else if (v == truncf(v) && (float)(stop - lo) <= 16777216.0f - fabsf(v)) {
                v = __fadd_rn(v, (float)(stop - lo));        // every sum on the way is exact
            } else {
#pragma unroll 1
                for (; lo < stop; lo++) v = __fadd_rn(v, 1.0f);
            }
        } else {
            for (; lo < end && cell(lo) == z; lo++) v = __fadd_rn(v, WEIGHTED ? __ldg(spos + lo).w : 1.0f);
        }
        if (fold) out[i] = v;
        else if (v != 0.0f) out[i] = __fadd_rn(out[i], __fmul_rn(v, scale));
    }
}

inline size_t al(size_t v) { return (v + 255) / 256 * 256; }

struct SortedWs {
    float4 *rec[2];
    unsigned *hist, *partial, *start, *n_gaps;
    SdGap *gaps;
    unsigned tiles;
    long long hist_len, parts, entries;      // entries: dims^2 * segments of a column
    size_t bytes;
};

SortedWs sorted_layout(void *base, long long n, int dims)
{
    SortedWs w;
    w.entries = (long long)dims * dims * ((dims + SD_Z - 1) / SD_Z);
    w.tiles = (unsigned)((n + RS_TILE - 1) / RS_TILE);
    w.hist_len = 256LL * w.tiles;
    w.parts = (w.hist_len + SCAN_BLOCK - 1) / SCAN_BLOCK;
    char *b = (char *)base;
    size_t o = 0;
    w.rec[0] = (float4 *)(b + o); o = al(o + 16 * (size_t)n);
    w.rec[1] = (float4 *)(b + o); o = al(o + 16 * (size_t)n);
    w.hist = (unsigned *)(b + o); o = al(o + 4 * (size_t)w.hist_len);
    w.partial = (unsigned *)(b + o); o = al(o + 4 * (size_t)w.parts);
    w.start = (unsigned *)(b + o); o = al(o + 4 * (size_t)(w.entries + 1));
    w.n_gaps = (unsigned *)(b + o); o = al(o + 4);
    w.gaps = (SdGap *)(b + o); o = al(o + sizeof(SdGap) * (size_t)sd_max_gaps(w.entries + 1));
    w.bytes = o;
    return w;
}

inline unsigned blocks_for(long long n, int threads, int per_sm)
{
    long long b = (n + threads - 1) / threads;
    const long long cap = (long long)num_sms() * per_sm;
    return (unsigned)(b < 1 ? 1 : (b > cap ? cap : b));
}

// One pass of the sort: histogram, scan, scatter.
template <int MAS, bool FIRST, bool SHIFT, bool WEIGHTED>
int sort_pass(const RsSource &src, long long n, int shift, const SortedWs &ws, float4 *out, cudaStream_t st)
{
    rs_hist_kernel<MAS, FIRST, SHIFT, WEIGHTED><<<ws.tiles, RS_THREADS, 0, st>>>(src, n, shift, ws.tiles, ws.hist);
    PYL_LAUNCH_CHECK();
    scan_reduce_kernel<<<(unsigned)ws.parts, SCAN_THREADS, 0, st>>>(ws.hist, ws.hist_len, ws.partial);
    PYL_LAUNCH_CHECK();
    scan_partials_kernel<<<1, SCAN_THREADS, 0, st>>>(ws.partial, ws.parts);
    PYL_LAUNCH_CHECK();
    scan_apply_kernel<<<(unsigned)ws.parts, SCAN_THREADS, 0, st>>>(ws.hist, ws.hist_len, ws.partial);
    PYL_LAUNCH_CHECK();
    auto kern = rs_scatter_kernel<MAS, FIRST, SHIFT, WEIGHTED>;
    PYL_CUDA(ensure_smem(kern, sizeof(RsSmem)));
    kern<<<ws.tiles, RS_THREADS, sizeof(RsSmem), st>>>(src, n, shift, ws.tiles, ws.hist, out);
    PYL_LAUNCH_CHECK();
    return PYL_OK;
}

// One grid: stable radix sort of the (shifted, for SHIFT) particles by cell, column starts,
// deposit.
template <int MAS, bool SHIFT, bool WEIGHTED>
int sorted_pass(const float *pos, const float *w, long long n, float *out, int dims, float inv, float halfcell,
                const SortedWs &ws, float scale_h, const float *scale_d, bool fold, cudaStream_t st)
{
    const long long cells = (long long)dims * dims * dims;
    stage_mark(PYL_STAGE_SORT, true, st);
    int bits = 1;
    while (bits < 32 && (1ull << bits) < (unsigned long long)cells) bits++;
    RsSource src{pos, w, nullptr, inv, halfcell, dims};
    for (int pass = 0; 8 * pass < bits; pass++) {
        float4 *to = ws.rec[pass & 1];
        const int rc = pass == 0 ? sort_pass<MAS, true, SHIFT, WEIGHTED>(src, n, 0, ws, to, st)
                                 : sort_pass<MAS, false, false, WEIGHTED>(src, n, 8 * pass, ws, to, st);
        if (rc) return rc;
        src.rec = to;
    }
    const float4 *spos = src.rec;
    const int nseg = (dims + SD_Z - 1) / SD_Z;
    PYL_CUDA(cudaMemsetAsync(ws.n_gaps, 0, sizeof(unsigned), st));
    sd_start_kernel<MAS, WEIGHTED><<<blocks_for(n + 1, 256, 16), 256, 0, st>>>(src, n, (unsigned)nseg, ws.entries, ws.start,
                                                                               ws.n_gaps, ws.gaps);
    PYL_LAUNCH_CHECK();
    sd_gap_kernel<<<(unsigned)num_sms() * 8, 256, 0, st>>>(ws.n_gaps, ws.gaps, ws.start);
    PYL_LAUNCH_CHECK();
    stage_mark(PYL_STAGE_SORT, false, st);
    stage_mark(PYL_STAGE_DEPOSIT, true, st);
    const int f = fold ? 1 : 0;
    if constexpr (MAS == PYL_MAS_NGP) {
        sd_ngp_kernel<WEIGHTED><<<blocks_for(cells, 256, 32), 256, 0, st>>>(spos, ws.start, dims, nseg, inv, cells, out,
                                                                            scale_h, scale_d, f);
    } else {
        constexpr int H = MAS - 1;
        // layers per CTA: SD_CTA_LAYERS, or fewer (each CTA brings its own S-1 halo layers)
        // until the CTAs are two per SM, below eight until they are one: a thread's walk is as
        // long as its layers (2^20 particles on 32^3, CIC, eight 221 us, two 138)
        const unsigned gy = (unsigned)((dims + SDY - H - 1) / (SDY - H)), gx = (unsigned)((dims + SDX - H - 1) / (SDX - H));
        int zs = SD_CTA_LAYERS;
        while (zs > 2 && (long long)gx * gy * ((dims + zs - 1) / zs) < (zs > 8 ? 2LL : 1LL) * num_sms()) zs /= 2;
        constexpr size_t smem = SdShape<MAS>::SMEM;
        const SdCrowd crowd = sd_crowd_layout(spos == ws.rec[0] ? ws.rec[1] : ws.rec[0], n);
        if (crowd.at) {
            PYL_CUDA(cudaMemsetAsync(crowd.count, 0, sizeof(unsigned), st));
            sd_crowd_find_kernel<MAS, WEIGHTED><<<blocks_for(n / SD_BLOCK + 2, 256, 16), 256, 0, st>>>(src, n, crowd);
            PYL_LAUNCH_CHECK();
            sd_crowd_sum_kernel<MAS, WEIGHTED><<<(unsigned)num_sms() * 4, 256, 0, st>>>(spos, inv, crowd);
            PYL_LAUNCH_CHECK();
        }
        auto kern = sd_deposit_kernel<MAS, WEIGHTED>;
        PYL_CUDA(ensure_smem(kern, smem));
        kern<<<dim3((unsigned)((dims + zs - 1) / zs), gy, gx), dim3(SDY, SDX), smem, st>>>(
            spos, ws.start, dims, nseg, zs, inv, out, scale_h, scale_d, f, crowd);
    }
    PYL_LAUNCH_CHECK();
    stage_mark(PYL_STAGE_DEPOSIT, false, st);
    return PYL_OK;
}

template <int MAS>
int sorted_run(const float *pos, const float *w, long long n, float *grid, float *grid2, int dims, float inv,
               float halfcell, void *workspace, float scale_h, const float *scale_d, bool fold, cudaStream_t st)
{
    const SortedWs ws = sorted_layout(workspace, n, dims);
    auto plain = w ? sorted_pass<MAS, false, true> : sorted_pass<MAS, false, false>;
    auto shifted = w ? sorted_pass<MAS, true, true> : sorted_pass<MAS, true, false>;
    const int rc = plain(pos, w, n, grid, dims, inv, halfcell, ws, scale_h, scale_d, fold, st);
    if (rc || !grid2) return rc;
    return shifted(pos, w, n, grid2, dims, inv, halfcell, ws, scale_h, scale_d, fold, st);
}

}  // namespace

bool sorted_supported(long long n, int dims)
{
    return n >= 0 && n < 0xFFFFFFFFLL && dims >= 1 && (long long)dims * dims * dims <= 0xFFFFFFFFLL;
}

size_t sorted_workspace_bytes(long long n, int dims)
{
    return sorted_layout(nullptr, n, dims).bytes;
}

int launch_sorted(int mas, const float *pos, const float *w, long long n, float *grid, float *grid2, int dims,
                  float inv, float halfcell, void *workspace, float scale_h, const float *scale_d, bool fold,
                  cudaStream_t st)
{
    if (!sorted_supported(n, dims)) {
        set_error("sorted strategy: needs dims^3 <= 2^32 and fewer than 2^32 particles");
        return PYL_ERR_UNSUPPORTED;
    }
    if (n == 0) return PYL_OK;
    switch (mas) {
        case PYL_MAS_NGP: return sorted_run<PYL_MAS_NGP>(pos, w, n, grid, grid2, dims, inv, halfcell, workspace,
                                                         scale_h, scale_d, fold, st);
        case PYL_MAS_CIC: return sorted_run<PYL_MAS_CIC>(pos, w, n, grid, grid2, dims, inv, halfcell, workspace,
                                                         scale_h, scale_d, fold, st);
        case PYL_MAS_TSC: return sorted_run<PYL_MAS_TSC>(pos, w, n, grid, grid2, dims, inv, halfcell, workspace,
                                                         scale_h, scale_d, fold, st);
        case PYL_MAS_PCS: return sorted_run<PYL_MAS_PCS>(pos, w, n, grid, grid2, dims, inv, halfcell, workspace,
                                                         scale_h, scale_d, fold, st);
    }
    set_error("sorted strategy: bad MAS");
    return PYL_ERR_INVALID;
}

}  // namespace pyl

// The deposit stages no particles any more: every limit gives the same sums.
extern "C" int pyl_sorted_set_stage_limit(int max_particles)
{
    PYL_CHECK_ARG(max_particles <= 1024, "max_particles above the stage capacity (1024)");
    return PYL_OK;
}
