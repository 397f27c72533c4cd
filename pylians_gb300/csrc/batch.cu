// Batched realizations: one persistent launch deposits a whole batch of
// particle sets with uneven particle counts, grid sizes, MAS and interlacing.
//
// Work is a device list of items (realization, first particle, count); the
// CTAs of the persistent kernel take items from a device counter until the
// list is exhausted, so long and short realizations balance across SMs.  Each
// item deposits its particles with red.global.add into its realization's
// grid(s) (grids of <= 256^3 cells stay resident in L2 while their items run),
// scaled by dims^3 / N so that grids pre-filled with -1 end as the overdensity
// delta = n/mean - 1 (library/Pk_library/Pk_snapshot.py:70-88).  The per-particle
// arithmetic is the one of mas.cu (MAS_library.pyx:123-545).
#include <cuda_runtime.h>

#include <algorithm>
#include <string>

#include "common.cuh"
#include "deposit.cuh"

namespace pyl {
namespace {

template <int MAS>
__device__ __forceinline__ void ba_deposit(const float *p, const pyl_batch_real &r, float shift, float *out)
{
    constexpr int S = MAS == PYL_MAS_NGP ? 1 : MAS;
    const int dims = r.dims;
    const long long d = dims;
    float C[3][S];
    int idx[3][S];
#pragma unroll
    for (int a = 0; a < 3; a++) {
        const int f = axis_weights<MAS>(__fadd_rn(p[a], shift), r.inv, C[a]);
#pragma unroll
        for (int j = 0; j < S; j++) idx[a][j] = wrap_index((long long)f + j, dims);
    }
#pragma unroll
    for (int l = 0; l < S; l++)
#pragma unroll
        for (int m = 0; m < S; m++) {
            const float c01 = __fmul_rn(C[0][l], C[1][m]);
            const long long row = ((long long)idx[0][l] * d + idx[1][m]) * d;
#pragma unroll
            for (int q = 0; q < S; q++)
                atomicAdd(out + row + idx[2][q], __fmul_rn(__fmul_rn(c01, C[2][q]), r.scale));
        }
}

__global__ void __launch_bounds__(256) batch_deposit_kernel(const pyl_batch_real *__restrict__ reals,
                                                            const pyl_batch_item *__restrict__ items,
                                                            int n_items, unsigned *counter)
{
    __shared__ int cur;
    for (;;) {
        if (threadIdx.x == 0) cur = (int)atomicAdd(counter, 1u);
        __syncthreads();
        const int it = cur;
        __syncthreads();
        if (it >= n_items) break;
        const pyl_batch_item item = items[it];
        const pyl_batch_real r = reals[item.real];
        for (long long i = item.first + threadIdx.x; i < item.first + item.count; i += blockDim.x) {
            const float p[3] = {__ldg(r.pos + 3 * i), __ldg(r.pos + 3 * i + 1), __ldg(r.pos + 3 * i + 2)};
            for (int g = 0; g < (r.grid_interlaced ? 2 : 1); g++) {
                float *out = g ? r.grid_interlaced : r.grid;
                const float sh = g ? r.halfcell : 0.0f;
                switch (r.mas) {
                    case PYL_MAS_NGP: ba_deposit<PYL_MAS_NGP>(p, r, sh, out); break;
                    case PYL_MAS_CIC: ba_deposit<PYL_MAS_CIC>(p, r, sh, out); break;
                    case PYL_MAS_TSC: ba_deposit<PYL_MAS_TSC>(p, r, sh, out); break;
                    default:          ba_deposit<PYL_MAS_PCS>(p, r, sh, out); break;
                }
            }
        }
    }
}

__global__ void __launch_bounds__(256) fill_value_kernel(float *g, long long n, float v)
{
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) g[i] = v;
}

__global__ void __launch_bounds__(256) scale_value_kernel(float *g, long long n, float f)
{
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) g[i] = __fmul_rn(g[i], f);
}

// ---- batched tiled path ------------------------------------------------------
// The same binning as pyl_ma's TILED strategy, over all realizations of a batch
// at once: every realization's grid is cut into 32^3-cell bins, numbered
// tile_base[r] + (tx*nt + ty)*nt + tz in one global list.
//   bt_count:   persistent over the items: per-item shared-memory histogram of
//               its realization's bins, flushed into the global bin counts;
//   bt_scan:    exclusive scan of the counts (bin offsets and cursors);
//   bt_place:   persistent over the items: per 4096-particle batch, shared-memory
//               ranks per bin, one global atomic per bin to reserve a range,
//               records (x, y, z, 1) written into their bins' ranges;
//   bt_list:    the deposit's work list: every bin of every grid (the
//               interlaced one apart), those of more than a quarter of an SM's share
//               of all corner additions in parts of that size (BinShare), so that
//               the crowded bins of a small grid (7.9 million particles in the 8 bins
//               of 64^3) do not keep a few SMs busy after all others are done;
//   bt_deposit: persistent over the parts: 10.22 fixed-point shared-memory
//               accumulation of the bin (+ halo) for its realization's MAS,
//               red.global into the realization's grid scaled to the overdensity.
//               24 realizations up to 256^3: 3.0 ms with whole bins (2.3 ms of it
//               one bin of a 64^3 grid), 1.9 ms in parts.
constexpr int BT_MAX_TILES = 4096;        // bins per realization (dims <= 512)
// Count and placement: threads per CTA, CTAs per SM.  One CTA of 1024 threads (its 50
// registers leave no room for a second) stood still at every barrier and reservation: 24
// realizations of 70 million particles 823 us for the placement, 236 for the count; three
// of 512 threads 733 and 202 (five of 256: 826 and 242).  The placement is bound by the
// random shared-memory accesses of its sort (60 % of the wavefronts) and by barriers.
constexpr int BT_THREADS = 512, BT_CTAS = 3;
constexpr int BT_BATCH = 4 * BT_THREADS;     // placement batch (particles)

// Count and placement take an item in `split` parts while the items are fewer than two per
// resident CTA (a CTA of 512 threads takes an item of 65536 particles in 32 batches): two
// realizations of 3 million particles (92 items) 222 us for the placement and 54 for the
// count with whole items, 63 and 25 in parts (CTAs of 1024 threads: 89 and 27).
constexpr int BT_MAX_SPLIT = 16;

inline int bt_split(int n_items)
{
    const int units = 2 * BT_CTAS * num_sms();
    return std::max(1, std::min(BT_MAX_SPLIT, (units + n_items - 1) / n_items));
}

// The unit-th part of all items, of whole groups of four particles.
__device__ __forceinline__ pyl_batch_item bt_part(const pyl_batch_item *__restrict__ items, unsigned unit, unsigned split)
{
    pyl_batch_item it = items[unit / split];
    const unsigned part = unit % split;
    const unsigned long long quads = ((unsigned long long)it.count + 3) / 4;
    const unsigned a = (unsigned)min(4 * (quads * part / split), (unsigned long long)it.count);
    const unsigned b = (unsigned)min(4 * (quads * (part + 1) / split), (unsigned long long)it.count);
    it.first += a;
    it.count = b - a;
    return it;
}

__device__ __forceinline__ int bt_nt(int dims) { return (dims + TB - 1) / TB; }

template <int MAS>
__device__ __forceinline__ int bt_key(const float *p, float inv, int dims, int nt)
{
    const int cx = wrap_index(axis_first<MAS>(p[0], inv), dims) / TB;
    const int cy = wrap_index(axis_first<MAS>(p[1], inv), dims) / TB;
    const int cz = wrap_index(axis_first<MAS>(p[2], inv), dims) / TB;
    return (cx * nt + cy) * nt + cz;
}

__device__ __forceinline__ int bt_key_rt(int mas, const float *p, float inv, int dims, int nt)
{
    switch (mas) {
        case PYL_MAS_NGP: return bt_key<PYL_MAS_NGP>(p, inv, dims, nt);
        case PYL_MAS_CIC: return bt_key<PYL_MAS_CIC>(p, inv, dims, nt);
        case PYL_MAS_TSC: return bt_key<PYL_MAS_TSC>(p, inv, dims, nt);
        default:          return bt_key<PYL_MAS_PCS>(p, inv, dims, nt);
    }
}

// Positions of particles q .. q+3 (q a multiple of 4, so 48 bytes from a 16-byte
// aligned base): three 16-byte loads instead of twelve 4-byte ones; lanes of a
// warp read consecutive 48-byte groups.  Particles at or past `end` are not read.
__device__ __forceinline__ void load_quad(const float *pos, long long q, long long end, bool vec, float p[4][3])
{
    if (vec && q + 4 <= end) {
        const float4 *g = reinterpret_cast<const float4 *>(pos + 3 * q);
        const float4 a = __ldg(g), b = __ldg(g + 1), c = __ldg(g + 2);
        p[0][0] = a.x; p[0][1] = a.y; p[0][2] = a.z;
        p[1][0] = a.w; p[1][1] = b.x; p[1][2] = b.y;
        p[2][0] = b.z; p[2][1] = b.w; p[2][2] = c.x;
        p[3][0] = c.y; p[3][1] = c.z; p[3][2] = c.w;
    } else {
#pragma unroll
        for (int u = 0; u < 4; u++)
            if (q + u < end) {
                p[u][0] = __ldg(pos + 3 * (q + u));
                p[u][1] = __ldg(pos + 3 * (q + u) + 1);
                p[u][2] = __ldg(pos + 3 * (q + u) + 2);
            }
    }
}

__host__ __device__ inline unsigned bt_corners(int mas)
{
    const unsigned s = mas == PYL_MAS_NGP ? 1u : (unsigned)mas;
    return s * s * s;
}

__global__ void __launch_bounds__(BT_THREADS, BT_CTAS) bt_count_kernel(const pyl_batch_real *__restrict__ reals,
                                                        const pyl_batch_item *__restrict__ items, int n_items, int split,
                                                        const unsigned *__restrict__ tile_base,
                                                        unsigned *__restrict__ counts, unsigned long long *adds,
                                                        unsigned *counter)
{
    __shared__ unsigned h[BT_MAX_TILES];
    __shared__ int cur;
    for (;;) {
        if (threadIdx.x == 0) cur = (int)atomicAdd(counter, 1u);
        __syncthreads();
        const int it = cur;
        if ((unsigned)it >= (unsigned)n_items * (unsigned)split) break;
        const pyl_batch_item item = bt_part(items, (unsigned)it, (unsigned)split);
        const pyl_batch_real r = reals[item.real];
        const int nt = bt_nt(r.dims), ntiles = nt * nt * nt;
        if (ntiles > BT_MAX_TILES) {                   // dims > 512: not binned here
            __syncthreads();
            continue;
        }
        for (int t = threadIdx.x; t < ntiles; t += blockDim.x) h[t] = 0u;
        __syncthreads();
        const long long end = item.first + item.count;
        const bool vec = (item.first & 3) == 0 && (((uintptr_t)r.pos) & 15) == 0;
        for (long long q = item.first + 4 * (long long)threadIdx.x; q < end; q += 4 * (long long)blockDim.x) {
            float p[4][3];
            load_quad(r.pos, q, end, vec, p);
#pragma unroll
            for (int u = 0; u < 4; u++)
                if (q + u < end) atomicAdd(h + bt_key_rt(r.mas, p[u], r.inv, r.dims, nt), 1u);
        }
        __syncthreads();
        if (threadIdx.x == 0 && item.count)
            atomicAdd(adds, (unsigned long long)item.count * bt_corners(r.mas) * (r.grid_interlaced ? 2u : 1u));
        const unsigned base = tile_base[item.real];
        for (int t = threadIdx.x; t < ntiles; t += blockDim.x)
            if (h[t]) atomicAdd(counts + base + t, h[t]);
        __syncthreads();
    }
}

// Parts of a batch of `adds` corner additions: at most BT_PARTS_PER_SM an SM, none below
// PART_ADDS.  Bins of less than two PART_ADDS stay whole: their longer part takes as long,
// and the words come on top (100 realizations of 20,000 particles on 32^3, PCS interlaced: 425
// us in parts, 368 whole, 383 before bins were divided).
constexpr unsigned BT_PARTS_PER_SM = 4;

__device__ __forceinline__ unsigned bt_part_len(unsigned long long adds, unsigned sms, int mas)
{
    const unsigned long long share = adds / (BT_PARTS_PER_SM * sms);
    return (unsigned)((share > PART_ADDS ? share : PART_ADDS) / bt_corners(mas)) + 1u;
}

// The most parts that a batch can have (its grids' bins, and the shares that all additions
// make, rounded up), and the most bins in parts: each has more than a share of all
// additions, and more than PART_ADDS of them, PART_ADDS / 64 particles at least.
inline size_t bt_max_parts(unsigned total_tiles)
{
    return 2 * (size_t)total_tiles + (BT_PARTS_PER_SM + 1) * (size_t)num_sms();
}
inline size_t bt_max_shared(unsigned total_tiles, long long total_particles)
{
    return std::min({(size_t)BT_PARTS_PER_SM * num_sms(), 2 * (size_t)total_tiles,
                     2 * (size_t)(total_particles / (PART_ADDS / 64))});
}

struct BtPart {
    unsigned tile, real;
    unsigned first, len;        // records of the bin
    unsigned inter;             // 1: the interlaced grid
    unsigned parts, shared;     // of the bin; with several, the index of their BinShare
    unsigned reserved;
};

// Words of a BinShare: the largest bin (PCS, interlaced).
constexpr size_t BT_SHARE_CELLS = FxShape<PYL_MAS_PCS, true>::CELLS;

// Realization of a bin: the last one with tile_base <= t.
__device__ __forceinline__ int bt_real_of(const unsigned *__restrict__ tile_base, int n_reals, unsigned t)
{
    int lo = 0, hi = n_reals;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (tile_base[mid] <= t) lo = mid; else hi = mid;
    }
    return lo;
}

// Parts of a bin of each grid of its realization, by the counts and the sum of additions.
struct BtBin {
    unsigned count, real, len, grids, parts;
};

__device__ __forceinline__ BtBin bt_bin(const pyl_batch_real *__restrict__ reals, int n_reals,
                                        const unsigned *__restrict__ tile_base, unsigned total_tiles,
                                        const unsigned *__restrict__ counts, unsigned long long adds, unsigned sms, unsigned t)
{
    if (t >= total_tiles) return BtBin{0u, 0u, 1u, 1u, 0u};
    const unsigned c = counts[t], real = (unsigned)bt_real_of(tile_base, n_reals, t);
    const unsigned len = bt_part_len(adds, sms, reals[real].mas);
    const bool whole = (unsigned long long)c * bt_corners(reals[real].mas) < 2 * PART_ADDS;
    return BtBin{c, real, len, reals[real].grid_interlaced ? 2u : 1u, whole ? (c != 0u) : c / len + (c % len != 0u)};
}

// CTA 0: exclusive scan of n counts into offsets[0..n] and cursor[0..n).  CTA b > 0: the
// list entries of its 1024 bins, into entries[b - 1].
__global__ void __launch_bounds__(1024) bt_scan_kernel(const pyl_batch_real *__restrict__ reals, int n_reals,
                                                       const unsigned *__restrict__ tile_base,
                                                       const unsigned *__restrict__ counts, unsigned n,
                                                       const unsigned long long *__restrict__ adds, unsigned sms,
                                                       unsigned *__restrict__ offsets, unsigned *__restrict__ cursor,
                                                       unsigned *__restrict__ entries)
{
    if (blockIdx.x) {
        __shared__ unsigned sum;
        if (threadIdx.x == 0) sum = 0u;
        __syncthreads();
        const BtBin b = bt_bin(reals, n_reals, tile_base, n, counts, *adds, sms, (blockIdx.x - 1) * 1024 + threadIdx.x);
        const unsigned w = __reduce_add_sync(0xffffffffu, b.parts * b.grids);
        if ((threadIdx.x & 31) == 0 && w) atomicAdd(&sum, w);
        __syncthreads();
        if (threadIdx.x == 0) entries[blockIdx.x - 1] = sum;
        return;
    }
    __shared__ unsigned long long part[1024];
    const unsigned per = (n + blockDim.x - 1) / blockDim.x;
    const unsigned b = threadIdx.x * per, e = min(n, b + per);
    unsigned long long sum = 0;
    for (unsigned i = b; i < e; i++) sum += counts[i];
    part[threadIdx.x] = sum;
    __syncthreads();
    for (int off = 1; off < (int)blockDim.x; off <<= 1) {
        const unsigned long long v = threadIdx.x >= (unsigned)off ? part[threadIdx.x - off] : 0ull;
        __syncthreads();
        part[threadIdx.x] += v;
        __syncthreads();
    }
    unsigned long long run = part[threadIdx.x] - sum;
    for (unsigned i = b; i < e; i++) {
        offsets[i] = (unsigned)run;
        cursor[i] = (unsigned)run;
        run += counts[i];
    }
    if (threadIdx.x == blockDim.x - 1) offsets[n] = (unsigned)part[threadIdx.x];
}

// The work list, in bin order: a bin's parts of the plain grid, then of the interlaced one.
// Each grid's bin in parts takes a BinShare.  (In any order, 24 realizations took 2 % longer:
// neighbouring bins add to the same cells.)  With kernels of their own for the sum of
// additions, the parts of each bin and their scan, four realizations of 512^3 took 27 us
// longer, one of 64^3 8.
__global__ void __launch_bounds__(1024) bt_list_kernel(const pyl_batch_real *__restrict__ reals, int n_reals,
                                                       const unsigned *__restrict__ tile_base, unsigned total_tiles,
                                                       const unsigned *__restrict__ counts,
                                                       const unsigned long long *__restrict__ adds, unsigned sms,
                                                       const unsigned *__restrict__ entries, unsigned max_parts,
                                                       unsigned max_shared, unsigned *n_parts, unsigned *shared_count,
                                                       BtPart *__restrict__ list)
{
    __shared__ unsigned before, warps[32];
    const unsigned t = blockIdx.x * 1024 + threadIdx.x, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) before = 0u;
    __syncthreads();
    unsigned sum = 0u;
    for (unsigned i = threadIdx.x; i < blockIdx.x; i += 1024) sum += entries[i];
    if (sum) atomicAdd(&before, sum);
    const BtBin bin = bt_bin(reals, n_reals, tile_base, total_tiles, counts, *adds, sms, t);
    const unsigned mine = bin.parts * bin.grids;
    unsigned end = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned v = __shfl_up_sync(0xffffffffu, end, o);
        if (lane >= (unsigned)o) end += v;
    }
    if (lane == 31u) warps[warp] = end;
    __syncthreads();
    unsigned first = before + end - mine;
    for (unsigned w = 0; w < warp; w++) first += warps[w];
    if (threadIdx.x == 1023u && blockIdx.x + 1 == gridDim.x) *n_parts = first + mine;
    unsigned shared = 0u;
    if (bin.parts > 1u) shared = atomicAdd(shared_count, bin.grids);
    // no BinShare left (bt_max_shared has one for every bin in parts, unless the items hold more
    // particles than the caller's total): whole bins, the other parts empty
    const bool whole = bin.parts > 1u && shared + bin.grids > max_shared;
    if (bin.parts == 1u)
        for (unsigned g = 0; g < bin.grids && first + g < max_parts; g++)
            list[first + g] = BtPart{t, bin.real, 0u, bin.count, g, 1u, 0u, 0u};
    for (unsigned many = __ballot_sync(0xffffffffu, bin.parts > 1u); many; many &= many - 1u) {
        const int s = __ffs(many) - 1;                       // bins in parts: a warp for each
        const unsigned b = __shfl_sync(0xffffffffu, first, s), p = __shfl_sync(0xffffffffu, bin.parts, s);
        const unsigned n = __shfl_sync(0xffffffffu, mine, s), r = __shfl_sync(0xffffffffu, bin.real, s);
        const unsigned c = __shfl_sync(0xffffffffu, bin.count, s), l = __shfl_sync(0xffffffffu, bin.len, s);
        const unsigned sh = __shfl_sync(0xffffffffu, shared, s), tile = __shfl_sync(0xffffffffu, t, s);
        const unsigned w = __shfl_sync(0xffffffffu, whole ? 1u : 0u, s);
        for (unsigned i = lane; i < n && b + i < max_parts; i += 32) {
            const unsigned from = (i % p) * l, g = i / p;
            list[b + i] = w ? BtPart{tile, r, 0u, from ? 0u : c, g, 1u, 0u, 0u}
                            : BtPart{tile, r, from, min(l, c - from), g, p, sh + g, 0u};
        }
    }
}

// Zeroes the words of the BinShares in use (blockIdx.y), gridDim.x CTAs each.
__global__ void __launch_bounds__(256) bt_share_zero_kernel(const unsigned *__restrict__ shared_count,
                                                            unsigned long long *__restrict__ share)
{
    if (blockIdx.y >= *shared_count) return;
    unsigned long long *z = share + blockIdx.y * BT_SHARE_CELLS;
    for (size_t i = blockIdx.x * blockDim.x + threadIdx.x; i < BT_SHARE_CELLS; i += gridDim.x * blockDim.x) z[i] = 0ull;
}

// Exclusive scan of v[0..n) in place (each thread n / blockDim.x consecutive entries);
// warp_tot: 32 entries of scratch.  All threads call it.
__device__ __forceinline__ void bt_block_scan(unsigned *v, int n, unsigned *warp_tot)
{
    const int t = threadIdx.x, lane = t & 31, w = t >> 5, nw = (blockDim.x + 31) >> 5;
    const int per = (n + blockDim.x - 1) / blockDim.x, first = per * t, last = min(n, first + per);
    unsigned tot = 0;
    for (int i = first; i < last; i++) tot += v[i];
    unsigned inc = tot;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
    }
    if (lane == 31) warp_tot[w] = inc;
    __syncthreads();
    if (w == 0) {
        const unsigned wt = lane < nw ? warp_tot[lane] : 0u;
        unsigned wi = wt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned y = __shfl_up_sync(0xffffffffu, wi, o);
            if (lane >= o) wi += y;
        }
        if (lane < nw) warp_tot[lane] = wi - wt;
    }
    __syncthreads();
    unsigned run = inc - tot + warp_tot[w];
    for (int i = first; i < last; i++) {
        const unsigned x = v[i];
        v[i] = run;
        run += x;
    }
    __syncthreads();
}

// Per BT_BATCH particles of an item: ranks per bin from shared-memory counters,
// one global atomic per bin touched reserves its run in the bin's range, the batch
// is sorted by bin in shared memory, and the runs are written out coalesced
// (consecutive threads, consecutive slots of a run).
constexpr size_t BT_PLACE_SMEM = sizeof(unsigned) * 2 * BT_MAX_TILES + sizeof(float4) * BT_BATCH +
                                 sizeof(unsigned short) * BT_BATCH;

__global__ void __launch_bounds__(BT_THREADS, BT_CTAS) bt_place_kernel(const pyl_batch_real *__restrict__ reals,
                                                        const pyl_batch_item *__restrict__ items, int n_items, int split,
                                                        const unsigned *__restrict__ tile_base,
                                                        unsigned *__restrict__ cursor, unsigned n_total,
                                                        float4 *__restrict__ rec, unsigned *counter)
{
    extern __shared__ __align__(16) unsigned char praw[];
    unsigned *bcnt = (unsigned *)praw, *gbase = bcnt + BT_MAX_TILES;
    float4 *stage = (float4 *)(gbase + BT_MAX_TILES);
    unsigned short *skey = (unsigned short *)(stage + BT_BATCH);
    __shared__ unsigned wt[32];
    __shared__ int cur;
    constexpr int U = BT_BATCH / BT_THREADS;
    static_assert(U == 4, "four particles per thread and batch");
    static_assert(BT_MAX_TILES <= 65536, "bin keys held as 16 bits");
    for (;;) {
        if (threadIdx.x == 0) cur = (int)atomicAdd(counter, 1u);
        __syncthreads();
        const int it = cur;
        if ((unsigned)it >= (unsigned)n_items * (unsigned)split) break;
        const pyl_batch_item item = bt_part(items, (unsigned)it, (unsigned)split);
        const pyl_batch_real r = reals[item.real];
        const int nt = bt_nt(r.dims), ntiles = nt * nt * nt;
        const unsigned base = tile_base[item.real];
        const long long end = item.first + item.count;
        if (ntiles > BT_MAX_TILES) {
            __syncthreads();
            continue;
        }
        const bool vec = (item.first & 3) == 0 && (((uintptr_t)r.pos) & 15) == 0;
        for (long long s0 = item.first; s0 < end; s0 += BT_BATCH) {
            const int c = (int)min((long long)BT_BATCH, end - s0);
            for (int t = threadIdx.x; t < ntiles; t += blockDim.x) bcnt[t] = 0u;
            __syncthreads();
            float4 v[U];
            int key[U];
            unsigned rank[U];
            // thread t takes particles s0 + 4t .. s0 + 4t + 3 (BT_BATCH = 4 BT_THREADS)
            float p[U][3];
            load_quad(r.pos, s0 + 4 * threadIdx.x, end, vec, p);
#pragma unroll
            for (int u = 0; u < U; u++) {
                const long long i = s0 + 4 * threadIdx.x + u;
                key[u] = -1;
                if (i < end) {
                    v[u] = make_float4(p[u][0], p[u][1], p[u][2], 1.0f);
                    key[u] = bt_key_rt(r.mas, p[u], r.inv, r.dims, nt);
                    rank[u] = atomicAdd(bcnt + key[u], 1u);
                }
            }
            __syncthreads();
            for (int t = threadIdx.x; t < ntiles; t += blockDim.x)
                if (bcnt[t]) gbase[t] = atomicAdd(cursor + base + t, bcnt[t]);
            __syncthreads();
            bt_block_scan(bcnt, ntiles, wt);                   // bcnt: the batch's run starts
#pragma unroll
            for (int u = 0; u < U; u++)
                if (key[u] >= 0) {
                    const unsigned slot = bcnt[key[u]] + rank[u];
                    stage[slot] = v[u];
                    skey[slot] = (unsigned short)key[u];
                }
            __syncthreads();
            for (int sidx = threadIdx.x; sidx < c; sidx += blockDim.x) {
                const unsigned k = skey[sidx];
                const unsigned dst = gbase[k] + ((unsigned)sidx - bcnt[k]);
                if (dst < n_total) rec[dst] = stage[sidx];
            }
            __syncthreads();
        }
        __syncthreads();
    }
}

// ---- bins in parts ---------------------------------------------------------------
// A bin whose records go to several CTAs keeps one 64-bit fixed-point word per cell in
// global memory: every CTA adds its cells there, and the last one to arrive converts
// the sums, so the grid gets the same value as from one CTA (integer sums do not depend
// on the order or the grouping of the adds; 64 bits cannot wrap).
struct BinShare {
    unsigned long long *acc;     // the bin's words (zeroed before the launch)
    unsigned *done;              // parts that have arrived (zeroed before the launch)
    unsigned parts;              // of the bin; 1: acc and done are not used
};

__device__ __forceinline__ void share_add(const BinShare &sh, const unsigned *smw, int cells)
{
    for (int c = threadIdx.x; c < cells; c += blockDim.x) {
        const unsigned w = smw[c];
        if (w != 0u) atomicAdd(sh.acc + c, (unsigned long long)w);
    }
}

// All threads, after share_add (or instead of it: a part summed in float32 goes to the
// grid by itself): true in the CTA that arrives last, which then sees every part's words.
__device__ __forceinline__ bool share_arrive(const BinShare &sh)
{
    __threadfence();
    __syncthreads();
    const bool last = threadIdx.x == 0 && atomicAdd(sh.done, 1u) + 1u == sh.parts;
    const bool mine = __syncthreads_or((int)last);
    __threadfence();
    return mine;
}

template <int MAS>
__device__ __forceinline__ float share_value(const BinShare &sh, int c)
{
    const float v = __ull2float_rn(__ldcg(sh.acc + c));
    return MAS == PYL_MAS_NGP ? v : __fmul_rn(v, FX_INV);
}

// Deposit of the records [begin, end) of one bin of realization r onto its plain grid or
// (PASS 1) its interlaced one; MAS and interlacing (the shape of the bin's cells) as
// template parameters; fixed point with the float32 redo of mode 1.
template <int MAS, bool INTER>
__device__ __forceinline__ void bt_deposit_bin(unsigned *smw, const float4 *__restrict__ rec, unsigned begin,
                                               unsigned end, const pyl_batch_real &r, const int *o, int pass,
                                               const BinShare &sh)
{
    using FS = FxShape<MAS, INTER>;
    constexpr int S = Support<MAS>::S, E = FS::E, CELLS = FS::CELLS;
    float *facc = (float *)smw;
    const long long d = r.dims;
    for (int mode = 0; mode < 2; mode++) {
        uint4 *z4 = (uint4 *)smw;
        for (int c = threadIdx.x; c < FS::SMEM / 16; c += blockDim.x) z4[c] = make_uint4(0u, 0u, 0u, 0u);
        __syncthreads();
        unsigned bad = 0u, seen = 0u;
        for (unsigned i = begin + threadIdx.x; i < end; i += blockDim.x) {
            const float4 p = rec[i];
            float C[3][S];
            const int b0 = INTER && pass ? fx_support<MAS, 1, E>(p, r.inv, r.halfcell, r.dims, o, C)
                                         : fx_support<MAS, 0, E>(p, r.inv, r.halfcell, r.dims, o, C);
            if (mode == 0) {
                if (MAS == PYL_MAS_CIC) bad |= (unsigned)!(C[0][1] >= 0.0f && C[1][1] >= 0.0f && C[2][1] >= 0.0f);
                // z weights times 2^22 (exact): each corner one FFMA into the fixed-point format
#pragma unroll
                for (int q = 0; q < S; q++) C[2][q] = __fmul_rn(C[2][q], FX_SCALE);
                seen |= fx_scatter_or<MAS, E, (MAS == PYL_MAS_NGP), true>(smw, b0, C);
            } else {
                float_scatter<MAS, E>(facc, b0, C);
            }
        }
        if (__syncthreads_or((int)(bad | (seen >> 31))) && mode == 0) {
            __syncthreads();
            continue;
        }
        float *out = INTER && pass ? r.grid_interlaced : r.grid;
        auto add = [&](int c, float v) {
            const int lz = c % E, ly = (c / E) % E, lx = c / (E * E);
            const long long gx = add_wrap(o[0], lx, d), gy = add_wrap(o[1], ly, d), gz = add_wrap(o[2], lz, d);
            atomicAdd(out + (gx * d + gy) * d + gz, __fmul_rn(v, r.scale));
        };
        if (sh.parts > 1 && mode == 0) {
            share_add(sh, smw, CELLS);
        } else {
            for (int c = threadIdx.x; c < CELLS; c += blockDim.x) {
                const unsigned w = smw[c];
                if (w == 0u) continue;
                add(c, mode == 1 ? __uint_as_float(w)
                                 : (MAS == PYL_MAS_NGP ? __uint2float_rn(w) : __fmul_rn(__uint2float_rn(w), FX_INV)));
            }
        }
        if (sh.parts > 1 && share_arrive(sh))
            for (int c = threadIdx.x; c < CELLS; c += blockDim.x) {
                const float v = share_value<MAS>(sh, c);
                if (v != 0.0f) add(c, v);
            }
        __syncthreads();
        break;
    }
}

constexpr size_t BT_DEPOSIT_SMEM = FxShape<PYL_MAS_PCS, true>::SMEM;

__global__ void __launch_bounds__(1024) bt_deposit_kernel(const pyl_batch_real *__restrict__ reals,
                                                          const unsigned *__restrict__ tile_base,
                                                          const BtPart *__restrict__ list,
                                                          const unsigned *__restrict__ n_parts, unsigned max_parts,
                                                          const unsigned *__restrict__ offsets, unsigned n_total,
                                                          const float4 *__restrict__ rec, unsigned long long *share,
                                                          unsigned *done, unsigned *counter)
{
    extern __shared__ __align__(16) unsigned bsm[];
    __shared__ int cur;
    const unsigned total = min(*n_parts, max_parts);
    for (;;) {
        if (threadIdx.x == 0) cur = (int)atomicAdd(counter, 1u);
        __syncthreads();
        const unsigned it = (unsigned)cur;
        __syncthreads();
        if (it >= total) break;
        const BtPart pt = list[it];
        const pyl_batch_real r = reals[pt.real];
        const unsigned bin_end = min(offsets[pt.tile + 1], n_total);
        const unsigned begin = min(offsets[pt.tile] + pt.first, bin_end);
        const unsigned end = min(begin + pt.len, bin_end);
        const BinShare sh{share + pt.shared * BT_SHARE_CELLS, done + pt.shared, pt.parts};
        const int nt = bt_nt(r.dims);
        const int local = (int)(pt.tile - tile_base[pt.real]);
        const int o[3] = {(local / (nt * nt)) * TB, ((local / nt) % nt) * TB, (local % nt) * TB};
        const int pass = (int)pt.inter;
        switch (r.mas * 2 + (r.grid_interlaced ? 1 : 0)) {
            case 2 * PYL_MAS_NGP:     bt_deposit_bin<PYL_MAS_NGP, false>(bsm, rec, begin, end, r, o, 0, sh); break;
            case 2 * PYL_MAS_NGP + 1: bt_deposit_bin<PYL_MAS_NGP, true>(bsm, rec, begin, end, r, o, pass, sh); break;
            case 2 * PYL_MAS_CIC:     bt_deposit_bin<PYL_MAS_CIC, false>(bsm, rec, begin, end, r, o, 0, sh); break;
            case 2 * PYL_MAS_CIC + 1: bt_deposit_bin<PYL_MAS_CIC, true>(bsm, rec, begin, end, r, o, pass, sh); break;
            case 2 * PYL_MAS_TSC:     bt_deposit_bin<PYL_MAS_TSC, false>(bsm, rec, begin, end, r, o, 0, sh); break;
            case 2 * PYL_MAS_TSC + 1: bt_deposit_bin<PYL_MAS_TSC, true>(bsm, rec, begin, end, r, o, pass, sh); break;
            case 2 * PYL_MAS_PCS:     bt_deposit_bin<PYL_MAS_PCS, false>(bsm, rec, begin, end, r, o, 0, sh); break;
            default:                  bt_deposit_bin<PYL_MAS_PCS, true>(bsm, rec, begin, end, r, o, pass, sh); break;
        }
    }
}

struct BtWs {
    unsigned *counts, *offsets, *cursor, *counters, *done, *entries;
    unsigned long long *adds, *share;
    BtPart *list;
    float4 *rec;
    size_t zero_bytes, bytes;
};

inline size_t bt_align(size_t v) { return (v + 255) / 256 * 256; }

BtWs bt_layout(void *base, unsigned total_tiles, long long total_particles)
{
    BtWs w;
    char *b = (char *)base;
    size_t o = 0;
    w.counts = (unsigned *)(b + o); o = bt_align(o + 4 * ((size_t)total_tiles + 1));
    w.offsets = (unsigned *)(b + o); o = bt_align(o + 4 * ((size_t)total_tiles + 1));
    w.cursor = (unsigned *)(b + o); o = bt_align(o + 4 * ((size_t)total_tiles + 1));
    // counters (of items, parts and BinShares), the count of additions and the parts'
    // arrivals: zeroed together
    const size_t shared = bt_max_shared(total_tiles, total_particles);
    w.counters = (unsigned *)(b + o);
    w.adds = (unsigned long long *)(b + o + 24);
    w.done = (unsigned *)(b + o + 32);
    w.zero_bytes = 32 + 4 * shared;
    o = bt_align(o + w.zero_bytes);
    w.share = (unsigned long long *)(b + o); o = bt_align(o + 8 * BT_SHARE_CELLS * shared);
    w.entries = (unsigned *)(b + o); o = bt_align(o + 4 * (((size_t)total_tiles + 1023) / 1024));
    w.list = (BtPart *)(b + o); o = bt_align(o + sizeof(BtPart) * bt_max_parts(total_tiles));
    w.rec = (float4 *)(b + o); o = bt_align(o + 16 * (size_t)total_particles);
    w.bytes = o;
    return w;
}

}  // namespace
}  // namespace pyl

using namespace pyl;

extern "C" int pyl_ma_batch(const pyl_batch_real *reals, int n_reals, const pyl_batch_item *items,
                            int n_items, unsigned *counter, int ctas_per_sm, void *stream)
{
    PYL_CHECK_ARG(reals != nullptr && items != nullptr && counter != nullptr, "null pointer");
    PYL_CHECK_ARG(n_reals >= 1 && n_items >= 0, "bad sizes");
    PYL_CHECK_ARG(ctas_per_sm >= 1 && ctas_per_sm <= 8, "ctas_per_sm must be 1..8");
    cudaStream_t st = (cudaStream_t)stream;
    PYL_CUDA(cudaMemsetAsync(counter, 0, sizeof(unsigned), st));
    if (n_items == 0) return PYL_OK;
    batch_deposit_kernel<<<num_sms() * ctas_per_sm, 256, 0, st>>>(reals, items, n_items, counter);
    PYL_LAUNCH_CHECK();
    return PYL_OK;
}

extern "C" int pyl_fill(float *p, int64_t n, float value, void *stream)
{
    PYL_CHECK_ARG(p != nullptr && n >= 0, "bad arguments");
    if (n == 0) return PYL_OK;
    long long b = (n + 255) / 256;
    if (b > (long long)num_sms() * 8) b = (long long)num_sms() * 8;
    fill_value_kernel<<<(unsigned)b, 256, 0, (cudaStream_t)stream>>>(p, n, value);
    PYL_LAUNCH_CHECK();
    return PYL_OK;
}

extern "C" int pyl_scale(float *p, int64_t n, float factor, void *stream)
{
    PYL_CHECK_ARG(p != nullptr && n >= 0, "bad arguments");
    if (n == 0) return PYL_OK;
    long long b = (n + 255) / 256;
    if (b > (long long)num_sms() * 8) b = (long long)num_sms() * 8;
    scale_value_kernel<<<(unsigned)b, 256, 0, (cudaStream_t)stream>>>(p, n, factor);
    PYL_LAUNCH_CHECK();
    return PYL_OK;
}

extern "C" size_t pyl_ma_batch_tiled_workspace_size(uint32_t total_tiles, int64_t total_particles)
{
    if (total_particles < 0) return 0;
    return bt_layout(nullptr, total_tiles, total_particles).bytes;
}

extern "C" int pyl_ma_batch_tiled(const pyl_batch_real *reals, int n_reals, const pyl_batch_item *items,
                                  int n_items, const uint32_t *tile_base, uint32_t total_tiles,
                                  int64_t total_particles, void *workspace, size_t workspace_bytes,
                                  int ctas_per_sm, void *stream)
{
    PYL_CHECK_ARG(reals != nullptr && items != nullptr && tile_base != nullptr, "null pointer");
    PYL_CHECK_ARG(n_reals >= 1 && n_items >= 0 && total_tiles >= 1, "bad sizes");
    PYL_CHECK_ARG(total_particles >= 0 && total_particles < 0xFFFFFFFFLL, "particle total out of range");
    PYL_CHECK_ARG(ctas_per_sm >= 1 && ctas_per_sm <= 8, "ctas_per_sm must be 1..8");
    const BtWs ws = bt_layout(workspace, total_tiles, total_particles);
    if (workspace == nullptr || workspace_bytes < ws.bytes) {
        set_error("pyl_ma_batch_tiled: needs " + std::to_string(ws.bytes) + " workspace bytes");
        return PYL_ERR_WORKSPACE;
    }
    cudaStream_t st = (cudaStream_t)stream;
    PYL_CUDA(cudaMemsetAsync(ws.counts, 0, 4 * ((size_t)total_tiles + 1), st));
    PYL_CUDA(cudaMemsetAsync(ws.counters, 0, ws.zero_bytes, st));
    if (n_items == 0) return PYL_OK;
    const unsigned grid = (unsigned)(num_sms() * BT_CTAS);
    const int split = bt_split(n_items);
    bt_count_kernel<<<grid, BT_THREADS, 0, st>>>(reals, items, n_items, split, tile_base, ws.counts, ws.adds,
                                                 ws.counters);
    PYL_LAUNCH_CHECK();
    const unsigned sms = (unsigned)num_sms(), groups = total_tiles / 1024 + (total_tiles % 1024 != 0);
    bt_scan_kernel<<<1 + groups, 1024, 0, st>>>(reals, n_reals, tile_base, ws.counts, total_tiles, ws.adds, sms, ws.offsets,
                                                ws.cursor, ws.entries);
    PYL_LAUNCH_CHECK();
    PYL_CUDA(ensure_smem(bt_place_kernel, BT_PLACE_SMEM));
    bt_place_kernel<<<grid, BT_THREADS, BT_PLACE_SMEM, st>>>(reals, items, n_items, split, tile_base, ws.cursor,
                                                       (unsigned)total_particles, ws.rec, ws.counters + 1);
    PYL_LAUNCH_CHECK();
    const unsigned max_parts = (unsigned)bt_max_parts(total_tiles);
    const size_t max_shared = bt_max_shared(total_tiles, total_particles);
    bt_list_kernel<<<groups, 1024, 0, st>>>(reals, n_reals, tile_base, total_tiles, ws.counts, ws.adds, sms, ws.entries,
                                            max_parts, (unsigned)max_shared, ws.counters + 4, ws.counters + 3, ws.list);
    PYL_LAUNCH_CHECK();
    if (max_shared) {
        bt_share_zero_kernel<<<dim3(8, (unsigned)max_shared), 256, 0, st>>>(ws.counters + 3, ws.share);
        PYL_LAUNCH_CHECK();
    }
    PYL_CUDA(ensure_smem(bt_deposit_kernel, BT_DEPOSIT_SMEM));
    bt_deposit_kernel<<<sms, 1024, BT_DEPOSIT_SMEM, st>>>(
        reals, tile_base, ws.list, ws.counters + 4, max_parts, ws.offsets, (unsigned)total_particles,
        ws.rec, ws.share, ws.done, ws.counters + 2);
    PYL_LAUNCH_CHECK();
    return PYL_OK;
}
