// LBVH Barnes-Hut: the replacement for Barnes_Hut::make_tree/compute_forces
// (src/solvers/barnes_hut.cpp:309-418, bh_specialization.cpp:30-46) and the
// OpenCL BH_hyper pipeline (src/solvers/full_GPU.cpp:54-339,519-527 with
// include/Aster/kernels/{morton_writer,radix,BHH_specific}.cl.h).
//
// Pipeline per force evaluation (all on one stream, no host sync):
//   box      max |coordinate| of the FP64 state (fused into the drift kernel
//            during time stepping, a separate reduction otherwise)
//   morton   30-bit code as the reference get_morton: x' = (x+B)/(2B),
//            q = min(trunc(x' * 1024), 1023), interleave z|y|x (63-bit: 21
//            bits per axis). IEEE FP64 add/div, no contraction: bit-exact.
//   sort     stable LSD radix sort of (code, body index), 8-bit digits:
//            per pass a tile histogram, a per-digit scan over tiles, a stable
//            scatter (ranked by warp ballots). Ties keep body-index order.
//   tree     Karras' (2012) tree exactly as barnes_hut.cpp:338-396 (tie-break
//            32 + clz(i ^ j) on sorted positions), built bottom up: climbs
//            meet at their parent's split and the second arrival merges the
//            children: FP64 mass and centre of mass in NodesArray::unite order
//            (barnes_hut.cpp:137-152, bit-exact), FP32 AABB, squared opening
//            radius r_crit = l/theta + |com - box centre| (rounded up to FP32).
//   walk     one warp per group (a subtree of <= 64 leaves whose parent holds
//            more): a shared-memory stack walk that opens a node for the whole
//            group unless its FP32 centre of mass lies farther than r_crit
//            from the group's FP32 box; accepted nodes are appended to a
//            shared interaction list and evaluated 32 at a time by every lane
//            (FP32 on group-relative double-single coordinates, or FP64).
// Node numbering is the reference's: leaves 0..n-1 (sorted order), internal
// n..2n-2, root n, -1 = no child.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>

#include <cooperative_groups.h>

#include "aster_internal.cuh"
#include "fp64_pair.cuh"
#include "pn.cuh"

namespace {

constexpr int SORT_THREADS = 256;
constexpr int SORT_ITEMS = 8;
constexpr int SORT_TILE = SORT_THREADS * SORT_ITEMS;  // 2048 keys per block
constexpr int SORT_WARPS = SORT_THREADS / 32;
constexpr int RADIX = 256;
static_assert(SORT_THREADS == RADIX, "the scan and scatter kernels give each thread one digit");
constexpr int MAX_CLIMB = 160;     // bottom-up level cap (tree depth <= 97 for 63-bit codes)
#ifndef ASTER_WALK_WARPS
#define ASTER_WALK_WARPS 4
#endif
#ifndef ASTER_WALK_MINBLOCKS
#define ASTER_WALK_MINBLOCKS 5
#endif
#ifndef ASTER_WALK_UNROLL
#define ASTER_WALK_UNROLL 8
#endif
constexpr int WALK_WARPS = ASTER_WALK_WARPS;  // warps (groups in flight) per block
constexpr int WALK_UNROLL = ASTER_WALK_UNROLL;
constexpr int WALK_STACK = 1024;   // nodes per warp
constexpr int GROUP_MAX = 64;      // leaves per walk group (1 or 2 per lane)
// Interaction list: evaluated (and its FP32 partial sums folded into the
// compensated accumulators) every WALK_FLUSH entries; capacity = flush - 1 +
// the 64 entries one round can append. The post-Newtonian mixed walk, whose
// entries also carry a velocity, flushes every WALK_FLUSH_PN.
constexpr int WALK_FLUSH_MIXED = 128, WALK_FLUSH_FP64 = 32, WALK_FLUSH_PN = 64;
constexpr int WALK_LIST_MIXED = 192, WALK_LIST_FP64 = 96, WALK_LIST_PN = 128;

// ----------------------------------------------------------------- box
__device__ __forceinline__ double warp_max_d(double v) {
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

__global__ void __launch_bounds__(256) k_box(int64_t n, const double4* __restrict__ pm,
                                             unsigned long long* __restrict__ box_bits) {
    __shared__ double red[8];
    double b = 0.0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        double4 p = pm[i];
        b = fmax(b, fmax(fabs(p.x), fmax(fabs(p.y), fabs(p.z))));
    }
    b = warp_max_d(b);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = b;
    __syncthreads();
    if (threadIdx.x < 32) {
        double v = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.0;
        v = warp_max_d(v);
        if (threadIdx.x == 0) atomicMax(box_bits, (unsigned long long)__double_as_longlong(v));
    }
}

// -------------------------------------------------------------- morton
__device__ __forceinline__ uint32_t part1by2_32(uint32_t n) {
    n = (n | (n << 16)) & 0x030000FFu;
    n = (n | (n << 8)) & 0x0300F00Fu;
    n = (n | (n << 4)) & 0x030C30C3u;
    n = (n | (n << 2)) & 0x09249249u;
    return n;
}

__device__ __forceinline__ uint64_t part1by2_64(uint64_t n) {
    n &= 0x1FFFFFull;
    n = (n | (n << 32)) & 0x001F00000000FFFFull;
    n = (n | (n << 16)) & 0x001F0000FF0000FFull;
    n = (n | (n << 8)) & 0x100F00F00F00F00Full;
    n = (n | (n << 4)) & 0x10C30C30C30C30C3ull;
    n = (n | (n << 2)) & 0x1249249249249249ull;
    return n;
}

// (x + B) / (2B) * scale truncated and clamped to maxv; NaN / negative -> 0.
__device__ __forceinline__ uint32_t quantize(double x, double B, double scale, uint32_t maxv) {
    double t = __ddiv_rn(__dadd_rn(x, B), __dmul_rn(2.0, B));
    double s = __dmul_rn(t, scale);
    if (!(s > 0.0)) return 0u;
    if (s >= 4294967296.0) return maxv;
    uint32_t q = (uint32_t)s;
    return q < maxv ? q : maxv;
}

// OpenCL gen_mortons (morton_writer.cl.h:72-122): clamp to [0,1], 1024 max,
// (ushort), so +B wraps to 0 through the 10-bit expansion mask.
__device__ __forceinline__ uint32_t quantize_compat(double x, double B) {
    double t = __ddiv_rn(__dadd_rn(x, B), __dmul_rn(2.0, B));
    t = fmin(fmax(t, 0.0), 1.0);
    uint32_t v = (uint32_t)__dmul_rn(t, 1024.0);
    v = v < 1024u ? v : 1024u;
    return (uint32_t)(uint16_t)v;
}

template <class KeyT, int MODE>  // MODE 0: 30-bit, 1: 63-bit, 2: 30-bit compat
__device__ __forceinline__ KeyT morton_code(const double4 p, double B) {
    if (MODE == 0) {
        uint32_t ix = quantize(p.x, B, 1024.0, 1023u), iy = quantize(p.y, B, 1024.0, 1023u),
                 iz = quantize(p.z, B, 1024.0, 1023u);
        return (KeyT)((part1by2_32(iz) << 2) | (part1by2_32(iy) << 1) | part1by2_32(ix));
    }
    if (MODE == 1) {
        uint64_t ix = quantize(p.x, B, 2097152.0, 2097151u), iy = quantize(p.y, B, 2097152.0, 2097151u),
                 iz = quantize(p.z, B, 2097152.0, 2097151u);
        return (KeyT)((part1by2_64(iz) << 2) | (part1by2_64(iy) << 1) | part1by2_64(ix));
    }
    uint32_t ix = quantize_compat(p.x, B), iy = quantize_compat(p.y, B), iz = quantize_compat(p.z, B);
    return (KeyT)(part1by2_32(ix) | (part1by2_32(iy) << 1) | (part1by2_32(iz) << 2));
}

// (and the build's counters, four from gcount, to zero)
template <class KeyT, int MODE>
__global__ void __launch_bounds__(256) k_morton(int64_t n, const double4* __restrict__ pm,
                                                const unsigned long long* __restrict__ box_bits,
                                                KeyT* __restrict__ codes, unsigned int* __restrict__ gcount) {
    if (blockIdx.x == 0 && threadIdx.x < 4) gcount[threadIdx.x] = 0u;
    const double B = __longlong_as_double((long long)*box_bits);
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        codes[i] = morton_code<KeyT, MODE>(pm[i], B);
}

// ---------------------------------------------------------------- sort
template <class KeyT>
__global__ void __launch_bounds__(SORT_THREADS) k_sort_hist(int64_t n, const KeyT* __restrict__ keys, int shift,
                                                            int nblocks, uint32_t* __restrict__ hist) {
    __shared__ uint32_t h[SORT_WARPS][RADIX];
    const int warp = threadIdx.x >> 5;
    for (int d = threadIdx.x; d < SORT_WARPS * RADIX; d += SORT_THREADS) (&h[0][0])[d] = 0;
    __syncthreads();
    const int64_t base = (int64_t)blockIdx.x * SORT_TILE;
    KeyT k[SORT_ITEMS];  // all loads in flight before the first count
#pragma unroll
    for (int r = 0; r < SORT_ITEMS; ++r) {
        const int64_t i = base + (int64_t)r * SORT_THREADS + threadIdx.x;
        k[r] = i < n ? keys[i] : (KeyT)0;
    }
#pragma unroll
    for (int r = 0; r < SORT_ITEMS; ++r) {
        const int64_t i = base + (int64_t)r * SORT_THREADS + threadIdx.x;
        if (i < n) atomicAdd(&h[warp][(uint32_t)(k[r] >> shift) & (RADIX - 1)], 1u);
    }
    __syncthreads();
    for (int d = threadIdx.x; d < RADIX; d += SORT_THREADS) {
        uint32_t s = 0;
        for (int w = 0; w < SORT_WARPS; ++w) s += h[w][d];
        hist[(int64_t)d * nblocks + blockIdx.x] = s;
    }
}

// Block-wide exclusive scan of one uint32 per thread (blockDim.x <= 1024,
// multiple of 32); returns the exclusive prefix, *total gets the block sum.
__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* smem32, uint32_t* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    uint32_t x = v;
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) smem32[warp] = x;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = lane < nw ? smem32[lane] : 0u;
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        if (lane < nw) smem32[lane] = w;  // inclusive warp sums
    }
    __syncthreads();
    const uint32_t before = warp ? smem32[warp - 1] : 0u;
    if (total) *total = smem32[nw - 1];
    __syncthreads();
    return before + x - v;
}

// Per digit d (one block each): exclusive scan of the per-tile counts
// hist[d*nblocks + b] over b, in place; digit_tot[d] = the digit's total.
__global__ void __launch_bounds__(1024) k_scan_digits(uint32_t* __restrict__ hist, int nblocks,
                                                      uint32_t* __restrict__ digit_tot) {
    __shared__ uint32_t s32[32];
    uint32_t* row = hist + (int64_t)blockIdx.x * nblocks;
    uint32_t carry = 0;
    for (int base = 0; base < nblocks; base += blockDim.x) {
        const int i = base + threadIdx.x;
        const uint32_t v = i < nblocks ? row[i] : 0u;
        uint32_t tot;
        const uint32_t ex = block_exclusive_scan(v, s32, &tot);
        if (i < nblocks) row[i] = carry + ex;
        carry += tot;
    }
    if (threadIdx.x == 0) digit_tot[blockIdx.x] = carry;
}

// The lanes of the warp whose keys have this lane's digit (ok: it has a key),
// from a ballot per bit: match-any takes longer (build of 2^20 bodies 267.6
// against 258.8 us, 32,768: 78.3 against 75.3).
__device__ __forceinline__ uint32_t digit_peers(uint32_t d, bool ok) {
    uint32_t peers = __ballot_sync(0xffffffffu, ok);
    if (!ok) peers = ~peers;
#pragma unroll
    for (int b = 0; b < 8; ++b) {
        const bool one = (d >> b) & 1u;
        const uint32_t m = __ballot_sync(0xffffffffu, one);
        peers &= one ? m : ~m;
    }
    return peers;
}

// Stable scatter of one 8-bit digit. Warp w of the block owns the 256 keys
// [w*256, w*256+256) of the tile and ranks them round by round (32 consecutive
// keys per round) by digit_peers, so ranks follow input order.
// Global position = (keys of smaller digits) + (same digit in earlier tiles)
// + (same digit earlier in this tile).
template <class KeyT, bool IDENTITY_VALS>
__global__ void __launch_bounds__(SORT_THREADS, 4) k_sort_scatter(int64_t n, const KeyT* __restrict__ kin,
                                                               const int32_t* __restrict__ vin, KeyT* __restrict__ kout,
                                                               int32_t* __restrict__ vout, int shift, int nblocks,
                                                               const uint32_t* __restrict__ tile_off,
                                                               const uint32_t* __restrict__ digit_tot) {
    __shared__ uint32_t wh[SORT_WARPS][RADIX];
    __shared__ uint32_t dstart[RADIX];
    __shared__ uint32_t gofs[RADIX];
    __shared__ uint32_t s32[32];
    __shared__ KeyT sk[SORT_TILE];
    __shared__ int32_t sv[SORT_TILE];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t tile0 = (int64_t)blockIdx.x * SORT_TILE;
    KeyT key[SORT_ITEMS];
    int32_t val[SORT_ITEMS];
    // the tile's keys and values: all loads in flight before the ranking
#pragma unroll
    for (int r = 0; r < SORT_ITEMS; ++r) {
        const int64_t i = tile0 + warp * (32 * SORT_ITEMS) + r * 32 + lane;
        const bool ok = i < n;
        key[r] = ok ? kin[i] : (KeyT)0;
        val[r] = ok ? (IDENTITY_VALS ? (int32_t)i : vin[i]) : 0;
    }
    const uint32_t toff = tile_off[(int64_t)threadIdx.x * nblocks + blockIdx.x];  // digit threadIdx.x
    for (int d = threadIdx.x; d < SORT_WARPS * RADIX; d += SORT_THREADS) (&wh[0][0])[d] = 0;
    // global base of each digit: exclusive scan of the digit totals
    const uint32_t gb = block_exclusive_scan(digit_tot[threadIdx.x], s32, nullptr);
    __syncthreads();
    const uint32_t lt = (1u << lane) - 1u;
    uint32_t rank[SORT_ITEMS];
    uint32_t dig[SORT_ITEMS];
#pragma unroll
    for (int r = 0; r < SORT_ITEMS; ++r) {
        const int64_t i = tile0 + warp * (32 * SORT_ITEMS) + r * 32 + lane;
        const bool ok = i < n;
        const uint32_t d = ok ? ((uint32_t)(key[r] >> shift) & (RADIX - 1)) : 0xFFFFu;
        dig[r] = d;
        const uint32_t peers = digit_peers(d, ok);
        uint32_t before = 0;
        if (ok) before = wh[warp][d];
        __syncwarp();
        rank[r] = before + __popc(peers & lt);
        if (ok && (peers & lt) == 0) wh[warp][d] = before + __popc(peers);
        __syncwarp();
    }
    __syncthreads();
    // per digit: exclusive prefix over warps, then over digits (block-local start)
    uint32_t tot = 0;
    for (int w = 0; w < SORT_WARPS; ++w) {
        const uint32_t t = wh[w][threadIdx.x];
        wh[w][threadIdx.x] = tot;
        tot += t;
    }
    const uint32_t ds = block_exclusive_scan(tot, s32, nullptr);
    dstart[threadIdx.x] = ds;
    // output position of the tile's p-th key (digit d) = gofs[d] + p
    gofs[threadIdx.x] = gb + toff - ds;
    __syncthreads();
#pragma unroll
    for (int r = 0; r < SORT_ITEMS; ++r) {
        if (dig[r] < RADIX) {
            const uint32_t pos = dstart[dig[r]] + wh[warp][dig[r]] + rank[r];
            sk[pos] = key[r];
            sv[pos] = val[r];
        }
    }
    __syncthreads();
    const int64_t valid = min((int64_t)SORT_TILE, n - tile0);
    for (int p = threadIdx.x; p < valid; p += SORT_THREADS) {
        const KeyT k = sk[p];
        const uint32_t d = (uint32_t)(k >> shift) & (RADIX - 1);
        const int64_t g = (int64_t)(uint32_t)(gofs[d] + (uint32_t)p);
        kout[g] = k;
        vout[g] = sv[p];
    }
}

// Morton codes and their whole stable sort in one launch, for up to 16 blocks'
// worth of bodies: a cluster of up to 16 blocks keeps the keys on chip (ITEMS
// per thread) and exchanges them through distributed shared memory, one 8-bit
// digit a pass. Per pass: warps rank their keys as k_sort_scatter
// does, every block publishes its digit counts to the others, and the keys go
// straight to their new block and place; the last pass writes to global memory.
// Bound by latency (two cluster barriers a pass) and by the number of stores into
// other blocks: a 32-bit key with its value in one store instead of two and counts
// eight to a store took the build of 32,768 bodies from 75.3 to 68.1 us (2000: 42.6
// to 41.0). The general sort takes three
// launches a pass, ~3.3 us each below 10^5 keys, whatever the size.
constexpr int CSORT_THREADS = 1024, CSORT_WARPS = CSORT_THREADS / 32, CSORT_BLOCKS = 16;

template <class KeyT>
constexpr size_t cluster_sort_smem(int items) {
    return (size_t)CSORT_THREADS * items * (sizeof(KeyT) + 4) + (size_t)CSORT_WARPS * RADIX * 2 +
           (size_t)CSORT_BLOCKS * RADIX * 2 + RADIX * 2 + RADIX * 4;
}

template <class KeyT, int MODE, int ITEMS>
__global__ void __launch_bounds__(CSORT_THREADS, 1) k_sort_cluster(int64_t n, const double4* __restrict__ pm,
                                                                   const unsigned long long* __restrict__ box_bits,
                                                                   KeyT* __restrict__ codes, KeyT* __restrict__ kout,
                                                                   int32_t* __restrict__ vout,
                                                                   unsigned int* __restrict__ gcount) {
    namespace cg = cooperative_groups;
    constexpr int PASSES = sizeof(KeyT) == 8 ? 8 : 4;
    constexpr int PER_BLOCK = CSORT_THREADS * ITEMS;
    extern __shared__ __align__(16) unsigned char csort_smem[];
    KeyT* bkey = reinterpret_cast<KeyT*>(csort_smem);
    uint32_t* bval = reinterpret_cast<uint32_t*>(bkey + PER_BLOCK);
    uint32_t* sbase = bval + PER_BLOCK;                          // [digit] place of this block's first key
    uint16_t* ctot = reinterpret_cast<uint16_t*>(sbase + RADIX);  // [block][digit] counts of every block (<= PER_BLOCK)
    uint16_t* stot = ctot + CSORT_BLOCKS * RADIX;                // [digit] this block's counts
    uint16_t* wh = stot + RADIX;                                 // [warp][digit]
    __shared__ uint32_t s32[32];
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank(), nblk = (int)cluster.num_blocks();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t lt = (1u << lane) - 1u;
    const int64_t tile0 = (int64_t)rank * PER_BLOCK;
    if (rank == 0 && threadIdx.x < 4) gcount[threadIdx.x] = 0u;  // the build's counters
    const int local0 = warp * 32 * ITEMS + lane;
    const double B = __longlong_as_double((long long)*box_bits);
    KeyT key[ITEMS];
    uint32_t val[ITEMS];
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
        const int64_t i = tile0 + local0 + 32 * r;
        key[r] = 0;
        val[r] = (uint32_t)i;
        if (i < n) {
            key[r] = morton_code<KeyT, MODE>(pm[i], B);
            if (codes) codes[i] = key[r];
        }
    }
    cluster.sync();  // every block runs before its shared memory is written from outside
#pragma unroll 1
    for (int pass = 0; pass < PASSES; ++pass) {
        if (pass > 0) {
#pragma unroll
            for (int r = 0; r < ITEMS; ++r) {
                if constexpr (sizeof(KeyT) == 4) {
                    const uint2 kv = reinterpret_cast<const uint2*>(csort_smem)[local0 + 32 * r];
                    key[r] = kv.x;
                    val[r] = kv.y;
                } else {
                    key[r] = bkey[local0 + 32 * r];
                    val[r] = bval[local0 + 32 * r];
                }
            }
        }
        for (int d = threadIdx.x; d < CSORT_WARPS * RADIX / 2; d += CSORT_THREADS) reinterpret_cast<uint32_t*>(wh)[d] = 0u;
        __syncthreads();
        uint32_t rk[ITEMS], dig[ITEMS];
        uint16_t* w = wh + warp * RADIX;
#pragma unroll
        for (int r = 0; r < ITEMS; ++r) {
            const bool ok = tile0 + local0 + 32 * r < n;
            const uint32_t d = ok ? (uint32_t)(key[r] >> (8 * pass)) & (RADIX - 1) : 0xFFFFu;
            dig[r] = d;
            const uint32_t peers = digit_peers(d, ok);
            uint32_t before = 0;
            if (ok) before = w[d];
            __syncwarp();
            rk[r] = before + __popc(peers & lt);
            if (ok && (peers & lt) == 0) w[d] = (uint16_t)(before + __popc(peers));
            __syncwarp();
        }
        __syncthreads();
        if (threadIdx.x < RADIX) {  // exclusive prefix of the digit over the warps
            uint32_t tot = 0;
#pragma unroll 8
            for (int q = 0; q < CSORT_WARPS; ++q) {
                const uint32_t t = wh[q * RADIX + threadIdx.x];
                wh[q * RADIX + threadIdx.x] = (uint16_t)tot;
                tot += t;
            }
            stot[threadIdx.x] = (uint16_t)tot;
        }
        __syncthreads();
        if (threadIdx.x < nblk * (RADIX / 8)) {  // eight counts a store, one row to each block
            const int to = threadIdx.x / (RADIX / 8), at = threadIdx.x % (RADIX / 8);
            reinterpret_cast<uint4*>(cluster.map_shared_rank(ctot, to) + rank * RADIX)[at] =
                reinterpret_cast<const uint4*>(stot)[at];
        }
        cluster.sync();  // every block's counts are here; every block has read its keys
        uint32_t all = 0, mine = 0;
        if (threadIdx.x < RADIX) {
            for (int q = 0; q < nblk; ++q) {
                const uint32_t t = ctot[q * RADIX + threadIdx.x];
                all += t;
                mine += q < rank ? t : 0u;
            }
        }
        const uint32_t start = block_exclusive_scan(all, s32, nullptr);
        if (threadIdx.x < RADIX) sbase[threadIdx.x] = start + mine;
        __syncthreads();
#pragma unroll
        for (int r = 0; r < ITEMS; ++r) {
            if (dig[r] >= RADIX) continue;
            const uint32_t g = sbase[dig[r]] + w[dig[r]] + rk[r];
            if (pass == PASSES - 1) {
                kout[g] = key[r];
                vout[g] = (int32_t)val[r];
            } else {
                const int to = (int)(g / PER_BLOCK), at = (int)(g % PER_BLOCK);
                if constexpr (sizeof(KeyT) == 4) {
                    cluster.map_shared_rank(reinterpret_cast<uint2*>(csort_smem), to)[at] = make_uint2(key[r], val[r]);
                } else {
                    cluster.map_shared_rank(bkey, to)[at] = key[r];
                    cluster.map_shared_rank(bval, to)[at] = val[r];
                }
            }
        }
        if (pass < PASSES - 1) cluster.sync();  // the keys have arrived
    }
}

template <class KeyT>
__global__ void k_reverse(int64_t n, const KeyT* __restrict__ kin, const int32_t* __restrict__ vin,
                          KeyT* __restrict__ kout, int32_t* __restrict__ vout) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        kout[i] = kin[n - 1 - i];
        vout[i] = vin[n - 1 - i];
    }
}

// A leaf's box: its position rounded outwards to FP32 (not stored: computed
// from the leaf's node_cm wherever it is needed).
__device__ __forceinline__ float4 leaf_lo(const double4 p) {
    return make_float4(__double2float_rd(p.x), __double2float_rd(p.y), __double2float_rd(p.z), 0.f);
}
__device__ __forceinline__ float4 leaf_hi(const double4 p) {
    return make_float4(__double2float_ru(p.x), __double2float_ru(p.y), __double2float_ru(p.z), 0.f);
}

// Traversal data of a node (the walk's view of it): h = (rn(com), rn(mass)),
// l = (com - rn(com), rcrit2). Internal node: the squared opening radius
// r_crit = l/theta + |com - box centre| (l = longest AABB side; FP64, rounded
// up to FP32). Leaf: rcrit2 = 0.
__device__ __forceinline__ void node_trav(const double4 c, const float4 lo, const float4 hi, double theta, float4& h,
                                          float4& l) {
    const double ex = __dsub_rn((double)hi.x, (double)lo.x), ey = __dsub_rn((double)hi.y, (double)lo.y),
                 ez = __dsub_rn((double)hi.z, (double)lo.z);
    double lmax = 0.0;
    lmax = ex > lmax ? ex : lmax;
    lmax = ey > lmax ? ey : lmax;
    lmax = ez > lmax ? ez : lmax;
    const double cx = __dmul_rn(0.5, __dadd_rn((double)lo.x, (double)hi.x));
    const double cy = __dmul_rn(0.5, __dadd_rn((double)lo.y, (double)hi.y));
    const double cz = __dmul_rn(0.5, __dadd_rn((double)lo.z, (double)hi.z));
    const double dx = __dsub_rn(c.x, cx), dy = __dsub_rn(c.y, cy), dz = __dsub_rn(c.z, cz);
    const double delta = __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz)));
    const double rc = __dadd_rn(__ddiv_rn(lmax, theta), delta);
    ds_split(c.x, h.x, l.x);
    ds_split(c.y, h.y, l.y);
    ds_split(c.z, h.z, l.z);
    h.w = __double2float_rn(c.w);
    l.w = __double2float_ru(__dmul_rn(rc, rc));
}
__device__ __forceinline__ void leaf_trav(const double4 c, float4& h, float4& l) {
    ds_split(c.x, h.x, l.x);
    ds_split(c.y, h.y, l.y);
    ds_split(c.z, h.z, l.z);
    h.w = __double2float_rn(c.w);
    l.w = 0.f;
}

// The child record of an internal node: the traversal data of both children
// in one contiguous 64 bytes, so opening a node costs one load, each field as
// a (left, right) pair so that the walk's paired FP32 opening test and
// list-entry arithmetic read aligned register pairs:
// (xL xR yL yR) (zL zR mL mR) (lxL lxR lyL lyR) (lzL lzR rcrit2L rcrit2R).
// Child ids below n are leaves (their boxes are not needed).
__device__ __forceinline__ void put_child_record(float4* __restrict__ dst, int64_t n, double theta, int32_t L,
                                                 const double4 cL, const float4 loL, const float4 hiL, int32_t R,
                                                 const double4 cR, const float4 loR, const float4 hiR) {
    float4 hL, lL, hR, lR;
    if (L < n) leaf_trav(cL, hL, lL);
    else node_trav(cL, loL, hiL, theta, hL, lL);
    if (R < n) leaf_trav(cR, hR, lR);
    else node_trav(cR, loR, hiR, theta, hR, lR);
    dst[0] = make_float4(hL.x, hR.x, hL.y, hR.y);
    dst[1] = make_float4(hL.z, hR.z, hL.w, hR.w);
    dst[2] = make_float4(lL.x, lR.x, lL.y, lR.y);
    dst[3] = make_float4(lL.z, lR.z, lL.w, lR.w);
}

// ---------------------------------------------------------------- tree
// The tree Karras (2012) builds top down (barnes_hut.cpp:338-396), built bottom
// up together with the node data: a node [lo, hi] of the radix tree over the
// sorted codes is its parent's left child when delta(hi, hi+1) > delta(lo-1, lo)
// (delta: common prefix of neighbouring augmented keys), so a climb finds its
// parent's split, hi or lo - 1, from two values, and the two children of a node
// meet at its split (Apetrei 2014). Node numbers are Karras': a left child has
// its last leaf's index, a right child its first leaf's, the root 0 (each + n).
// The same trees bit for bit, without the searches of the top-down form (57 us
// of the build at 2^20 bodies) and without links to read on the way up.
//
// k_tree_local: a block merges what it can of TREE_LEAVES consecutive leaves;
// the subtrees left over ("frontier": their sibling lies outside) go out in leaf
// order. k_tree_merge, launched until one block is left: a block takes the
// frontiers of several neighbouring blocks as items and merges on, climbs again
// meeting through shared memory. Rank r of an item and its first leaf lo(r)
// give every range: items tile their region. What bounds it: a chain of
// dependent merges (about 31 levels at 2^20 bodies, three divisions each);
// before, every level between the 64-leaf blocks and the root was an
// acquire-release atomic and a dependent load at L2 (54 us at 131,072 bodies,
// 59 at 2^20). Climbing through global memory in these kernels took as long
// again; with node data, deltas and exchanges in shared memory a level is about
// 0.5 us. Build per graph-replayed step, before and after: 2000 bodies 98.7 ->
// 71.6 us, 20,011 115.6 -> 93.7, 131,073 132.5 -> 108.9, 2^20 315 -> 273.
constexpr int TREE_LEAVES = 64;
constexpr int MERGE_FAN_MAX = 256;  // input blocks per block at most
// Items a merge holds in shared memory: 512 leave two blocks per SM, 256 (the
// first merge of up to MERGE_MANY input blocks, 32 blocks' worth of items) five.
// More items (clustered bodies) go through global memory. A merge's time grows
// with its items (400 items 28 us, 200 some 15), a further launch costs as much
// as those save: build per step with 512 / 256 in the first merge, us: 10,000
// bodies 72.8 / 67.0, 20,011 81.2 / 75.0, 262,144 136.0 / 132.2, 524,288 178.1 /
// 188.5, 2^20 265.7 / 284.0; one last merge of up to 1344 items instead of 512:
// 10,000 bodies 80.5, 262,144 140.9. 256 threads a merge are slower than 512
// (20,011 bodies 77.6, 262,144 142.4).
constexpr int MERGE_CAP0 = 256, MERGE_CAP = 512;
constexpr int64_t MERGE_MANY = 6000;
constexpr int MERGE_THREADS = 512;

// delta of the neighbours at sorted positions i, i + 1 (codes a, b, bodies pa, pb)
template <class KeyT, bool COMPAT>
__device__ __forceinline__ int neighbour_delta(KeyT a, KeyT b, int64_t i, int32_t pa, int32_t pb) {
    if (a == b) {
        const uint32_t t = COMPAT ? (uint32_t)(pa ^ pb) : (uint32_t)(i ^ (i + 1));
        return (sizeof(KeyT) == 8 ? 64 : 32) + __clz((int)t);
    }
    return sizeof(KeyT) == 8 ? __clzll((long long)(a ^ b)) : __clz((int)(uint32_t)(a ^ b));
}

// Walk groups: a node whose subtree holds at most GROUP_MAX leaves while its
// parent's holds more (the root when n <= GROUP_MAX). Its leaves are a
// contiguous sorted run sharing a Morton prefix, so the group is spatially
// compact (a fixed run of consecutive sorted bodies is not: it can straddle a
// Morton jump and span the whole system). Listed here as (first leaf, size)
// where the parent is merged. Groups of more than 32 bodies (a second pass over
// the list, or two bodies per lane) fill the array from the front, groups of at
// most 32 (one pass) from the back; the walk takes the front part first, so its
// last wave is made of the cheaper groups and warps finish closer together.
constexpr int GROUP_SMALL = 32;
__device__ __forceinline__ void list_group(int2* groups, unsigned int* ngroups, int64_t n, int64_t first,
                                           int64_t size) {
    if (size > GROUP_SMALL)
        groups[atomicAdd(&ngroups[0], 1u)] = make_int2((int32_t)first, (int32_t)size);
    else
        groups[n - 1 - atomicAdd(&ngroups[3], 1u)] = make_int2((int32_t)first, (int32_t)size);
}

// (x, y, z) / m, each correctly rounded as __ddiv_rn, from one correctly rounded
// reciprocal: q = a y, then q + (a - m q) y twice with fused multiply-adds. The
// first correction leaves q within an ulp of a / m, and from there, y being the
// rounded 1 / m, the second one gives the rounded quotient (Markstein 1990).
// Components or masses outside [2^-400, 2^400), where a step could leave the
// normal range, take the division itself. Three divisions were the longest part
// of a merge's serial chain.
__device__ __forceinline__ bool mid_range(double v) {
    return (unsigned)((__double2hiint(v) & 0x7fffffff) - ((1023 - 400) << 20)) < (800u << 20);
}
__device__ __forceinline__ void div3_rn(double& x, double& y, double& z, double m) {
    const double r = __drcp_rn(m);
    double qx = __dmul_rn(x, r), qy = __dmul_rn(y, r), qz = __dmul_rn(z, r);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        qx = __fma_rn(__fma_rn(-m, qx, x), r, qx);
        qy = __fma_rn(__fma_rn(-m, qy, y), r, qy);
        qz = __fma_rn(__fma_rn(-m, qz, z), r, qz);
    }
    if (!(mid_range(x) && mid_range(y) && mid_range(z) && mid_range(m))) {
        qx = __ddiv_rn(x, m);
        qy = __ddiv_rn(y, m);
        qz = __ddiv_rn(z, m);
    }
    x = qx;
    y = qy;
    z = qz;
}

// Exchange on a shared-memory slot where two climbs meet: its release half
// publishes the climb's node data (shared memory), its acquire half makes the
// first arrival's visible to the second.
__device__ __forceinline__ int meet(int* slot, int mine) {
    int old;
    asm volatile("atom.acq_rel.cta.shared.exch.b32 %0, [%1], %2;"
                 : "=r"(old)
                 : "r"((unsigned)__cvta_generic_to_shared(slot)), "r"(mine)
                 : "memory");
    return old;
}

__device__ __forceinline__ void bu_merge(const double4 cl, const double4 cr, const float4 l0, const float4 l1,
                                         const float4 h0, const float4 h1, double4& cm, float4& lo, float4& hi) {
    // NodesArray::unite order: M = m_R + m_L; c = (c_R m_R + c_L m_L) / M.
    // A node without mass (M <= 0: only massless bodies below it) takes the
    // midpoint (c_R + c_L) / 2, finite, so that its ancestors' centres stay
    // finite too (unite leaves such a node's previous contents in place).
    const double M = __dadd_rn(cr.w, cl.w);
    if (M > 0.0) {
        cm.x = __dadd_rn(__dmul_rn(cr.x, cr.w), __dmul_rn(cl.x, cl.w));
        cm.y = __dadd_rn(__dmul_rn(cr.y, cr.w), __dmul_rn(cl.y, cl.w));
        cm.z = __dadd_rn(__dmul_rn(cr.z, cr.w), __dmul_rn(cl.z, cl.w));
        div3_rn(cm.x, cm.y, cm.z, M);
    } else {
        cm.x = __dmul_rn(0.5, __dadd_rn(cr.x, cl.x));
        cm.y = __dmul_rn(0.5, __dadd_rn(cr.y, cl.y));
        cm.z = __dmul_rn(0.5, __dadd_rn(cr.z, cl.z));
    }
    cm.w = M;
    lo = make_float4(fminf(l0.x, l1.x), fminf(l0.y, l1.y), fminf(l0.z, l1.z), 0.f);
    hi = make_float4(fmaxf(h0.x, h1.x), fmaxf(h0.y, h1.y), fmaxf(h0.z, h1.z), 0.f);
}

// The node arrays. LINKS: also parent, sib (>= 0: a left child's sibling; < 0: a
// right child's, complemented) and the leaf ranges, which only the exported
// tree and the post-Newtonian node velocities read.
struct TreeOut {
    double4* node_cm;
    float4 *bmin, *bmax;
    int2* child;
    float4* crec;
    int32_t *parent, *sib, *rlo, *rhi;
    int2* groups;
    unsigned int* ngroups;
    int* err;
};

// lists the walk groups among a node's children [l0, l1) and [l1, l2)
__device__ __forceinline__ void list_children(const TreeOut& o, int64_t n, int64_t l0, int64_t l1, int64_t l2) {
    if (l2 - l0 <= GROUP_MAX) return;
    if (l1 - l0 <= GROUP_MAX) list_group(o.groups, o.ngroups, n, l0, l1 - l0);
    if (l2 - l1 <= GROUP_MAX) list_group(o.groups, o.ngroups, n, l1, l2 - l1);
}

template <bool LINKS>
__device__ __forceinline__ void put_links(const TreeOut& o, int32_t id, int32_t L, int32_t R, int64_t lo, int64_t hi) {
    if (LINKS) {
        o.parent[L] = id;
        o.parent[R] = id;
        o.sib[L] = R;
        o.sib[R] = ~L;
        o.rlo[id] = (int32_t)lo;
        o.rhi[id] = (int32_t)hi;
    }
}

// front[B0 + r] = (node, first leaf) of the block's r-th frontier subtree,
// nfront[block] their number; dl[k] = delta(k, k + 1), -1 at the end.
template <class KeyT, bool COMPAT, bool LINKS>
__global__ void __launch_bounds__(TREE_LEAVES, 1024 / TREE_LEAVES) k_tree_local(
    int64_t n, double theta, const KeyT* __restrict__ codes, const int32_t* __restrict__ perm,
    const double4* __restrict__ pm, TreeOut o, signed char* __restrict__ dl, int2* __restrict__ front,
    int32_t* __restrict__ nfront, unsigned long long* __restrict__ zero_box) {
    // [0][j]: leaf B0 + j; [1][j]: the node whose children meet between leaves B0 + j and B0 + j + 1
    __shared__ double4 s_cm[2][TREE_LEAVES];
    __shared__ float4 s_lo[2][TREE_LEAVES], s_hi[2][TREE_LEAVES];
    __shared__ int s_slot[TREE_LEAVES], s_kids[TREE_LEAVES];
    __shared__ int32_t s_id[TREE_LEAVES], s_fid[TREE_LEAVES];
    __shared__ int s_rng[TREE_LEAVES];
    __shared__ signed char s_dl[TREE_LEAVES + 1];  // [j]: delta(B0 + j - 1, B0 + j)
    __shared__ int s_warp[TREE_LEAVES / 32];
    const int j = threadIdx.x;
    const int64_t B0 = (int64_t)blockIdx.x * TREE_LEAVES, k = B0 + j;
    const int cnt = (int)(n - B0 < TREE_LEAVES ? n - B0 : TREE_LEAVES);
    const bool in = j < cnt;
    if (zero_box && k == 0) *zero_box = 0ull;  // read by the codes; the walk's fused drift refills it
    s_slot[j] = 0;
    s_id[j] = -1;
    s_fid[j] = -1;
    double4 cm = make_double4(0, 0, 0, 0);
    float4 blo = make_float4(0, 0, 0, 0), bhi = blo;
    if (in) {
        const int32_t pk = perm[k];
        const KeyT ck = codes[k];
        const int d = k == 0 ? -1 : neighbour_delta<KeyT, COMPAT>(codes[k - 1], ck, k - 1, COMPAT ? perm[k - 1] : 0, pk);
        s_dl[j] = (signed char)d;
        if (k > 0) dl[k - 1] = (signed char)d;
        if (k == n - 1) dl[k] = -1;
        if (j == cnt - 1)
            s_dl[cnt] = (signed char)(k == n - 1 ? -1
                                                 : neighbour_delta<KeyT, COMPAT>(ck, codes[k + 1], k, pk,
                                                                                 COMPAT ? perm[k + 1] : 0));
        cm = pm[pk];
        blo = leaf_lo(cm);
        bhi = leaf_hi(cm);
        o.node_cm[k] = cm;
        s_cm[0][j] = cm;
        s_lo[0][j] = blo;
        s_hi[0][j] = bhi;
        if (LINKS) o.rlo[k] = o.rhi[k] = (int32_t)k;
    }
    __syncthreads();
    int lo = j, hi = j, loc = j;
    int32_t id = (int32_t)k;
    for (int level = 0; in; ++level) {
        const int dL = s_dl[lo], dR = s_dl[hi + 1];
        if (dL < 0 && dR < 0) {  // the root
            if (n <= GROUP_MAX) list_group(o.groups, o.ngroups, n, 0, n);
            if (LINKS) {
                o.parent[n] = -1;
                if (n == 1) o.parent[0] = -1;
            }
            break;
        }
        const bool left = dR > dL;
        const int s = left ? hi : lo - 1;
        s_fid[lo] = id;  // on the frontier unless it is merged below
        if (s < 0 || s >= cnt - 1) break;
        if (level >= MAX_CLIMB) {
            atomicOr(o.err, ASTER_DEVERR_TREE);
            break;
        }
        const int old = meet(&s_slot[s], 1 + (left ? lo : hi) + TREE_LEAVES * loc);
        if (old == 0) break;  // the sibling merges
        const int e = (old - 1) % TREE_LEAVES, sl = (old - 1) / TREE_LEAVES;
        const int sw = sl / TREE_LEAVES, si = sl % TREE_LEAVES;
        const double4 oc = s_cm[sw][si];
        const float4 ol = s_lo[sw][si], oh = s_hi[sw][si];
        double4 pc;
        float4 plo, phi;
        bu_merge(left ? cm : oc, left ? oc : cm, left ? blo : ol, left ? ol : blo, left ? bhi : oh, left ? oh : bhi, pc,
                 plo, phi);
        s_fid[s + 1] = -1;
        s_kids[s] = left ? loc + 256 * sl : sl + 256 * loc;
        if (left) hi = e;
        else lo = e;
        loc = TREE_LEAVES + s;
        cm = pc;
        blo = plo;
        bhi = phi;
        s_cm[1][s] = cm;
        s_lo[1][s] = blo;
        s_hi[1][s] = bhi;
        s_rng[s] = lo + 256 * hi;
        const int nL = s_dl[lo], nR = s_dl[hi + 1];
        id = (int32_t)(n + (nL < 0 && nR < 0 ? 0 : B0 + (nR > nL ? hi : lo)));
        s_id[s] = id;
    }
    __syncthreads();
    const unsigned fm = __ballot_sync(0xffffffffu, s_fid[j] >= 0);
    if ((j & 31) == 0) s_warp[j >> 5] = __popc(fm);
    if (s_id[j] >= 0) {
        const int32_t v = s_id[j];
        const int kL = s_kids[j] & 255, kR = s_kids[j] >> 8;
        const int tL = kL / TREE_LEAVES, iL = kL % TREE_LEAVES, tR = kR / TREE_LEAVES, iR = kR % TREE_LEAVES;
        const int32_t L = tL ? s_id[iL] : (int32_t)(B0 + iL), R = tR ? s_id[iR] : (int32_t)(B0 + iR);
        o.node_cm[v] = s_cm[1][j];
        o.bmin[v] = s_lo[1][j];
        o.bmax[v] = s_hi[1][j];
        o.child[v] = make_int2(L, R);
        put_links<LINKS>(o, v, L, R, B0 + (s_rng[j] & 255), B0 + (s_rng[j] >> 8));
        put_child_record(o.crec + 4 * (v - n), n, theta, L, s_cm[tL][iL], s_lo[tL][iL], s_hi[tL][iL], R, s_cm[tR][iR],
                         s_lo[tR][iR], s_hi[tR][iR]);
    }
    __syncthreads();
    if (s_fid[j] >= 0) {
        const int r = (j >= 32 ? s_warp[0] : 0) + __popc(fm & ((1u << (j & 31)) - 1u));
        front[B0 + r] = make_int2(s_fid[j], (int32_t)(B0 + j));
    }
    if (j == 0) nfront[blockIdx.x] = s_warp[0] + s_warp[1];
}

// One block's share of a merge: `T` items (node, first leaf) in leaf order that
// tile the leaves [base, end).
struct MergeItems {
    int64_t n, end;
    int T;
    const signed char* dl;
};

// The climb of a merge whose items exceed the shared memory (`cap`): the same
// with node data, and the climb state per leaf of the region, in global memory.
struct MergeSpill {
    unsigned long long* slot;
    int32_t *lo, *done, *fid;
};
template <bool LINKS>
__device__ __noinline__ void merge_spilled(const MergeItems m, double theta, const TreeOut o, unsigned long long* slot,
                                           int32_t* ilo, int32_t* done, int32_t* fid) {
    const int64_t n = m.n;
    const int T = m.T;
    auto first = [&](int r) -> int64_t { return r < T ? (int64_t)ilo[r] : m.end; };
    auto delta = [&](int r) -> int {  // across the boundary before item r
        const int64_t l = first(r);
        return l == 0 ? -1 : (int)m.dl[l - 1];
    };
    for (int r = threadIdx.x; r < T; r += MERGE_THREADS) {
        int a = r, b = r;
        int32_t id = fid[r];
        double4 cm = o.node_cm[id];
        float4 lo = id < n ? leaf_lo(cm) : o.bmin[id], hi = id < n ? leaf_hi(cm) : o.bmax[id];
        int dL = delta(r), dR = delta(r + 1);
        for (int level = 0;; ++level) {
            if (dL < 0 && dR < 0) break;  // the root
            const bool left = dR > dL;
            const int s = left ? b : a - 1;
            fid[a] = id;
            if (s < 0 || s >= T - 1) break;
            if (level >= MAX_CLIMB) {
                atomicOr(o.err, ASTER_DEVERR_TREE);
                break;
            }
            __threadfence_block();
            const unsigned long long mine =
                ((unsigned long long)(unsigned)((left ? a : b) + 1) << 32) | (unsigned long long)(unsigned)id;
            const unsigned long long old = atomicExch(&slot[s], mine);
            if (old == 0ull) break;
            __threadfence_block();
            const int e = (int)(old >> 32) - 1;
            const int32_t so = (int32_t)(unsigned)old;
            const double4 oc = o.node_cm[so];
            const float4 ol = so < n ? leaf_lo(oc) : o.bmin[so], oh = so < n ? leaf_hi(oc) : o.bmax[so];
            if (left) b = e;
            else a = e;
            dL = delta(a);
            dR = delta(b + 1);
            double4 pc;
            float4 plo, phi;
            bu_merge(left ? cm : oc, left ? oc : cm, left ? lo : ol, left ? ol : lo, left ? hi : oh, left ? oh : hi, pc,
                     plo, phi);
            const int64_t l0 = first(a), l1 = first(s + 1), l2 = first(b + 1);  // children [l0, l1), [l1, l2)
            const int32_t L = left ? id : so, R = left ? so : id;
            id = (int32_t)(n + (dL < 0 && dR < 0 ? 0 : dR > dL ? l2 - 1 : l0));
            fid[s + 1] = -1;
            done[s] = id;
            cm = pc;
            lo = plo;
            hi = phi;
            o.node_cm[id] = cm;
            o.bmin[id] = lo;
            o.bmax[id] = hi;
            o.child[id] = make_int2(L, R);
            put_links<LINKS>(o, id, L, R, l0, l2 - 1);
            list_children(o, n, l0, l1, l2);
        }
    }
    __syncthreads();
    // the records of the nodes merged here, off the climbs' serial path
    for (int s = threadIdx.x; s < T - 1; s += MERGE_THREADS) {
        const int32_t v = done[s];
        if (v < 0) continue;
        const int2 ch = o.child[v];
        const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
        put_child_record(o.crec + 4 * (v - n), n, theta, ch.x, o.node_cm[ch.x], ch.x < n ? z : o.bmin[ch.x],
                         ch.x < n ? z : o.bmax[ch.x], ch.y, o.node_cm[ch.y], ch.y < n ? z : o.bmin[ch.y],
                         ch.y < n ? z : o.bmax[ch.y]);
    }
}

// Shared memory of a merge of up to `cap` items: per location (item r, or cap +
// the node whose children meet between items s and s + 1) the node's data and
// number; per item its first leaf and the climb state.
__host__ __device__ inline size_t merge_smem_bytes(int cap) {
    return (size_t)cap * (2 * (sizeof(double4) + 2 * sizeof(float4) + sizeof(int32_t)) + 5 * sizeof(int32_t) + 1) + 16;
}

template <bool LINKS>
__global__ void __launch_bounds__(MERGE_THREADS, 1) k_tree_merge(int64_t n, double theta, int64_t region, int64_t sub,
                                                                 int cap, const signed char* __restrict__ dl, TreeOut o,
                                                                 const int2* __restrict__ front_in,
                                                                 const int32_t* __restrict__ nfront_in,
                                                                 int2* __restrict__ front_out,
                                                                 int32_t* __restrict__ nfront_out, MergeSpill spill) {
    extern __shared__ double4 merge_smem[];
    __shared__ int s_off[MERGE_FAN_MAX];
    __shared__ uint32_t s32[32];
    const int64_t base = (int64_t)blockIdx.x * region, end = base + region < n ? base + region : n;
    const int nin = (int)((end - base + sub - 1) / sub);
    const int32_t* nf = nfront_in + base / sub;
    uint32_t total;
    const uint32_t off = block_exclusive_scan((int)threadIdx.x < nin ? (uint32_t)nf[threadIdx.x] : 0u, s32, &total);
    if ((int)threadIdx.x < nin) s_off[threadIdx.x] = (int)off;
    const int T = (int)total;
    const bool fits = T <= cap;
    double4* s_cm = merge_smem;
    float4* s_lo = reinterpret_cast<float4*>(s_cm + 2 * cap);
    float4* s_hi = s_lo + 2 * cap;
    int32_t* s_id = reinterpret_cast<int32_t*>(s_hi + 2 * cap);
    int32_t* s_kids = s_id + 2 * cap;
    int32_t* s_rng = s_kids + cap;
    int32_t* s_slot = s_rng + cap;
    int32_t* ilo = fits ? s_slot + cap : spill.lo + base;
    int32_t* fid = fits ? s_slot + 2 * cap : spill.fid + base;
    signed char* s_dl = reinterpret_cast<signed char*>(s_slot + 3 * cap);  // [r]: delta before item r
    __syncthreads();
    for (int q = threadIdx.x >> 5; q < nin; q += MERGE_THREADS / 32) {
        const int2* f = front_in + base + q * sub;
        const int c = (q + 1 < nin ? s_off[q + 1] : T) - s_off[q];
        for (int i = threadIdx.x & 31; i < c; i += 32) {
            const int2 it = f[i];
            const int r = s_off[q] + i;
            ilo[r] = it.y;
            fid[r] = fits ? -1 : it.x;
            if (fits) {
                const double4 cm = o.node_cm[it.x];
                s_cm[r] = cm;
                s_lo[r] = it.x < n ? leaf_lo(cm) : o.bmin[it.x];
                s_hi[r] = it.x < n ? leaf_hi(cm) : o.bmax[it.x];
                s_dl[r] = it.y == 0 ? (signed char)-1 : dl[it.y - 1];
                s_id[r] = it.x;
                s_id[cap + r] = -1;
                s_slot[r] = 0;
            } else {
                spill.slot[base + r] = 0ull;
                spill.done[base + r] = -1;
            }
        }
    }
    if (fits && threadIdx.x == 0) s_dl[T] = dl[end - 1];
    __syncthreads();
    if (!fits) {
        merge_spilled<LINKS>(MergeItems{n, end, T, dl}, theta, o, spill.slot + base, ilo, spill.done + base, fid);
    } else {
        for (int r = threadIdx.x; r < T; r += MERGE_THREADS) {
            int a = r, b = r, loc = r;
            int32_t id = s_id[r];
            double4 cm = s_cm[r];
            float4 lo = s_lo[r], hi = s_hi[r];
            int dL = s_dl[r], dR = s_dl[r + 1];
            for (int level = 0;; ++level) {
                if (dL < 0 && dR < 0) break;  // the root
                const bool left = dR > dL;
                const int s = left ? b : a - 1;
                fid[a] = id;  // on the frontier unless it is merged below
                if (s < 0 || s >= T - 1) break;
                if (level >= MAX_CLIMB) {
                    atomicOr(o.err, ASTER_DEVERR_TREE);
                    break;
                }
                const int old = meet(&s_slot[s], 1 + (left ? a : b) + (loc << 12));
                if (old == 0) break;  // the sibling merges
                const int e = (old - 1) & 4095, sl = (old - 1) >> 12;
                const double4 oc = s_cm[sl];
                const float4 ol = s_lo[sl], oh = s_hi[sl];
                if (left) b = e;
                else a = e;
                dL = s_dl[a];
                dR = s_dl[b + 1];
                double4 pc;
                float4 plo, phi;
                bu_merge(left ? cm : oc, left ? oc : cm, left ? lo : ol, left ? ol : lo, left ? hi : oh, left ? oh : hi,
                         pc, plo, phi);
                fid[s + 1] = -1;
                s_kids[s] = left ? loc | sl << 16 : sl | loc << 16;
                s_rng[s] = a | b << 16;
                id = (int32_t)(n + (dL < 0 && dR < 0 ? 0 : dR > dL ? (b + 1 < T ? (int64_t)ilo[b + 1] : end) - 1 : ilo[a]));
                loc = cap + s;
                cm = pc;
                lo = plo;
                hi = phi;
                s_id[loc] = id;
                s_cm[loc] = cm;
                s_lo[loc] = lo;
                s_hi[loc] = hi;
            }
        }
        __syncthreads();
        // the merged nodes to global memory, their records, groups and links
        for (int s = threadIdx.x; s < T - 1; s += MERGE_THREADS) {
            const int32_t v = s_id[cap + s];
            if (v < 0) continue;
            const int kL = s_kids[s] & 0xffff, kR = s_kids[s] >> 16, a = s_rng[s] & 0xffff, b = s_rng[s] >> 16;
            const int32_t L = s_id[kL], R = s_id[kR];
            const int64_t l0 = ilo[a], l1 = ilo[s + 1], l2 = b + 1 < T ? (int64_t)ilo[b + 1] : end;
            o.node_cm[v] = s_cm[cap + s];
            o.bmin[v] = s_lo[cap + s];
            o.bmax[v] = s_hi[cap + s];
            o.child[v] = make_int2(L, R);
            put_links<LINKS>(o, v, L, R, l0, l2 - 1);
            list_children(o, n, l0, l1, l2);
            put_child_record(o.crec + 4 * (v - n), n, theta, L, s_cm[kL], s_lo[kL], s_hi[kL], R, s_cm[kR], s_lo[kR],
                             s_hi[kR]);
        }
    }
    if (gridDim.x == 1) {  // the root is done
        if (LINKS && threadIdx.x == 0) o.parent[n] = -1;
        return;
    }
    uint32_t at = 0;
    for (int r0 = 0; r0 < T; r0 += MERGE_THREADS) {
        const int r = r0 + (int)threadIdx.x;
        const bool f = r < T && fid[r] >= 0;
        uint32_t sum;
        const uint32_t p = block_exclusive_scan(f ? 1u : 0u, s32, &sum);
        if (f) front_out[base + at + p] = make_int2(fid[r], ilo[r]);
        at += sum;
    }
    if (threadIdx.x == 0) nfront_out[blockIdx.x] = (int32_t)at;
}

// Arrival at a node of the node-velocity climb: one atomic with
// acquire-release semantics at GPU scope. Its release half publishes this
// climb's node data (written before it) to the climb that arrives second; its
// acquire half makes the sibling's data, published by the first arrival's
// release, visible to the loads that follow.
__device__ __forceinline__ unsigned int bu_arrive(unsigned int* counter) {
    unsigned int old;
    asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(old) : "l"(counter) : "memory");
    return old;
}
__device__ __forceinline__ double4 ld_cg(const double4* p) {
    const double2 a = __ldcg(reinterpret_cast<const double2*>(p));
    const double2 b = __ldcg(reinterpret_cast<const double2*>(p) + 1);
    return make_double4(a.x, a.y, b.x, b.y);
}

// Node velocities for the post-Newtonian walk, in NodesArray::unite form
// (src/solvers/barnes_hut.cpp:150): leaf k holds the velocity of sorted body k,
// an internal node the mass-weighted mean of its children,
// v = (v_R m_R + v_L m_L) / M, with M the node mass from the bottom-up pass
// (M <= 0: (v_R + v_L) / 2). One climb per leaf with the arrival counters of
// the internal nodes (zero on entry); the second arrival merges. Only the
// post-Newtonian walk needs it, so it is a pass of its own.
__global__ void __launch_bounds__(256) k_node_vel(int64_t n, const int32_t* __restrict__ parent,
                                                  const int32_t* __restrict__ sib, const int32_t* __restrict__ perm,
                                                  const double4* __restrict__ vel, const double4* __restrict__ node_cm,
                                                  uint32_t* __restrict__ counters, double4* __restrict__ node_v,
                                                  int* __restrict__ err) {
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x) {
        double4 v = vel[perm[k]];
        v.w = 0.0;
        node_v[k] = v;
        int32_t cur = (int32_t)k;
        int32_t par = n >= 2 ? parent[cur] : -1, sb = n >= 2 ? sib[cur] : 0;
        for (int level = 0; par >= 0; ++level) {
            if (level >= MAX_CLIMB) {
                atomicOr(err, ASTER_DEVERR_TREE);
                break;
            }
            if (bu_arrive(&counters[par - n]) == 0u) break;  // first arrival: the sibling finishes it
            const int32_t so = sb >= 0 ? sb : ~sb;
            const double4 ov = ld_cg(node_v + so);
            const double mc = node_cm[cur].w, mo = node_cm[so].w, M = node_cm[par].w;
            const bool right = sb < 0;  // cur is the right child
            const double4 vR = right ? v : ov, vL = right ? ov : v;
            const double mR = right ? mc : mo, mL = right ? mo : mc;
            double4 pv;
            if (M > 0.0) {
                pv.x = __ddiv_rn(__dadd_rn(__dmul_rn(vR.x, mR), __dmul_rn(vL.x, mL)), M);
                pv.y = __ddiv_rn(__dadd_rn(__dmul_rn(vR.y, mR), __dmul_rn(vL.y, mL)), M);
                pv.z = __ddiv_rn(__dadd_rn(__dmul_rn(vR.z, mR), __dmul_rn(vL.z, mL)), M);
            } else {
                pv.x = __dmul_rn(0.5, __dadd_rn(vR.x, vL.x));
                pv.y = __dmul_rn(0.5, __dadd_rn(vR.y, vL.y));
                pv.z = __dmul_rn(0.5, __dadd_rn(vR.z, vL.z));
            }
            pv.w = 0.0;
            node_v[par] = pv;
            v = pv;
            cur = par;
            par = parent[cur];
            sb = sib[cur];
        }
    }
}

// ----------------------------------------------------------------- walk
template <bool MIXED>
struct WalkShared {
    int stack[WALK_WARPS][WALK_STACK];
    // mixed list, two entries per slot so that each paired FP32 operand is an
    // aligned register pair: lpa = (x0, x1, y0, y1), lpb = (z0, z1, m0, m1),
    // positions relative to the group centre
    float4 lpa[WALK_WARPS][MIXED ? WALK_LIST_MIXED / 2 : 1];
    float4 lpb[WALK_WARPS][MIXED ? WALK_LIST_MIXED / 2 : 1];
    double4 lcm[WALK_WARPS][MIXED ? 1 : WALK_LIST_FP64];  // FP64 (com, mass)
};

// Post-Newtonian walk: each list entry also carries the node's velocity
// (vx, vy, vz, |v|^2), FP32 for the mixed walk and FP64 for the FP64 walk.
template <bool MIXED>
struct WalkSharedPn : WalkShared<MIXED> {
    // mixed: paired like lpa/lpb, lva = (vx0, vx1, vy0, vy1), lvb = (vz0, vz1, w0, w1), w = |v|^2
    float4 lva[WALK_WARPS][MIXED ? WALK_LIST_PN / 2 : 1];
    float4 lvb[WALK_WARPS][MIXED ? WALK_LIST_PN / 2 : 1];
    double4 lvd[WALK_WARPS][MIXED ? 1 : WALK_LIST_FP64];
};

__device__ __forceinline__ void prefetch_l1(const void* p) {
    asm volatile("prefetch.global.L1 [%0];" ::"l"(p));
}
__device__ __forceinline__ float warp_min_f(float v) {
    for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ float warp_max_f(float v) {
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Two interactions at once with the paired FP32 instructions of sm_100
// (add/mul/fma .f32x2): list entries (A.x|A.y, A.z|A.w, B.x|B.y) positions,
// B.z|B.w masses; nb = -(body position) broadcast to both halves.
template <bool GUARD>
__device__ __forceinline__ void interact2_f32(const float4 A, const float4 B, const float2 nbx, const float2 nby,
                                              const float2 nbz, const float2 eps2, float2& ax, float2& ay, float2& az) {
    const float2 dx = __fadd2_rn(make_float2(A.x, A.y), nbx);
    const float2 dy = __fadd2_rn(make_float2(A.z, A.w), nby);
    const float2 dz = __fadd2_rn(make_float2(B.x, B.y), nbz);
    float2 r2 = __ffma2_rn(dz, dz, eps2);
    r2 = __ffma2_rn(dy, dy, r2);
    r2 = __ffma2_rn(dx, dx, r2);
    float2 inv = make_float2(rsqrt_approx(r2.x), rsqrt_approx(r2.y));
    if (GUARD) {
        inv.x = r2.x > 0.f ? inv.x : 0.f;
        inv.y = r2.y > 0.f ? inv.y : 0.f;
    }
    const float2 inv2 = __fmul2_rn(inv, inv);
    const float2 sN = __fmul2_rn(__fmul2_rn(make_float2(B.z, B.w), inv), inv2);
    ax = __ffma2_rn(dx, sN, ax);
    ay = __ffma2_rn(dy, sN, ay);
    az = __ffma2_rn(dz, sN, az);
}

// `count` entries first, first + step, ... of a shared list on one body, FP64,
// Q at a time so that their dependent chains overlap. CHECK: some r^2 may lie
// outside the range of the series step (fp64_pair.cuh); one branch for the Q.
template <bool CHECK, int Q>
__device__ __forceinline__ void interact_list_f64(const double4* __restrict__ list, int first, int step, int count,
                                                  const double4 b, double eps2, double& ax, double& ay, double& az) {
#pragma unroll 1
    for (int e = 0; e < count; e += Q) {
        const double4* l = list + first + e * step;
        double dx[Q], dy[Q], dz[Q], s[Q];
        bool odd = false;
#pragma unroll
        for (int k = 0; k < Q; ++k) {
            const double4 c = l[k * step];
            dx[k] = c.x - b.x; dy[k] = c.y - b.y; dz[k] = c.z - b.z;
            const double r2 = fma(dx[k], dx[k], fma(dy[k], dy[k], fma(dz[k], dz[k], eps2)));
            s[k] = inv_r3_fast(r2) * c.w;
            if (CHECK) odd = odd || !r2_ordinary(r2);
        }
        if (CHECK && odd) {
#pragma unroll 1
            for (int k = 0; k < Q; ++k) {
                const double4 c = l[k * step];
                const double x = c.x - b.x, y = c.y - b.y, z = c.z - b.z;
                const double t = m_inv_r3(c.w, fma(x, x, fma(y, y, fma(z, z, eps2))));
                ax = fma(x, t, ax); ay = fma(y, t, ay); az = fma(z, t, az);
            }
        } else {
#pragma unroll
            for (int k = 0; k < Q; ++k) {
                ax = fma(dx[k], s[k], ax); ay = fma(dy[k], s[k], ay); az = fma(dz[k], s[k], az);
            }
        }
    }
}

// 32 list entries (the ones past the list's end massless) on a lane's two
// bodies: c0 by all of them, c1 (when `two`) by every lps-th from `sub`.
template <bool CHECK>
__device__ __forceinline__ void interact32_f64(const double4* __restrict__ list, const double4 c0, const double4 c1,
                                               bool two, int lps, int sub, double eps2, double& x0, double& y0,
                                               double& z0, double& x1, double& y1, double& z1) {
    interact_list_f64<CHECK, 4>(list, 0, 1, 32, c0, eps2, x0, y0, z0);
    if (!two) return;
    if (lps <= 8) interact_list_f64<CHECK, 4>(list, sub, lps, 32 / lps, c1, eps2, x1, y1, z1);
    else interact_list_f64<CHECK, 1>(list, sub, lps, 32 / lps, c1, eps2, x1, y1, z1);
}

// Softened, and the root's box far inside FP64's range: every r^2 of the walk
// lies in [1e-200, 1e200] and needs no test.
__device__ __forceinline__ bool walk_r2_ordinary(int64_t n, const float4* __restrict__ bmin,
                                                 const float4* __restrict__ bmax, double eps2) {
    if (n < 2 || !(eps2 >= 1e-199 && eps2 < 1e199)) return false;
    const float4 a = bmin[n], b = bmax[n];
    return fmaxf(fmaxf(fmaxf(fabsf(a.x), fabsf(a.y)), fabsf(a.z)), fmaxf(fmaxf(fabsf(b.x), fabsf(b.y)), fabsf(b.z))) <
           1e30f;
}

// One entry with a post-Newtonian force law, FP64: the Newtonian term and the
// terms pk selects (pn.cuh), all divided by G.
// Entry e (position, mass; velocity ev) acts on the body b (velocity vi).
template <int PNL>
__device__ __forceinline__ void interact_pn_f64(const double4 e, const double4 ev, const double4 b, const double4 vi,
                                                double eps2, double G, const PnK<double>& k, double& ax, double& ay,
                                                double& az) {
    const double dx = e.x - b.x, dy = e.y - b.y, dz = e.z - b.z;
    const double r2 = fma(dx, dx, fma(dy, dy, fma(dz, dz, eps2)));
    newton_pn_f64<PNL>(k, dx, dy, dz, inv_r(r2), b.w, e.w, vi, ev, G, ax, ay, az);
}

// Two entries at once with the paired FP32 instructions, force law Newton +
// 1PN: the Newtonian term into (ax, ay, az) as interact2_f32 forms it and the
// 1PN sum of newton_pn1_x2 into (px, py, pz) (the 1PN term divided by G is
// -c^-2 times it). A, B: entry positions and masses as in interact2_f32;
// VA = (vx0, vx1, vy0, vy1), VB = (vz0, vz1, |v0|^2, |v1|^2) the entries'
// velocities. Per body, broadcast to both halves: nb = -(position),
// vi = velocity, vi4 = 4 vi, nvi2 = -|vi|^2, mi5G = 5 G m_i; G4 = 4 G.
template <bool GUARD>
__device__ __forceinline__ void interact2_pn1_f32(const float4 A, const float4 B, const float4 VA, const float4 VB,
                                                  const float2 nbx, const float2 nby, const float2 nbz,
                                                  const float2 vix, const float2 viy, const float2 viz,
                                                  const float2 vi4x, const float2 vi4y, const float2 vi4z,
                                                  const float2 nvi2, const float2 mi5G, const float2 eps2,
                                                  const float2 G4, float2& ax, float2& ay, float2& az, float2& px,
                                                  float2& py, float2& pz) {
    const float2 dx = __fadd2_rn(make_float2(A.x, A.y), nbx);  // entry - body
    const float2 dy = __fadd2_rn(make_float2(A.z, A.w), nby);
    const float2 dz = __fadd2_rn(make_float2(B.x, B.y), nbz);
    newton_pn1_x2<GUARD>(dx, dy, dz, make_float2(B.z, B.w), make_float2(VA.x, VA.y), make_float2(VA.z, VA.w),
                         make_float2(VB.x, VB.y), make_float2(VB.z, VB.w), vix, viy, viz, vi4x, vi4y, vi4z, nvi2,
                         mi5G, eps2, G4, ax, ay, az, px, py, pz);
}

__device__ __forceinline__ float4 vel_f4(const double4 v) {
    return make_float4((float)v.x, (float)v.y, (float)v.z, (float)(v.x * v.x + v.y * v.y + v.z * v.z));
}
__device__ __forceinline__ double4 vel_d4(const double4 v) {
    return make_double4(v.x, v.y, v.z, v.x * v.x + v.y * v.y + v.z * v.z);
}

__device__ __forceinline__ float max3_f32(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// Pairs q0i, q0i + step, ... < np of a list with velocities acting on one body,
// two entries per paired FP32 instruction: the Newtonian sum into sx, sy, sz,
// the 1PN sum into p and the 2PN + 2.5PN sum into qq. PNL = 1: Newton + 1PN;
// 2: the terms that pk.f selects.
template <int PNL, bool GUARD>
__device__ __forceinline__ void pn_list(const float4* LA, const float4* LB, const float4* LVA, const float4* LVB,
                                        int np, int q0i, int step, const float2 nbx, const float2 nby,
                                        const float2 nbz, const float4 vf, float mi, const float2 e2, double G,
                                        const PnK<double>& pk, CompSum& sx, CompSum& sy, CompSum& sz, float3& p,
                                        float3& qq) {
    const float Gf = (float)G, mc2 = -(float)pk.c2;
    const float2 G4 = make_float2(4.f * Gf, 4.f * Gf);
    const float2 vix = make_float2(vf.x, vf.x), viy = make_float2(vf.y, vf.y), viz = make_float2(vf.z, vf.z),
                 nvi2 = make_float2(-vf.w, -vf.w), vi4x = make_float2(4.f * vf.x, 4.f * vf.x),
                 vi4y = make_float2(4.f * vf.y, 4.f * vf.y), vi4z = make_float2(4.f * vf.z, 4.f * vf.z),
                 mi5G = make_float2(5.f * Gf * mi, 5.f * Gf * mi);
    float2 ax = make_float2(0.f, 0.f), ay = ax, az = ax, px = ax, py = ax, pz = ax;
    if constexpr (PNL == 1) {
#pragma unroll 2
        for (int q = q0i; q < np; q += step)
            interact2_pn1_f32<GUARD>(LA[q], LB[q], LVA[q], LVB[q], nbx, nby, nbz, vix, viy, viz, vi4x, vi4y, vi4z,
                                     nvi2, mi5G, e2, G4, ax, ay, az, px, py, pz);
    } else {
        const float mc4 = -(float)pk.c4, nkf = -0.8f * (float)pk.ic;
        const float2 G2 = make_float2(Gf, Gf), nk = make_float2(nkf, nkf), vi2 = make_float2(vf.w, vf.w),
                     Gmi = make_float2(Gf * mi, Gf * mi);
        float2 qx = make_float2(0.f, 0.f), qy = qx, qz = qx;
        for (int q = q0i; q < np; q += step) {
            const float4 A = LA[q], B = LB[q], VA = LVA[q], VB = LVB[q];
            const float2 dx = __fadd2_rn(make_float2(A.x, A.y), nbx);  // entry - body
            const float2 dy = __fadd2_rn(make_float2(A.z, A.w), nby);
            const float2 dz = __fadd2_rn(make_float2(B.x, B.y), nbz);
            newton_pn_all_x2<GUARD>(dx, dy, dz, make_float2(B.z, B.w), make_float2(VA.x, VA.y),
                                    make_float2(VA.z, VA.w), make_float2(VB.x, VB.y), make_float2(VB.z, VB.w), vix,
                                    viy, viz, vi4x, vi4y, vi4z, nvi2, vi2, mi5G, Gmi, e2, G4, G2, nk, pk.f, ax, ay,
                                    az, px, py, pz, qx, qy, qz);
        }
        qq.x = fmaf(mc4, qx.x + qx.y, qq.x);
        qq.y = fmaf(mc4, qy.x + qy.y, qq.y);
        qq.z = fmaf(mc4, qz.x + qz.y, qq.z);
    }
    sx.add(ax.x + ax.y); sy.add(ay.x + ay.y); sz.add(az.x + az.y);
    p.x = fmaf(mc2, px.x + px.y, p.x);
    p.y = fmaf(mc2, py.x + py.y, p.y);
    p.z = fmaf(mc2, pz.x + pz.y, p.z);
}

// Opening test of both children of a node for the whole group, FP32
// round-to-nearest without FMA (the CPU restatement reproduces it bit for
// bit), the two children in the halves of paired FP32 operations: the squared
// distance from a child's FP32 centre of mass to the group box is
// sum over axes of max(lo - c, c - hi, 0)^2; the child is accepted when it
// exceeds the child's r_crit^2. lo - c is formed as fma(c, -1, lo), which is
// the correctly rounded difference; nhi = -hi.
__device__ __forceinline__ float2 box_dist2_pair(const float2 cx, const float2 cy, const float2 cz, const float2 lox,
                                                 const float2 loy, const float2 loz, const float2 nhix,
                                                 const float2 nhiy, const float2 nhiz) {
    const float2 m1 = make_float2(-1.f, -1.f);
    const float2 ux = __ffma2_rn(cx, m1, lox), wx = __fadd2_rn(cx, nhix);
    const float2 uy = __ffma2_rn(cy, m1, loy), wy = __fadd2_rn(cy, nhiy);
    const float2 uz = __ffma2_rn(cz, m1, loz), wz = __fadd2_rn(cz, nhiz);
    const float2 tx = make_float2(max3_f32(ux.x, wx.x, 0.f), max3_f32(ux.y, wx.y, 0.f));
    const float2 ty = make_float2(max3_f32(uy.x, wy.x, 0.f), max3_f32(uy.y, wy.y, 0.f));
    const float2 tz = make_float2(max3_f32(uz.x, wz.x, 0.f), max3_f32(uz.y, wz.y, 0.f));
    return __fadd2_rn(__fadd2_rn(__fmul2_rn(tx, tx), __fmul2_rn(ty, ty)), __fmul2_rn(tz, tz));
}

// Persistent walk: each warp takes groups from a global work counter until
// none are left. Per group: lane l holds sorted leaf l of the group; the r
// leaves beyond 32 are each shared by 32/r (rounded down to a power of two)
// lanes that split the interaction list between them, so groups of 33..64
// bodies keep every lane busy. The warp pops up to 32 opened internal nodes
// per round from its shared stack; each lane loads the contiguous record of
// its node's two children (centres of mass, masses, opening radii: one
// 64-byte load, issued together with the child indices) and tests both:
// leaves and accepted cells go to the shared interaction list, opened
// internal children to the stack. The list is evaluated 32 entries at a
// time by every lane.
// Mixed precision: list entries and bodies are stored relative to the group
// centre cg (FP32 of hi - cg plus the double-single low part), so an
// interaction needs one subtraction per axis; the group is compact, so the
// relative coordinates keep FP32 precision of the separation.
// PNL > 0: the post-Newtonian walk (the terms pk selects, with the nodes'
// velocities node_v); PNL == 0 is the Newtonian kernel. GUARD (mixed): unsoftened,
// a zero distance contributes nothing (the FP64 sums see to that by themselves).
template <bool MIXED, bool GUARD, bool KICK, int PNL = 0>
__global__ void __launch_bounds__(WALK_WARPS * 32, PNL ? 4 : ASTER_WALK_MINBLOCKS) k_walk(
    int64_t n, const int2* __restrict__ groups, const unsigned int* __restrict__ ngroups_p,
    unsigned int* __restrict__ work,
    const float4* __restrict__ crec, const double4* __restrict__ node_cm, const int2* __restrict__ child,
    const int32_t* __restrict__ perm, double G, double eps2, double half_dt, double4* __restrict__ acc,
    double4* __restrict__ vel, int* __restrict__ err, int* __restrict__ stack_hw, int stack_limit,
    int32_t* __restrict__ body_counts, unsigned long long* __restrict__ inter_count,
    const double4* __restrict__ node_v, PnK<double> pk, double4* __restrict__ pm_next, double dt_next,
    unsigned long long* __restrict__ box_next, const float4* __restrict__ bmin, const float4* __restrict__ bmax) {
    using Shared = typename std::conditional<PNL != 0, WalkSharedPn<MIXED>, WalkShared<MIXED>>::type;
    __shared__ Shared sm;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t lt = (1u << lane) - 1u;
    // ngroups_p[0] groups of more than GROUP_SMALL bodies at groups[0..), then
    // ngroups_p[3] smaller ones at groups[n - 1], groups[n - 2], ...
    const unsigned int nbig = ngroups_p[0], ngroups = nbig + ngroups_p[3];
    int* stack = sm.stack[warp];
    int hw = 1;
    unsigned long long wtotal = 0;
    double box = 0.0;  // fused next drift: max |coordinate| of the drifted bodies
    const bool plain = !MIXED && PNL == 0 && walk_r2_ordinary(n, bmin, bmax, eps2);

    for (;;) {
        unsigned int g = 0;
        if (lane == 0) g = atomicAdd(work, 1u);
        g = __shfl_sync(0xffffffffu, g, 0);
        if (g >= ngroups) break;
        const int2 gr = groups[g < nbig ? (int64_t)g : n - 1 - (int64_t)(g - nbig)];
        // Bodies 0..31 of the group: one per lane (primary). Bodies 32.. (r of
        // them, "secondary"): each shared by lps lanes that split the list.
        const int r = gr.y > 32 ? gr.y - 32 : 0;
        const bool two = r > 0;  // warp-uniform
        int lps = 32;
        while (lps > 1 && lps * r > 32) lps >>= 1;
        const int sb = lane / lps, sub = lane & (lps - 1);
        const bool v0 = lane < gr.y, v1 = two && sb < r;
        const int64_t k0 = (int64_t)gr.x + (v0 ? lane : 0);
        const int64_t k1 = (int64_t)gr.x + (v1 ? 32 + sb : 0);
        // the bodies' input indices, for the results (loaded now, used at the end)
        const int32_t pb0 = perm[k0], pb1 = perm[k1];

        float4 h0, l0, h1, l1;  // the bodies' traversal data, from their leaves
        leaf_trav(node_cm[k0], h0, l0);
        if (two) {
            leaf_trav(node_cm[k1], h1, l1);
        } else {
            h1 = h0;
            l1 = l0;
        }
        const float glox = warp_min_f(fminf(v0 ? h0.x : INFINITY, v1 ? h1.x : INFINITY));
        const float gloy = warp_min_f(fminf(v0 ? h0.y : INFINITY, v1 ? h1.y : INFINITY));
        const float gloz = warp_min_f(fminf(v0 ? h0.z : INFINITY, v1 ? h1.z : INFINITY));
        const float ghix = warp_max_f(fmaxf(v0 ? h0.x : -INFINITY, v1 ? h1.x : -INFINITY));
        const float ghiy = warp_max_f(fmaxf(v0 ? h0.y : -INFINITY, v1 ? h1.y : -INFINITY));
        const float ghiz = warp_max_f(fmaxf(v0 ? h0.z : -INFINITY, v1 ? h1.z : -INFINITY));
        const float cgx = 0.5f * (glox + ghix), cgy = 0.5f * (gloy + ghiy), cgz = 0.5f * (gloz + ghiz);
        const float3 b0 = make_float3((h0.x - cgx) + l0.x, (h0.y - cgy) + l0.y, (h0.z - cgz) + l0.z);
        const float3 b1 = make_float3((h1.x - cgx) + l1.x, (h1.y - cgy) + l1.y, (h1.z - cgz) + l1.z);
        const float2 nb0x = make_float2(-b0.x, -b0.x), nb0y = make_float2(-b0.y, -b0.y), nb0z = make_float2(-b0.z, -b0.z);
        const float2 nb1x = make_float2(-b1.x, -b1.x), nb1y = make_float2(-b1.y, -b1.y), nb1z = make_float2(-b1.z, -b1.z);
        const float2 eps2f2 = make_float2((float)eps2, (float)eps2);
        double4 c0 = make_double4(0, 0, 0, 0), c1 = c0;
        if (!MIXED) {
            c0 = node_cm[k0];
            c1 = two ? node_cm[k1] : c0;
        }
        // post-Newtonian walk: the bodies' own velocities and the running
        // 1PN (p) and 2PN + 2.5PN (q) sums of the mixed walk
        float4 vf0 = make_float4(0.f, 0.f, 0.f, 0.f), vf1 = vf0;
        double4 vd0 = make_double4(0, 0, 0, 0), vd1 = vd0;
        float3 p0 = make_float3(0.f, 0.f, 0.f), q0 = p0, p1 = p0, q1 = p0;
        if constexpr (PNL > 0) {
            if (MIXED) {
                vf0 = vel_f4(node_v[k0]);
                vf1 = two ? vel_f4(node_v[k1]) : vf0;
            } else {
                vd0 = vel_d4(node_v[k0]);
                vd1 = two ? vel_d4(node_v[k1]) : vd0;
            }
        }

        CompSum sx0, sy0, sz0, sx1, sy1, sz1;
        double dx0 = 0, dy0 = 0, dz0 = 0, dx1 = 0, dy1 = 0, dz1 = 0;
        int top = 0, lc = 0;
        int total = 0;
        bool overflow = false;

        // store list entry `pos` (lane-private): mixed = group-relative position and mass
        auto put = [&](int pos, float x, float y, float z, float mass) {
            float* A = reinterpret_cast<float*>(&sm.lpa[warp][0]);
            float* B = reinterpret_cast<float*>(&sm.lpb[warp][0]);
            const int o = ((pos >> 1) << 2) | (pos & 1);
            A[o] = x;
            A[o + 2] = y;
            B[o] = z;
            B[o + 2] = mass;
        };

        // post-Newtonian walk: the velocity of list entry `pos`
        auto put_v = [&](int pos, const double4 v) {
            if constexpr (PNL > 0) {
                if (MIXED) {
                    const float4 f = vel_f4(v);
                    float* VA = reinterpret_cast<float*>(&sm.lva[warp][0]);
                    float* VB = reinterpret_cast<float*>(&sm.lvb[warp][0]);
                    const int o = ((pos >> 1) << 2) | (pos & 1);
                    VA[o] = f.x;
                    VA[o + 2] = f.y;
                    VB[o] = f.z;
                    VB[o + 2] = f.w;
                } else {
                    sm.lvd[warp][pos] = vel_d4(v);
                }
            }
        };

        auto evaluate = [&](int cnt) __attribute__((always_inline)) {
            if constexpr (PNL > 0) {
                if constexpr (MIXED) {
                    const int np = (cnt + 1) >> 1;  // an odd cnt: last slot half zero-padded by the caller
                    pn_list<PNL, GUARD>(sm.lpa[warp], sm.lpb[warp], sm.lva[warp], sm.lvb[warp], np, 0, 1, nb0x, nb0y,
                                        nb0z, vf0, h0.w, eps2f2, G, pk, sx0, sy0, sz0, p0, q0);
                    if (two)
                        pn_list<PNL, GUARD>(sm.lpa[warp], sm.lpb[warp], sm.lva[warp], sm.lvb[warp], np, sub, lps, nb1x,
                                            nb1y, nb1z, vf1, h1.w, eps2f2, G, pk, sx1, sy1, sz1, p1, q1);
                } else {
                    for (int e = 0; e < cnt; ++e)
                        interact_pn_f64<PNL>(sm.lcm[warp][e], sm.lvd[warp][e], c0, vd0, eps2, G, pk, dx0, dy0,
                                                    dz0);
                    if (two)
                        for (int e = sub; e < cnt; e += lps)
                            interact_pn_f64<PNL>(sm.lcm[warp][e], sm.lvd[warp][e], c1, vd1, eps2, G, pk, dx1,
                                                        dy1, dz1);
                }
                total += cnt;
                return;
            }
            if (MIXED) {
                // an odd cnt has its last slot half zero-padded by the caller
                const int np = (cnt + 1) >> 1;
                float2 ax0 = make_float2(0.f, 0.f), ay0 = ax0, az0 = ax0;
                if (two && lps == 1) {  // 49..64 bodies: both bodies of a lane share each list load
                    float2 ax1 = make_float2(0.f, 0.f), ay1 = ax1, az1 = ax1;
#pragma unroll 4
                    for (int q = 0; q < np; ++q) {
                        const float4 A = sm.lpa[warp][q], B = sm.lpb[warp][q];
                        interact2_f32<GUARD>(A, B, nb0x, nb0y, nb0z, eps2f2, ax0, ay0, az0);
                        interact2_f32<GUARD>(A, B, nb1x, nb1y, nb1z, eps2f2, ax1, ay1, az1);
                    }
                    sx0.add(ax0.x + ax0.y); sy0.add(ay0.x + ay0.y); sz0.add(az0.x + az0.y);
                    sx1.add(ax1.x + ax1.y); sy1.add(ay1.x + ay1.y); sz1.add(az1.x + az1.y);
                    total += cnt;
                    return;
                }
#pragma unroll WALK_UNROLL
                for (int q = 0; q < np; ++q)
                    interact2_f32<GUARD>(sm.lpa[warp][q], sm.lpb[warp][q], nb0x, nb0y, nb0z, eps2f2, ax0, ay0, az0);
                sx0.add(ax0.x + ax0.y); sy0.add(ay0.x + ay0.y); sz0.add(az0.x + az0.y);
                if (two) {
                    float2 ax1 = make_float2(0.f, 0.f), ay1 = ax1, az1 = ax1;
#pragma unroll 4
                    for (int q = sub; q < np; q += lps)
                        interact2_f32<GUARD>(sm.lpa[warp][q], sm.lpb[warp][q], nb1x, nb1y, nb1z, eps2f2, ax1, ay1, az1);
                    sx1.add(ax1.x + ax1.y); sy1.add(ay1.x + ay1.y); sz1.add(az1.x + az1.y);
                }
            } else {
                // cnt = 32, or the rest of the list, padded to 32 by the caller
                if (plain) interact32_f64<false>(sm.lcm[warp], c0, c1, two, lps, sub, eps2, dx0, dy0, dz0, dx1, dy1, dz1);
                else interact32_f64<true>(sm.lcm[warp], c0, c1, two, lps, sub, eps2, dx0, dy0, dz0, dx1, dy1, dz1);
            }
            total += cnt;
        };

        const int nI = (int)n;  // node ids are int32: leaves < nI <= internal nodes
        if (n >= 2) {
            if (lane == 0) stack[0] = nI;  // the root is internal: start by opening it
            top = 1;
        } else {
            if (lane == 0) {  // a single body: its own leaf
                if (MIXED) {
                    float4 h, l;
                    leaf_trav(node_cm[0], h, l);
                    put(0, (h.x - cgx) + l.x, (h.y - cgy) + l.y, (h.z - cgz) + l.z, h.w);
                } else {
                    sm.lcm[warp][0] = node_cm[0];
                }
                put_v(0, PNL > 0 ? node_v[0] : make_double4(0, 0, 0, 0));
            }
            lc = 1;
        }
        __syncwarp();
        const float2 lox2 = make_float2(glox, glox), loy2 = make_float2(gloy, gloy), loz2 = make_float2(gloz, gloz);
        const float2 nhix2 = make_float2(-ghix, -ghix), nhiy2 = make_float2(-ghiy, -ghiy),
                     nhiz2 = make_float2(-ghiz, -ghiz);
        const float2 ncgx2 = make_float2(-cgx, -cgx), ncgy2 = make_float2(-cgy, -cgy), ncgz2 = make_float2(-cgz, -cgz);

        while (top > 0) {
            const int cnt = top < 32 ? top : 32;
            const bool act = lane < cnt;
            // inactive lanes read the root's record (valid memory) and are masked off
            int v = nI;
            if (act) v = stack[top - 1 - lane];
            __syncwarp();
            top -= cnt;
            const float4* rec = crec + 4 * (int64_t)(v - nI);
            const float4 r0 = rec[0], r1 = rec[1], r2 = rec[2], r3 = rec[3];
            const int2 ch = child[v];
            const float2 cx = make_float2(r0.x, r0.y), cy = make_float2(r0.z, r0.w), cz = make_float2(r1.x, r1.y);
            const float2 d2 = box_dist2_pair(cx, cy, cz, lox2, loy2, loz2, nhix2, nhiy2, nhiz2);
            const bool fL = ch.x < nI || d2.x > r3.z, fR = ch.y < nI || d2.y > r3.w;  // leaf or far enough
            const bool aL = act && fL, aR = act && fR, oL = act && !fL, oR = act && !fR;
            const uint32_t mAL = __ballot_sync(0xffffffffu, aL), mAR = __ballot_sync(0xffffffffu, aR);
            const uint32_t mOL = __ballot_sync(0xffffffffu, oL), mOR = __ballot_sync(0xffffffffu, oR);
            const int npush = __popc(mOL) + __popc(mOR);
            if (top + npush > stack_limit) {
                overflow = true;
                break;
            }
            {
                const int pos = top + __popc(mOL & lt) + __popc(mOR & lt);
                if (oL) stack[pos] = ch.x;
                if (oR) stack[pos + (oL ? 1 : 0)] = ch.y;
            }
            top += npush;
            hw = top > hw ? top : hw;
            {
                const int pos = lc + __popc(mAL & lt) + __popc(mAR & lt);
                if (MIXED) {
                    // both children's group-relative positions: (c - cg) + remainder
                    const float2 ex = __fadd2_rn(__fadd2_rn(cx, ncgx2), make_float2(r2.x, r2.y));
                    const float2 ey = __fadd2_rn(__fadd2_rn(cy, ncgy2), make_float2(r2.z, r2.w));
                    const float2 ez = __fadd2_rn(__fadd2_rn(cz, ncgz2), make_float2(r3.x, r3.y));
                    if (aL) put(pos, ex.x, ey.x, ez.x, r1.z);
                    if (aR) put(pos + (aL ? 1 : 0), ex.y, ey.y, ez.y, r1.w);
                } else {
                    if (aL) sm.lcm[warp][pos] = node_cm[ch.x];
                    if (aR) sm.lcm[warp][pos + (aL ? 1 : 0)] = node_cm[ch.y];
                }
                if constexpr (PNL > 0) {
                    if (aL) put_v(pos, node_v[ch.x]);
                    if (aR) put_v(pos + (aL ? 1 : 0), node_v[ch.y]);
                }
            }
            lc += __popc(mAL) + __popc(mAR);
            __syncwarp();
            constexpr int FL = MIXED ? (PNL ? WALK_FLUSH_PN : WALK_FLUSH_MIXED) : WALK_FLUSH_FP64;
            while (lc >= FL) {
                evaluate(FL);
                __syncwarp();
                const int rest = lc - FL;  // < 64
                if (MIXED) {  // whole slots (FL is even), at most 32; read all, then write
                    const int ns = (rest + 1) >> 1;
                    float4 a = make_float4(0, 0, 0, 0), b = a;
                    if (lane < ns) { a = sm.lpa[warp][FL / 2 + lane]; b = sm.lpb[warp][FL / 2 + lane]; }
                    __syncwarp();
                    if (lane < ns) { sm.lpa[warp][lane] = a; sm.lpb[warp][lane] = b; }
                } else {
                    const bool m0 = lane < rest, m1 = lane + 32 < rest;
                    double4 x0 = make_double4(0, 0, 0, 0), x1 = x0;
                    if (m0) x0 = sm.lcm[warp][32 + lane];
                    if (m1) x1 = sm.lcm[warp][64 + lane];
                    __syncwarp();
                    if (m0) sm.lcm[warp][lane] = x0;
                    if (m1) sm.lcm[warp][32 + lane] = x1;
                }
                if constexpr (PNL > 0) {  // the entries' velocities: [FL, FL + rest) -> [0, rest), rest < 64
                    const bool m0 = lane < rest, m1 = lane + 32 < rest;
                    if (MIXED) {  // whole slots, as for the positions
                        const int ns = (rest + 1) >> 1;
                        float4 a = make_float4(0, 0, 0, 0), b = a;
                        if (lane < ns) { a = sm.lva[warp][FL / 2 + lane]; b = sm.lvb[warp][FL / 2 + lane]; }
                        __syncwarp();
                        if (lane < ns) { sm.lva[warp][lane] = a; sm.lvb[warp][lane] = b; }
                    } else {
                        double4 x0 = make_double4(0, 0, 0, 0), x1 = x0;
                        if (m0) x0 = sm.lvd[warp][FL + lane];
                        if (m1) x1 = sm.lvd[warp][FL + 32 + lane];
                        __syncwarp();
                        if (m0) sm.lvd[warp][lane] = x0;
                        if (m1) sm.lvd[warp][32 + lane] = x1;
                    }
                }
                lc = rest;
                __syncwarp();
            }
        }
        if (overflow) {
            if (lane == 0) atomicOr(err, ASTER_DEVERR_STACK);
            break;
        }
        if (!MIXED && PNL == 0 && lane >= lc) sm.lcm[warp][lane] = make_double4(0, 0, 0, 0);  // the last 32, padded
        if (MIXED && (lc & 1) && lane == 0) {  // zero mass, zero offset: contributes nothing
            float* A = reinterpret_cast<float*>(&sm.lpa[warp][0]);
            float* B = reinterpret_cast<float*>(&sm.lpb[warp][0]);
            const int q = lc >> 1;
            A[4 * q + 1] = 0.f; A[4 * q + 3] = 0.f; B[4 * q + 1] = 0.f; B[4 * q + 3] = 0.f;
            if constexpr (PNL > 0) {  // and zero velocity, so the 1PN term is 0 * finite
                float* VA = reinterpret_cast<float*>(&sm.lva[warp][0]);
                float* VB = reinterpret_cast<float*>(&sm.lvb[warp][0]);
                VA[4 * q + 1] = 0.f; VA[4 * q + 3] = 0.f; VB[4 * q + 1] = 0.f; VB[4 * q + 3] = 0.f;
            }
        }
        __syncwarp();
        if (KICK) {  // the closing kick's operands into L1 while the last list is evaluated
            prefetch_l1(vel + pb0);
            if (pm_next) prefetch_l1(pm_next + pb0);
            if (v1 && sub == 0) {
                prefetch_l1(vel + pb1);
                if (pm_next) prefetch_l1(pm_next + pb1);
            }
        }
        if (lc > 0) evaluate(lc);
        __syncwarp();
        wtotal += (unsigned long long)total * (unsigned long long)gr.y;
        // secondary bodies: add the lps partial sums (aligned lane groups)
        double s1x = MIXED ? sx1.value() : dx1, s1y = MIXED ? sy1.value() : dy1, s1z = MIXED ? sz1.value() : dz1;
        if constexpr (PNL > 0) {
            if (MIXED) {
                s1x += (double)p1.x + (double)q1.x;
                s1y += (double)p1.y + (double)q1.y;
                s1z += (double)p1.z + (double)q1.z;
            }
        }
        if (two) {
            for (int o = lps >> 1; o >= 1; o >>= 1) {
                s1x += __shfl_xor_sync(0xffffffffu, s1x, o);
                s1y += __shfl_xor_sync(0xffffffffu, s1y, o);
                s1z += __shfl_xor_sync(0xffffffffu, s1z, o);
            }
        }
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const bool vq = q ? (v1 && sub == 0) : v0;
            if (!vq) continue;
            double ax, ay, az;
            if (q) {
                ax = G * s1x; ay = G * s1y; az = G * s1z;
            } else if (MIXED) {
                if constexpr (PNL > 0) {
                    ax = G * (sx0.value() + ((double)p0.x + (double)q0.x));
                    ay = G * (sy0.value() + ((double)p0.y + (double)q0.y));
                    az = G * (sz0.value() + ((double)p0.z + (double)q0.z));
                } else {
                    ax = G * sx0.value(); ay = G * sy0.value(); az = G * sz0.value();
                }
            } else {
                ax = G * dx0; ay = G * dy0; az = G * dz0;
            }
            const int32_t b = q ? pb1 : pb0;
            acc[b] = make_double4(ax, ay, az, 0.0);
            if (body_counts) body_counts[b] = total;
            if (KICK) {
                double4 vv = vel[b];
                vv.x += ax * half_dt; vv.y += ay * half_dt; vv.z += az * half_dt;
                if (pm_next) {
                    // the next step's opening kick and drift, the same operations
                    // in the same order as its kick-drift kernel would apply them
                    // (that kernel does not run then); other bodies' positions
                    // are read from the tree, never from pm
                    vv.x += ax * half_dt; vv.y += ay * half_dt; vv.z += az * half_dt;
                    double4 pp = pm_next[b];
                    pp.x += vv.x * dt_next; pp.y += vv.y * dt_next; pp.z += vv.z * dt_next;
                    pm_next[b] = pp;
                    box = fmax(box, fmax(fabs(pp.x), fmax(fabs(pp.y), fabs(pp.z))));
                }
                vel[b] = vv;
            }
        }
    }
    if (box_next) {
        for (int o = 16; o > 0; o >>= 1) box = fmax(box, __shfl_xor_sync(0xffffffffu, box, o));
        // non-negative doubles order like their bit patterns
        if (lane == 0) atomicMax(box_next, (unsigned long long)__double_as_longlong(box));
    }
    if (lane == 0) {
        atomicMax(stack_hw, hw);
        atomicAdd(inter_count, wtotal);
    }
}

// Team walk: a block of TEAM_WARPS warps per group, for trees with too few
// groups to fill the GPU with one warp each. Warp 0 traverses (the rounds of
// k_walk, the same lists in the same order) and hands the list over in batches
// of WARPS - 1 chunks through a double buffer; the other warps evaluate
// one chunk each while it goes on. A chunk is WALK_FLUSH_MIXED entries, as in
// k_walk, so that every FP32 partial sum is the same as there; only the order
// in which the chunks' sums are added differs (compensated FP32 per warp, FP64
// over the warps). FP64: the list holds node ids, and each evaluating warp
// gathers the nodes of its chunk 32 at a time, so that the traversal does not
// wait for them; post-Newtonian velocities come the same way in both
// precisions. Bound by the traversal's ~85 dependent rounds a group (mixed)
// or by the FP64 pipe (FP64); chunk, warps and resident teams are the best of
// 64 / 96 / 128 entries, 3 to 8 warps and 2 to 6 teams per SM at 1000 to
// 262,144 bodies (fewer teams leave FP64 the registers it would spill).
template <bool MIXED, int PNL = 0>
struct TeamSize {
    static constexpr int WARPS = MIXED ? 4 : 5;
    static constexpr int PER_SM = MIXED ? (PNL ? 4 : 5) : 3;
    static constexpr int CHUNK = MIXED && PNL == 0 ? WALK_FLUSH_MIXED : 64;
    static constexpr int BATCH = (WARPS - 1) * CHUNK;
    static constexpr int LIST = BATCH + 64;  // a round appends up to 64 entries
    static_assert(CHUNK >= 64 && CHUNK % 32 == 0, "the rest of a list is at most WARPS chunks");
};

template <bool MIXED, int PNL>
struct TeamShared {
    using Size = TeamSize<MIXED, PNL>;
    int stack[WALK_STACK];
    float4 lpa[2][MIXED ? Size::LIST / 2 : 1];  // as WalkShared::lpa, lpb
    float4 lpb[2][MIXED ? Size::LIST / 2 : 1];
    int lid[2][MIXED && PNL == 0 ? 1 : Size::LIST];  // node ids
    double4 lcm[Size::WARPS][MIXED ? 1 : 32];        // the entries a warp evaluates
    double4 lvd[Size::WARPS][!MIXED && PNL ? 32 : 1];  // and their velocities
    float4 lva[Size::WARPS][MIXED && PNL ? Size::CHUNK / 2 : 1];  // mixed: paired as in WalkSharedPn
    float4 lvb[Size::WARPS][MIXED && PNL ? Size::CHUNK / 2 : 1];
    double sum[Size::WARPS][6][32];
    int cnt[2];    // entries in each buffer
    int state[2];  // of each buffer: 0 more to come, 1 last batch, 2 stack overflow
    unsigned int next;
};

template <bool MIXED, bool GUARD, bool KICK, int PNL>
__global__ void __launch_bounds__(TeamSize<MIXED, PNL>::WARPS * 32, TeamSize<MIXED, PNL>::PER_SM) k_walk_team(
    int64_t n, const int2* __restrict__ groups, const unsigned int* __restrict__ ngroups_p,
    unsigned int* __restrict__ work, const float4* __restrict__ crec, const double4* __restrict__ node_cm,
    const int2* __restrict__ child, const int32_t* __restrict__ perm, double G, double eps2, double half_dt,
    double4* __restrict__ acc, double4* __restrict__ vel, int* __restrict__ err, int* __restrict__ stack_hw,
    int stack_limit, int32_t* __restrict__ body_counts, unsigned long long* __restrict__ inter_count,
    const double4* __restrict__ node_v, PnK<double> pk, double4* __restrict__ pm_next, double dt_next,
    unsigned long long* __restrict__ box_next, const float4* __restrict__ bmin, const float4* __restrict__ bmax) {
    __shared__ TeamShared<MIXED, PNL> sm;
    using Size = TeamSize<MIXED, PNL>;
    constexpr int TEAM_WARPS = Size::WARPS, TEAM_CHUNK = Size::CHUNK, TEAM_BATCH = Size::BATCH;
    const bool plain = !MIXED && PNL == 0 && walk_r2_ordinary(n, bmin, bmax, eps2);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t lt = (1u << lane) - 1u;
    const unsigned int nbig = ngroups_p[0], ngroups = nbig + ngroups_p[3];
    const int nI = (int)n;
    int hw = 1;
    unsigned long long wtotal = 0;
    double box = 0.0;
    if (threadIdx.x == 0) sm.next = atomicAdd(work, 1u);
    __syncthreads();
    for (;;) {
        const unsigned int g = sm.next;
        __syncthreads();
        if (g >= ngroups) break;
        if (threadIdx.x == 32) sm.next = atomicAdd(work, 1u);  // read after this group's barriers
        const int2 gr = groups[g < nbig ? (int64_t)g : n - 1 - (int64_t)(g - nbig)];
        const int r = gr.y > 32 ? gr.y - 32 : 0;
        const bool two = r > 0;
        int lps = 32;
        while (lps > 1 && lps * r > 32) lps >>= 1;
        const int sb = lane / lps, sub = lane & (lps - 1);
        const bool v0 = lane < gr.y, v1 = two && sb < r;
        const int64_t k0 = (int64_t)gr.x + (v0 ? lane : 0);
        const int64_t k1 = (int64_t)gr.x + (v1 ? 32 + sb : 0);
        const double4 c0 = node_cm[k0], c1 = two ? node_cm[k1] : c0;
        float4 h0, l0, h1, l1;
        leaf_trav(c0, h0, l0);
        leaf_trav(c1, h1, l1);
        const float glox = warp_min_f(fminf(v0 ? h0.x : INFINITY, v1 ? h1.x : INFINITY));
        const float gloy = warp_min_f(fminf(v0 ? h0.y : INFINITY, v1 ? h1.y : INFINITY));
        const float gloz = warp_min_f(fminf(v0 ? h0.z : INFINITY, v1 ? h1.z : INFINITY));
        const float ghix = warp_max_f(fmaxf(v0 ? h0.x : -INFINITY, v1 ? h1.x : -INFINITY));
        const float ghiy = warp_max_f(fmaxf(v0 ? h0.y : -INFINITY, v1 ? h1.y : -INFINITY));
        const float ghiz = warp_max_f(fmaxf(v0 ? h0.z : -INFINITY, v1 ? h1.z : -INFINITY));
        const float cgx = 0.5f * (glox + ghix), cgy = 0.5f * (gloy + ghiy), cgz = 0.5f * (gloz + ghiz);
        const float3 b0 = make_float3((h0.x - cgx) + l0.x, (h0.y - cgy) + l0.y, (h0.z - cgz) + l0.z);
        const float3 b1 = make_float3((h1.x - cgx) + l1.x, (h1.y - cgy) + l1.y, (h1.z - cgz) + l1.z);
        CompSum sx0, sy0, sz0, sx1, sy1, sz1;
        double dx0 = 0, dy0 = 0, dz0 = 0, dx1 = 0, dy1 = 0, dz1 = 0;
        // the bodies' velocities and the 1PN (p) and 2PN + 2.5PN (q) sums, as in k_walk
        float4 vf0 = make_float4(0.f, 0.f, 0.f, 0.f), vf1 = vf0;
        double4 vd0 = make_double4(0, 0, 0, 0), vd1 = vd0;
        float3 p0 = make_float3(0.f, 0.f, 0.f), q0 = p0, p1 = p0, q1 = p0;
        if constexpr (PNL > 0) {
            if (MIXED) {
                vf0 = vel_f4(node_v[k0]);
                vf1 = two ? vel_f4(node_v[k1]) : vf0;
            } else {
                vd0 = vel_d4(node_v[k0]);
                vd1 = two ? vel_d4(node_v[k1]) : vd0;
            }
        }

        // one chunk: cnt entries from entry `from` of buffer b
        auto evaluate = [&](int b, int from, int cnt) __attribute__((always_inline)) {
            if constexpr (MIXED) {
                const float4* A = sm.lpa[b] + from / 2;
                const float4* B = sm.lpb[b] + from / 2;
                const float2 e2 = make_float2((float)eps2, (float)eps2);
                const float2 nb0x = make_float2(-b0.x, -b0.x), nb0y = make_float2(-b0.y, -b0.y),
                             nb0z = make_float2(-b0.z, -b0.z);
                const float2 nb1x = make_float2(-b1.x, -b1.x), nb1y = make_float2(-b1.y, -b1.y),
                             nb1z = make_float2(-b1.z, -b1.z);
                const int np = (cnt + 1) >> 1;  // an odd list has its last half slot zeroed
                if constexpr (PNL > 0) {  // the warp fetches its chunk's velocities, the traversal only lists the nodes
                    const int* id = sm.lid[b] + from;
                    float* VA = reinterpret_cast<float*>(sm.lva[warp]);
                    float* VB = reinterpret_cast<float*>(sm.lvb[warp]);
                    __syncwarp();
#pragma unroll
                    for (int e = lane; e < TEAM_CHUNK; e += 32) {
                        const float4 v = vel_f4(e < cnt ? node_v[id[e]] : make_double4(0, 0, 0, 0));
                        const int o = ((e >> 1) << 2) | (e & 1);
                        VA[o] = v.x;
                        VA[o + 2] = v.y;
                        VB[o] = v.z;
                        VB[o + 2] = v.w;
                    }
                    __syncwarp();
                    pn_list<PNL, GUARD>(A, B, sm.lva[warp], sm.lvb[warp], np, 0, 1, nb0x, nb0y, nb0z, vf0, h0.w, e2, G,
                                        pk, sx0, sy0, sz0, p0, q0);
                    if (two)
                        pn_list<PNL, GUARD>(A, B, sm.lva[warp], sm.lvb[warp], np, sub, lps, nb1x, nb1y, nb1z, vf1,
                                            h1.w, e2, G, pk, sx1, sy1, sz1, p1, q1);
                    return;
                }
                float2 ax0 = make_float2(0.f, 0.f), ay0 = ax0, az0 = ax0, ax1 = ax0, ay1 = ax0, az1 = ax0;
                if (two && lps == 1) {
#pragma unroll 4
                    for (int q = 0; q < np; ++q) {
                        interact2_f32<GUARD>(A[q], B[q], nb0x, nb0y, nb0z, e2, ax0, ay0, az0);
                        interact2_f32<GUARD>(A[q], B[q], nb1x, nb1y, nb1z, e2, ax1, ay1, az1);
                    }
                } else {
#pragma unroll WALK_UNROLL
                    for (int q = 0; q < np; ++q)
                        interact2_f32<GUARD>(A[q], B[q], nb0x, nb0y, nb0z, e2, ax0, ay0, az0);
                    if (two) {
#pragma unroll 4
                        for (int q = sub; q < np; q += lps)
                            interact2_f32<GUARD>(A[q], B[q], nb1x, nb1y, nb1z, e2, ax1, ay1, az1);
                    }
                }
                sx0.add(ax0.x + ax0.y); sy0.add(ay0.x + ay0.y); sz0.add(az0.x + az0.y);
                if (two) { sx1.add(ax1.x + ax1.y); sy1.add(ay1.x + ay1.y); sz1.add(az1.x + az1.y); }
            } else {
                const int* id = sm.lid[b] + from;
                double4* st = sm.lcm[warp];
                if constexpr (PNL > 0) {
                    double4* sv = sm.lvd[warp];
                    for (int e0 = 0; e0 < cnt; e0 += 32) {
                        __syncwarp();
                        if (e0 + lane < cnt) {
                            st[lane] = node_cm[id[e0 + lane]];
                            sv[lane] = vel_d4(node_v[id[e0 + lane]]);
                        }
                        __syncwarp();
                        const int m = cnt - e0 < 32 ? cnt - e0 : 32;
                        for (int e = 0; e < m; ++e)
                            interact_pn_f64<PNL>(st[e], sv[e], c0, vd0, eps2, G, pk, dx0, dy0, dz0);
                        if (two)
                            for (int e = sub; e < m; e += lps)
                                interact_pn_f64<PNL>(st[e], sv[e], c1, vd1, eps2, G, pk, dx1, dy1, dz1);
                    }
                    return;
                }
                double4 nx = lane < cnt ? node_cm[id[lane]] : make_double4(0, 0, 0, 0);
                for (int e0 = 0; e0 < cnt; e0 += 32) {
                    __syncwarp();
                    st[lane] = nx;
                    __syncwarp();
                    nx = e0 + 32 + lane < cnt ? node_cm[id[e0 + 32 + lane]] : make_double4(0, 0, 0, 0);
                    if (plain) interact32_f64<false>(st, c0, c1, two, lps, sub, eps2, dx0, dy0, dz0, dx1, dy1, dz1);
                    else interact32_f64<true>(st, c0, c1, two, lps, sub, eps2, dx0, dy0, dz0, dx1, dy1, dz1);
                }
            }
        };
        auto put = [&](int b, int pos, float x, float y, float z, float mass) {
            float* A = reinterpret_cast<float*>(sm.lpa[b]);
            float* B = reinterpret_cast<float*>(sm.lpb[b]);
            const int o = ((pos >> 1) << 2) | (pos & 1);
            A[o] = x;
            A[o + 2] = y;
            B[o] = z;
            B[o + 2] = mass;
        };

        // the traversing warp's state
        int top = 0, lc = 0, total = 0;
        bool overflow = false;
        const float2 lox2 = make_float2(glox, glox), loy2 = make_float2(gloy, gloy), loz2 = make_float2(gloz, gloz);
        const float2 nhix2 = make_float2(-ghix, -ghix), nhiy2 = make_float2(-ghiy, -ghiy),
                     nhiz2 = make_float2(-ghiz, -ghiz);
        const float2 ncgx2 = make_float2(-cgx, -cgx), ncgy2 = make_float2(-cgy, -cgy), ncgz2 = make_float2(-cgz, -cgz);
        if (warp == 0) {
            if (n >= 2) {
                if (lane == 0) sm.stack[0] = nI;
                top = 1;
            } else {
                if (lane == 0) {
                    if (MIXED) put(0, 0, b0.x, b0.y, b0.z, h0.w);
                    if (!MIXED || PNL > 0) sm.lid[0][0] = 0;
                }
                lc = 1;
            }
            __syncwarp();
        }
        // traverses until buffer b holds a batch or nothing is left to open
        auto fill = [&](int b) {
            while (top > 0 && lc < TEAM_BATCH) {
                const int cnt = top < 32 ? top : 32;
                const bool act = lane < cnt;
                int v = nI;
                if (act) v = sm.stack[top - 1 - lane];
                __syncwarp();
                top -= cnt;
                const float4* rec = crec + 4 * (int64_t)(v - nI);
                const float4 r0 = rec[0], r1 = rec[1], r2 = rec[2], r3 = rec[3];
                const int2 ch = child[v];
                const float2 cx = make_float2(r0.x, r0.y), cy = make_float2(r0.z, r0.w), cz = make_float2(r1.x, r1.y);
                const float2 d2 = box_dist2_pair(cx, cy, cz, lox2, loy2, loz2, nhix2, nhiy2, nhiz2);
                const bool fL = ch.x < nI || d2.x > r3.z, fR = ch.y < nI || d2.y > r3.w;
                const bool aL = act && fL, aR = act && fR, oL = act && !fL, oR = act && !fR;
                const uint32_t mAL = __ballot_sync(0xffffffffu, aL), mAR = __ballot_sync(0xffffffffu, aR);
                const uint32_t mOL = __ballot_sync(0xffffffffu, oL), mOR = __ballot_sync(0xffffffffu, oR);
                const int npush = __popc(mOL) + __popc(mOR);
                if (top + npush > stack_limit) {
                    overflow = true;
                    return;
                }
                {
                    const int pos = top + __popc(mOL & lt) + __popc(mOR & lt);
                    if (oL) sm.stack[pos] = ch.x;
                    if (oR) sm.stack[pos + (oL ? 1 : 0)] = ch.y;
                }
                top += npush;
                hw = top > hw ? top : hw;
                const int pos = lc + __popc(mAL & lt) + __popc(mAR & lt);
                if (MIXED) {
                    const float2 ex = __fadd2_rn(__fadd2_rn(cx, ncgx2), make_float2(r2.x, r2.y));
                    const float2 ey = __fadd2_rn(__fadd2_rn(cy, ncgy2), make_float2(r2.z, r2.w));
                    const float2 ez = __fadd2_rn(__fadd2_rn(cz, ncgz2), make_float2(r3.x, r3.y));
                    if (aL) put(b, pos, ex.x, ey.x, ez.x, r1.z);
                    if (aR) put(b, pos + (aL ? 1 : 0), ex.y, ey.y, ez.y, r1.w);
                }
                if (!MIXED || PNL > 0) {
                    if (aL) sm.lid[b][pos] = ch.x;
                    if (aR) sm.lid[b][pos + (aL ? 1 : 0)] = ch.y;
                }
                lc += __popc(mAL) + __popc(mAR);
                __syncwarp();
            }
        };
        int b = 0;
        bool fail = false;
        for (;;) {
            if (warp == 0) {
                fill(b);
                const bool last = overflow || top == 0;
                if (MIXED && top == 0 && (lc & 1) && lane == 0) put(b, lc, 0.f, 0.f, 0.f, 0.f);
                if (lane == 0) {
                    sm.cnt[b] = lc;
                    sm.state[b] = overflow ? 2 : last ? 1 : 0;
                }
            }
            __syncthreads();  // buffer b is full; the other one has been evaluated
            const int cnt = sm.cnt[b], state = sm.state[b];
            if (state != 0) {
                fail = state == 2;
                // the rest: up to TEAM_WARPS chunks (warp 0 takes the fourth)
                const int from = ((warp + TEAM_WARPS - 1) % TEAM_WARPS) * TEAM_CHUNK;
                if (!fail && from < cnt) evaluate(b, from, cnt - from < TEAM_CHUNK ? cnt - from : TEAM_CHUNK);
                total += cnt;
                break;
            }
            total += TEAM_BATCH;
            if (warp == 0) {  // carry the entries beyond the batch over
                const int rest = lc - TEAM_BATCH;  // < 64
                if (MIXED) {
                    if (lane < (rest + 1) >> 1) {
                        sm.lpa[b ^ 1][lane] = sm.lpa[b][TEAM_BATCH / 2 + lane];
                        sm.lpb[b ^ 1][lane] = sm.lpb[b][TEAM_BATCH / 2 + lane];
                    }
                }
                if (!MIXED || PNL > 0) {
                    if (lane < rest) sm.lid[b ^ 1][lane] = sm.lid[b][TEAM_BATCH + lane];
                    if (lane + 32 < rest) sm.lid[b ^ 1][lane + 32] = sm.lid[b][TEAM_BATCH + 32 + lane];
                }
                lc = rest;
                __syncwarp();
            } else {
                evaluate(b, (warp - 1) * TEAM_CHUNK, TEAM_CHUNK);
            }
            b ^= 1;  // (sm.cnt, sm.state of a buffer are rewritten two barriers after they are read)
        }
        if (fail) {
            if (threadIdx.x == 0) atomicOr(err, ASTER_DEVERR_STACK);
            break;
        }
        {
            double(*s)[32] = sm.sum[warp];
            s[0][lane] = MIXED ? sx0.value() : dx0; s[1][lane] = MIXED ? sy0.value() : dy0;
            s[2][lane] = MIXED ? sz0.value() : dz0; s[3][lane] = MIXED ? sx1.value() : dx1;
            s[4][lane] = MIXED ? sy1.value() : dy1; s[5][lane] = MIXED ? sz1.value() : dz1;
            if (MIXED && PNL > 0) {
                s[0][lane] += (double)p0.x + (double)q0.x; s[1][lane] += (double)p0.y + (double)q0.y;
                s[2][lane] += (double)p0.z + (double)q0.z; s[3][lane] += (double)p1.x + (double)q1.x;
                s[4][lane] += (double)p1.y + (double)q1.y; s[5][lane] += (double)p1.z + (double)q1.z;
            }
        }
        __syncthreads();
        if (warp == 0) wtotal += (unsigned long long)total * (unsigned long long)gr.y;
        // warp 0: bodies 0..31; warp 1: the secondary bodies
        if (warp < 2 && (warp == 0 || two)) {
            double ax = 0, ay = 0, az = 0;
#pragma unroll
            for (int w = 0; w < TEAM_WARPS; ++w) {
                ax += sm.sum[w][3 * warp][lane];
                ay += sm.sum[w][3 * warp + 1][lane];
                az += sm.sum[w][3 * warp + 2][lane];
            }
            if (warp == 1)
                for (int o = lps >> 1; o >= 1; o >>= 1) {
                    ax += __shfl_xor_sync(0xffffffffu, ax, o);
                    ay += __shfl_xor_sync(0xffffffffu, ay, o);
                    az += __shfl_xor_sync(0xffffffffu, az, o);
                }
            if (warp == 0 ? v0 : (v1 && sub == 0)) {
                ax *= G; ay *= G; az *= G;
                const int32_t body = perm[warp == 0 ? k0 : k1];
                acc[body] = make_double4(ax, ay, az, 0.0);
                if (body_counts) body_counts[body] = total;
                if (KICK) {
                    double4 vv = vel[body];
                    vv.x += ax * half_dt; vv.y += ay * half_dt; vv.z += az * half_dt;
                    if (pm_next) {  // the next step's opening kick and drift, as in k_walk
                        vv.x += ax * half_dt; vv.y += ay * half_dt; vv.z += az * half_dt;
                        double4 pp = pm_next[body];
                        pp.x += vv.x * dt_next; pp.y += vv.y * dt_next; pp.z += vv.z * dt_next;
                        pm_next[body] = pp;
                        box = fmax(box, fmax(fabs(pp.x), fmax(fabs(pp.y), fabs(pp.z))));
                    }
                    vel[body] = vv;
                }
            }
        }
        // the next group's first barrier orders these reads of sm.sum before its writes
    }
    if (box_next && warp < 2) {
        for (int o = 16; o > 0; o >>= 1) box = fmax(box, __shfl_xor_sync(0xffffffffu, box, o));
        if (lane == 0) atomicMax(box_next, (unsigned long long)__double_as_longlong(box));
    }
    if (threadIdx.x == 0) {
        atomicMax(stack_hw, hw);
        atomicAdd(inter_count, wtotal);
    }
}

// Up to these sizes a tree has too few groups for one warp each (mixed: 740
// resident teams against 2960 warps, about 3000 groups at 10^5 bodies).
// Walk at theta = 0.5, k_walk against the team, us: mixed 5000 bodies 82, 46;
// 20,011: 125, 66; 60,000: 196, 135; 100,000: 238, 201; 131,073: 244, 248;
// 262,144: 432, 480. FP64 5000: 164, 64; 20,011: 225, 98; 60,000: 391, 236;
// 131,073: 580, 492; 262,144: 942, 948; 1,048,576: 3556, 4002. 1PN mixed 3000:
// 183, 120; 20,011: 429, 191; 60,000: 595, 366; 119,000: 681, 622; FP64 20,011:
// 796, 386; 119,000: 1465, 1379; 190,000: 2274, 2178. Every term, mixed 20,011:
// 867, 419; 119,000: 1738, 1521; FP64 20,011: 1355, 597; 119,000: 2749, 2266;
// 190,000: 3942, 3599. (At theta = 0.8 the two meet somewhat earlier: Newton mixed
// 119,000 113, 119, FP64 190,000 309, 332.)
constexpr int64_t TEAM_MAX_MIXED = 120000, TEAM_MAX_FP64 = 200000;

template <bool MIXED, bool GUARD, bool KICK, int PNL>
int launch_team(aster_ctx* c, const aster_params* p, int32_t* counts, bool fuse_next) {
    LbvhBufs& t = c->tree;
    auto kern = k_walk_team<MIXED, GUARD, KICK, PNL>;
    int per_sm = 0;
    ASTER_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, TeamSize<MIXED, PNL>::WARPS * 32, 0));
    if (per_sm < 1) per_sm = 1;
    const int64_t blocks = std::min<int64_t>((int64_t)c->sm_count * per_sm, c->n);  // groups <= n
    unsigned int* gcount = red_groups(c);
    kern<<<(unsigned)blocks, TeamSize<MIXED, PNL>::WARPS * 32, 0, c->stream>>>(
        c->n, t.groups.as<int2>(), gcount, gcount + 1, t.crec.as<float4>(), t.node_cm.as<double4>(),
        t.child.as<int2>(), t.perm.as<int32_t>(), p->G, p->eps2, 0.5 * p->dt, c->acc.as<double4>(),
        c->vel.as<double4>(), c->err_dev, c->stack_hw_dev, c->walk_stack_limit, counts, red_inter(c),
        PNL > 0 ? t.node_v.as<double4>() : nullptr, make_pn(p), KICK && fuse_next ? c->pm.as<double4>() : nullptr, p->dt, KICK && fuse_next ? red_box(c) : nullptr,
        t.bmin.as<float4>(), t.bmax.as<float4>());
    ASTER_CUDA(cudaGetLastError());
    return ASTER_OK;
}

template <bool MIXED, bool GUARD, bool KICK, int PNL = 0>
int launch_walk(aster_ctx* c, const aster_params* p, int32_t* counts, bool fuse_next) {
    LbvhBufs& t = c->tree;
    if (c->n <= std::min(c->walk_team_limit, MIXED ? TEAM_MAX_MIXED : TEAM_MAX_FP64))
        return launch_team<MIXED, GUARD, KICK, PNL>(c, p, counts, fuse_next);
    auto kern = k_walk<MIXED, GUARD, KICK, PNL>;
    int per_sm = 0;
    ASTER_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, WALK_WARPS * 32, 0));
    if (per_sm < 1) per_sm = 1;
    int64_t blocks = (int64_t)c->sm_count * per_sm;
    const int64_t need = (c->n + WALK_WARPS - 1) / WALK_WARPS;  // groups <= n
    if (blocks > need) blocks = need;
    unsigned int* gcount = red_groups(c);
    kern<<<(unsigned)blocks, WALK_WARPS * 32, 0, c->stream>>>(
        c->n, t.groups.as<int2>(), gcount, gcount + 1,
        t.crec.as<float4>(), t.node_cm.as<double4>(), t.child.as<int2>(), t.perm.as<int32_t>(), p->G, p->eps2, 0.5 * p->dt,
        c->acc.as<double4>(), c->vel.as<double4>(), c->err_dev, c->stack_hw_dev, c->walk_stack_limit, counts,
        red_inter(c), PNL > 0 ? t.node_v.as<double4>() : nullptr, make_pn(p),
        KICK && fuse_next ? c->pm.as<double4>() : nullptr, p->dt, KICK && fuse_next ? red_box(c) : nullptr,
        t.bmin.as<float4>(), t.bmax.as<float4>());
    ASTER_CUDA(cudaGetLastError());
    return ASTER_OK;
}

template <class KeyT>
int run_sort(aster_ctx* c, int bits) {
    LbvhBufs& t = c->tree;
    const int64_t n = c->n;
    const int nblocks = (int)((n + SORT_TILE - 1) / SORT_TILE);
    const int passes = (bits + 7) / 8;  // 30 -> 4, 63 -> 8 (even: result lands in sorted_codes)
    uint32_t* hist = t.hist.as<uint32_t>();
    uint32_t* dtot = t.digit_off.as<uint32_t>();
    const KeyT* kin = t.codes.as<KeyT>();
    const int32_t* vin = nullptr;
    for (int ps = 0; ps < passes; ++ps) {
        KeyT* kout = (ps & 1) ? t.sorted_codes.as<KeyT>() : t.codes_alt.as<KeyT>();
        int32_t* vout = (ps & 1) ? t.perm.as<int32_t>() : t.perm_alt.as<int32_t>();
        const int shift = 8 * ps;
        k_sort_hist<KeyT><<<nblocks, SORT_THREADS, 0, c->stream>>>(n, kin, shift, nblocks, hist);
        k_scan_digits<<<RADIX, 1024, 0, c->stream>>>(hist, nblocks, dtot);
        if (ps == 0)
            k_sort_scatter<KeyT, true><<<nblocks, SORT_THREADS, 0, c->stream>>>(n, kin, nullptr, kout, vout, shift,
                                                                             nblocks, hist, dtot);
        else
            k_sort_scatter<KeyT, false><<<nblocks, SORT_THREADS, 0, c->stream>>>(n, kin, vin, kout, vout, shift,
                                                                              nblocks, hist, dtot);
        ASTER_CUDA(cudaGetLastError());
        c->stats.kernels += 3;
        kin = kout;
        vin = vout;
    }
    return ASTER_OK;
}

// One cluster's launch; false (nothing launched) where the device cannot hold
// such a cluster.
template <class KeyT, int MODE, int ITEMS>
bool launch_sort_cluster(aster_ctx* c, bool want_codes, int* st) {
    LbvhBufs& t = c->tree;
    auto kern = k_sort_cluster<KeyT, MODE, ITEMS>;
    const size_t smem = cluster_sort_smem<KeyT>(ITEMS);
    const int blocks = (int)((c->n + (int64_t)CSORT_THREADS * ITEMS - 1) / ((int64_t)CSORT_THREADS * ITEMS));
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)blocks);
    cfg.blockDim = dim3(CSORT_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = c->stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)blocks;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int fit = 0;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
        cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&fit, kern, &cfg) != cudaSuccess || fit < 1) {
        cudaGetLastError();
        return false;
    }
    const cudaError_t e =
        cudaLaunchKernelEx(&cfg, kern, c->n, (const double4*)c->pm.as<double4>(),
                           (const unsigned long long*)red_box(c), want_codes ? t.codes.as<KeyT>() : (KeyT*)nullptr,
                           t.sorted_codes.as<KeyT>(), t.perm.as<int32_t>(), red_groups(c));
    *st = e == cudaSuccess ? ASTER_OK : aster_cuda_fail(e, "k_sort_cluster", __FILE__, __LINE__);
    c->stats.kernels += 1;
    return true;
}
template <class KeyT, int MODE>
bool sort_cluster(aster_ctx* c, bool want_codes, int* st) {
    const int64_t per = (c->n + (int64_t)CSORT_THREADS * CSORT_BLOCKS - 1) / ((int64_t)CSORT_THREADS * CSORT_BLOCKS);
    if (per <= 1) return launch_sort_cluster<KeyT, MODE, 1>(c, want_codes, st);
    if (per <= 2) return launch_sort_cluster<KeyT, MODE, 2>(c, want_codes, st);
    return false;  // four keys a thread: 98 us a build at 40,000 bodies, as the general sort's
}

template <class KeyT, bool COMPAT, bool LINKS>
int run_tree(aster_ctx* c, const aster_params* p, bool zero_box) {
    LbvhBufs& t = c->tree;
    const int64_t n = c->n;
    int64_t nb = (n + TREE_LEAVES - 1) / TREE_LEAVES, sub = TREE_LEAVES;
    const TreeOut o{t.node_cm.as<double4>(), t.bmin.as<float4>(), t.bmax.as<float4>(), t.child.as<int2>(),
                    t.crec.as<float4>(), LINKS ? t.parent.as<int32_t>() : nullptr, LINKS ? t.sib.as<int32_t>() : nullptr,
                    LINKS ? t.rlo.as<int32_t>() : nullptr, LINKS ? t.rhi.as<int32_t>() : nullptr,
                    t.groups.as<int2>(), red_groups(c), c->err_dev};
    // frontiers alternate between two arrays; the sort's alternate keys, histogram and the leaves' unused boxes are free
    int2* fr[2] = {t.front.as<int2>(), t.codes_alt.as<int2>()};
    int32_t* nfr[2] = {t.hist.as<int32_t>(), t.hist.as<int32_t>() + nb};
    const MergeSpill spill{t.bmax.as<unsigned long long>(), t.perm_alt.as<int32_t>(), t.counters.as<int32_t>(),
                           t.bmin.as<int32_t>()};
    signed char* dl = t.dl.as<signed char>();
    k_tree_local<KeyT, COMPAT, LINKS><<<(unsigned)nb, TREE_LEAVES, 0, c->stream>>>(
        n, p->theta, t.sorted_codes.as<KeyT>(), t.perm.as<int32_t>(), c->pm.as<double4>(), o, dl, fr[0], nfr[0],
        zero_box ? red_box(c) : nullptr);
    ASTER_CUDA(cudaGetLastError());
    c->stats.kernels += 1;
    ASTER_CUDA(cudaFuncSetAttribute(k_tree_merge<LINKS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)merge_smem_bytes(MERGE_CAP)));
    for (int cur = 0; nb > 1; cur ^= 1) {
        // a block of R leaves leaves about log2(R) + 0.3 subtrees over (Plummer, 2^20 bodies: 6.3 of 64 leaves, 8.3 of
        // 256): one block takes the rest when its items fit, else each takes as many as fit
        const double items = 1.2 * (std::log2((double)sub) + 0.3);
        const bool last = nb <= MERGE_FAN_MAX && (double)nb * items <= MERGE_CAP;
        const int cap = last || sub > TREE_LEAVES || nb > MERGE_MANY ? MERGE_CAP : MERGE_CAP0;
        int64_t fan = nb;
        if (!last)
            for (fan = 4; 2 * fan * items <= cap && fan < 64;) fan *= 2;
        const int64_t region = sub * fan, out = (n + region - 1) / region;
        k_tree_merge<LINKS><<<(unsigned)out, MERGE_THREADS, merge_smem_bytes(cap), c->stream>>>(
            n, p->theta, region, sub, cap, dl, o, fr[cur], nfr[cur], fr[cur ^ 1], nfr[cur ^ 1], spill);
        ASTER_CUDA(cudaGetLastError());
        c->stats.kernels += 1;
        sub = region;
        nb = out;
    }
    return ASTER_OK;
}

template <class KeyT>
int run_build(aster_ctx* c, const aster_params* p, bool links, bool zero_box) {
    LbvhBufs& t = c->tree;
    const int64_t n = c->n;
    const int grid = (int)std::min<int64_t>((n + 255) / 256, (int64_t)c->sm_count * 16);
    const unsigned long long* box = red_box(c);
    const int mode = p->compat_mode ? 2 : (p->morton_bits == 63 ? 1 : 0);
    unsigned int* gcount = red_groups(c);  // [0] large groups, [1] walk work counter, [3] small groups: zeroed with
                                           // the codes
    int cst = ASTER_OK;
    bool sorted = false;
    if constexpr (sizeof(KeyT) == 8) sorted = sort_cluster<KeyT, 1>(c, links, &cst);
    else sorted = mode == 2 ? sort_cluster<KeyT, 2>(c, links, &cst) : sort_cluster<KeyT, 0>(c, links, &cst);
    if (cst != ASTER_OK) return cst;
    if (!sorted) {
        const double4* pm = c->pm.as<double4>();
        KeyT* codes = t.codes.as<KeyT>();
        if constexpr (sizeof(KeyT) == 8) k_morton<KeyT, 1><<<grid, 256, 0, c->stream>>>(n, pm, box, codes, gcount);
        else if (mode == 2) k_morton<KeyT, 2><<<grid, 256, 0, c->stream>>>(n, pm, box, codes, gcount);
        else k_morton<KeyT, 0><<<grid, 256, 0, c->stream>>>(n, pm, box, codes, gcount);
        ASTER_CUDA(cudaGetLastError());
        c->stats.kernels += 1;
        ASTER_TRY(run_sort<KeyT>(c, p->morton_bits == 63 ? 64 : 32));
    }
    if (p->compat_mode) {
        // OpenCL order is descending by (code, index): reverse the ascending sort
        k_reverse<KeyT><<<grid, 256, 0, c->stream>>>(n, t.sorted_codes.as<KeyT>(), t.perm.as<int32_t>(),
                                                     t.codes_alt.as<KeyT>(), t.perm_alt.as<int32_t>());
        ASTER_CUDA(cudaMemcpyAsync(t.sorted_codes.ptr, t.codes_alt.ptr, (size_t)n * sizeof(KeyT),
                                   cudaMemcpyDeviceToDevice, c->stream));
        ASTER_CUDA(cudaMemcpyAsync(t.perm.ptr, t.perm_alt.ptr, (size_t)n * sizeof(int32_t), cudaMemcpyDeviceToDevice,
                                   c->stream));
        c->stats.kernels += 1;
    }
    ASTER_TRY(aster_apply_pending_mass(c));  // the leaf gather below is the first reader of the masses
    if (p->compat_mode) return links ? run_tree<KeyT, true, true>(c, p, zero_box)
                                        : run_tree<KeyT, true, false>(c, p, zero_box);
    return links ? run_tree<KeyT, false, true>(c, p, zero_box) : run_tree<KeyT, false, false>(c, p, zero_box);
}

int ensure_tree(aster_ctx* c, bool links) {
    LbvhBufs& t = c->tree;
    const int64_t n = c->n, m = 2 * n;  // 2n-1 nodes, +1 slot so parent[n] exists for n == 1
    const int64_t nblocks = (n + SORT_TILE - 1) / SORT_TILE;
    ASTER_TRY(t.codes.ensure((size_t)n * 8));
    ASTER_TRY(t.codes_alt.ensure((size_t)n * 8));
    ASTER_TRY(t.sorted_codes.ensure((size_t)n * 8));
    ASTER_TRY(t.perm.ensure((size_t)n * 4));
    ASTER_TRY(t.perm_alt.ensure((size_t)n * 4));
    ASTER_TRY(t.hist.ensure((size_t)nblocks * RADIX * 4));
    ASTER_TRY(t.digit_off.ensure((size_t)RADIX * 4));
    if (links) {
        ASTER_TRY(t.parent.ensure((size_t)m * 4));
        ASTER_TRY(t.sib.ensure((size_t)m * 4));
        ASTER_TRY(t.rlo.ensure((size_t)m * 4));
        ASTER_TRY(t.rhi.ensure((size_t)m * 4));
    }
    ASTER_TRY(t.front.ensure((size_t)n * sizeof(int2)));
    ASTER_TRY(t.dl.ensure((size_t)n));
    ASTER_TRY(t.counters.ensure((size_t)n * 4));
    ASTER_TRY(t.node_cm.ensure((size_t)m * sizeof(double4)));
    ASTER_TRY(t.bmin.ensure((size_t)m * sizeof(float4)));
    ASTER_TRY(t.bmax.ensure((size_t)m * sizeof(float4)));
    ASTER_TRY(t.child.ensure((size_t)m * sizeof(int2)));
    ASTER_TRY(t.groups.ensure((size_t)n * sizeof(int2)));
    ASTER_TRY(t.crec.ensure((size_t)4 * n * sizeof(float4)));
    ASTER_TRY(c->red.ensure(4096));
    t.n = n;
    return ASTER_OK;
}

}  // namespace

int aster_lbvh_build_dev(aster_ctx* c, const aster_params* p, bool box_ready, bool links, bool zero_box) {
    links = links || pn_level(p) > 0;  // the node velocities climb by parent and sibling
    ASTER_TRY(ensure_tree(c, links));
    if (!box_ready) {
        unsigned long long* box = red_box(c);
        ASTER_CUDA(cudaMemsetAsync(box, 0, sizeof(unsigned long long), c->stream));
        const int grid = (int)std::min<int64_t>((c->n + 255) / 256, (int64_t)c->sm_count * 8);
        k_box<<<grid, 256, 0, c->stream>>>(c->n, c->pm.as<double4>(), box);
        ASTER_CUDA(cudaGetLastError());
        c->stats.kernels += 1;
    }
    if (p->morton_bits == 63) ASTER_TRY(run_build<uint64_t>(c, p, links, zero_box));
    else ASTER_TRY(run_build<uint32_t>(c, p, links, zero_box));
    c->tree.built = true;
    return ASTER_OK;
}

int aster_lbvh_walk_launch(aster_ctx* c, const aster_params* p, int precision, bool kick, int32_t* counts,
                           bool fuse_next) {
    if (kick) c->mixed_valid = false;  // the closing kick moves the velocities
    fuse_next = fuse_next && kick;
    // the work counter and, with fuse_next, the box are zero: the build that just ran left them so
    const bool guard = !(p->eps2 > 0.0);
    if (precision != ASTER_MIXED && precision != ASTER_FP64) return ASTER_ERR_INVALID_ARG;
    const bool mixed = precision == ASTER_MIXED;
    if (pn_level(p) > 0) {
        // post-Newtonian law: node velocities from the current body velocities
        // (one climb, fresh arrival counters), then the walk with the pair law
        LbvhBufs& t = c->tree;
        const int64_t n = c->n;
        ASTER_TRY(t.node_v.ensure((size_t)2 * n * sizeof(double4)));
        if (n >= 2) ASTER_CUDA(cudaMemsetAsync(t.counters.ptr, 0, (size_t)(n - 1) * sizeof(uint32_t), c->stream));
        const int grid = (int)std::min<int64_t>((n + 255) / 256, (int64_t)c->sm_count * 8);
        k_node_vel<<<grid, 256, 0, c->stream>>>(n, t.parent.as<int32_t>(), t.sib.as<int32_t>(), t.perm.as<int32_t>(),
                                                c->vel.as<double4>(), t.node_cm.as<double4>(),
                                                t.counters.as<uint32_t>(), t.node_v.as<double4>(), c->err_dev);
        ASTER_CUDA(cudaGetLastError());
        c->stats.kernels += 1;
        if (mixed && pn_level(p) == 1) {  // Newton + 1PN: the paired-FP32 list evaluation
            if (guard) { ASTER_TRY(kick ? launch_walk<true, true, true, 1>(c, p, counts, fuse_next) : launch_walk<true, true, false, 1>(c, p, counts, fuse_next)); }
            else       { ASTER_TRY(kick ? launch_walk<true, false, true, 1>(c, p, counts, fuse_next) : launch_walk<true, false, false, 1>(c, p, counts, fuse_next)); }
        } else if (mixed) {
            if (guard) { ASTER_TRY(kick ? launch_walk<true, true, true, 2>(c, p, counts, fuse_next) : launch_walk<true, true, false, 2>(c, p, counts, fuse_next)); }
            else       { ASTER_TRY(kick ? launch_walk<true, false, true, 2>(c, p, counts, fuse_next) : launch_walk<true, false, false, 2>(c, p, counts, fuse_next)); }
        } else {
            ASTER_TRY(kick ? launch_walk<false, false, true, 2>(c, p, counts, fuse_next) : launch_walk<false, false, false, 2>(c, p, counts, fuse_next));
        }
        c->stats.kernels += 1;
        return ASTER_OK;
    }
    if (mixed) {
        if (guard) { ASTER_TRY(kick ? launch_walk<true, true, true>(c, p, counts, fuse_next) : launch_walk<true, true, false>(c, p, counts, fuse_next)); }
        else       { ASTER_TRY(kick ? launch_walk<true, false, true>(c, p, counts, fuse_next) : launch_walk<true, false, false>(c, p, counts, fuse_next)); }
    } else {
        ASTER_TRY(kick ? launch_walk<false, false, true>(c, p, counts, fuse_next) : launch_walk<false, false, false>(c, p, counts, fuse_next));
    }
    c->stats.kernels += 1;
    return ASTER_OK;
}

// ---- tree export -------------------------------------------------------------
namespace {
// Node i of m = 2n - 1 in the view's layout: leaves (i < n) have no children
// and the box of their position; internal nodes' children come from child[].
__global__ void k_export_nodes(int64_t n, int64_t m, double theta, const double4* __restrict__ cm,
                               const float4* __restrict__ bmin, const float4* __restrict__ bmax,
                               const int2* __restrict__ child, double* __restrict__ mass, double* __restrict__ com,
                               float* __restrict__ fmin3, float* __restrict__ fmax3, float* __restrict__ rc2,
                               int32_t* __restrict__ left, int32_t* __restrict__ right) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < m; i += (int64_t)gridDim.x * blockDim.x) {
        const double4 c = cm[i];
        mass[i] = c.w;
        com[3 * i] = c.x; com[3 * i + 1] = c.y; com[3 * i + 2] = c.z;
        const bool leaf = i < n;
        const float4 a = leaf ? leaf_lo(c) : bmin[i], b = leaf ? leaf_hi(c) : bmax[i];
        const int2 ch = leaf ? make_int2(-1, -1) : child[i];
        left[i] = ch.x;
        right[i] = ch.y;
        fmin3[3 * i] = a.x; fmin3[3 * i + 1] = a.y; fmin3[3 * i + 2] = a.z;
        fmax3[3 * i] = b.x; fmax3[3 * i + 1] = b.y; fmax3[3 * i + 2] = b.z;
        float4 h, l;
        if (leaf) leaf_trav(c, h, l);
        else node_trav(c, a, b, theta, h, l);
        rc2[i] = l.w;
    }
}
template <class KeyT>
__global__ void k_widen(int64_t n, const KeyT* __restrict__ in, uint64_t* __restrict__ out) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = (uint64_t)in[i];
}
}  // namespace

static int export_tree(aster_ctx* c, const aster_params* p, aster_tree_view* v) {
    LbvhBufs& t = c->tree;
    const int64_t n = c->n, m = 2 * n - 1;
    cudaStream_t st = c->stream;
    const size_t need = (size_t)m * (8 + 24 + 12 + 12 + 4 + 8) + (size_t)n * 16 + 1024;
    ASTER_TRY(c->stage.ensure(need));
    char* base = c->stage.as<char>();
    double* mass = (double*)base;
    double* com = mass + m;
    float* fmin3 = (float*)(com + 3 * m);
    float* fmax3 = fmin3 + 3 * m;
    float* rc2 = fmax3 + 3 * m;
    int32_t* lft = (int32_t*)(rc2 + m);
    int32_t* rgt = lft + m;
    uint64_t* wide = (uint64_t*)(((uintptr_t)(rgt + m) + 15) & ~(uintptr_t)15);
    uint64_t* wide2 = wide + n;
    const int grid = (int)std::min<int64_t>((m + 255) / 256, (int64_t)c->sm_count * 16);
    k_export_nodes<<<grid, 256, 0, st>>>(n, m, p->theta, t.node_cm.as<double4>(), t.bmin.as<float4>(),
                                         t.bmax.as<float4>(), t.child.as<int2>(), mass, com, fmin3, fmax3, rc2, lft,
                                         rgt);
    if (p->morton_bits == 63) {
        k_widen<uint64_t><<<grid, 256, 0, st>>>(n, t.codes.as<uint64_t>(), wide);
        k_widen<uint64_t><<<grid, 256, 0, st>>>(n, t.sorted_codes.as<uint64_t>(), wide2);
    } else {
        k_widen<uint32_t><<<grid, 256, 0, st>>>(n, t.codes.as<uint32_t>(), wide);
        k_widen<uint32_t><<<grid, 256, 0, st>>>(n, t.sorted_codes.as<uint32_t>(), wide2);
    }
    ASTER_CUDA(cudaGetLastError());
    auto cp = [&](void* dst, const void* src, size_t bytes) -> int {
        if (dst) ASTER_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, st));
        return ASTER_OK;
    };
    ASTER_TRY(cp(v->codes, wide, (size_t)n * 8));
    ASTER_TRY(cp(v->sorted_codes, wide2, (size_t)n * 8));
    ASTER_TRY(cp(v->perm, t.perm.ptr, (size_t)n * 4));
    ASTER_TRY(cp(v->left, lft, (size_t)m * 4));
    ASTER_TRY(cp(v->right, rgt, (size_t)m * 4));
    ASTER_TRY(cp(v->parent, t.parent.ptr, (size_t)m * 4));
    ASTER_TRY(cp(v->range_lo, t.rlo.ptr, (size_t)m * 4));
    ASTER_TRY(cp(v->range_hi, t.rhi.ptr, (size_t)m * 4));
    ASTER_TRY(cp(v->node_mass, mass, (size_t)m * 8));
    ASTER_TRY(cp(v->node_com, com, (size_t)m * 24));
    ASTER_TRY(cp(v->node_bmin, fmin3, (size_t)m * 12));
    ASTER_TRY(cp(v->node_bmax, fmax3, (size_t)m * 12));
    ASTER_TRY(cp(v->node_rcrit2, rc2, (size_t)m * 4));
    unsigned long long bits = 0;
    ASTER_CUDA(cudaMemcpyAsync(&bits, red_box(c), 8, cudaMemcpyDeviceToHost, st));
    ASTER_CUDA(cudaStreamSynchronize(st));
    double box;
    memcpy(&box, &bits, 8);
    v->box = box;
    return ASTER_OK;
}

extern "C" int aster_lbvh_build(aster_ctx* c, const aster_params* p, aster_tree_view* view) {
    if (!c) return ASTER_ERR_INVALID_ARG;
    ASTER_TRY(aster_check_params(p));
    if (c->n <= 0) return ASTER_ERR_NO_STATE;
    ASTER_TRY(aster_begin(c));
    c->stats = aster_stats{};
    cudaEventRecord(c->ev[0], c->stream);
    ASTER_TRY(aster_lbvh_build_dev(c, p, false, view != nullptr));
    cudaEventRecord(c->ev[1], c->stream);
    ASTER_TRY(aster_finish(c));
    float ms = 0.f;
    cudaEventElapsedTime(&ms, c->ev[0], c->ev[1]);
    c->stats.ms_build = c->stats.ms_total = ms;
    if (view) ASTER_TRY(export_tree(c, p, view));
    return ASTER_OK;
}

extern "C" int aster_lbvh_forces(aster_ctx* c, const aster_params* p, int precision, double* acc_out,
                                 int32_t* list_counts) {
    if (!c) return ASTER_ERR_INVALID_ARG;
    ASTER_TRY(aster_check_params(p));
    if (c->n <= 0) return ASTER_ERR_NO_STATE;
    if (precision != ASTER_FP64 && precision != ASTER_MIXED) return ASTER_ERR_INVALID_ARG;
    ASTER_TRY(aster_begin(c));
    c->stats = aster_stats{};
    int32_t* cnt = nullptr;
    if (list_counts) {
        ASTER_TRY(c->targets.ensure((size_t)c->n * 4));
        cnt = c->targets.as<int32_t>();
    }
    ASTER_TRY(ensure_tree(c, pn_level(p) > 0));
    unsigned long long* inter = red_inter(c);
    ASTER_CUDA(cudaMemsetAsync(inter, 0, 8, c->stream));
    cudaEventRecord(c->ev[0], c->stream);
    ASTER_TRY(aster_lbvh_build_dev(c, p, false));
    cudaEventRecord(c->ev[1], c->stream);
    ASTER_TRY(aster_lbvh_walk_launch(c, p, precision, false, cnt));
    cudaEventRecord(c->ev[2], c->stream);
    unsigned long long ic = 0;
    ASTER_CUDA(cudaMemcpyAsync(&ic, inter, 8, cudaMemcpyDeviceToHost, c->stream));
    if (list_counts)
        ASTER_CUDA(cudaMemcpyAsync(list_counts, cnt, (size_t)c->n * 4, cudaMemcpyDeviceToHost, c->stream));
    ASTER_TRY(aster_finish(c));
    float a = 0.f, b = 0.f;
    cudaEventElapsedTime(&a, c->ev[0], c->ev[1]);
    cudaEventElapsedTime(&b, c->ev[1], c->ev[2]);
    c->stats.ms_build = a;
    c->stats.ms_force = b;
    c->stats.ms_total = a + b;
    c->stats.interactions = (double)ic;
    c->acc_valid = true;
    return aster_copy_acc_out(c, acc_out);
}
