// Pippenger MSM kernels and engine (see msm.cuh for the pipeline).
#include "msm.cuh"
#include <type_traits>
#include "common.cuh"
#include "lanes.cuh"
#include <algorithm>
#include <cstdlib>
#include <atomic>
#include <vector>

namespace g16d {

using g16::MSM_DEAD;
using g16::MSM_MAX_SETS;
using g16::MSM_CHUNK;
using g16::MSM_PLAN_TILE;
using g16::MsmPlanGrid;
using g16::MSM_SPREAD_THREADS;
using g16::MSM_MAX_TARGETS;

// Bits [off, off + width) of a 256-bit little-endian scalar held in shared
// memory (8 words, row stride 9 to spread banks); reads past bit 255 are 0.
__device__ __forceinline__ uint32_t read_bits(const uint32_t* s, int off, int width) {
    int idx = off >> 5;
    if (idx >= 8) return 0;
    int sh = off & 31;
    uint64_t w = s[idx];
    if (idx + 1 < 8) w |= (uint64_t)s[idx + 1] << 32;
    return (uint32_t)(w >> sh) & ((1u << width) - 1u);
}

// Window w's digit of the carry-free signed recoding, in [-2^(c-1), 2^(c-1)]:
// the raw window b borrows 2^c when its top bit is set, and the bit just below
// the window repays the borrow of the window beneath.  255 recoding bits keep
// the top window's borrow zero for every scalar below 2^254.
__device__ __forceinline__ int signed_digit(const uint32_t* s, int w, int c) {
    int off = w * c;
    int b = (int)read_bits(s, off, c);
    int d = b - ((b >> (c - 1)) << c);
    int carry = off ? (int)read_bits(s, off - 1, 1) : 0;
    return d + carry;
}

constexpr uint32_t NO_KEY = 0xffffffffu;

// Scalar i into a shared-memory row of 8 words (zeros when not valid),
// converted to standard form when mont is set, with a copy to std_out if given.
__device__ __forceinline__ void stage_scalar(const uint4* __restrict__ scalars, int mont, uint32_t i, bool valid,
                                             uint4* __restrict__ std_out, uint32_t* row) {
    Fr s = Fr::zero();
    if (valid) {
        uint4 a = __ldg(scalars + 2 * (size_t)i), b = __ldg(scalars + 2 * (size_t)i + 1);
        s.v[0] = a.x; s.v[1] = a.y; s.v[2] = a.z; s.v[3] = a.w;
        s.v[4] = b.x; s.v[5] = b.y; s.v[6] = b.z; s.v[7] = b.w;
        if (mont) s = from_mont(s);
        if (std_out) {
            std_out[2 * (size_t)i] = make_uint4(s.v[0], s.v[1], s.v[2], s.v[3]);
            std_out[2 * (size_t)i + 1] = make_uint4(s.v[4], s.v[5], s.v[6], s.v[7]);
        }
    }
#pragma unroll
    for (int j = 0; j < 8; j++) row[j] = s.v[j];
}

// A block of 256 threads takes 256 / WPG scalars: WPG warps share 32 scalars
// and split their windows.  One warp per 32 scalars (WPG = 1) keeps every lane
// busy in the conversion but runs through the windows alone, waiting for an
// atomic in each; eight warps wait side by side.  Digits and scatter together,
// one warp / eight, us (uniform scalars; 70% zeros and ones): 2^10 44 / 17, 38 /
// 17; 2^14 44 / 26, 36 / 19; 2^16 57 / 46, 35 / 26; 2^17 102 / 82, 56 / 46; 2^18
// 108 / 104, 57 / 55; 2^19 198 / 198, 86 / 93; 2^20 358 / 364, 145 / 157.  From
// 2^19 on there are warps enough, and the conversion on one warp in eight costs.
constexpr uint32_t DIGITS_SPLIT = 1u << 18;

template <int WPG>
struct DigitsPlace {
    static constexpr uint32_t SCALARS = 256 / WPG;   // per block
    uint32_t slot;    // this thread's scalar in the block
    uint32_t i;       // and in the vector
    int w0;           // its warp's first window; the next ones follow in steps of WPG
    __device__ __forceinline__ DigitsPlace() {
        const uint32_t wid = threadIdx.x >> 5;
        slot = (wid / WPG) * 32 + (threadIdx.x & 31);
        i = blockIdx.x * SCALARS + slot;
        w0 = (int)(wid % WPG);
    }
};

// kw: key stride per window (B when every window has its own buckets, 0 when
// all windows share one bucket set over window-shifted bases)
// sink: the key of a zero digit (NO_KEY: not sorted; the constant-work sink bucket otherwise)
template <int WPG>
__global__ void __launch_bounds__(256) k_digits_count(const uint4* __restrict__ scalars, int mont, uint32_t n, int c,
                                                      int W, uint32_t kw, uint32_t sink, uint4* __restrict__ scalars_std,
                                                      uint32_t* __restrict__ counts) {
    __shared__ uint32_t sh[DigitsPlace<WPG>::SCALARS * 9];
    const DigitsPlace<WPG> at;
    const uint32_t i = at.i;
    bool valid = i < n;
    uint32_t* row = sh + at.slot * 9;
    if (at.w0 == 0) stage_scalar(scalars, mont, i, valid, scalars_std, row);
    if (WPG > 1) __syncthreads();
    unsigned lane = threadIdx.x & 31;
    for (int w = at.w0; w < W; w += WPG) {
        int d = signed_digit(row, w, c);
        uint32_t key = !valid ? NO_KEY : d != 0 ? (uint32_t)w * kw + (uint32_t)(d < 0 ? -d : d) - 1u : sink;
        unsigned mask = __match_any_sync(0xffffffffu, key);
        if (key != NO_KEY && lane == (unsigned)(__ffs(mask) - 1)) atomicAdd(&counts[key], (uint32_t)__popc(mask));
    }
}

// ew: entry-index stride per window (0, or n for window-shifted bases: entry
// w*n + i names base 2^(c w) P_i)
template <int WPG>
__global__ void __launch_bounds__(256) k_scatter(const uint4* __restrict__ scalars_std, uint32_t n, int c, int W,
                                                 uint32_t kw, uint32_t ew, uint32_t sink, uint32_t* __restrict__ cursor,
                                                 uint32_t* __restrict__ entries) {
    __shared__ uint32_t sh[DigitsPlace<WPG>::SCALARS * 9];
    const DigitsPlace<WPG> at;
    const uint32_t i = at.i;
    bool valid = i < n;
    uint32_t* row = sh + at.slot * 9;
    if (at.w0 == 0) stage_scalar(scalars_std, 0, i, valid, nullptr, row);
    if (WPG > 1) __syncthreads();
    unsigned lane = threadIdx.x & 31;
    unsigned lt = (1u << lane) - 1u;
    for (int w = at.w0; w < W; w += WPG) {
        int d = signed_digit(row, w, c);
        uint32_t key = !valid ? NO_KEY : d != 0 ? (uint32_t)w * kw + (uint32_t)(d < 0 ? -d : d) - 1u : sink;
        unsigned mask = __match_any_sync(0xffffffffu, key);
        int leader = __ffs(mask) - 1;
        uint32_t base = 0;
        if (key != NO_KEY && (int)lane == leader) base = atomicAdd(&cursor[key], (uint32_t)__popc(mask));
        base = __shfl_sync(0xffffffffu, base, leader);
        if (key != NO_KEY) entries[base + __popc(mask & lt)] = ((uint32_t)w * ew + i) | (d < 0 ? 0x80000000u : 0u);
    }
}

// ---- one scalar vector sorted for several live sets (the prover's witness MSMs) ----
// Set j keeps scalar i when rank[j][i] != MSM_DEAD; its entries name row
// rank[j][i] of the set's own window-shifted table: w * rows[j] + rank[j][i].
// The digits are computed once and sorted into every set the scalar is live
// in, so a base at infinity never becomes an entry.
// With per-window bucket sets instead (plain bases, a compact key) window w's
// digit d goes to bucket w B + |d| - 1 and its entry is rank[j][i] itself:
// key_stride = B and rows = 0.
struct LiveSetArgs {
    const uint32_t* rank[MSM_MAX_SETS];
    uint32_t* counts[MSM_MAX_SETS];
    uint32_t* cursor[MSM_MAX_SETS];
    uint32_t* entries[MSM_MAX_SETS];
    uint32_t rows[MSM_MAX_SETS];   // entry stride per window: the table rows, or 0
    uint32_t key_stride;           // bucket offset per window: 0 (one shared set), or B
};

template <int WPG>
__global__ void __launch_bounds__(256) k_digits_count_sets(const uint4* __restrict__ scalars, int mont, uint32_t n,
                                                           int c, int W, uint32_t sink, int nsets, LiveSetArgs a,
                                                           uint4* __restrict__ scalars_std) {
    __shared__ uint32_t sh[DigitsPlace<WPG>::SCALARS * 9];
    const DigitsPlace<WPG> at;
    const uint32_t i = at.i;
    bool valid = i < n;
    bool live[MSM_MAX_SETS];
#pragma unroll
    for (int j = 0; j < MSM_MAX_SETS; j++) live[j] = valid && j < nsets && __ldg(a.rank[j] + i) != MSM_DEAD;
    uint32_t* row = sh + at.slot * 9;
    if (at.w0 == 0) stage_scalar(scalars, mont, i, valid, scalars_std, row);
    if (WPG > 1) __syncthreads();
    unsigned lane = threadIdx.x & 31;
    for (int w = at.w0; w < W; w += WPG) {
        int d = signed_digit(row, w, c);
        uint32_t key = d != 0 ? (uint32_t)w * a.key_stride + (uint32_t)(d < 0 ? -d : d) - 1u : sink;
#pragma unroll
        for (int j = 0; j < MSM_MAX_SETS; j++) {
            if (j >= nsets) break;
            uint32_t kj = live[j] ? key : NO_KEY;
            unsigned mask = __match_any_sync(0xffffffffu, kj);
            if (kj != NO_KEY && lane == (unsigned)(__ffs(mask) - 1)) atomicAdd(&a.counts[j][kj], (uint32_t)__popc(mask));
        }
    }
}

template <int WPG>
__global__ void __launch_bounds__(256) k_scatter_sets(const uint4* __restrict__ scalars_std, uint32_t n, int c, int W,
                                                      uint32_t sink, int nsets, LiveSetArgs a) {
    __shared__ uint32_t sh[DigitsPlace<WPG>::SCALARS * 9];
    const DigitsPlace<WPG> at;
    const uint32_t i = at.i;
    bool valid = i < n;
    uint32_t rank[MSM_MAX_SETS];
#pragma unroll
    for (int j = 0; j < MSM_MAX_SETS; j++) rank[j] = valid && j < nsets ? __ldg(a.rank[j] + i) : MSM_DEAD;
    uint32_t* row = sh + at.slot * 9;
    if (at.w0 == 0) stage_scalar(scalars_std, 0, i, valid, nullptr, row);
    if (WPG > 1) __syncthreads();
    unsigned lane = threadIdx.x & 31;
    unsigned lt = (1u << lane) - 1u;
    for (int w = at.w0; w < W; w += WPG) {
        int d = signed_digit(row, w, c);
        uint32_t key = d != 0 ? (uint32_t)w * a.key_stride + (uint32_t)(d < 0 ? -d : d) - 1u : sink;
        const uint32_t sign = d < 0 ? 0x80000000u : 0u;
#pragma unroll
        for (int j = 0; j < MSM_MAX_SETS; j++) {
            if (j >= nsets) break;
            uint32_t kj = rank[j] != MSM_DEAD ? key : NO_KEY;
            unsigned mask = __match_any_sync(0xffffffffu, kj);
            int leader = __ffs(mask) - 1;
            uint32_t base = 0;
            if (kj != NO_KEY && (int)lane == leader) base = atomicAdd(&a.cursor[j][kj], (uint32_t)__popc(mask));
            base = __shfl_sync(0xffffffffu, base, leader);
            if (kj != NO_KEY) a.entries[j][base + __popc(mask & lt)] = ((uint32_t)w * a.rows[j] + rank[j]) | sign;
        }
    }
}

// ---- exclusive scans ----
__device__ __forceinline__ uint32_t block_excl_scan(uint32_t v, uint32_t* warp_tot, uint32_t& total) {
    unsigned lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= (unsigned)o) x += y;
    }
    if (lane == 31) warp_tot[wid] = x;
    __syncthreads();
    unsigned nw = blockDim.x >> 5;
    if (wid == 0) {
        uint32_t t = lane < nw ? warp_tot[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t y = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= (unsigned)o) t += y;
        }
        if (lane < nw) warp_tot[lane] = t;
    }
    __syncthreads();
    uint32_t before = wid ? warp_tot[wid - 1] : 0;
    total = warp_tot[nw - 1];
    __syncthreads();
    return before + x - v;
}

// Partial sums per bucket (one per chunk the bucket touches).  Buckets with
// more than FAT_PARTIALS of them -- a repeated scalar, most often 1 -- go on
// the fat list and are folded in parallel before the bucket sums.
constexpr uint32_t FAT_PARTIALS = 16;
constexpr uint32_t FAT_JOBS = 64;

// partials per job of a fat bucket: FAT_JOB_MIN or more, two or four for each of
// the folding block's 64 (G1) or 32 (G2) groups of lanes, at most FAT_JOBS jobs
constexpr uint32_t FAT_JOB_MIN = 128;
__device__ __forceinline__ uint32_t fat_job_len(uint32_t ns) {
    uint32_t j = (ns + FAT_JOBS - 1) / FAT_JOBS;
    return j < FAT_JOB_MIN ? FAT_JOB_MIN : j;
}

// Entries per accumulate thread, chosen on the device from the sorted count
// M and the K real buckets: at least L_min, no more than ACC_THREADS threads,
// and about M / (4 K) or more, so that an average bucket gets at most ~4
// partial sums and only skewed buckets (a repeated scalar such as 1) take the
// fat-bucket path.  Sparse scalars (witnesses of zeros and ones) still spread
// over the whole GPU.  Last, the chunks are fitted to whole waves of `wave`
// threads (the G1 accumulate's 512 threads an SM) when that saves 5% or more: a
// launch takes about (waves x L) additions per thread, so 2.4 waves of 16
// entries lose to 2 waves of 20 (a sparse witness MSM of the 2^21 prove).  A
// sort that only a G2 accumulate reads is fitted to the same wave although that
// kernel holds 384 threads an SM: G2 MSMs with a wave of 512 / 384 / no fitting,
// us: 2^18 uniform 3520 / 3570 / 3560, 200007 2993 / 2994 / 3068, 100003 1998 /
// 2010 / 2048, 2^17 sparse 1448 / 1403 / 1446; neither wins throughout.
constexpr uint32_t ACC_THREADS = 1u << 19;

__device__ __forceinline__ uint32_t chunk_len(uint32_t M, uint32_t K, uint32_t L_min, uint32_t wave) {
    uint32_t L = (uint32_t)(((uint64_t)M + ACC_THREADS - 1) / ACC_THREADS);
    uint32_t per_bucket = (uint32_t)(((uint64_t)M + 4ull * K - 1) / (4ull * K));
    if (per_bucket > L) L = per_bucket;
    if (L < L_min) L = L_min;
    if (wave && M) {
        const uint64_t chunks = ((uint64_t)M + L - 1) / L;
        const uint64_t waves = (chunks + wave - 1) / wave;
        if (waves > 1) {
            const uint64_t L2 = ((uint64_t)M + (waves - 1) * wave - 1) / ((waves - 1) * wave);
            // only for a clear gain: block times vary, and more, shorter waves balance better
            if (20 * (waves - 1) * L2 < 19 * waves * L) L = (uint32_t)L2;
        }
    }
    return L;
}

// Smallest chunk for M entries: down to `floor` (4) entries a thread when 16
// would leave SMs empty.  A chunk's additions run one after another while its
// bucket's partial sums cost the bucket-sum step one (dearer) addition each, so
// the chunks stop shrinking once every SM has its 512 threads.  The four G1
// accumulates of a 500-constraint prove 0.73 -> 0.12 ms, of a 2^15-constraint
// one 0.83 -> 0.29 ms, of 1000 uniform points 0.20 -> 0.03 ms.
__device__ __forceinline__ uint32_t min_chunk(uint32_t M, uint32_t floor) {
    const uint32_t spread = (M + MSM_SPREAD_THREADS - 1) / MSM_SPREAD_THREADS;
    const uint32_t L = spread < MSM_CHUNK ? spread : MSM_CHUNK;
    return L > floor ? L : floor;
}

// ---- from bucket counts to the accumulate's plan, for up to MSM_MAX_SETS sorts a launch ----
// Three kernels, blockIdx.y picking the sort, a block's buckets in tiles of 1024
// (msm_plan_grid): block sums of the counts; offsets (and the scatter's cursors),
// the chunk length L, each bucket's partial-sum count and the fat list; the
// partial sums' bases.  A block adds up the block sums before its own itself (at
// most 4096 words from L2) instead of waiting for a kernel that scans them: three
// launches where scanning twice, copying and counting took eight a sort (a
// prove's four sorts 32 launches and 0.21 ms serialised, now 6 and 0.05 ms).
struct SortPlanArgs {
    uint32_t* counts;     // in: entries per bucket; out: partial sums per bucket
    uint32_t* offsets;    // Ks + 1
    uint32_t* cursor;
    uint32_t* seg_base;   // Ks + 1
    uint32_t* fat_list;
    uint32_t* sums;       // block sums of the counts, then those of the partial sums
    uint32_t* total;      // [0] M, [1] partial sums, [2] fat buckets, [3] L
    uint32_t Ks, K;       // sorted and real buckets (the constant-work sink is sorted, never reduced)
    uint32_t L_floor;
    MsmPlanGrid grid;     // of Ks
    // this block's tiles
    __device__ __forceinline__ uint32_t first_tile() const { return blockIdx.x * grid.per_block; }
    __device__ __forceinline__ uint32_t end_tile() const {
        const uint32_t e = first_tile() + grid.per_block;
        return e < grid.tiles ? e : grid.tiles;
    }
};
struct SortPlanSets {
    SortPlanArgs s[MSM_MAX_SETS];
    uint32_t wave;
};

// sums[0 .. b) and sums[0 .. nb), by the whole block
__device__ __forceinline__ uint32_t sums_before(const uint32_t* sums, uint32_t b, uint32_t nb, uint32_t* warp_tot,
                                                uint32_t& all) {
    uint32_t before = 0, every = 0;
    for (uint32_t j = threadIdx.x; j < nb; j += blockDim.x) {
        const uint32_t x = sums[j];
        every += x;
        before += j < b ? x : 0;
    }
    uint32_t total;
    block_excl_scan(every, warp_tot, total);
    all = total;
    block_excl_scan(before, warp_tot, total);
    return total;
}

__global__ void __launch_bounds__(256) k_plan_sums(SortPlanSets a) {
    const SortPlanArgs& s = a.s[blockIdx.y];
    if (blockIdx.x >= s.grid.blocks) return;   // uniform across the block
    __shared__ uint32_t wt[32];
    uint32_t v = 0, total;
    for (uint32_t tile = s.first_tile(); tile < s.end_tile(); tile++) {
        const size_t base = (size_t)tile * MSM_PLAN_TILE + threadIdx.x * 4;
#pragma unroll
        for (int j = 0; j < 4; j++) v += base + j < s.Ks ? s.counts[base + j] : 0;
    }
    block_excl_scan(v, wt, total);
    if (threadIdx.x == 0) {
        s.sums[blockIdx.x] = total;
        if (blockIdx.x == 0) s.total[2] = 0;
    }
}

__global__ void __launch_bounds__(256) k_plan_offsets(SortPlanSets a) {
    const SortPlanArgs& s = a.s[blockIdx.y];
    if (blockIdx.x >= s.grid.blocks) return;   // uniform across the block
    __shared__ uint32_t wt[32];
    const uint32_t nb = s.grid.blocks;
    uint32_t M, total, segs = 0;
    uint32_t before = sums_before(s.sums, blockIdx.x, nb, wt, M);
    const uint32_t L = chunk_len(M, s.K, min_chunk(M, s.L_floor), a.wave);
    for (uint32_t tile = s.first_tile(); tile < s.end_tile(); tile++) {
        const size_t base = (size_t)tile * MSM_PLAN_TILE + threadIdx.x * 4;
        uint32_t v[4], sum = 0;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            v[j] = base + j < s.Ks ? s.counts[base + j] : 0;
            sum += v[j];
        }
        uint32_t off = before + block_excl_scan(sum, wt, total);
        before += total;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const size_t g = base + j;
            if (g >= s.Ks) break;
            s.offsets[g] = off;
            s.cursor[g] = off;
            const uint32_t hi = off + v[j], ns = v[j] ? ((hi - 1) / L - off / L + 1) : 0;
            s.counts[g] = ns;
            if (g < s.K && ns > FAT_PARTIALS) s.fat_list[atomicAdd(s.total + 2, 1u)] = (uint32_t)g;
            off = hi;
            segs += ns;
        }
    }
    block_excl_scan(segs, wt, total);
    if (threadIdx.x == 0) {
        s.sums[nb + blockIdx.x] = total;
        if (blockIdx.x == 0) {
            s.total[0] = M;
            s.total[3] = L;
            s.offsets[s.Ks] = M;
        }
    }
}

__global__ void __launch_bounds__(256) k_plan_segments(SortPlanSets a) {
    const SortPlanArgs& s = a.s[blockIdx.y];
    if (blockIdx.x >= s.grid.blocks) return;   // uniform across the block
    __shared__ uint32_t wt[32];
    const uint32_t nb = s.grid.blocks;
    uint32_t S, total;
    uint32_t before = sums_before(s.sums + nb, blockIdx.x, nb, wt, S);
    for (uint32_t tile = s.first_tile(); tile < s.end_tile(); tile++) {
        const size_t base = (size_t)tile * MSM_PLAN_TILE + threadIdx.x * 4;
        uint32_t v[4], sum = 0;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            v[j] = base + j < s.Ks ? s.counts[base + j] : 0;
            sum += v[j];
        }
        uint32_t off = before + block_excl_scan(sum, wt, total);
        before += total;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            if (base + j >= s.Ks) break;
            s.seg_base[base + j] = off;
            off += v[j];
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        s.total[1] = S;
        s.seg_base[s.Ks] = S;
    }
}

// One MSM of a multi-segment space, as the accumulate kernel reads it.
struct MsmSegDev {
    const uint4* bases;   // window-shifted base table
    uint32_t key_start;   // first bucket of the segment in the space
    uint32_t n_bases;     // table entries
};

// ---- accumulate: one thread per chunk of L sorted entries ----
// Bound by the issue of multiply-adds.  A G1 mixed addition takes 1160 wide ones
// and 72 low halves at half their cost, 1196 in all, a G2 one 3072 and 160, 3152
// (eight products of 320 + 16 and two squares of 256 + 16): at 32 a clock on an
// SM at most 7.78 and 2.95 G additions/s.  Measured 6.7 to 6.8 over G1 (MSMs of
// 2^20 to 2^22), 0.87 of that, and 2.2 over G2, 0.76, where 392 bytes of spills
// and 12 warps an SM leave the pipe idle.  Warps run freely; a block-wide barrier after
// every entry, which kept a longer body in the instruction cache, costs 12% now.
// MULTI: the buckets belong to several MSMs (segments, msm_space_*), each
// with its own base table; the segment of bucket g is the last one whose
// key_start is <= g, followed forward as g grows.
template <class F, bool MULTI = false>
__device__ __forceinline__ void accumulate_chunks(const uint32_t* __restrict__ entries,
                                                  const uint32_t* __restrict__ offsets,
                                                  const uint32_t* __restrict__ seg_base, uint32_t K, uint32_t M,
                                                  uint32_t L, const uint4* __restrict__ bases, uint32_t base_offset,
                                                  uint32_t n_bases, uint4* __restrict__ partials,
                                                  unsigned long long* __restrict__ work,
                                                  const MsmSegDev* __restrict__ segs = nullptr, uint32_t nsegs = 0) {
    const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x, start = t * L;
    if (start >= M) return;
    const size_t end = start + L < M ? start + L : M;
    // last bucket g with offsets[g] <= start; then offsets[g+1] > start
    uint32_t lo = 0, hi = K;
    while (hi - lo > 1) {
        uint32_t mid = (lo + hi) >> 1;
        if (offsets[mid] <= start) lo = mid; else hi = mid;
    }
    uint32_t g = lo, next = offsets[g + 1];
    uint32_t si = 0, seg_end = 0xffffffffu;
    if (MULTI) {
        lo = 0;
        hi = nsegs;
        while (hi - lo > 1) {
            uint32_t mid = (lo + hi) >> 1;
            if (segs[mid].key_start <= g) lo = mid; else hi = mid;
        }
        si = lo;
        bases = segs[si].bases;
        n_bases = segs[si].n_bases;
        base_offset = 0;
        seg_end = si + 1 < nsegs ? segs[si + 1].key_start : 0xffffffffu;
    }
    Xyzz<F> acc = Xyzz<F>::identity();
    unsigned adds = 0;
    for (size_t k = start; k < end; k++) {
        if (k == next) {
            st_xyzz<F>(partials, seg_base[g] + (uint32_t)(t - offsets[g] / L), acc);
            acc = Xyzz<F>::identity();
            do {
                g++;
                next = offsets[g + 1];
            } while (next <= k);
            if (MULTI) {
                while (g >= seg_end) {
                    si++;
                    bases = segs[si].bases;
                    n_bases = segs[si].n_bases;
                    seg_end = si + 1 < nsegs ? segs[si + 1].key_start : 0xffffffffu;
                }
            }
        }
        uint32_t e = entries[k];
        if (k + 1 < end) {   // bring the next entry's base towards L1 while this one is added
            uint32_t nx = (entries[k + 1] & 0x7fffffffu) - base_offset;
            if (nx < n_bases)
                asm volatile("prefetch.global.L1 [%0];" ::"l"(bases + (size_t)nx * (2 * Codec<F>::U4)));
        }
        uint32_t idx = e & 0x7fffffffu;
        if (idx >= base_offset && idx - base_offset < n_bases) {
            Affine<F> p = ld_affine<F>(bases, idx - base_offset);
            if (!p.is_inf()) {
                if (e >> 31) p.y = neg(p.y);
                // G1 keeps its products inlined; the Fq2 body is large enough
                // that one out-of-line Fq2 product (three Fq chains) runs
                // faster than inlined code that misses the instruction cache
                // (G2 MSM 2^18: 2.18 against 2.44 ms)
                acc = xyzz_add_affine<F, !std::is_same<F, Fq2>::value>(acc, p.x, p.y);
                adds++;
            }
        }
    }
    st_xyzz<F>(partials, seg_base[g] + (uint32_t)(t - offsets[g] / L), acc);
    // mixed additions performed, one atomic per warp
    unsigned mask = __activemask();
    unsigned total = __reduce_add_sync(mask, adds);
    if ((threadIdx.x & 31) == (unsigned)(__ffs(mask) - 1) && total) atomicAdd(work, (unsigned long long)total);
}

// Small blocks: a thread's time varies with its bucket boundaries, and a small
// MSM's chunks spread over the SMs.  Registers allow 16 warps an SM over G1
// (four blocks at 128 registers) and 12 over G2 (three at 168).
constexpr int ACC_BLOCK_G1 = 128;
constexpr int ACC_BLOCK_G2 = 128;
constexpr int ACC_G1_BLOCKS = 4;
constexpr int ACC_G2_BLOCKS = 3;

// Multiprocessors of the current device (148 on a B200), cached per device.
static uint32_t device_sms() {
    static std::atomic<uint32_t> cache[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
    uint32_t v = cache[dev].load(std::memory_order_relaxed);
    if (!v) {
        int sms = 0;
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) return 148;
        v = (uint32_t)sms;
        cache[dev].store(v, std::memory_order_relaxed);
    }
    return v;
}

// Threads in one wave of G1 accumulate blocks on the current device, for chunk_len; 0 (no fitting) if the device cannot be read.
static uint32_t accumulate_wave() {
    static std::atomic<uint32_t> cache[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
    uint32_t w = cache[dev].load(std::memory_order_relaxed);
    if (!w) {
        int sms = 0;
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) return 0;
        w = (uint32_t)sms * ACC_BLOCK_G1 * ACC_G1_BLOCKS;
        cache[dev].store(w, std::memory_order_relaxed);
    }
    return w;
}

__global__ void __launch_bounds__(ACC_BLOCK_G1, ACC_G1_BLOCKS) k_accumulate_g1(const uint32_t* __restrict__ entries,
                                                                   const uint32_t* __restrict__ offsets,
                                                                   const uint32_t* __restrict__ seg_base, uint32_t K,
                                                                   const uint32_t* __restrict__ d_M,
                                                                   const uint32_t* __restrict__ d_L,
                                                                   const uint4* __restrict__ bases, uint32_t base_offset,
                                                                   uint32_t n_bases, uint4* __restrict__ partials,
                                                                   unsigned long long* __restrict__ work) {
    accumulate_chunks<Fq>(entries, offsets, seg_base, K, *d_M, *d_L, bases, base_offset, n_bases, partials, work);
}

__global__ void __launch_bounds__(ACC_BLOCK_G2, ACC_G2_BLOCKS) k_accumulate_g2(const uint32_t* __restrict__ entries,
                                                               const uint32_t* __restrict__ offsets,
                                                               const uint32_t* __restrict__ seg_base, uint32_t K,
                                                               const uint32_t* __restrict__ d_M,
                                                               const uint32_t* __restrict__ d_L,
                                                               const uint4* __restrict__ bases, uint32_t base_offset,
                                                               uint32_t n_bases, uint4* __restrict__ partials,
                                                               unsigned long long* __restrict__ work) {
    accumulate_chunks<Fq2>(entries, offsets, seg_base, K, *d_M, *d_L, bases, base_offset, n_bases, partials, work);
}

__device__ __forceinline__ uint32_t n_partials(const uint32_t* offsets, uint32_t g, uint32_t L) {
    uint32_t lo = offsets[g], hi = offsets[g + 1];
    return hi > lo ? ((hi - 1) / L - lo / L + 1) : 0;
}

// ---- bucket reduction: point operations by groups of lanes (lanes.cuh) ----
constexpr unsigned LANES_BLOCK = 256;   // threads per block of the kernels below
template <class F>
constexpr uint32_t LANES_GROUPS = LANES_BLOCK / Lanes<F>::N;   // points a block works on at a time

// Fat buckets, stage 1: each of a fat bucket's partials is assigned to one of
// FAT_JOBS contiguous jobs; a block folds one job into the job's first slot.
template <class F>
__global__ void __launch_bounds__(LANES_BLOCK) k_fat_merge_jobs(uint4* __restrict__ partials,
                                                                const uint32_t* __restrict__ offsets,
                                                                const uint32_t* __restrict__ seg_base,
                                                                const uint32_t* __restrict__ fat_list,
                                                                const uint32_t* __restrict__ fat_count,
                                                                const uint32_t* __restrict__ d_L) {
    constexpr uint32_t G = LANES_GROUPS<F>;
    __shared__ uint4 smem[LANES_BLOCK * 2];
    const uint32_t L = *d_L, grp = threadIdx.x / Lanes<F>::N;
    uint32_t items = *fat_count * FAT_JOBS;
    for (uint32_t item = blockIdx.x; item < items; item += gridDim.x) {
        uint32_t g = fat_list[item / FAT_JOBS], j = item % FAT_JOBS;
        uint32_t ns = n_partials(offsets, g, L), J = fat_job_len(ns);
        uint32_t a = j * J;
        if (a >= ns) continue;   // uniform across the block
        uint32_t b = min(a + J, ns), base = seg_base[g];
        Fq acc = a + grp < b ? ld_lane<F>(partials, base + a + grp) : Fq::zero();
        for (uint32_t i0 = a + G; i0 < b; i0 += G)
            acc = lanes_add<F>(acc, i0 + grp < b ? ld_lane<F>(partials, base + i0 + grp) : Fq::zero());
        acc = block_sum_lanes<F>(acc, smem, G);
        if (grp == 0) st_lane<F>(partials, base + a, acc);
        __syncthreads();
    }
}

// Fat buckets, stage 2: fold the (at most FAT_JOBS) job results into the
// bucket's first partial slot.
template <class F>
__global__ void __launch_bounds__(LANES_BLOCK) k_fat_merge_final(uint4* __restrict__ partials,
                                                                 const uint32_t* __restrict__ offsets,
                                                                 const uint32_t* __restrict__ seg_base,
                                                                 const uint32_t* __restrict__ fat_list,
                                                                 const uint32_t* __restrict__ fat_count,
                                                                 const uint32_t* __restrict__ d_L) {
    constexpr uint32_t G = LANES_GROUPS<F>;
    __shared__ uint4 smem[LANES_BLOCK * 2];
    const uint32_t L = *d_L, grp = threadIdx.x / Lanes<F>::N;
    uint32_t nf = *fat_count;
    for (uint32_t f = blockIdx.x; f < nf; f += gridDim.x) {
        uint32_t g = fat_list[f];
        uint32_t ns = n_partials(offsets, g, L), J = fat_job_len(ns);
        uint32_t base = seg_base[g];
        Fq acc = grp * J < ns ? ld_lane<F>(partials, base + grp * J) : Fq::zero();
        for (uint32_t t0 = G; t0 < FAT_JOBS; t0 += G) {
            const uint32_t a = (t0 + grp) * J;
            acc = lanes_add<F>(acc, a < ns ? ld_lane<F>(partials, base + a) : Fq::zero());
        }
        acc = block_sum_lanes<F>(acc, smem, G);
        if (grp == 0) st_lane<F>(partials, base, acc);
        __syncthreads();
    }
}

// Bucket sums S_g: one group of lanes per bucket folds its few partials (a fat
// bucket's total already sits in its first slot).  A warp's groups run as many
// steps as its longest bucket needs.
template <class F>
__global__ void __launch_bounds__(LANES_BLOCK) k_bucket_sums(const uint4* __restrict__ partials,
                                                             const uint32_t* __restrict__ offsets,
                                                             const uint32_t* __restrict__ seg_base, uint32_t K,
                                                             const uint32_t* __restrict__ d_L,
                                                             uint4* __restrict__ buckets) {
    const uint32_t g = (blockIdx.x * LANES_BLOCK + threadIdx.x) / Lanes<F>::N;
    uint32_t ns = 0, base = 0;
    if (g < K) {
        ns = n_partials(offsets, g, *d_L);
        base = seg_base[g];
        if (ns > FAT_PARTIALS) ns = 1;
    }
    const uint32_t steps = __reduce_max_sync(FULL_WARP, ns);
    Fq acc = ns ? ld_lane<F>(partials, base) : Fq::zero();
    for (uint32_t s = 1; s < steps; s++)
        acc = lanes_add<F>(acc, s < ns ? ld_lane<F>(partials, base + s) : Fq::zero());
    if (g < K) st_lane<F>(buckets, g, acc);
}

// Bucket reduction, step 1.  A set's buckets S_0 .. S_{B-1} (S_b holds the
// points whose digit is b + 1) are cut into pieces of seg buckets; piece
// p = j 2^LB + t of block j gives
//   run_p = sum_i S_{p seg + i},   tot_p = sum_i (i + 1) S_{p seg + i},
// so that the set's sum_b (b + 1) S_b = sum_p tot_p + seg sum_p p run_p.
// Two groups of lanes share a piece: the first runs run += S_i, the second
// tot += run one step behind it, so a bucket costs one addition of latency.
// The weights p are split over their bits instead of being multiplied out (a
// double-and-add per piece costs more than the piece's running sums): the
// block halves its 2^LB run values LB times in shared memory, v_t += v_(t+h)
// for h = 2^(LB-1) .. 1, and the upper half [h, 2h) that a halving reads holds
// exactly the folded values whose piece index has bit log2(h) set.  Once
// frozen, each upper half is summed by a tree that runs alongside the later
// halvings, so G_j = sum over the pieces with bit j set of run_p ends in slot
// 2^j after LB steps.  The second groups halve the tot values into T meanwhile
// (with seg = 1, tot = run and T = R).  Each step is one addition deep: depth
// is what counts here, the device has lanes to spare.
// The block writes T, G_0 .. G_(LB-1) and its run total R (LB + 2 points).
template <class F, int LB>
__device__ __forceinline__ void reduce_piece_block(const uint4* __restrict__ buckets, size_t g0, bool in_range,
                                                   uint32_t seg, uint4* __restrict__ out, size_t o0) {
    constexpr uint32_t N = 1u << LB;
    __shared__ uint4 s_pts[2][N * Lanes<F>::N * 2];   // run, tot
    const uint32_t t = threadIdx.x / (2 * Lanes<F>::N);
    const bool second = (threadIdx.x / Lanes<F>::N) & 1u;
    const bool weighted = seg > 1;   // uniform: tot differs from run
    const bool reads = in_range && !second;
    Fq acc = Fq::zero(), next = reads ? ld_lane<F>(buckets, g0 + seg - 1) : Fq::zero();
    const uint32_t steps = weighted ? seg + 1 : 1;
#pragma unroll 1
    for (uint32_t j = 0; j < steps; j++) {
        const Fq o = pick(second, shfl_xor(acc, Lanes<F>::N), next);
        next = reads && j + 1 < seg ? ld_lane<F>(buckets, g0 + seg - 2 - j) : Fq::zero();
        acc = lanes_add<F>(acc, o);
    }
    uint4* mine = s_pts[second];
    // acc stays equal to this group's slot t: no other group writes it
    st_lane<F>(mine, t, acc);
    const uint32_t lg = t ? 31 - __clz(t) : 0;   // slot t lies in the upper half [2^lg, 2^(lg+1))
#pragma unroll 1
    for (uint32_t k = 1; k <= (uint32_t)LB; k++) {
        __syncthreads();
        const uint32_t h = N >> k;
        // a step reads no slot that another group writes in the same step: the
        // halvings read [h, 2h) and write [0, h); the trees stay at 2h and above
        uint32_t src = t;   // t: nothing to add in this step
        if (t < h) {
            if (!second || weighted) src = t + h;
        } else if (t >= 2 * h && !second) {
            // the half [2^lg, 2^(lg+1)) froze at step LB - lg; tree level k - (LB - lg) - 1 now
            const uint32_t hs = 1u << lg, s = 1u << (k - (LB - lg) - 1), o = t - hs;
            if ((o & (2 * s - 1)) == 0 && o + s < hs) src = t + s;
        }
        const bool adds = src != t;
        if (__any_sync(FULL_WARP, adds)) {
            acc = lanes_add<F>(acc, adds ? ld_lane<F>(mine, src) : Fq::zero());
            if (adds) st_lane<F>(mine, t, acc);
        }
    }
    if (second) {
        if (t == 0 && weighted) st_lane<F>(out, o0, acc);   // T
    } else if (t == 0) {
        if (!weighted) st_lane<F>(out, o0, acc);
        st_lane<F>(out, o0 + LB + 1, acc);
    } else if ((t & (t - 1)) == 0) {
        st_lane<F>(out, o0 + 1 + lg, acc);   // G_lg
    }
}

// threads of a reduction block: two groups for each of its 2^LB pieces
template <class F, int LB>
constexpr unsigned REDUCE_BLOCK = (2u * Lanes<F>::N) << LB;

template <class F, int LB>
__global__ void __launch_bounds__(REDUCE_BLOCK<F, LB>) k_reduce_pieces(const uint4* __restrict__ buckets, uint32_t B,
                                                                       uint32_t seg, uint4* __restrict__ out) {
    const uint32_t p = (blockIdx.x << LB) + threadIdx.x / (2 * Lanes<F>::N), set = blockIdx.y;
    reduce_piece_block<F, LB>(buckets, (size_t)set * B + (size_t)p * seg, (size_t)p * seg < B, seg, out,
                              ((size_t)set * gridDim.x + blockIdx.x) * (LB + 2));
}

// Bucket reduction, step 2 (when a set has more than a couple of blocks):
// block (o, set) sums one term over the set's nb blocks: o = 0 gives T,
// o = 1 .. LB gives G_(o-1), o = LB + 1 + i gives Gb_i, the sum of the run
// totals R of the blocks whose index has bit i set.
template <class F, int LB>
__device__ __forceinline__ void reduce_set_term(const uint4* __restrict__ in, size_t base, uint32_t nb, uint32_t o,
                                                uint4* __restrict__ out, size_t to) {
    __shared__ uint4 smem[LANES_BLOCK * 2];
    const uint32_t grp = threadIdx.x / Lanes<F>::N, groups = blockDim.x / Lanes<F>::N;
    const bool bits = o > (uint32_t)LB;
    const uint32_t i = bits ? o - LB - 1 : 0, count = bits ? nb / 2 : nb;
    auto at = [&](uint32_t x) {   // the x-th point of the term
        const uint32_t j = bits ? ((x >> i) << (i + 1)) | (1u << i) | (x & ((1u << i) - 1u)) : x;
        return base + (size_t)j * (LB + 2) + (bits ? LB + 1 : o);
    };
    Fq acc = grp < count ? ld_lane<F>(in, at(grp)) : Fq::zero();
    for (uint32_t x0 = groups; x0 < count; x0 += groups)
        acc = lanes_add<F>(acc, x0 + grp < count ? ld_lane<F>(in, at(x0 + grp)) : Fq::zero());
    acc = block_sum_lanes<F>(acc, smem, groups);
    if (grp == 0) st_lane<F>(out, to, acc);
}

template <class F, int LB>
__global__ void __launch_bounds__(LANES_BLOCK) k_reduce_sets(const uint4* __restrict__ in, uint32_t nb,
                                                             uint4* __restrict__ out) {
    const uint32_t o = blockIdx.x, set = blockIdx.y;
    reduce_set_term<F, LB>(in, (size_t)set * nb * (LB + 2), nb, o, out, (size_t)set * gridDim.x + o);
}

// Bucket reduction, step 3: a set's sum from its terms,
//   T + seg (sum_j 2^j G_j + 2^LB sum_i 2^i Gb_i),
// by one block.  With e_g the g-th bit term (G_0 .., then Gb_0 ..), groups
// combine in a tree, e_g + 2^s e_(g+s) for s = 1, 2, 4, ..: the s doublings of
// a level run in all of its groups at once, so the chain is at most 31
// doublings and 5 additions for up to 31 bits, then log2(seg) doublings and T.
// Latency-bound: 27 us over G1 and 8 bits, 57 us over 15, 87 us over G2 and 14,
// for any number of sets.  The host's combination took about 8 us a set over G1
// and 35 us over G2, one set after another: a standalone MSM has one per window
// (G2 MSM 2^18 4.22 -> 3.68 ms, G1 MSM of 1000 points 606 -> 473 us, 2^20 4.31
// -> 4.23 ms); a single prove, one set in each of five MSMs, is level.
// terms: nb points at `in` (stride LB + 2 per block; the blocks' own points,
// nb at most 2) when direct, else one point per term from step 2.
constexpr uint32_t FINISH_GROUPS = 32;

template <class F, int LB>
__device__ __forceinline__ void reduce_finish(const uint4* __restrict__ in, size_t base, uint32_t nb, uint32_t hb,
                                              bool direct, uint32_t seg, uint4* __restrict__ out, size_t to) {
    __shared__ uint4 smem[FINISH_GROUPS * Lanes<F>::N * 2];
    const uint32_t g = threadIdx.x / Lanes<F>::N, m = LB + hb;
    const bool is_t = g == FINISH_GROUPS - 1;   // m < 31: the last group holds T
    Fq acc = Fq::zero();
    if (!direct) {
        if (g < m || is_t) acc = ld_lane<F>(in, base + (is_t ? 0 : 1 + g));
    } else {
        // block j's points: T, G_0 .. G_(LB-1), R
        const uint32_t o = is_t ? 0 : 1 + g;
        const bool low = is_t || g < (uint32_t)LB;
        if (low) acc = ld_lane<F>(in, base + o);
        else if (g < m) acc = ld_lane<F>(in, base + (LB + 2) + LB + 1);   // Gb_0 = R of block 1
        if (nb > 1) acc = lanes_add<F>(acc, low ? ld_lane<F>(in, base + (LB + 2) + o) : Fq::zero());
    }
    for (uint32_t s = 1; s < m; s *= 2) {
        const bool up = (g & (2 * s - 1)) == s && g < m, down = (g & (2 * s - 1)) == 0 && g + s < m;
        if (__any_sync(FULL_WARP, up)) {
            for (uint32_t i = 0; i < s; i++) acc = pick(up, lanes_dbl<F>(acc), acc);
            if (up) st_lane<F>(smem, g, acc);
        }
        __syncthreads();
        if (__any_sync(FULL_WARP, down)) acc = lanes_add<F>(acc, down ? ld_lane<F>(smem, g + s) : Fq::zero());
    }
    if (is_t) st_lane<F>(smem, g, acc);
    __syncthreads();
    if (threadIdx.x < 32) {
        for (uint32_t s = seg; s > 1; s >>= 1) acc = lanes_dbl<F>(acc);
        acc = lanes_add<F>(acc, g == 0 ? ld_lane<F>(smem, FINISH_GROUPS - 1) : Fq::zero());
        if (g == 0) st_lane<F>(out, to, acc);
    }
}

template <class F>
constexpr unsigned FINISH_BLOCK = FINISH_GROUPS * Lanes<F>::N;

template <class F, int LB>
__global__ void __launch_bounds__(FINISH_BLOCK<F>) k_reduce_finish(const uint4* __restrict__ in, uint32_t stride,
                                                                   uint32_t nb, uint32_t hb, int direct, uint32_t seg,
                                                                   uint4* __restrict__ out) {
    reduce_finish<F, LB>(in, (size_t)blockIdx.x * stride, nb, hb, direct, seg, out, blockIdx.x);
}

// ---- batched MSMs: several scalar vectors, many MSMs, one launch per step ----
// A space holds the buckets of many MSMs (segments) back to back; sources are
// scalar vectors, each feeding up to MSM_MAX_TARGETS segments (the witness
// feeds A, B1 and L in the G1 space and B2 in the G2 space; an H vector feeds
// its H segment).  One digits pass and one scatter pass sort every source into
// every space; one accumulate launch per space adds every entry.

struct MsmTargetDev {
    uint32_t* counts;        // the space's sort buffers
    uint32_t* cursor;
    uint32_t* entries;
    const uint32_t* rank;    // scalar -> table row, MSM_DEAD where the base is infinity; nullptr: the scalar's index
    uint32_t key_start;      // the segment's first bucket in its space
    uint32_t rows;           // the segment's table rows
};

struct MsmSourceDev {
    const uint4* scalars;    // Montgomery Fr
    uint4* std_out;          // standard-form copy, for the scatter pass
    uint32_t n, c, W, ntargets;
    MsmTargetDev t[MSM_MAX_TARGETS];
};

// the source of block b: the last s with blk_start[s] <= b
__device__ __forceinline__ uint32_t source_of(const uint32_t* __restrict__ blk_start, uint32_t nsrc, uint32_t b) {
    uint32_t lo = 0, hi = nsrc;
    while (hi - lo > 1) {
        uint32_t mid = (lo + hi) >> 1;
        if (blk_start[mid] <= b) lo = mid; else hi = mid;
    }
    return lo;
}

__global__ void __launch_bounds__(256) k_digits_multi(const MsmSourceDev* __restrict__ srcs,
                                                      const uint32_t* __restrict__ blk_start, uint32_t nsrc) {
    __shared__ uint32_t sh[256 * 9];
    const uint32_t si = source_of(blk_start, nsrc, blockIdx.x);
    const MsmSourceDev& S = srcs[si];
    const uint32_t i = (blockIdx.x - blk_start[si]) * 256 + threadIdx.x;
    const bool valid = i < S.n;
    const uint32_t nt = S.ntargets, c = S.c, W = S.W;
    Fr x = Fr::zero();
    bool live[MSM_MAX_TARGETS];
#pragma unroll
    for (int j = 0; j < MSM_MAX_TARGETS; j++)
        live[j] = valid && (uint32_t)j < nt && (!S.t[j].rank || __ldg(S.t[j].rank + i) != MSM_DEAD);
    if (valid) {
        uint4 a = __ldg(S.scalars + 2 * (size_t)i), b = __ldg(S.scalars + 2 * (size_t)i + 1);
        x.v[0] = a.x; x.v[1] = a.y; x.v[2] = a.z; x.v[3] = a.w;
        x.v[4] = b.x; x.v[5] = b.y; x.v[6] = b.z; x.v[7] = b.w;
        x = from_mont(x);
        S.std_out[2 * (size_t)i] = make_uint4(x.v[0], x.v[1], x.v[2], x.v[3]);
        S.std_out[2 * (size_t)i + 1] = make_uint4(x.v[4], x.v[5], x.v[6], x.v[7]);
    }
    uint32_t* row = sh + threadIdx.x * 9;
#pragma unroll
    for (int j = 0; j < 8; j++) row[j] = x.v[j];
    const unsigned lane = threadIdx.x & 31;
    for (uint32_t w = 0; w < W; w++) {
        const int d = signed_digit(row, (int)w, (int)c);
        const uint32_t key = d != 0 ? (uint32_t)(d < 0 ? -d : d) - 1u : NO_KEY;
#pragma unroll
        for (int j = 0; j < MSM_MAX_TARGETS; j++) {
            if ((uint32_t)j >= nt) break;
            const uint32_t kj = live[j] && key != NO_KEY ? S.t[j].key_start + key : NO_KEY;
            const unsigned mask = __match_any_sync(0xffffffffu, kj);
            if (kj != NO_KEY && lane == (unsigned)(__ffs(mask) - 1)) atomicAdd(&S.t[j].counts[kj], (uint32_t)__popc(mask));
        }
    }
}

__global__ void __launch_bounds__(256) k_scatter_multi(const MsmSourceDev* __restrict__ srcs,
                                                       const uint32_t* __restrict__ blk_start, uint32_t nsrc) {
    __shared__ uint32_t sh[256 * 9];
    const uint32_t si = source_of(blk_start, nsrc, blockIdx.x);
    const MsmSourceDev& S = srcs[si];
    const uint32_t i = (blockIdx.x - blk_start[si]) * 256 + threadIdx.x;
    const bool valid = i < S.n;
    const uint32_t nt = S.ntargets, c = S.c, W = S.W;
    uint32_t rowi[MSM_MAX_TARGETS];
#pragma unroll
    for (int j = 0; j < MSM_MAX_TARGETS; j++)
        rowi[j] = valid && (uint32_t)j < nt ? (S.t[j].rank ? __ldg(S.t[j].rank + i) : i) : MSM_DEAD;
    uint32_t* row = sh + threadIdx.x * 9;
    if (valid) {
        uint4 a = S.std_out[2 * (size_t)i], b = S.std_out[2 * (size_t)i + 1];
        row[0] = a.x; row[1] = a.y; row[2] = a.z; row[3] = a.w;
        row[4] = b.x; row[5] = b.y; row[6] = b.z; row[7] = b.w;
    } else {
#pragma unroll
        for (int j = 0; j < 8; j++) row[j] = 0;
    }
    const unsigned lane = threadIdx.x & 31, lt = (1u << lane) - 1u;
    for (uint32_t w = 0; w < W; w++) {
        const int d = signed_digit(row, (int)w, (int)c);
        const uint32_t key = d != 0 ? (uint32_t)(d < 0 ? -d : d) - 1u : NO_KEY;
        const uint32_t sign = d < 0 ? 0x80000000u : 0u;
#pragma unroll
        for (int j = 0; j < MSM_MAX_TARGETS; j++) {
            if ((uint32_t)j >= nt) break;
            const uint32_t kj = rowi[j] != MSM_DEAD && key != NO_KEY ? S.t[j].key_start + key : NO_KEY;
            const unsigned mask = __match_any_sync(0xffffffffu, kj);
            const int leader = __ffs(mask) - 1;
            uint32_t base = 0;
            if (kj != NO_KEY && (int)lane == leader) base = atomicAdd(&S.t[j].cursor[kj], (uint32_t)__popc(mask));
            base = __shfl_sync(0xffffffffu, base, leader);
            if (kj != NO_KEY) S.t[j].entries[base + __popc(mask & lt)] = (w * S.t[j].rows + rowi[j]) | sign;
        }
    }
}

__global__ void __launch_bounds__(ACC_BLOCK_G1, ACC_G1_BLOCKS) k_accumulate_multi_g1(const uint32_t* __restrict__ entries,
                                                                         const uint32_t* __restrict__ offsets,
                                                                         const uint32_t* __restrict__ seg_base,
                                                                         uint32_t K, const uint32_t* __restrict__ d_M,
                                                                         const uint32_t* __restrict__ d_L,
                                                                         const MsmSegDev* __restrict__ segs,
                                                                         uint32_t nsegs, uint4* __restrict__ partials,
                                                                         unsigned long long* __restrict__ work) {
    accumulate_chunks<Fq, true>(entries, offsets, seg_base, K, *d_M, *d_L, nullptr, 0, 0, partials, work, segs, nsegs);
}

__global__ void __launch_bounds__(ACC_BLOCK_G2, ACC_G2_BLOCKS) k_accumulate_multi_g2(const uint32_t* __restrict__ entries,
                                                                     const uint32_t* __restrict__ offsets,
                                                                     const uint32_t* __restrict__ seg_base,
                                                                     uint32_t K, const uint32_t* __restrict__ d_M,
                                                                     const uint32_t* __restrict__ d_L,
                                                                     const MsmSegDev* __restrict__ segs,
                                                                     uint32_t nsegs, uint4* __restrict__ partials,
                                                                     unsigned long long* __restrict__ work) {
    accumulate_chunks<Fq2, true>(entries, offsets, seg_base, K, *d_M, *d_L, nullptr, 0, 0, partials, work, segs, nsegs);
}

// The bucket reduction of one segment of a space (msm_reduce_plan with one set).
struct MsmReduceDev {
    uint32_t key_start, B, seg, nb, hb;
    uint32_t block_start;   // its first k_reduce_pieces_multi block
    uint32_t out_block;     // its first point in the blocks' output
    uint32_t out_set;       // its first point in the sets' output
};

// k_reduce_pieces for many segments: block b works on block b - block_start
// of the segment that owns it, with that segment's B and seg.
template <class F, int LB>
__global__ void __launch_bounds__(REDUCE_BLOCK<F, LB>) k_reduce_pieces_multi(const uint4* __restrict__ buckets,
                                                                             const MsmReduceDev* __restrict__ segs,
                                                                             uint32_t nsegs, uint4* __restrict__ out) {
    uint32_t lo = 0, hi = nsegs;
    while (hi - lo > 1) {
        uint32_t mid = (lo + hi) >> 1;
        if (segs[mid].block_start <= blockIdx.x) lo = mid; else hi = mid;
    }
    const MsmReduceDev sd = segs[lo];
    const uint32_t jb = blockIdx.x - sd.block_start, p = (jb << LB) + threadIdx.x / (2 * Lanes<F>::N);
    reduce_piece_block<F, LB>(buckets, (size_t)sd.key_start + (size_t)p * sd.seg, (size_t)p * sd.seg < sd.B, sd.seg,
                              out, (size_t)sd.out_block + (size_t)jb * (LB + 2));
}

// k_reduce_sets for many segments: blockIdx.y picks the segment, blockIdx.x
// the term (T, G_0 .. G_(LB-1), Gb_0 .. Gb_(hb-1)); terms past the segment's
// own hb leave at once.
template <class F, int LB>
__global__ void __launch_bounds__(LANES_BLOCK) k_reduce_sets_multi(const uint4* __restrict__ in,
                                                                   const MsmReduceDev* __restrict__ segs,
                                                                   uint4* __restrict__ out) {
    const MsmReduceDev sd = segs[blockIdx.y];
    const uint32_t o = blockIdx.x;
    if (o >= (uint32_t)LB + 1 + sd.hb) return;   // uniform across the block
    reduce_set_term<F, LB>(in, sd.out_block, sd.nb, o, out, (size_t)sd.out_set + o);
}

// k_reduce_finish for many segments, one block each.
template <class F, int LB>
__global__ void __launch_bounds__(FINISH_BLOCK<F>) k_reduce_finish_multi(const uint4* __restrict__ in,
                                                                         const MsmReduceDev* __restrict__ segs,
                                                                         uint4* __restrict__ out) {
    const MsmReduceDev sd = segs[blockIdx.x];
    reduce_finish<F, LB>(in, sd.out_set, sd.nb, sd.hb, false, sd.seg, out, blockIdx.x);
}

// Window-shifted base table: out[w n + i] = 2^(c w) P_i (affine).  Built once
// per prepared key in two steps, so that the normalisations share inversions.
//
// Step 1, one thread per point: window 0 is P_i itself (written affine), and
// the XYZZ multiples 2^(c w) P_i for w >= 1 (c doublings each) go to tmp at
// (w - 1) n + i; a point at infinity (or below skip) gives zeros / identity.
template <class F>
__global__ void __launch_bounds__(128) k_window_xyzz(const uint4* __restrict__ in, uint32_t n, uint32_t skip, int c,
                                                     int W, uint4* __restrict__ out, uint4* __restrict__ tmp) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    Affine<F> p;
    bool inf = i < skip;
    if (!inf) {
        p = ld_affine<F>(in, i - skip);
        inf = p.is_inf();
    }
    if (inf) {
        st_affine<F>(out, i, F::zero(), F::zero());
        for (int w = 1; w < W; w++) st_xyzz<F>(tmp, (size_t)(w - 1) * n + i, Xyzz<F>::identity());
        return;
    }
    st_affine<F>(out, i, p.x, p.y);
    Xyzz<F> acc;
    acc.x = p.x;
    acc.y = p.y;
    acc.zz = F::one();
    acc.zzz = F::one();
    for (int w = 1; w < W; w++) {
        for (int j = 0; j < c; j++) acc = xyzz_dbl<F, false>(acc);
        st_xyzz<F>(tmp, (size_t)(w - 1) * n + i, acc);
    }
}

// Step 2, Montgomery's batch inversion over runs of NORM_RUN consecutive
// entries: one inversion per run instead of one per entry.  With
// d_j = ZZ_j ZZZ_j, x = X ZZZ / d and y = Y ZZ / d.  The output slots hold the
// running products (x) and d_j (y) between the forward and the backward pass;
// an identity entry (ZZ = 0) takes d = 1 and is written as zeros.
constexpr uint32_t NORM_RUN = 32;

template <class F>
__global__ void __launch_bounds__(128) k_window_normalize(const uint4* __restrict__ tmp, size_t count,
                                                          uint4* __restrict__ out) {
    size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    size_t a = t * NORM_RUN;
    if (a >= count) return;
    size_t b = a + NORM_RUN < count ? a + NORM_RUN : count;
    F acc = F::one();
    for (size_t j = a; j < b; j++) {
        Xyzz<F> q = ld_xyzz<F>(tmp, j);
        F d = q.zz.is_zero() ? F::one() : fmul<false>(q.zz, q.zzz);
        acc = fmul<false>(acc, d);
        st_affine<F>(out, j, acc, d);
    }
    F inv_acc = inv(acc);   // 1 / (d_a ... d_(b-1))
    for (size_t j = b; j-- > a;) {
        Affine<F> slot = ld_affine_rw<F>(out, j);   // (running product through j, d_j)
        F before = j > a ? ld_affine_rw<F>(out, j - 1).x : F::one();
        F inv_d = fmul<false>(inv_acc, before);   // 1 / d_j
        inv_acc = fmul<false>(inv_acc, slot.y);   // 1 / (d_a ... d_(j-1))
        Xyzz<F> q = ld_xyzz<F>(tmp, j);
        if (q.zz.is_zero()) {
            st_affine<F>(out, j, F::zero(), F::zero());
        } else {
            F x, y;
            fmul2<false>(q.x, q.zzz, q.y, q.zz, x, y);
            fmul2<false>(x, inv_d, y, inv_d, x, y);
            st_affine<F>(out, j, x, y);
        }
    }
}

// Fixed-base multiplication for key generation: P_i = k_i G with 8-bit windows,
// table[w * 256 + d] = d 2^(8 w) G (affine; d = 0 unused), k_i Montgomery Fr.
// The XYZZ result goes to tmp for k_window_normalize.
template <class F>
__global__ void __launch_bounds__(128) k_fixed_base(const uint4* __restrict__ table, const uint4* __restrict__ scalars,
                                                    size_t n, uint4* __restrict__ tmp) {
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    Fr k;
    uint4 a = __ldg(scalars + 2 * i), b = __ldg(scalars + 2 * i + 1);
    k.v[0] = a.x; k.v[1] = a.y; k.v[2] = a.z; k.v[3] = a.w;
    k.v[4] = b.x; k.v[5] = b.y; k.v[6] = b.z; k.v[7] = b.w;
    k = from_mont(k);
    Xyzz<F> acc = Xyzz<F>::identity();
    for (int w = 0; w < 32; w++) {
        uint32_t d = (k.v[w >> 2] >> (8 * (w & 3))) & 255u;
        if (d) {
            Affine<F> p = ld_affine<F>(table, (size_t)w * 256 + d);
            acc = xyzz_add_affine<F, !std::is_same<F, Fq2>::value>(acc, p.x, p.y);
        }
    }
    st_xyzz<F>(tmp, i, acc);
}

}  // namespace g16d

namespace g16 {

using namespace g16d;

void MsmSort::release() {
    cudaFree(d_scalars_std);
    cudaFree(d_counts);
    cudaFree(d_offsets);
    cudaFree(d_cursor);
    cudaFree(d_seg_base);
    cudaFree(d_fat_list);
    cudaFree(d_scan_tmp);
    cudaFree(d_entries);
    cudaFree(d_total);
    *this = MsmSort();
}

void MsmAccum::release() {
    cudaFree(d_work);
    cudaFree(d_buckets);
    cudaFree(d_partials);
    cudaFree(d_segments);
    cudaFree(d_terms);
    cudaFree(d_windows);
    *this = MsmAccum();
}

int msm_shared_window_bits(size_t m) {
    // A bucket costs about six mixed additions over one shared set: two additions
    // of the reduction, of four products on a group of lanes, and its share of
    // the bucket sums.  Below 10 bits the buckets are so few that chunks run
    // long and the small MSM loses its threads.  Witness widths of the default
    // circuits against three additions a bucket: 2^15 constraints 15 -> 13 bits,
    // prove 1139 -> 1034 us; 2^17 16 -> 15, 2301 -> 2254 us; 1.1M 17 either way.
    int best = 10;
    double best_cost = 1e300;
    for (int c = 10; c <= 22; c++) {
        double cost = (double)m * msm_windows(c) + 6.0 * (double)(1u << (c - 1));
        if (cost < best_cost) {
            best_cost = cost;
            best = c;
        }
    }
    return best;
}

template <class F>
static cudaError_t window_table(const void* d_in, size_t n, uint32_t skip, int c, void* d_out, cudaStream_t st,
                                size_t xyzz_bytes) {
    const int W = msm_windows(c);
    const size_t count = n * (size_t)(W - 1);
    void* tmp = nullptr;
    G16_CUDA(g16::dev_malloc(&tmp, (count ? count : 1) * xyzz_bytes));
    cudaError_t e = cudaSuccess;
    {
        TimedLaunch tl("msm_window_table", st);
        k_window_xyzz<F><<<blocks_for(n, 128), 128, 0, st>>>((const uint4*)d_in, (uint32_t)n, skip, c, W,
                                                            (uint4*)d_out, (uint4*)tmp);
    }
    e = cudaGetLastError();
    if (e == cudaSuccess && count) {
        TimedLaunch tl("msm_window_table", st);
        uint4* out1 = (uint4*)((uint8_t*)d_out + n * (xyzz_bytes / 2));   // window 1 onwards
        k_window_normalize<F><<<blocks_for((count + NORM_RUN - 1) / NORM_RUN, 128), 128, 0, st>>>(
            (const uint4*)tmp, count, out1);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    cudaFree(tmp);
    return e;
}

template <class F>
static cudaError_t fixed_base(const void* d_table, const void* d_scalars, size_t n, void* d_out, cudaStream_t st,
                              size_t xyzz_bytes) {
    if (!n) return cudaSuccess;
    void* tmp = nullptr;
    G16_CUDA(g16::dev_malloc(&tmp, n * xyzz_bytes));
    cudaError_t e;
    {
        TimedLaunch tl("fixed_base", st);
        k_fixed_base<F><<<blocks_for(n, 128), 128, 0, st>>>((const uint4*)d_table, (const uint4*)d_scalars, n,
                                                            (uint4*)tmp);
    }
    e = cudaGetLastError();
    if (e == cudaSuccess) {
        TimedLaunch tl("fixed_base", st);
        k_window_normalize<F><<<blocks_for((n + NORM_RUN - 1) / NORM_RUN, 128), 128, 0, st>>>((const uint4*)tmp, n,
                                                                                            (uint4*)d_out);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    cudaFree(tmp);
    return e;
}

cudaError_t fixed_base_g1(const void* d_table, const void* d_scalars, size_t n, void* d_out, cudaStream_t st) {
    return fixed_base<g16d::Fq>(d_table, d_scalars, n, d_out, st, XYZZ_G1_BYTES);
}

cudaError_t fixed_base_g2(const void* d_table, const void* d_scalars, size_t n, void* d_out, cudaStream_t st) {
    return fixed_base<g16d::Fq2>(d_table, d_scalars, n, d_out, st, XYZZ_G2_BYTES);
}

cudaError_t msm_window_table_g1(const void* d_in, size_t n, uint32_t skip, int c, void* d_out, cudaStream_t st) {
    return window_table<g16d::Fq>(d_in, n, skip, c, d_out, st, XYZZ_G1_BYTES);
}

cudaError_t msm_window_table_g2(const void* d_in, size_t n, uint32_t skip, int c, void* d_out, cudaStream_t st) {
    return window_table<g16d::Fq2>(d_in, n, skip, c, d_out, st, XYZZ_G2_BYTES);
}

int msm_window_bits(size_t m) {
    // cost ~ windows * (m + 3.75 * buckets), a bucket at about four mixed additions.
    // us by width, the model's choice in brackets, G1: 2^14 9: 389, [10: 416], 11:
    // 450; 2^16 11: 643, [12: 629], 13: 690; 2^17 12: 891, [13: 939], 14: 937; 2^18
    // 14: 1394, [15: 1326], 16: 1513; 2^20 15: 3625, [16: 3692], 17: 3894.  G2: 2^14
    // 9: 905, [10: 903], 11: 1012; 2^16 11: 1596, [12: 1589], 13: 1641; 2^18 14: 3613,
    // [15: 3522], 16: 4074.  A step to either side is at most 7% better (2^14).  For
    // scalars of which 70% are 0 or 1 it is one to three bits too wide, since it
    // counts all of them: 2^18 836 at 15 bits, 719 at 12.
    int best = 8;
    double best_cost = 1e300;
    for (int c = 8; c <= 18; c++) {
        double windows = (255 + c - 1) / c;
        double cost = windows * ((double)m + 3.75 * (double)(1u << (c - 1)));
        if (cost < best_cost) {
            best_cost = cost;
            best = c;
        }
    }
    return best;
}

// Buffers that are views (fixed) are never reallocated: too small is an error.
static cudaError_t fixed_too_small(size_t need_bytes, size_t cap_bytes) {
    set_error("fixed MSM scratch holds %zu bytes where %zu are needed", cap_bytes, need_bytes);
    return cudaErrorInvalidValue;
}

// Grow-only scratch, reallocated in stream order on st (dev_realloc_async).
template <class T>
static cudaError_t grow(cudaStream_t st, T*& p, size_t& cap, size_t need_elems, bool fixed = false) {
    if (need_elems <= cap && p) return cudaSuccess;
    if (fixed) return fixed_too_small(need_elems * sizeof(T), cap * sizeof(T));
    cap = 0;
    size_t n = need_elems + need_elems / 8 + 64;
    cudaError_t e = g16::dev_realloc_async(&p, n * sizeof(T), st, false);
    if (e != cudaSuccess) {
        cap = 0;
        set_error("cudaMalloc of %zu bytes for MSM scratch failed: %s", n * sizeof(T), cudaGetErrorString(e));
        return e;
    }
    cap = n;
    return cudaSuccess;
}

static cudaError_t grow_bytes(cudaStream_t st, void*& p, size_t& cap, size_t need, bool fixed = false) {
    if (need <= cap && p) return cudaSuccess;
    if (fixed) return fixed_too_small(need, cap);
    cap = 0;
    size_t n = need + need / 8 + 256;
    cudaError_t e = g16::dev_realloc_async(&p, n, st, true);
    if (e != cudaSuccess) {
        cap = 0;
        set_error("cudaMalloc of %zu bytes for MSM scratch failed: %s", n, cudaGetErrorString(e));
        return e;
    }
    cap = n;
    return cudaSuccess;
}

// Scratch words for a plan over Ks buckets: two block sums each.
static size_t plan_tmp_words(size_t Ks) { return 2 * (size_t)msm_plan_grid(Ks).blocks; }

// The accumulate's plan from the bucket counts of `count` sorts (d_counts
// filled); the scatter follows.
static cudaError_t sort_plan(MsmSort* const* sorts, int count, cudaStream_t st) {
    SortPlanSets a = {};
    a.wave = accumulate_wave();
    uint32_t nb = 1;
    for (int j = 0; j < count; j++) {
        const MsmSort& s = *sorts[j];
        a.s[j] = {s.d_counts, s.d_offsets, s.d_cursor, s.d_seg_base, s.d_fat_list, s.d_scan_tmp, s.d_total, s.Ks, s.K,
                  s.chunk, msm_plan_grid(s.Ks)};
        nb = std::max(nb, a.s[j].grid.blocks);
    }
    const dim3 grid(nb, count);
    {
        TimedLaunch tl("msm_plan", st);
        k_plan_sums<<<grid, 256, 0, st>>>(a);
    }
    {
        TimedLaunch tl("msm_plan", st);
        k_plan_offsets<<<grid, 256, 0, st>>>(a);
    }
    {
        TimedLaunch tl("msm_plan", st);
        k_plan_segments<<<grid, 256, 0, st>>>(a);
    }
    return cudaGetLastError();
}

cudaError_t msm_sort(MsmSort& s, const void* d_scalars, size_t n, bool montgomery, int c, cudaStream_t st,
                     bool shared_windows, bool constant_work) {
    if (c == 0) c = msm_window_bits(n);
    if (c < 4 || c > 24) {
        set_error("MSM window of %d bits outside [4, 24]", c);
        return cudaErrorInvalidValue;
    }
    s.c = c;
    s.W = (255 + c - 1) / c;
    s.B = 1u << (c - 1);
    s.shared = shared_windows;
    s.K = shared_windows ? s.B : (uint32_t)s.W * s.B;
    s.constant_work = constant_work;
    s.Ks = s.K + (constant_work ? 1u : 0u);
    s.n = n;
    if ((shared_windows ? n * (size_t)s.W : n) >= 0x80000000ull) {
        set_error("MSM of %zu points x %d windows exceeds the 2^31 entry-index limit", n, s.W);
        return cudaErrorInvalidValue;
    }
    // the smallest chunk the accumulate may use (fixed scratch is sized for MSM_CHUNK);
    // the one it does use is chosen on the device from the entry count
    s.chunk = s.fixed ? MSM_CHUNK : s.chunk_floor;
    const uint32_t kw = shared_windows ? 0u : s.B, ew = shared_windows ? (uint32_t)n : 0u;
    const uint32_t sink = constant_work ? s.K : NO_KEY;
    size_t nn = n ? n : 1;
    G16_CUDA(grow(st, s.d_scalars_std, s.cap_scalars, nn * 8, s.fixed));
    size_t kk = (size_t)s.Ks + 1;
    if (s.fixed && (kk > s.cap_k || !s.d_counts || !s.d_offsets || !s.d_cursor || !s.d_seg_base || !s.d_fat_list))
        G16_CUDA(fixed_too_small(kk * sizeof(uint32_t), s.cap_k * sizeof(uint32_t)));
    if (kk > s.cap_k || !s.d_counts) {
        size_t cap = 0;
        G16_CUDA(grow(st, s.d_counts, cap, kk));
        cap = 0;
        G16_CUDA(grow(st, s.d_offsets, cap, kk));
        cap = 0;
        G16_CUDA(grow(st, s.d_cursor, cap, kk));
        cap = 0;
        G16_CUDA(grow(st, s.d_seg_base, cap, kk));
        cap = 0;
        G16_CUDA(grow(st, s.d_fat_list, cap, kk));
        s.cap_k = cap;
    }
    G16_CUDA(grow(st, s.d_scan_tmp, s.cap_tmp, plan_tmp_words(s.Ks), s.fixed));
    G16_CUDA(grow(st, s.d_entries, s.cap_entries, nn * s.W, s.fixed));
    if (!s.d_total) {
        if (s.fixed) G16_CUDA(fixed_too_small(4 * sizeof(uint32_t), 0));
        G16_CUDA(g16::dev_realloc_async(&s.d_total, 4 * sizeof(uint32_t), st, false));
    }

    G16_CUDA(cudaMemsetAsync(s.d_counts, 0, kk * sizeof(uint32_t), st));
    if (n) {
        timer().add_bytes("msm_digits", 64.0 * n);   // scalars in, standard-form copy out
        TimedLaunch tl("msm_digits", st);
        if (n < DIGITS_SPLIT)
            k_digits_count<8><<<blocks_for(n, 32), 256, 0, st>>>((const uint4*)d_scalars, montgomery ? 1 : 0,
                                                               (uint32_t)n, c, s.W, kw, sink,
                                                               (uint4*)s.d_scalars_std, s.d_counts);
        else
            k_digits_count<1><<<blocks_for(n, 256), 256, 0, st>>>((const uint4*)d_scalars, montgomery ? 1 : 0,
                                                                (uint32_t)n, c, s.W, kw, sink,
                                                                (uint4*)s.d_scalars_std, s.d_counts);
    }
    G16_CUDA(cudaGetLastError());
    MsmSort* const one[1] = {&s};
    G16_CUDA(sort_plan(one, 1, st));
    if (n) {
        TimedLaunch tl("msm_scatter", st);
        if (n < DIGITS_SPLIT)
            k_scatter<8><<<blocks_for(n, 32), 256, 0, st>>>((const uint4*)s.d_scalars_std, (uint32_t)n, c, s.W, kw, ew,
                                                          sink, s.d_cursor, s.d_entries);
        else
            k_scatter<1><<<blocks_for(n, 256), 256, 0, st>>>((const uint4*)s.d_scalars_std, (uint32_t)n, c, s.W, kw,
                                                           ew, sink, s.d_cursor, s.d_entries);
    }
    G16_CUDA(cudaGetLastError());
    return cudaSuccess;
}

cudaError_t msm_sort_sets(MsmSort* sorts, const MsmLiveSets& sets, const void* d_scalars, size_t n, bool montgomery,
                          int c, cudaStream_t st, bool constant_work, bool shared) {
    if (sets.count < 1 || sets.count > MSM_MAX_SETS) {
        set_error("%d live sets (1 to %d)", sets.count, MSM_MAX_SETS);
        return cudaErrorInvalidValue;
    }
    if (c < 4 || c > 24) {
        set_error("MSM window of %d bits outside [4, 24]", c);
        return cudaErrorInvalidValue;
    }
    const int W = (255 + c - 1) / c;
    if (n >= 0x80000000ull) {
        set_error("MSM of %zu scalars exceeds the 2^31 index limit", n);
        return cudaErrorInvalidValue;
    }
    LiveSetArgs a = {};
    for (int j = 0; j < sets.count; j++) {
        MsmSort& s = sorts[j];
        s.c = c;
        s.W = W;
        s.B = 1u << (c - 1);
        s.shared = shared;
        s.K = shared ? s.B : (uint32_t)W * s.B;
        s.constant_work = constant_work;
        s.Ks = s.K + (constant_work ? 1u : 0u);
        s.n = sets.rows[j];
        s.chunk = s.chunk_floor;
        if ((size_t)sets.rows[j] * (size_t)W >= 0x80000000ull || sets.rows[j] > n) {
            set_error("live set of %u rows x %d windows exceeds the 2^31 entry-index limit", sets.rows[j], W);
            return cudaErrorInvalidValue;
        }
        const size_t kk = (size_t)s.Ks + 1;
        if (kk > s.cap_k || !s.d_counts) {
            size_t cap = 0;
            G16_CUDA(grow(st, s.d_counts, cap, kk));
            cap = 0;
            G16_CUDA(grow(st, s.d_offsets, cap, kk));
            cap = 0;
            G16_CUDA(grow(st, s.d_cursor, cap, kk));
            cap = 0;
            G16_CUDA(grow(st, s.d_seg_base, cap, kk));
            cap = 0;
            G16_CUDA(grow(st, s.d_fat_list, cap, kk));
            s.cap_k = cap;
        }
        G16_CUDA(grow(st, s.d_scan_tmp, s.cap_tmp, plan_tmp_words(s.Ks)));
        G16_CUDA(grow(st, s.d_entries, s.cap_entries, (size_t)(sets.rows[j] ? sets.rows[j] : 1) * W));
        if (!s.d_total) G16_CUDA(g16::dev_realloc_async(&s.d_total, 4 * sizeof(uint32_t), st, false));
        G16_CUDA(cudaMemsetAsync(s.d_counts, 0, kk * sizeof(uint32_t), st));
        a.rank[j] = sets.d_rank[j];
        a.counts[j] = s.d_counts;
        a.cursor[j] = s.d_cursor;
        a.entries[j] = s.d_entries;
        a.rows[j] = shared ? sets.rows[j] : 0u;
    }
    a.key_stride = shared ? 0u : (1u << (c - 1));
    // the standard-form copy of the scalars, shared by the sets, lives in the first
    MsmSort& s0 = sorts[0];
    G16_CUDA(grow(st, s0.d_scalars_std, s0.cap_scalars, (n ? n : 1) * 8));
    const uint32_t sink = constant_work ? sorts[0].K : NO_KEY;
    if (n) {
        timer().add_bytes("msm_digits", 64.0 * n);   // scalars in, standard-form copy out
        TimedLaunch tl("msm_digits", st);
        if (n < DIGITS_SPLIT)
            k_digits_count_sets<8><<<blocks_for(n, 32), 256, 0, st>>>((const uint4*)d_scalars, montgomery ? 1 : 0,
                                                                    (uint32_t)n, c, W, sink, sets.count, a,
                                                                    (uint4*)s0.d_scalars_std);
        else
            k_digits_count_sets<1><<<blocks_for(n, 256), 256, 0, st>>>((const uint4*)d_scalars, montgomery ? 1 : 0,
                                                                     (uint32_t)n, c, W, sink, sets.count, a,
                                                                     (uint4*)s0.d_scalars_std);
    }
    G16_CUDA(cudaGetLastError());
    MsmSort* all[MSM_MAX_SETS] = {};
    for (int j = 0; j < sets.count; j++) all[j] = &sorts[j];
    G16_CUDA(sort_plan(all, sets.count, st));
    if (n) {
        TimedLaunch tl("msm_scatter", st);
        if (n < DIGITS_SPLIT)
            k_scatter_sets<8><<<blocks_for(n, 32), 256, 0, st>>>((const uint4*)s0.d_scalars_std, (uint32_t)n, c, W, sink,
                                                               sets.count, a);
        else
            k_scatter_sets<1><<<blocks_for(n, 256), 256, 0, st>>>((const uint4*)s0.d_scalars_std, (uint32_t)n, c, W,
                                                                sink, sets.count, a);
    }
    G16_CUDA(cudaGetLastError());
    return cudaSuccess;
}

// threads of a k_reduce_sets block: a group per point of a term (nb a power of
// two), a warp at least
template <class F>
static unsigned reduce_sets_threads(uint32_t nb) {
    const uint32_t t = nb * Lanes<F>::N;
    return t < 32 ? 32 : t < LANES_BLOCK ? t : LANES_BLOCK;
}

template <class F>
static cudaError_t accumulate(const MsmSort& s, MsmAccum& acc, const void* d_bases, uint32_t base_offset,
                              uint32_t n_bases, cudaStream_t st, size_t xyzz_bytes, const char* tag) {
    size_t max_entries = (s.n ? s.n : 1) * (size_t)s.W;
    const size_t chunks = msm_max_chunks(max_entries, s.chunk);
    size_t max_partials = (size_t)s.Ks + chunks + 1;
    G16_CUDA(grow_bytes(st, acc.d_partials, acc.cap_partials, max_partials * xyzz_bytes, acc.fixed));
    const uint32_t Wr = s.shared ? 1u : (uint32_t)s.W;   // bucket sets to reduce
    constexpr bool G2 = !std::is_same<F, g16d::Fq>::value;
    constexpr int LB = G2 ? MSM_REDUCE_LB_G2 : MSM_REDUCE_LB_G1;   // pieces per reduction block: 2^LB
    const MsmReducePlan plan =
        msm_reduce_plan(Wr, s.B, G2, s.reduce_pieces ? s.reduce_pieces : msm_reduce_pieces(s.shared));
    acc.plan = plan;
    G16_CUDA(grow_bytes(st, acc.d_buckets, acc.cap_buckets, (size_t)s.K * xyzz_bytes, acc.fixed));
    G16_CUDA(grow_bytes(st, acc.d_segments, acc.cap_segments, plan.block_points() * xyzz_bytes, acc.fixed));
    if (!plan.direct)
        G16_CUDA(grow_bytes(st, acc.d_terms, acc.cap_terms, plan.result_points() * xyzz_bytes, acc.fixed));
    G16_CUDA(grow_bytes(st, acc.d_windows, acc.cap_windows, (size_t)plan.sets * xyzz_bytes, acc.fixed));
    if (!acc.d_work) {
        if (acc.fixed) G16_CUDA(fixed_too_small(sizeof(unsigned long long), 0));
        G16_CUDA(g16::dev_realloc_async(&acc.d_work, sizeof(unsigned long long), st, false));
    }
    G16_CUDA(cudaMemsetAsync(acc.d_work, 0, sizeof(unsigned long long), st));
    uint4* partials = (uint4*)acc.d_partials;
    {
        TimedLaunch tl(tag, st);
        if (std::is_same<F, g16d::Fq>::value)
            k_accumulate_g1<<<blocks_for(chunks, ACC_BLOCK_G1), ACC_BLOCK_G1, 0, st>>>(
                s.d_entries, s.d_offsets, s.d_seg_base, s.Ks, s.d_total, s.d_total + 3, (const uint4*)d_bases,
                base_offset, n_bases, partials, acc.d_work);
        else
            k_accumulate_g2<<<blocks_for(chunks, ACC_BLOCK_G2), ACC_BLOCK_G2, 0, st>>>(
                s.d_entries, s.d_offsets, s.d_seg_base, s.Ks, s.d_total, s.d_total + 3, (const uint4*)d_bases,
                base_offset, n_bases, partials, acc.d_work);
    }
    G16_CUDA(cudaGetLastError());
    {
        TimedLaunch tl("msm_fat_merge", st);
        k_fat_merge_jobs<F><<<2 * device_sms(), LANES_BLOCK, 0, st>>>(partials, s.d_offsets, s.d_seg_base, s.d_fat_list,
                                                                      s.d_total + 2, s.d_total + 3);
    }
    {
        TimedLaunch tl("msm_fat_merge", st);
        k_fat_merge_final<F><<<device_sms(), LANES_BLOCK, 0, st>>>(partials, s.d_offsets, s.d_seg_base, s.d_fat_list,
                                                                   s.d_total + 2, s.d_total + 3);
    }
    G16_CUDA(cudaGetLastError());
    {
        TimedLaunch tl("msm_bucket_sums", st);
        k_bucket_sums<F><<<blocks_for(s.K, LANES_GROUPS<F>), LANES_BLOCK, 0, st>>>(
            partials, s.d_offsets, s.d_seg_base, s.K, s.d_total + 3, (uint4*)acc.d_buckets);
    }
    {
        TimedLaunch tl("msm_reduce", st);
        k_reduce_pieces<F, LB><<<dim3(plan.nb, Wr), REDUCE_BLOCK<F, LB>, 0, st>>>((const uint4*)acc.d_buckets, s.B,
                                                                                plan.seg, (uint4*)acc.d_segments);
    }
    if (!plan.direct) {
        TimedLaunch tl("msm_reduce_sets", st);
        k_reduce_sets<F, LB><<<dim3(LB + 1 + plan.hb, Wr), reduce_sets_threads<F>(plan.nb), 0, st>>>(
            (const uint4*)acc.d_segments, plan.nb, (uint4*)acc.d_terms);
    }
    {
        TimedLaunch tl("msm_reduce_finish", st);
        k_reduce_finish<F, LB><<<Wr, FINISH_BLOCK<F>, 0, st>>>((const uint4*)(plan.direct ? acc.d_segments : acc.d_terms),
                                                              plan.set_terms(), plan.nb, plan.hb, plan.direct, plan.seg,
                                                              (uint4*)acc.d_windows);
    }
    G16_CUDA(cudaGetLastError());
    return cudaSuccess;
}

cudaError_t msm_accumulate_g1(const MsmSort& s, MsmAccum& acc, const void* d_bases, uint32_t base_offset,
                              uint32_t n_bases, cudaStream_t st) {
    return accumulate<g16d::Fq>(s, acc, d_bases, base_offset, n_bases, st, XYZZ_G1_BYTES, "msm_accumulate_g1");
}

cudaError_t msm_accumulate_g2(const MsmSort& s, MsmAccum& acc, const void* d_bases, uint32_t base_offset,
                              uint32_t n_bases, cudaStream_t st) {
    return accumulate<g16d::Fq2>(s, acc, d_bases, base_offset, n_bases, st, XYZZ_G2_BYTES, "msm_accumulate_g2");
}

// ---- batched MSMs ----
void MsmSpace::release() {
    sort.release();
    acc.release();
    cudaFree(d_segdev);
    cudaFree(d_reduce);
    d_segdev = d_reduce = nullptr;
    cap_segdev = cap_reduce = 0;
}

void MsmSources::release() {
    cudaFree(d_desc);
    cudaFree(d_blk);
    cudaFree(d_std);
    d_desc = nullptr;
    d_blk = nullptr;
    d_std = nullptr;
    cap_desc = cap_blk = cap_std = 0;
}

// Upload a descriptor table into a device buffer that only grows (cap in bytes).
template <class T>
static cudaError_t upload_vec(void*& d, size_t& cap, const std::vector<T>& v, cudaStream_t st) {
    G16_CUDA(grow_bytes(st, d, cap, (v.empty() ? 1 : v.size()) * sizeof(T)));
    if (!v.empty()) G16_CUDA(cudaMemcpyAsync(d, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice, st));
    return cudaSuccess;
}

cudaError_t msm_batch_setup(MsmSources& so, MsmSpace* const* spaces, int nspaces, cudaStream_t st) {
    // entries each space can receive: every live row of every target, once per window
    for (int i = 0; i < nspaces; i++) spaces[i]->max_entries = 0;
    for (auto& src : so.srcs) {
        if (src.c < 4 || src.c > 24 || src.ntargets < 0 || src.ntargets > MSM_MAX_TARGETS) {
            set_error("batched MSM source with window %d bits and %d targets", src.c, src.ntargets);
            return cudaErrorInvalidValue;
        }
        const uint32_t W = (uint32_t)msm_windows(src.c);
        for (int j = 0; j < src.ntargets; j++) {
            const MsmSourceTgt& t = src.t[j];
            if (t.space < 0 || t.space >= nspaces || t.seg < 0 || (size_t)t.seg >= spaces[t.space]->segs.size() ||
                spaces[t.space]->segs[t.seg].B != (1u << (src.c - 1)) || (uint64_t)t.rows * W >= 0x80000000ull) {
                set_error("batched MSM target does not match its segment");
                return cudaErrorInvalidValue;
            }
            spaces[t.space]->max_entries += (size_t)(t.d_rank ? t.rows : src.n) * W;
        }
    }
    for (int i = 0; i < nspaces; i++) {
        MsmSpace& sp = *spaces[i];
        const size_t pb = sp.g2 ? XYZZ_G2_BYTES : XYZZ_G1_BYTES;
        uint32_t piece_len = 0;
        if (const char* e = std::getenv("G16_BATCH_PIECE_LEN")) piece_len = (uint32_t)std::max(0, std::atoi(e));   // tuning knob: 1, 2, 4, ..., 32
        std::vector<uint32_t> seg_B;
        for (auto& g : sp.segs) seg_B.push_back(g.B);
        const MsmSpaceReduceLayout L = msm_space_reduce_layout(seg_B, sp.g2, sp.pieces_target, device_sms(), piece_len);
        std::vector<MsmSegDev> segdev;
        std::vector<MsmReduceDev> red;
        for (size_t j = 0; j < sp.segs.size(); j++) {
            MsmSpaceSeg& g = sp.segs[j];
            g.key_start = L.key_start[j];
            g.plan = L.plans[j];
            g.block_start = L.block_start[j];
            g.out_block = L.out_block[j];
            g.out_set = L.out_set[j];
            segdev.push_back({(const uint4*)g.table, g.key_start, g.n_bases});
            red.push_back({g.key_start, g.B, g.plan.seg, g.plan.nb, g.plan.hb, g.block_start, g.out_block, g.out_set});
        }
        sp.max_hb = L.max_hb;
        const uint64_t K = L.K, blocks = L.blocks, out_block = L.block_points, out_set = L.result_points;
        if (K >= 0x80000000ull || sp.max_entries >= 0x80000000ull) {
            set_error("batched MSM space of %llu buckets and %zu entries exceeds 32-bit indices",
                      (unsigned long long)K, sp.max_entries);
            return cudaErrorInvalidValue;
        }
        sp.K = (uint32_t)K;
        sp.blocks = (uint32_t)blocks;
        sp.result_points = (uint32_t)sp.segs.size();
        MsmSort& s = sp.sort;
        s.K = s.Ks = sp.K;
        s.B = 0;
        s.shared = true;
        s.chunk = s.chunk_floor;
        s.n = sp.max_entries;   // accumulate sizes its partials by entries, W = 1 below
        s.W = 1;
        const size_t kk = (size_t)sp.K + 1;
        if (kk > s.cap_k || !s.d_counts) {
            size_t cap = 0;
            G16_CUDA(grow(st, s.d_counts, cap, kk));
            cap = 0;
            G16_CUDA(grow(st, s.d_offsets, cap, kk));
            cap = 0;
            G16_CUDA(grow(st, s.d_cursor, cap, kk));
            cap = 0;
            G16_CUDA(grow(st, s.d_seg_base, cap, kk));
            cap = 0;
            G16_CUDA(grow(st, s.d_fat_list, cap, kk));
            s.cap_k = cap;
        }
        G16_CUDA(grow(st, s.d_scan_tmp, s.cap_tmp, plan_tmp_words(s.Ks)));
        G16_CUDA(grow(st, s.d_entries, s.cap_entries, sp.max_entries ? sp.max_entries : 1));
        if (!s.d_total) G16_CUDA(g16::dev_realloc_async(&s.d_total, 4 * sizeof(uint32_t), st, false));
        MsmAccum& a = sp.acc;
        const size_t chunks = msm_max_chunks(sp.max_entries, s.chunk);
        G16_CUDA(grow_bytes(st, a.d_partials, a.cap_partials, ((size_t)sp.K + chunks + 1) * pb));
        G16_CUDA(grow_bytes(st, a.d_buckets, a.cap_buckets, ((size_t)sp.K + 1) * pb));
        G16_CUDA(grow_bytes(st, a.d_segments, a.cap_segments, (out_block + 1) * pb));
        G16_CUDA(grow_bytes(st, a.d_terms, a.cap_terms, (out_set + 1) * pb));
        G16_CUDA(grow_bytes(st, a.d_windows, a.cap_windows, (sp.segs.size() + 1) * pb));
        if (!a.d_work) G16_CUDA(g16::dev_realloc_async(&a.d_work, sizeof(unsigned long long), st, false));
        G16_CUDA(upload_vec(sp.d_segdev, sp.cap_segdev, segdev, st));
        G16_CUDA(upload_vec(sp.d_reduce, sp.cap_reduce, red, st));
    }
    // sources: one block of 256 scalars never straddles two sources
    std::vector<MsmSourceDev> desc;
    std::vector<uint32_t> blk;
    size_t std_elems = 0;
    for (auto& src : so.srcs) std_elems += src.n;
    G16_CUDA(grow_bytes(st, so.d_std, so.cap_std, (std_elems ? std_elems : 1) * 32));
    uint64_t blocks = 0, off = 0;
    for (auto& src : so.srcs) {
        MsmSourceDev d = {};
        d.scalars = (const uint4*)src.d_scalars;
        d.std_out = (uint4*)((uint8_t*)so.d_std + off * 32);
        d.n = src.n;
        d.c = (uint32_t)src.c;
        d.W = (uint32_t)msm_windows(src.c);
        d.ntargets = (uint32_t)src.ntargets;
        for (int j = 0; j < src.ntargets; j++) {
            MsmSpace& sp = *spaces[src.t[j].space];
            d.t[j] = {sp.sort.d_counts, sp.sort.d_cursor, sp.sort.d_entries, src.t[j].d_rank,
                      sp.segs[src.t[j].seg].key_start, src.t[j].d_rank ? src.t[j].rows : src.n};
        }
        desc.push_back(d);
        blk.push_back((uint32_t)blocks);
        blocks += (src.n + 255) / 256;
        off += src.n;
    }
    if (blocks >= 0x80000000ull) {
        set_error("batched MSM sources of %llu blocks", (unsigned long long)blocks);
        return cudaErrorInvalidValue;
    }
    so.total_blocks = (uint32_t)blocks;
    G16_CUDA(upload_vec(so.d_desc, so.cap_desc, desc, st));
    void* dblk = so.d_blk;
    G16_CUDA(upload_vec(dblk, so.cap_blk, blk, st));
    so.d_blk = (uint32_t*)dblk;
    G16_CUDA(cudaStreamSynchronize(st));
    return cudaSuccess;
}

cudaError_t msm_batch_sort(MsmSources& so, MsmSpace* const* spaces, int nspaces, cudaStream_t st) {
    for (int i = 0; i < nspaces; i++) {
        MsmSort& s = spaces[i]->sort;
        G16_CUDA(cudaMemsetAsync(s.d_counts, 0, ((size_t)s.K + 1) * sizeof(uint32_t), st));
    }
    const uint32_t nsrc = (uint32_t)so.srcs.size();
    if (so.total_blocks) {
        TimedLaunch tl("msm_digits", st);
        k_digits_multi<<<so.total_blocks, 256, 0, st>>>((const MsmSourceDev*)so.d_desc, so.d_blk, nsrc);
    }
    G16_CUDA(cudaGetLastError());
    MsmSort* all[MSM_MAX_SETS] = {};
    if (nspaces > MSM_MAX_SETS) {
        set_error("%d MSM spaces in one sort (at most %d)", nspaces, MSM_MAX_SETS);
        return cudaErrorInvalidValue;
    }
    for (int i = 0; i < nspaces; i++) all[i] = &spaces[i]->sort;
    G16_CUDA(sort_plan(all, nspaces, st));
    if (so.total_blocks) {
        TimedLaunch tl("msm_scatter", st);
        k_scatter_multi<<<so.total_blocks, 256, 0, st>>>((const MsmSourceDev*)so.d_desc, so.d_blk, nsrc);
    }
    G16_CUDA(cudaGetLastError());
    return cudaSuccess;
}

template <class F, int LB>
static cudaError_t space_accumulate(MsmSpace& sp, cudaStream_t st, size_t xyzz_bytes, const char* tag) {
    MsmSort& s = sp.sort;
    MsmAccum& a = sp.acc;
    const size_t chunks = msm_max_chunks(sp.max_entries, s.chunk);
    G16_CUDA(cudaMemsetAsync(a.d_work, 0, sizeof(unsigned long long), st));
    uint4* partials = (uint4*)a.d_partials;
    const uint32_t nsegs = (uint32_t)sp.segs.size();
    // the blocks' output was laid out from the plans: they must use this LB
    for (const auto& g : sp.segs)
        if (g.plan.lb != (uint32_t)LB) {
            set_error("batched MSM reduction planned with 2^%u pieces per block, launched with 2^%d", g.plan.lb, LB);
            return cudaErrorInvalidValue;
        }
    if (chunks) {
        TimedLaunch tl(tag, st);
        if (std::is_same<F, g16d::Fq>::value)
            k_accumulate_multi_g1<<<blocks_for(chunks, ACC_BLOCK_G1), ACC_BLOCK_G1, 0, st>>>(
                s.d_entries, s.d_offsets, s.d_seg_base, s.K, s.d_total, s.d_total + 3, (const MsmSegDev*)sp.d_segdev,
                nsegs, partials, a.d_work);
        else
            k_accumulate_multi_g2<<<blocks_for(chunks, ACC_BLOCK_G2), ACC_BLOCK_G2, 0, st>>>(
                s.d_entries, s.d_offsets, s.d_seg_base, s.K, s.d_total, s.d_total + 3, (const MsmSegDev*)sp.d_segdev,
                nsegs, partials, a.d_work);
    }
    G16_CUDA(cudaGetLastError());
    const uint32_t sms = device_sms();
    {
        TimedLaunch tl("msm_fat_merge", st);
        k_fat_merge_jobs<F><<<2 * sms, LANES_BLOCK, 0, st>>>(partials, s.d_offsets, s.d_seg_base, s.d_fat_list,
                                                            s.d_total + 2, s.d_total + 3);
    }
    {
        TimedLaunch tl("msm_fat_merge", st);
        k_fat_merge_final<F><<<sms, LANES_BLOCK, 0, st>>>(partials, s.d_offsets, s.d_seg_base, s.d_fat_list,
                                                          s.d_total + 2, s.d_total + 3);
    }
    G16_CUDA(cudaGetLastError());
    if (s.K) {
        TimedLaunch tl("msm_bucket_sums", st);
        k_bucket_sums<F><<<blocks_for(s.K, LANES_GROUPS<F>), LANES_BLOCK, 0, st>>>(
            partials, s.d_offsets, s.d_seg_base, s.K, s.d_total + 3, (uint4*)a.d_buckets);
    }
    if (sp.blocks) {
        TimedLaunch tl("msm_reduce", st);
        k_reduce_pieces_multi<F, LB><<<sp.blocks, REDUCE_BLOCK<F, LB>, 0, st>>>(
            (const uint4*)a.d_buckets, (const MsmReduceDev*)sp.d_reduce, nsegs, (uint4*)a.d_segments);
    }
    if (nsegs) {
        TimedLaunch tl("msm_reduce_sets", st);
        k_reduce_sets_multi<F, LB><<<dim3(LB + 1 + sp.max_hb, nsegs), LANES_BLOCK, 0, st>>>(
            (const uint4*)a.d_segments, (const MsmReduceDev*)sp.d_reduce, (uint4*)a.d_terms);
    }
    if (nsegs) {
        TimedLaunch tl("msm_reduce_finish", st);
        k_reduce_finish_multi<F, LB><<<nsegs, FINISH_BLOCK<F>, 0, st>>>(
            (const uint4*)a.d_terms, (const MsmReduceDev*)sp.d_reduce, (uint4*)a.d_windows);
    }
    G16_CUDA(cudaGetLastError());
    return cudaSuccess;
}

cudaError_t msm_space_accumulate(MsmSpace& sp, cudaStream_t st) {
    if (sp.g2) return space_accumulate<g16d::Fq2, MSM_REDUCE_LB_G2>(sp, st, XYZZ_G2_BYTES, "msm_accumulate_g2");
    return space_accumulate<g16d::Fq, MSM_REDUCE_LB_G1>(sp, st, XYZZ_G1_BYTES, "msm_accumulate_g1");
}

// ---- host: window sums -> Horner ----
static Fq fq_at(const uint8_t* p) {
    uint64_t v[4];
    std::memcpy(v, p, 32);
    return Fq::raw(v);
}

template <class F>
static F read_coord(const uint8_t* p);
template <>
Fq read_coord<Fq>(const uint8_t* p) { return fq_at(p); }
template <>
Fq2 read_coord<Fq2>(const uint8_t* p) { return {fq_at(p), fq_at(p + 32)}; }

// XYZZ (x = X / ZZ, y = Y / ZZZ) -> Jacobian (x = X' / Z^2, y = Y' / Z^3)
// without an inversion: Z = ZZ ZZZ, X' = X ZZ ZZZ^2, Y' = Y ZZ^3 ZZZ^2.
template <class F>
static Jac<F> xyzz_to_jac(const uint8_t* p) {
    const size_t cs = sizeof(F) == sizeof(Fq) ? 32 : 64;   // coordinate bytes
    F X = read_coord<F>(p), Y = read_coord<F>(p + cs), zz = read_coord<F>(p + 2 * cs), zzz = read_coord<F>(p + 3 * cs);
    if (zz.is_zero()) return Jac<F>::identity();
    F zzz2 = zzz.sqr();
    Jac<F> r;
    r.z = zz * zzz;
    r.x = X * zz * zzz2;
    r.y = Y * zz.sqr() * zz * zzz2;
    return r;
}

// Horner over the sets' sums
template <class F>
static Jac<F> combine(const uint8_t* sums, uint32_t sets, int c) {
    const size_t pb = 4 * (sizeof(F) == sizeof(Fq) ? 32 : 64);
    Jac<F> acc = Jac<F>::identity();
    for (uint32_t i = sets; i-- > 0;) {
        if (i + 1 < sets)
            for (int j = 0; j < c; j++) acc = acc.dbl();
        acc = acc + xyzz_to_jac<F>(sums + i * pb);
    }
    return acc;
}

G1J msm_combine_g1(const uint8_t* sums_xyzz, const MsmReducePlan& plan, int c) {
    return combine<Fq>(sums_xyzz, plan.sets, c);
}
G2J msm_combine_g2(const uint8_t* sums_xyzz, const MsmReducePlan& plan, int c) {
    return combine<Fq2>(sums_xyzz, plan.sets, c);
}

}  // namespace g16

namespace g16 {

G1J msm_space_combine_g1(const uint8_t* results, const MsmSpace& sp, size_t s) {
    return msm_combine_g1(results + s * XYZZ_G1_BYTES, sp.segs[s].plan, 1);
}

G2J msm_space_combine_g2(const uint8_t* results, const MsmSpace& sp, size_t s) {
    return msm_combine_g2(results + s * XYZZ_G2_BYTES, sp.segs[s].plan, 1);
}

}  // namespace g16
