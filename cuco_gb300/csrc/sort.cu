// Cell keys, stable LSD radix sort, and the reorder / cell-bound kernels.
//
// Reference: calcHashD (gravlist_kernel.cu:92-118), RadixSort::sort ->
// radixSort (radixsort.h:170-187, radixsort.cu:1048-1145), and
// reorderDataAndFindCellStartD (gravlist_kernel.cu:121-160).
//
// The sort is a three-kernel-per-pass LSD radix sort designed for sm_103a:
//   1. k_sort_hist:   per tile, a digit histogram (one shared-memory counter
//                     row per warp);
//   2. k_sort_scan:   one CTA per digit turns its tile counts into inclusive
//                     prefixes over the tiles (the digit's total is the last);
//   3. k_sort_scatter: each tile ranks its keys stably with warp ballots
//                     (the lanes sharing a digit are found from RB ballots, the
//                     rank is a popcount below the lane), takes each run's
//                     global offset from the digit totals and its own
//                     prefix, stages the tile in digit order in shared memory
//                     and writes out digit runs with coalesced stores.
// Digits are 4..8 bits; a pass count of ceil(bits/8) with equal digit widths
// is used (18-bit keys: three 6-bit passes).
//
// What bounds it: memory traffic at millions of keys, latency below.  Every
// kernel issues all of a thread's loads before it uses the first: the ranking
// loop used to load a key per round, behind the round's warp barriers, and
// the scatter counted the next pass's digits with global atomics, which cost
// more than reading the keys again.  A tile is 4096 keys, or 2048 or 1024
// where that would leave SMs without four tiles (sort_items).  Measured alone,
// before and after, a pass over 4M pairs: histogram 27 -> 6, scan 5 -> 4,
// scatter 33 -> 26 us; three passes over 32K pairs 93 -> 36 us.
//
// Up to kClusterMax keys take one launch instead: a cluster of eight CTAs holds
// every key in shared memory, ranks each pass's digits, exchanges the digit
// totals and scatters the pairs through distributed shared memory.  What
// bounds such a sort is launches: 32K pairs of 18 bits were nine of them and
// 36 us of kernels, and two copies back where the pass count is odd.
#include <cooperative_groups.h>

#include "common.cuh"
#include "shortrange_plan.cuh"

namespace cg = cooperative_groups;

namespace cuco {

namespace {

constexpr int kSortThreads = 256;
constexpr int kSortWarps = kSortThreads / 32;
constexpr unsigned kFull = 0xffffffffu;

__device__ __forceinline__ int cell_coord(float t, int G) {
    int c = (int)t;  // truncation toward zero (cvt.rzi), as calcHashD's int3 assignment
    c = c < 0 ? 0 : c;
    return c >= G ? G - 1 : c;
}

__global__ void k_cell_keys(const float4 *__restrict__ pos, uint32_t *__restrict__ keys,
                            uint32_t *__restrict__ idx, uint32_t n, float gridfac, int G) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        float4 p = pos[i];
        int ix = cell_coord(__fmul_rn(gridfac, p.x), G);
        int iy = cell_coord(__fmul_rn(gridfac, p.y), G);
        int iz = cell_coord(__fmul_rn(gridfac, p.z), G);
        keys[i] = ((uint32_t)ix * G + iy) * G + iz;
        if (idx) idx[i] = i;
    }
}

// Digit counts of each tile of kSortThreads * ITEMS keys.
template <int RB, int ITEMS>
__global__ void __launch_bounds__(kSortThreads)
    k_sort_hist(const uint32_t *__restrict__ keys, uint32_t n, int shift, uint32_t *__restrict__ hist,
                uint32_t tiles) {
    constexpr int RADIX = 1 << RB;
    __shared__ uint32_t h[kSortWarps][RADIX];
    const int warp = threadIdx.x >> 5;
    const uint32_t tile = blockIdx.x, base = tile * (kSortThreads * ITEMS) + threadIdx.x;
    uint32_t key[ITEMS];
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        const uint32_t i = base + k * kSortThreads;
        key[k] = i < n ? keys[i] : 0u;
    }
    for (int e = threadIdx.x; e < kSortWarps * RADIX; e += kSortThreads) (&h[0][0])[e] = 0;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < ITEMS; ++k)
        if (base + k * kSortThreads < n) atomicAdd(&h[warp][(key[k] >> shift) & (RADIX - 1)], 1u);
    __syncthreads();
    for (int d = threadIdx.x; d < RADIX; d += kSortThreads) {
        uint32_t c = 0;
#pragma unroll
        for (int w = 0; w < kSortWarps; ++w) c += h[w][d];
        hist[(size_t)d * tiles + tile] = c;
    }
}

// hist[d*tiles + t] (count of digit d in tile t) -> the inclusive prefix of
// those counts over the tiles, one CTA per digit.  A digit's total is then its
// last entry, and the scatter derives every run's global offset from these
// (no second pass over the table, no scratch beyond it).  Four counts a
// thread and round are in flight together.
constexpr int kScanThreads = 512, kScanWarps = kScanThreads / 32, kScanItems = 4;
__global__ void __launch_bounds__(kScanThreads) k_sort_scan(uint32_t *__restrict__ hist, uint32_t tiles) {
    __shared__ uint32_t wsum[kScanItems][kScanWarps];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint32_t *h = hist + (size_t)blockIdx.x * tiles;
    uint32_t carry = 0;
    for (uint32_t t0 = 0; t0 < tiles; t0 += kScanThreads * kScanItems) {
        uint32_t incl[kScanItems];
#pragma unroll
        for (int j = 0; j < kScanItems; ++j) {
            const uint32_t t = t0 + j * kScanThreads + threadIdx.x;
            incl[j] = t < tiles ? h[t] : 0u;
        }
#pragma unroll
        for (int j = 0; j < kScanItems; ++j) {
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const uint32_t y = __shfl_up_sync(kFull, incl[j], off);
                if (lane >= off) incl[j] += y;
            }
            if (lane == 31) wsum[j][warp] = incl[j];
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < kScanItems; ++j) {
            uint32_t before = carry;
#pragma unroll
            for (int w = 0; w < kScanWarps; ++w) {
                const uint32_t x = wsum[j][w];
                before += w < warp ? x : 0u;
                carry += x;
            }
            const uint32_t t = t0 + j * kScanThreads + threadIdx.x;
            if (t < tiles) h[t] = before + incl[j];
        }
        __syncthreads();  // wsum is rewritten by the next round
    }
}

// The values are read when the ranks are known: held through the ranking they
// took 88 registers, two CTAs an SM.  (At 16 keys a thread three CTAs without
// spills beat four: 4 passes over 4M pairs 132 against 140 us.)
template <int RB, int ITEMS, bool WITH_VALS>
__global__ void __launch_bounds__(kSortThreads, ITEMS == 16 ? 3 : 4)
    k_sort_scatter(const uint32_t *__restrict__ kin, const uint32_t *__restrict__ vin, uint32_t *__restrict__ kout,
                   uint32_t *__restrict__ vout, uint32_t n, int shift, const uint32_t *__restrict__ hist,
                   uint32_t tiles) {
    constexpr int RADIX = 1 << RB;
    constexpr uint32_t TILE = kSortThreads * ITEMS;
    static_assert(RADIX <= kSortThreads, "a thread per digit");
    __shared__ uint32_t wcnt[kSortWarps][RADIX];
    __shared__ uint32_t dstart[RADIX];  // digit's start in the staged tile
    __shared__ uint32_t gofs[RADIX];    // staged position -> global position
    __shared__ uint32_t wsum[2][kSortWarps];
    __shared__ uint32_t skeys[TILE];
    __shared__ uint32_t svals[WITH_VALS ? TILE : 1];

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t tile = blockIdx.x;
    const uint32_t base = tile * TILE;
    const uint32_t lt = (1u << lane) - 1u;
    // Warp w owns tile elements [w * 32 * ITEMS, ...); item k covers 32 of
    // them in lane order, so (k, lane) order is input order and the ranks are
    // stable.
    const uint32_t first = base + warp * (32 * ITEMS) + lane;
    uint32_t key[ITEMS];
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        const uint32_t i = first + k * 32;
        key[k] = i < n ? kin[i] : 0xffffffffu;
    }
    // this thread's digit: the prefix over the tiles up to this one, the total
    uint32_t gp = 0, gt = 0;
    if (tid < RADIX) {
        gp = hist[(size_t)tid * tiles + tile];
        gt = hist[(size_t)tid * tiles + tiles - 1];
    }
    for (int d = lane; d < RADIX; d += 32) wcnt[warp][d] = 0;
    __syncwarp();
    // the ranks (below 4096) two to a register
    uint32_t rank2[(ITEMS + 1) / 2];
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        const bool valid = first + k * 32 < n;
        const uint32_t d = (key[k] >> shift) & (RADIX - 1);
        uint32_t peers = __ballot_sync(kFull, valid);
#pragma unroll
        for (int b = 0; b < RB; ++b) {
            const uint32_t bit = (d >> b) & 1u;
            const uint32_t m = __ballot_sync(kFull, bit);
            peers &= bit ? m : ~m;
        }
        if (!valid) peers = 1u << lane;
        // the lowest lane of a digit's group keeps the warp's counter
        const int lead = __ffs(peers) - 1;
        uint32_t c = 0;
        if (valid && lane == lead) {
            c = wcnt[warp][d];
            wcnt[warp][d] = c + __popc(peers);
        }
        const uint32_t r = __shfl_sync(kFull, c, lead) + __popc(peers & lt);
        if (k & 1)
            rank2[k >> 1] |= r << 16;
        else
            rank2[k >> 1] = r;
        __syncwarp();
    }
    __syncthreads();
    uint32_t val[WITH_VALS ? ITEMS : 1];
    if (WITH_VALS) {
#pragma unroll
        for (int k = 0; k < ITEMS; ++k) {
            const uint32_t i = first + k * 32;
            val[k] = vin && i < n ? vin[i] : i;
        }
    }
    // thread d: the digit's counts over the warps, then two exclusive scans
    // over the digits (this tile's counts, the global totals)
    uint32_t v = 0;
    if (tid < RADIX) {
#pragma unroll
        for (int w = 0; w < kSortWarps; ++w) {
            const uint32_t c = wcnt[w][tid];
            wcnt[w][tid] = v;
            v += c;
        }
    }
    uint32_t incl = v, tincl = gt;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const uint32_t y = __shfl_up_sync(kFull, incl, off), ty = __shfl_up_sync(kFull, tincl, off);
        if (lane >= off) incl += y, tincl += ty;
    }
    if (RADIX > 32) {
        if (lane == 31) wsum[0][warp] = incl, wsum[1][warp] = tincl;
        __syncthreads();
#pragma unroll
        for (int w = 0; w < kSortWarps; ++w) {
            incl += w < warp ? wsum[0][w] : 0u;
            tincl += w < warp ? wsum[1][w] : 0u;
        }
    }
    if (tid < RADIX) {
        dstart[tid] = incl - v;
        // the digit's run from this tile starts after the lower digits'
        // totals and this digit's runs from earlier tiles
        gofs[tid] = (tincl - gt) + (gp - v) - (incl - v);
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        if (first + k * 32 < n) {
            const uint32_t d = (key[k] >> shift) & (RADIX - 1);
            const uint32_t lp = dstart[d] + wcnt[warp][d] + ((rank2[k >> 1] >> (16 * (k & 1))) & 0xffffu);
            skeys[CUCO_IDX(lp, TILE)] = key[k];
            if (WITH_VALS) svals[CUCO_IDX(lp, TILE)] = val[k];
        }
    }
    __syncthreads();
    const uint32_t tile_n = min(TILE, n - base);
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        const uint32_t j = k * kSortThreads + tid;
        if (j < tile_n) {
            const uint32_t kk = skeys[j];
            const uint32_t o = gofs[(kk >> shift) & (RADIX - 1)] + j;
            kout[CUCO_IDX(o, n)] = kk;
            if (WITH_VALS) vout[CUCO_IDX(o, n)] = svals[j];
        }
    }
}

// Keys per thread of a tile: the most that leave four tiles for each of ~150
// SMs (2M pairs, three passes: 8 keys 70 us, 16 keys 83 us; at 4M they are
// level), in a table of at most hist_words counts (16 always fits).
int sort_items(uint32_t n, int rb, size_t hist_words) {
    for (int items : {4, 8}) {
        const uint32_t next = kSortThreads * items * 2;
        const size_t tiles = (n + kSortThreads * items - 1) / (kSortThreads * items);
        if (n / next < 608u && (tiles << rb) <= hist_words) return items;
    }
    return 16;
}

// One pass.
template <int RB, int ITEMS>
cuco_status_t sort_pass_items(const uint32_t *kin, const uint32_t *vin, uint32_t *kout, uint32_t *vout,
                              bool with_vals, uint32_t *hist, uint32_t n, int shift, cudaStream_t stream,
                              int *launches) {
    const uint32_t tiles = (n + kSortThreads * ITEMS - 1) / (kSortThreads * ITEMS);
    k_sort_hist<RB, ITEMS><<<tiles, kSortThreads, 0, stream>>>(kin, n, shift, hist, tiles);
    k_sort_scan<<<1u << RB, kScanThreads, 0, stream>>>(hist, tiles);
    if (with_vals)
        k_sort_scatter<RB, ITEMS, true><<<tiles, kSortThreads, 0, stream>>>(kin, vin, kout, vout, n, shift, hist, tiles);
    else
        k_sort_scatter<RB, ITEMS, false><<<tiles, kSortThreads, 0, stream>>>(kin, vin, kout, vout, n, shift, hist, tiles);
    *launches += 3;
    CUCO_TRY_CUDA(cudaGetLastError());
    return CUCO_OK;
}

template <int RB>
cuco_status_t sort_pass(int items, const uint32_t *kin, const uint32_t *vin, uint32_t *kout, uint32_t *vout,
                        bool with_vals, uint32_t *hist, uint32_t n, int shift, cudaStream_t stream, int *launches) {
    switch (items) {
        case 4: return sort_pass_items<RB, 4>(kin, vin, kout, vout, with_vals, hist, n, shift, stream, launches);
        case 8: return sort_pass_items<RB, 8>(kin, vin, kout, vout, with_vals, hist, n, shift, stream, launches);
        default: return sort_pass_items<RB, 16>(kin, vin, kout, vout, with_vals, hist, n, shift, stream, launches);
    }
}

// ---- the one-launch sort of up to kClusterMax keys
constexpr int kClusterCtas = 8, kClusterThreads = 1024, kClusterWarps = kClusterThreads / 32;
constexpr uint32_t kClusterMax = 8u * kClusterCtas * kClusterThreads;

// Cells (prev, cur] start at sorted index i: a lane's few by itself, a long
// gap by the whole warp.  Every lane of the warp calls it together (`has`: it
// holds an index; prev + 1 = first for the first).
__device__ __forceinline__ void fill_offsets(uint32_t *__restrict__ cell_off, bool has, uint32_t first, uint32_t cur,
                                             uint32_t i) {
    const bool is_long = has && cur >= first && cur - first >= 8u;
    if (has && !is_long)
        for (uint32_t c = first; c <= cur; ++c) cell_off[c] = i;
    for (uint32_t rest = __ballot_sync(kFull, is_long); rest; rest &= rest - 1) {
        const int src = __ffs(rest) - 1;
        const uint32_t a = __shfl_sync(kFull, first, src), b = __shfl_sync(kFull, cur, src), v = __shfl_sync(kFull, i, src);
        for (uint32_t c = a + (threadIdx.x & 31); c <= b; c += 32) cell_off[c] = v;
    }
}

// Shared memory of a CTA: its pairs, the same staged in digit order (so that
// the pairs a warp sends to another CTA are runs: single pairs sent as they
// came took 10 us a pass), each warp's digit counts, the CTA's digit totals
// (read by the others), each digit's first place in the stage and its offset
// to the global order.
template <int ITEMS>
struct ClusterMem {
    uint2 pair[kClusterThreads * ITEMS], stage[kClusterThreads * ITEMS];
    uint16_t cnt[kClusterWarps][256];
    uint32_t total[256], lstart[256], gofs[256], wsum[2][8];
};

// In place: (keys, vals) sorted by the low passes * rb bits, vals_in null: the
// input positions; vals null: keys only.  cell_off (or null): also the cells'
// first sorted indices, cell_off[c] for c in [0, ncells].
template <int ITEMS>
__global__ void __cluster_dims__(kClusterCtas, 1, 1) __launch_bounds__(kClusterThreads, 1)
    k_sort_cluster(uint32_t *keys, uint32_t *vals, const uint32_t *vals_in, uint32_t n, int passes, int rb,
                   uint32_t *__restrict__ cell_off, uint32_t ncells, uint32_t *__restrict__ plan_ctl) {
    constexpr uint32_t E = kClusterThreads * ITEMS;  // keys of a CTA
    extern __shared__ __align__(16) unsigned char cluster_smem[];
    ClusterMem<ITEMS> &sm = *reinterpret_cast<ClusterMem<ITEMS> *>(cluster_smem);
    cg::cluster_group cluster = cg::this_cluster();
    const uint32_t rank = cluster.block_rank();
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, lt = (1u << lane) - 1u;
    const uint32_t radix = 1u << rb;
    if (plan_ctl && rank == 0 && tid < 3) plan_ctl[tid] = 0u;
    // item k of this thread: CTA position `first + 32 k`, input order over
    // (CTA, warp, item, lane)
    const uint32_t first = warp * (32 * ITEMS) + lane, g0 = rank * E + first;
    uint32_t key[ITEMS], val[ITEMS];
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        const uint32_t g = g0 + 32 * k;
        key[k] = g < n ? keys[g] : 0xffffffffu;
        val[k] = vals && vals_in && g < n ? vals_in[g] : g;
    }
    for (int p = 0; p < passes; ++p) {
        const int shift = p * rb;
        for (uint32_t d = lane; d < radix; d += 32) sm.cnt[warp][d] = 0;
        __syncwarp();
        uint32_t place[ITEMS];  // rank within the warp's keys of the digit
#pragma unroll
        for (int k = 0; k < ITEMS; ++k) {
            const bool valid = g0 + 32 * k < n;
            const uint32_t d = (key[k] >> shift) & (radix - 1);
            uint32_t peers = __ballot_sync(kFull, valid);
#pragma unroll
            for (int b = 0; b < 8; ++b)
                if (b < rb) {
                    const uint32_t bit = (d >> b) & 1u;
                    const uint32_t m = __ballot_sync(kFull, bit);
                    peers &= bit ? m : ~m;
                }
            if (!valid) peers = 1u << lane;
            const int lead = __ffs(peers) - 1;
            uint32_t c = 0;
            if (valid && lane == (uint32_t)lead) {
                c = sm.cnt[warp][d];
                sm.cnt[warp][d] = (uint16_t)(c + __popc(peers));
            }
            place[k] = __shfl_sync(kFull, c, lead) + __popc(peers & lt);
            __syncwarp();
        }
        __syncthreads();
        uint32_t mine = 0;  // thread d: this CTA's keys of digit d
        if (tid < radix) {
#pragma unroll
            for (int w0 = 0; w0 < kClusterWarps; w0 += 8) {
                uint32_t c[8];
#pragma unroll
                for (int w = 0; w < 8; ++w) c[w] = sm.cnt[w0 + w][tid];
#pragma unroll
                for (int w = 0; w < 8; ++w) {
                    sm.cnt[w0 + w][tid] = (uint16_t)mine;
                    mine += c[w];
                }
            }
            sm.total[tid] = mine;
        }
        cluster.sync();  // totals complete, and the last pass's pairs read
        uint32_t all = 0, before = 0, incl = 0, lincl = mine;
        if (tid < 256) {
            if (tid < radix) {
#pragma unroll
                for (uint32_t c = 0; c < (uint32_t)kClusterCtas; ++c) {
                    const uint32_t v = cluster.map_shared_rank(sm.total, c)[tid];
                    all += v;
                    if (c < rank) before += v;
                }
            }
            incl = all;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const uint32_t y = __shfl_up_sync(kFull, incl, off), ly = __shfl_up_sync(kFull, lincl, off);
                if (lane >= (uint32_t)off) incl += y, lincl += ly;
            }
            if (lane == 31) sm.wsum[0][warp] = incl, sm.wsum[1][warp] = lincl;
        }
        __syncthreads();
        if (tid < radix) {
#pragma unroll
            for (uint32_t w = 0; w < 8; ++w)
                if (w < warp) incl += sm.wsum[0][w], lincl += sm.wsum[1][w];
            sm.lstart[tid] = lincl - mine;
            sm.gofs[tid] = (incl - all + before) - (lincl - mine);
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < ITEMS; ++k) {
            if (g0 + 32 * k < n) {
                const uint32_t d = (key[k] >> shift) & (radix - 1);
                sm.stage[CUCO_IDX(sm.lstart[d] + sm.cnt[warp][d] + place[k], E)] = make_uint2(key[k], val[k]);
            }
        }
        __syncthreads();
        const uint32_t held = n > rank * E ? min(n - rank * E, E) : 0u;
#pragma unroll
        for (int k = 0; k < ITEMS; ++k) {
            const uint32_t j = k * kClusterThreads + tid;
            if (j < held) {
                const uint2 kv = sm.stage[j];
                const uint32_t o = CUCO_IDX(sm.gofs[(kv.x >> shift) & (radix - 1)] + j, n);
                cluster.map_shared_rank(sm.pair, o / E)[o & (E - 1)] = kv;
            }
        }
        cluster.sync();
#pragma unroll
        for (int k = 0; k < ITEMS; ++k) {
            const uint2 kv = sm.pair[first + 32 * k];
            key[k] = kv.x, val[k] = kv.y;
        }
    }
    chain_next();  // (the cell-order launch, which waits for the stores below)
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        const uint32_t g = g0 + 32 * k;
        if (g < n) {
            keys[g] = key[k];
            if (vals) vals[g] = val[k];
        }
    }
    if (cell_off) {
        // the key before a thread's item (the previous CTA's last for a CTA's
        // first), and the cells past the last key
#pragma unroll
        for (int k = 0; k < ITEMS; ++k) {
            const uint32_t e = first + 32 * k, g = g0 + 32 * k;
            uint32_t from = 0;
            if (g && g < n) from = 1u + (e ? sm.pair[e - 1].x : cluster.map_shared_rank(sm.pair, rank - 1)[E - 1].x);
            fill_offsets(cell_off, g < n, from, key[k], g);
            fill_offsets(cell_off, g == n - 1, key[k] + 1u, ncells, n);
        }
        cluster.sync();  // no CTA leaves while its keys may be read
    }
}

template <int ITEMS>
cuco_status_t launch_sort_cluster(uint32_t *keys, uint32_t *vals, const uint32_t *vals_in, uint32_t n, int passes,
                                  int rb, uint32_t *cell_off, uint32_t ncells, uint32_t *plan_ctl,
                                  cudaStream_t stream) {
    static OncePerDevice limit;
    CUCO_TRY_CUDA(limit.run([] { return raise_smem_limit(k_sort_cluster<ITEMS>, sizeof(ClusterMem<ITEMS>)); }));
    k_sort_cluster<ITEMS><<<kClusterCtas, kClusterThreads, sizeof(ClusterMem<ITEMS>), stream>>>(
        keys, vals, vals_in, n, passes, rb, cell_off, ncells, plan_ctl);
    CUCO_TRY_CUDA(cudaGetLastError());
    return CUCO_OK;
}

void split_bits(int key_bits, int max_radix_bits, int *passes, int *rb) {
    if (key_bits < 1) key_bits = 1;
    if (max_radix_bits > 8) max_radix_bits = 8;
    if (max_radix_bits < 4) max_radix_bits = 4;
    *passes = (key_bits + max_radix_bits - 1) / max_radix_bits;
    *rb = (key_bits + *passes - 1) / *passes;
    if (*rb < 4) *rb = 4;
}

__global__ void k_reorder_start_end(uint32_t *__restrict__ cell_start, uint32_t *__restrict__ cell_end,
                                    float4 *__restrict__ sorted_pos,
                                    const uint32_t *__restrict__ skeys,
                                    const uint32_t *__restrict__ perm,
                                    const float4 *__restrict__ pos, uint32_t n) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint32_t k = skeys[i];
    if (i == 0 || k != skeys[i - 1]) {
        cell_start[k] = i;
        if (i > 0) cell_end[skeys[i - 1]] = i;
    }
    if (i == n - 1) cell_end[k] = i + 1;
    sorted_pos[i] = pos[perm[i]];
}

__global__ void k_reorder_offsets(uint32_t *__restrict__ cell_off, const uint32_t *__restrict__ skeys, uint32_t n,
                                  uint32_t ncells, uint32_t *__restrict__ plan_ctl) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (plan_ctl && i < 3) plan_ctl[i] = 0u;
    // cells (prev, cur] start at i; thread n closes the tail up to ncells
    const uint32_t first = i == 0 || i > n ? 0u : skeys[i - 1] + 1u;
    const uint32_t cur = i >= n ? ncells : skeys[i];
    fill_offsets(cell_off, i <= n, first, cur, i);
}

// A stable counting sort of each cell's particles by z slice.  A lane's
// slice is spelled out by four ballots (three slice bits and "no particle"),
// so the lanes of each slice, their counts and each lane's rank among equal
// slices are popcounts of the ballots masked to the cell's lanes, and one
// lane per slice keeps the slice's running offset.  The order is fixed by the
// input order alone.  A warp takes four consecutive cells: eight lanes per
// cell, eight particles at a time, which keeps four cells' dependent loads
// (bounds, permutation, position) in flight where cells hold a few particles
// (one warp per cell left most lanes idle waiting on them); where one of the
// four holds more than 32, the warp sorts them one after the other with all
// 32 lanes, so a dense cell does not leave three groups of lanes idle.
constexpr uint32_t kSubLanes = 8;  // lanes per cell in the four-cell mode
static_assert(kZSub == (int)kSubLanes, "one lane per slice within a cell's lanes");

// The cell box of cell c: `one`, or the box of a many-box launch holding c.
__device__ __forceinline__ CellBox cell_box(uint32_t c, const CellBox &one, const CellBox *__restrict__ boxes,
                                            int nbox) {
    if (!boxes) return one;
    int lo = 0, hi = nbox;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(&boxes[mid].cell_base) <= c)
            lo = mid;
        else
            hi = mid;
    }
    return boxes[lo];
}

// slice of z within cell cz: plain, of the key rule's product G/L * z (in
// [cz, cz + 1) but for the clamped top face); fixed point, the three bits
// below the cell index of z * G / 2^32
__device__ __forceinline__ uint32_t z_slice(float4 p, const CellBox &d, uint32_t cz, int fixed) {
    if (fixed) return (uint32_t)(((uint64_t)__float_as_uint(p.z) * d.G) >> (32 - kZSubBits)) & (kZSub - 1);
    const float t = __fmul_rn(p.z, d.gridfac);
    const int s = __float2int_rd(__fmul_rn(__fsub_rn(t, (float)cz), (float)kZSub));
    return (uint32_t)min(max(s, 0), kZSub - 1);
}

// One cell [a, b) sorted by the lanes of gmask (W = 8 or 32 consecutive
// lanes; gl = lane within them); every lane of the warp calls it together.
// `valid`: whether this lane's group has a cell (c < ncells).
template <uint32_t W>
__device__ __forceinline__ void subsort_cell(bool valid, uint32_t c, uint32_t a, uint32_t b, const CellBox &d,
                                             uint32_t gmask, uint32_t gl, const uint32_t *__restrict__ perm,
                                             const float4 *__restrict__ pos, float4 *__restrict__ sorted_pos,
                                             uint32_t *__restrict__ perm_s, uint4 *__restrict__ slices,
                                             int fixed) {
    const uint32_t lane = threadIdx.x & 31, lt = (1u << lane) - 1u;
    const uint32_t n_cell = b - a;
    const uint32_t cz = valid ? (c - d.cell_base) % d.G : 0u;
    // lanes gl < kZSub write the cell's inclusive slice counts as u16
    uint16_t *sl = reinterpret_cast<uint16_t *>(slices + (valid ? c : 0u));
    auto put_counts = [&](uint32_t incl) {
        if (valid && gl < kZSub) sl[gl] = n_cell >= 0xffffu ? (uint16_t)0xffffu : (uint16_t)incl;
    };
    // the lanes of gmask holding slice k (k = kZSub: no particle)
    auto lanes_of = [&](uint32_t k, uint32_t b0, uint32_t b1, uint32_t b2, uint32_t none) {
        return ((k & 1) ? b0 : ~b0) & ((k & 2) ? b1 : ~b1) & ((k & 4) ? b2 : ~b2) & ~none & gmask;
    };
    // inclusive scan over the group's first kZSub lanes
    auto scan = [&](uint32_t v) {
#pragma unroll
        for (uint32_t off = 1; off < (uint32_t)kZSub; off <<= 1) {
            const uint32_t u = __shfl_up_sync(0xffffffffu, v, off, W);
            if (gl >= off) v += u;
        }
        return v;
    };
    const uint32_t chunks = (n_cell + W - 1) / W;
    const uint32_t chunks_max = __reduce_max_sync(0xffffffffu, chunks);
    const bool multi = chunks > 1;
    if (n_cell == 0) put_counts(0);
    const uint32_t gbase = lane - gl;  // the group's first lane
    uint32_t base = 0;                  // lane gl < kZSub: slice gl's next offset in the cell
    // Chunks are loaded kAhead at a time: a chunk's two dependent loads (the
    // permutation, then the position) are most of a dense cell's time.
    constexpr uint32_t kAhead = W == 32 ? 4 : 1;
    if (__any_sync(0xffffffffu, multi)) {
        // cells of more than one chunk count their slices first
        for (uint32_t j = 0; j < chunks_max; j += kAhead) {
            uint32_t o[kAhead], s[kAhead];
#pragma unroll
            for (uint32_t u = 0; u < kAhead; ++u) {
                const uint32_t i = a + (j + u) * W + gl;
                o[u] = multi && i < b ? perm[i] : 0xffffffffu;
            }
#pragma unroll
            for (uint32_t u = 0; u < kAhead; ++u)
                s[u] = o[u] != 0xffffffffu ? z_slice(pos[o[u]], d, cz, fixed) : (uint32_t)kZSub;
#pragma unroll
            for (uint32_t u = 0; u < kAhead; ++u) {
                const uint32_t b0 = __ballot_sync(0xffffffffu, s[u] & 1), b1 = __ballot_sync(0xffffffffu, s[u] & 2),
                               b2 = __ballot_sync(0xffffffffu, s[u] & 4), none = __ballot_sync(0xffffffffu, s[u] == kZSub);
                if (gl < kZSub) base += __popc(lanes_of(gl, b0, b1, b2, none));
            }
        }
        const uint32_t incl = scan(base);
        if (multi) put_counts(incl);
        base = incl - base;
    }
    for (uint32_t j = 0; j < chunks_max; j += kAhead) {
        uint32_t o[kAhead];
        float4 p[kAhead];
#pragma unroll
        for (uint32_t u = 0; u < kAhead; ++u) {
            const uint32_t i = a + (j + u) * W + gl;
            o[u] = i < b ? perm[i] : 0u;
        }
#pragma unroll
        for (uint32_t u = 0; u < kAhead; ++u)
            p[u] = a + (j + u) * W + gl < b ? pos[o[u]] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (uint32_t u = 0; u < kAhead; ++u) {
            const bool in = a + (j + u) * W + gl < b;
            const uint32_t s = in ? z_slice(p[u], d, cz, fixed) : (uint32_t)kZSub;
            const uint32_t b0 = __ballot_sync(0xffffffffu, s & 1), b1 = __ballot_sync(0xffffffffu, s & 2),
                           b2 = __ballot_sync(0xffffffffu, s & 4), none = __ballot_sync(0xffffffffu, s == kZSub);
            const uint32_t mine = lanes_of(s, b0, b1, b2, none);
            const uint32_t cnt = gl < kZSub ? __popc(lanes_of(gl, b0, b1, b2, none)) : 0u;
            if (j + u == 0) {
                // one chunk: the offsets are the exclusive scan of its counts
                const uint32_t incl = scan(cnt);
                if (!multi) {
                    if (n_cell) put_counts(incl);
                    base = incl - cnt;
                }
            }
            const uint32_t at = __shfl_sync(0xffffffffu, base, gbase + (s & (kZSub - 1))) + __popc(mine & lt);
            if (in) {
                sorted_pos[CUCO_IDX(a + at, b)] = make_float4(p[u].x, p[u].y, p[u].z, (float)s);
                perm_s[CUCO_IDX(a + at, b)] = o[u];
            }
            base += cnt;
        }
    }
}

__global__ void k_cell_subsort(const uint32_t *__restrict__ cell_off, const uint32_t *__restrict__ perm,
                               const float4 *__restrict__ pos, float4 *__restrict__ sorted_pos,
                               uint32_t *__restrict__ perm_s, uint4 *__restrict__ slices, uint32_t ncells,
                               const __grid_constant__ CellBox one, const CellBox *__restrict__ boxes, int nbox,
                               int fixed, uint32_t plan_blocks, const __grid_constant__ SRPlan plan,
                               const __grid_constant__ SRWork work) {
    chain_wait();
    // the first blocks write the short range's work plan (a launch less)
    if (blockIdx.x < plan_blocks) {
        plan_box_segment(plan, blockIdx.x * blockDim.x + threadIdx.x, cell_off, 0u, 0u, work);
        return;
    }
    constexpr uint32_t kCells = 32 / kSubLanes;
    const uint32_t lane = threadIdx.x & 31, grp = lane / kSubLanes;
    const uint32_t c0 = (((blockIdx.x - plan_blocks) * blockDim.x + threadIdx.x) >> 5) * kCells;
    if (c0 >= ncells) return;  // warp-uniform
    const uint32_t c = c0 + grp;
    const bool valid = c < ncells;
    const uint32_t a = valid ? cell_off[c] : 0u, b = valid ? cell_off[c + 1] : 0u;
    if (__any_sync(0xffffffffu, b - a > 32u)) {
        // the four cells one after the other, all 32 lanes on each
        for (uint32_t g = 0; g < kCells; ++g) {
            const uint32_t cg = c0 + g;
            if (cg >= ncells) break;  // warp-uniform
            const uint32_t ag = __shfl_sync(0xffffffffu, a, g * kSubLanes), bg = __shfl_sync(0xffffffffu, b, g * kSubLanes);
            subsort_cell<32>(true, cg, ag, bg, cell_box(cg, one, boxes, nbox), 0xffffffffu, lane, perm, pos,
                             sorted_pos, perm_s, slices, fixed);
        }
    } else {
        const CellBox d = valid ? cell_box(c, one, boxes, nbox) : one;
        subsort_cell<kSubLanes>(valid, c, a, b, d, 0xffu << (grp * kSubLanes), lane % kSubLanes, perm, pos,
                                sorted_pos, perm_s, slices, fixed);
    }
}

}  // namespace

cuco_status_t launch_cell_subsort(const uint32_t *cell_off, const uint32_t *perm, const float4 *pos,
                                  float4 *sorted_pos, uint32_t *perm_s, uint4 *slices, uint32_t ncells,
                                  const CellBox &one, const CellBox *boxes, int nbox, bool fixed,
                                  cudaStream_t stream, const SRPlan *plan, const SRWork *work) {
    if (ncells == 0) return CUCO_OK;
    const uint64_t threads = 32ull * ((ncells + 32 / kSubLanes - 1) / (32 / kSubLanes));
    const uint32_t plan_blocks = plan ? (plan->nseg + 255) / 256 : 0u;
    CUCO_TRY_CUDA(launch_chained(!boxes, k_cell_subsort, plan_blocks + (unsigned)((threads + 255) / 256), 256, 0, stream,
                                 cell_off, perm, pos, sorted_pos, perm_s, slices, ncells, one, boxes, nbox, fixed ? 1 : 0,
                                 plan_blocks, plan ? *plan : SRPlan{}, work ? *work : SRWork{}));
    return CUCO_OK;
}

size_t sort_hist_entries(uint32_t n, int key_bits, int max_radix_bits) {
    int passes, rb;
    split_bits(key_bits, max_radix_bits, &passes, &rb);
    const uint32_t tile = (uint32_t)kSortThreads * sort_items(n, rb, ~(size_t)0);
    const size_t tiles = (n + tile - 1) / tile;
    return (size_t)(1u << rb) * (tiles ? tiles : 1);
}

cuco_status_t sort_pairs(uint32_t *keys, uint32_t *vals, const uint32_t *vals_in,
                         uint32_t *keys_alt, uint32_t *vals_alt, uint32_t *hist, size_t hist_words, uint32_t n,
                         int key_bits, int max_radix_bits, cudaStream_t stream,
                         bool *result_in_alt, int *launches, uint32_t *cell_off, uint32_t ncells,
                         bool *offsets_done, uint32_t *plan_ctl) {
    int passes, rb;
    split_bits(key_bits, max_radix_bits, &passes, &rb);
    bool with_vals = vals != nullptr;
    *result_in_alt = false;
    if (offsets_done) *offsets_done = false;
    if (n == 0) return CUCO_OK;
    if (n <= kClusterMax) {
        uint32_t *off = offsets_done ? cell_off : nullptr;
        if (offsets_done) *offsets_done = true;
        *launches += 1;
        const uint32_t ctas = kClusterCtas * kClusterThreads;
        auto launch = n <= ctas ? launch_sort_cluster<1>
                                : (n <= 2 * ctas ? launch_sort_cluster<2>
                                                 : (n <= 4 * ctas ? launch_sort_cluster<4> : launch_sort_cluster<8>));
        return launch(keys, vals, vals_in, n, passes, rb, off, ncells, plan_ctl, stream);
    }
    uint32_t *kbuf[2] = {keys, keys_alt};
    uint32_t *vbuf[2] = {vals, vals_alt};
    const int items = sort_items(n, rb, hist_words);
    int cur = 0;
    for (int p = 0; p < passes; ++p) {
        const uint32_t *vin = (p == 0) ? vals_in : vbuf[cur];
        const int shift = p * rb;
        cuco_status_t s;
        switch (rb) {
#define CUCO_SORT_PASS(R)                                                                                         \
    s = sort_pass<R>(items, kbuf[cur], vin, kbuf[cur ^ 1], vbuf[cur ^ 1], with_vals, hist, n, shift, stream, \
                     launches)
            case 4: CUCO_SORT_PASS(4); break;
            case 5: CUCO_SORT_PASS(5); break;
            case 6: CUCO_SORT_PASS(6); break;
            case 7: CUCO_SORT_PASS(7); break;
            default: CUCO_SORT_PASS(8); break;
#undef CUCO_SORT_PASS
        }
        if (s != CUCO_OK) return s;
        cur ^= 1;
    }
    *result_in_alt = cur == 1;
    return CUCO_OK;
}

cuco_status_t launch_cell_keys(const float4 *pos, uint32_t *keys, uint32_t *idx, uint32_t n,
                               float gridfac, int G, cudaStream_t stream) {
    if (n == 0) return CUCO_OK;
    int blocks = (int)((n + 255) / 256);
    k_cell_keys<<<blocks, 256, 0, stream>>>(pos, keys, idx, n, gridfac, G);
    CUCO_TRY_CUDA(cudaGetLastError());
    return CUCO_OK;
}

cuco_status_t launch_reorder_start_end(uint32_t *cell_start, uint32_t *cell_end,
                                       float4 *sorted_pos, const uint32_t *sorted_keys,
                                       const uint32_t *perm, const float4 *pos, uint32_t n,
                                       uint32_t ncells, cudaStream_t stream) {
    CUCO_TRY_CUDA(cudaMemsetAsync(cell_start, 0xff, sizeof(uint32_t) * ncells, stream));
    if (n == 0) return CUCO_OK;
    k_reorder_start_end<<<(n + 255) / 256, 256, 0, stream>>>(cell_start, cell_end, sorted_pos,
                                                           sorted_keys, perm, pos, n);
    CUCO_TRY_CUDA(cudaGetLastError());
    return CUCO_OK;
}

cuco_status_t launch_reorder_offsets(uint32_t *cell_off, const uint32_t *sorted_keys, uint32_t n, uint32_t ncells,
                                     cudaStream_t stream, uint32_t *plan_ctl) {
    k_reorder_offsets<<<(unsigned)(((size_t)n + 1 + 255) / 256), 256, 0, stream>>>(cell_off, sorted_keys, n, ncells,
                                                                                   plan_ctl);
    CUCO_TRY_CUDA(cudaGetLastError());
    return CUCO_OK;
}

// ---- start/end -> offsets: where the cells' ranges follow one another without
// gaps (as reorderDataAndFindCellStart leaves them), off[c] is the largest end
// of the cells before c, a running maximum; a range that does not start there is
// reported.  Where they do not, off[c] is the particles that the cells before c
// hold, a running sum, for a copy of the particles in that order.  Either takes
// two launches: each block's value, then every block its cells after the values
// of the blocks before it.  Up to kDirectBlocks blocks, each reads those values
// itself; beyond, which would be quadratic in the cells, the last block of the
// first launch to finish turns them into running values (at few blocks that
// costs 5 us of latency).  Bound by memory: both bounds read twice.  A force on
// 1000 particles in 512^3, 768^3 and 1024^3 cells: 1.81, 21.0 and 116 ms with
// every block reading all values before it, 0.54, 1.66 and 3.86 so; on 32^3
// particles in 64^3 and 256^3 cells 0.108 and 0.206 ms, 0.108 and 0.195.
namespace {
constexpr unsigned kDirectBlocks = 4096;
// 4 cells a thread; 16 from kOffWideCells cells
constexpr uint32_t kOffWideCells = 1u << 20;

struct RunningEnd {
    static __device__ __forceinline__ uint32_t of(uint32_t s, uint32_t e) { return e > s ? e : 0u; }
    static __device__ __forceinline__ uint32_t join(uint32_t a, uint32_t b) { return max(a, b); }
    static __device__ __forceinline__ uint32_t warp(uint32_t v) { return __reduce_max_sync(kFull, v); }
};
struct RunningCount {
    static __device__ __forceinline__ uint32_t of(uint32_t s, uint32_t e) { return e > s ? e - s : 0u; }
    static __device__ __forceinline__ uint32_t join(uint32_t a, uint32_t b) { return a + b; }
    static __device__ __forceinline__ uint32_t warp(uint32_t v) { return __reduce_add_sync(kFull, v); }
};

// The caller's bounds; wide: both on 16 bytes.
struct CellBounds {
    const uint32_t *start, *end;
    uint32_t ncells;
    bool wide;
};

// Cells c .. c + 3 of an array, `past` beyond the last.
__device__ __forceinline__ uint4 load_four(const uint32_t *__restrict__ p, uint32_t c, const CellBounds &b, uint32_t past) {
    if (b.wide && c + 3 < b.ncells) return *reinterpret_cast<const uint4 *>(p + c);
    return make_uint4(c < b.ncells ? p[c] : past, c + 1 < b.ncells ? p[c + 1] : past, c + 2 < b.ncells ? p[c + 2] : past,
                      c + 3 < b.ncells ? p[c + 3] : past);
}

// A warp takes ROUNDS times 128 consecutive cells, a lane four neighbours of
// each: their starts and values, 0 for a cell that is empty (kEmptyCell for a
// start, or an end not above it).
template <uint32_t ROUNDS>
__device__ __forceinline__ uint32_t first_cell() {
    return (blockIdx.x * kSortWarps + (threadIdx.x >> 5)) * (128 * ROUNDS) + (threadIdx.x & 31) * 4;
}
template <typename Op, uint32_t ROUNDS>
__device__ __forceinline__ void load_cells(const CellBounds &b, uint4 (&s)[ROUNDS], uint4 (&v)[ROUNDS]) {
    const uint32_t c0 = first_cell<ROUNDS>();
#pragma unroll
    for (uint32_t k = 0; k < ROUNDS; ++k) {
        s[k] = load_four(b.start, c0 + 128 * k, b, kEmptyCell);
        v[k] = load_four(b.end, c0 + 128 * k, b, 0u);
    }
    auto value = [](uint32_t st, uint32_t e) { return st != kEmptyCell ? Op::of(st, e) : 0u; };
#pragma unroll
    for (uint32_t k = 0; k < ROUNDS; ++k)
        v[k] = make_uint4(value(s[k].x, v[k].x), value(s[k].y, v[k].y), value(s[k].z, v[k].z), value(s[k].w, v[k].w));
}
template <typename Op>
__device__ __forceinline__ uint32_t joined(const uint4 &v) {
    return Op::join(Op::join(v.x, v.y), Op::join(v.z, v.w));
}
template <typename Op, uint32_t ROUNDS>
__device__ __forceinline__ uint32_t warp_joined(const uint4 (&v)[ROUNDS]) {
    uint32_t m = 0;
#pragma unroll
    for (uint32_t k = 0; k < ROUNDS; ++k) m = Op::join(m, joined<Op>(v[k]));
    return Op::warp(m);
}

// The joined v of the block's warps before this one (0 for the first), v being
// the warp's own; *all: of the whole block.  Every thread calls it together.
template <typename Op>
__device__ __forceinline__ uint32_t warps_before(uint32_t v, uint32_t *all) {
    __shared__ uint32_t s_warp[kSortWarps];
    const uint32_t warp = threadIdx.x >> 5;
    uint32_t before = 0;
    __syncthreads();  // s_warp of a call before is read
    if ((threadIdx.x & 31) == 0) s_warp[warp] = v;
    __syncthreads();
    *all = 0;
#pragma unroll
    for (uint32_t w = 0; w < (uint32_t)kSortWarps; ++w) {
        const uint32_t x = s_warp[w];
        before = Op::join(before, w < warp ? x : 0u);
        *all = Op::join(*all, x);
    }
    return before;
}

// The joined v of the lanes before this one (0 for the first); *all: of the warp.
template <typename Op>
__device__ __forceinline__ uint32_t lanes_before(uint32_t v, uint32_t *all) {
    const uint32_t lane = threadIdx.x & 31;
#pragma unroll
    for (uint32_t off = 1; off < 32; off <<= 1) {
        const uint32_t u = __shfl_up_sync(kFull, v, off);
        if (lane >= off) v = Op::join(v, u);
    }
    *all = __shfl_sync(kFull, v, 31);
    const uint32_t before = __shfl_up_sync(kFull, v, 1);
    return lane ? before : 0u;
}

// values[b] = block b's value; with `finished`, which counts the blocks that
// have written theirs and is 0 between launches, the value before block b.
template <typename Op, uint32_t ROUNDS>
__global__ void __launch_bounds__(kSortThreads)
    k_block_values(const __grid_constant__ CellBounds bounds, uint32_t *values, uint32_t *finished) {
    __shared__ bool s_last;
    uint4 s[ROUNDS], v[ROUNDS];
    uint32_t all;
    load_cells<Op>(bounds, s, v);
    warps_before<Op>(warp_joined<Op>(v), &all);
    if (threadIdx.x == 0) {
        __stcg(&values[blockIdx.x], all);
        if (finished) {
            __threadfence();
            s_last = atomicAdd(finished, 1u) == gridDim.x - 1;
        }
    }
    if (!finished) return;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    // the last block: the value before each block, 8 rounds' loads in flight
    constexpr uint32_t kAhead = 8;
    uint32_t carry = 0;
    for (uint32_t b0 = 0; b0 < gridDim.x; b0 += kAhead * kSortThreads) {
        uint32_t x[kAhead];
#pragma unroll
        for (uint32_t k = 0; k < kAhead; ++k) {
            const uint32_t b = b0 + k * kSortThreads + threadIdx.x;
            x[k] = b < gridDim.x ? __ldcg(&values[b]) : 0u;
        }
#pragma unroll
        for (uint32_t k = 0; k < kAhead; ++k) {
            const uint32_t b = b0 + k * kSortThreads + threadIdx.x;
            uint32_t warp_all, round_all;
            const uint32_t lanes = lanes_before<Op>(x[k], &warp_all);
            const uint32_t at = Op::join(Op::join(carry, warps_before<Op>(warp_all, &round_all)), lanes);
            if (b < gridDim.x) __stcg(&values[b], at);
            carry = Op::join(carry, round_all);
        }
    }
    if (threadIdx.x == 0) *finished = 0;
}

// running: values[b] is the value before block b, else block b's own.  gap (or
// null): gap_bit is set where a cell's range does not start at its offset.
// cell_off lies on 16 bytes.
template <typename Op, uint32_t ROUNDS>
__global__ void __launch_bounds__(kSortThreads)
    k_cell_offsets(const __grid_constant__ CellBounds bounds, const uint32_t *__restrict__ values, bool running,
                   uint32_t *__restrict__ cell_off, uint32_t *gap, uint32_t gap_bit) {
    uint4 s[ROUNDS], v[ROUNDS];
    uint32_t all, carry = 0;
    load_cells<Op>(bounds, s, v);
    if (running) {
        carry = values[blockIdx.x];
    } else {
#pragma unroll 4
        for (uint32_t b = threadIdx.x; b < blockIdx.x; b += kSortThreads) carry = Op::join(carry, values[b]);
        warps_before<Op>(Op::warp(carry), &all);
        carry = all;
    }
    carry = Op::join(carry, warps_before<Op>(warp_joined<Op>(v), &all));
    const uint32_t c0 = first_cell<ROUNDS>();
    bool apart = false;
#pragma unroll
    for (uint32_t k = 0; k < ROUNDS; ++k) {
        const uint32_t c = c0 + 128 * k;
        uint4 o;
        o.x = Op::join(carry, lanes_before<Op>(joined<Op>(v[k]), &all));
        o.y = Op::join(o.x, v[k].x);
        o.z = Op::join(o.y, v[k].y);
        o.w = Op::join(o.z, v[k].z);
        if (c + 3 < bounds.ncells) {
            *reinterpret_cast<uint4 *>(cell_off + c) = o;
        } else {
            if (c < bounds.ncells) cell_off[c] = o.x;
            if (c + 1 < bounds.ncells) cell_off[c + 1] = o.y;
            if (c + 2 < bounds.ncells) cell_off[c + 2] = o.z;
        }
        apart |= (v[k].x && s[k].x != o.x) || (v[k].y && s[k].y != o.y) || (v[k].z && s[k].z != o.z) ||
                 (v[k].w && s[k].w != o.w);
        // (cells past the last have no value: theirs is the offset of the end)
        if (c <= bounds.ncells - 1 && bounds.ncells - 1 <= c + 3) cell_off[bounds.ncells] = Op::join(o.w, v[k].w);
        carry = Op::join(carry, all);
    }
    if (gap && __any_sync(kFull, apart) && (threadIdx.x & 31) == 0) atomicOr(gap, gap_bit);
}

template <typename Op, uint32_t ROUNDS>
cuco_status_t cell_offsets(const CellBounds &bounds, uint32_t *cell_off, uint32_t *scratch, uint32_t *finished,
                           uint32_t *gap, uint32_t gap_bit, cudaStream_t stream) {
    constexpr uint32_t kCells = kSortThreads * 4 * ROUNDS;
    const unsigned blocks = bounds.ncells / kCells + (bounds.ncells % kCells != 0);
    const bool running = blocks > kDirectBlocks;
    k_block_values<Op, ROUNDS><<<blocks, kSortThreads, 0, stream>>>(bounds, scratch, running ? finished : nullptr);
    k_cell_offsets<Op, ROUNDS><<<blocks, kSortThreads, 0, stream>>>(bounds, scratch, running, cell_off, gap, gap_bit);
    CUCO_TRY_CUDA(cudaGetLastError());
    return CUCO_OK;
}

CellBounds cell_bounds(const uint32_t *start, const uint32_t *end, uint32_t ncells) {
    return {start, end, ncells, ((uintptr_t)start | (uintptr_t)end) % sizeof(uint4) == 0};
}

// The particles of the cells' ranges, in cell order, to where cell_off says: a
// warp takes 32 cells, and copies one cell after the other.
__global__ void k_gather_cells(const uint32_t *__restrict__ start, const uint32_t *__restrict__ end,
                               const uint32_t *__restrict__ cell_off, uint32_t ncells, const float4 *__restrict__ pos,
                               const uint32_t *__restrict__ perm, float4 *__restrict__ pos_out,
                               uint32_t *__restrict__ perm_out) {
    const uint32_t lane = threadIdx.x & 31, c = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t s = c < ncells ? start[c] : kEmptyCell, e = s != kEmptyCell ? end[c] : 0u;
    const uint32_t to = c < ncells ? cell_off[c] : 0u;
    for (uint32_t rest = __ballot_sync(kFull, s != kEmptyCell && e > s); rest; rest &= rest - 1) {
        const int src = __ffs(rest) - 1;
        const uint32_t from = __shfl_sync(kFull, s, src), count = __shfl_sync(kFull, e, src) - from,
                       at = __shfl_sync(kFull, to, src);
        for (uint32_t k = lane; k < count; k += 32) {
            pos_out[at + k] = pos[from + k];
            perm_out[at + k] = perm[from + k];
        }
    }
}
}  // namespace

size_t offsets_scratch(uint32_t ncells) { return (size_t)ncells / (kSortThreads * 4) + 1; }

cuco_status_t launch_start_end_offsets(const uint32_t *cell_start, const uint32_t *cell_end, uint32_t *cell_off,
                                       uint32_t ncells, uint32_t *scratch, uint32_t *finished, uint32_t *gap,
                                       uint32_t gap_bit, cudaStream_t stream) {
    if (!ncells) return CUCO_OK;
    auto launch = ncells < kOffWideCells ? cell_offsets<RunningEnd, 1> : cell_offsets<RunningEnd, 4>;
    return launch(cell_bounds(cell_start, cell_end, ncells), cell_off, scratch, finished, gap, gap_bit, stream);
}

cuco_status_t launch_start_end_counts(const uint32_t *cell_start, const uint32_t *cell_end, uint32_t *cell_off,
                                      uint32_t ncells, uint32_t *scratch, uint32_t *finished, cudaStream_t stream) {
    if (!ncells) return CUCO_OK;
    auto launch = ncells < kOffWideCells ? cell_offsets<RunningCount, 1> : cell_offsets<RunningCount, 4>;
    return launch(cell_bounds(cell_start, cell_end, ncells), cell_off, scratch, finished, nullptr, 0u, stream);
}

cuco_status_t launch_gather_cells(const uint32_t *cell_start, const uint32_t *cell_end, const uint32_t *cell_off,
                                  uint32_t ncells, const float4 *pos, const uint32_t *perm, float4 *pos_out,
                                  uint32_t *perm_out, cudaStream_t stream) {
    if (!ncells) return CUCO_OK;
    k_gather_cells<<<ncells / 256 + (ncells % 256 != 0), 256, 0, stream>>>(cell_start, cell_end, cell_off, ncells, pos,
                                                                         perm, pos_out, perm_out);
    CUCO_TRY_CUDA(cudaGetLastError());
    return CUCO_OK;
}

uint32_t bounds_violations_sort() { return bounds_violations_take(); }

}  // namespace cuco
