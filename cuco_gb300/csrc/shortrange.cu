// Short-range P3M pair force on the cell grid.
//
// Reference: cudaForceEvaluateShortrangeD + calcForce (gravlist_kernel.cu:20-88,
// 162-234) and the CPU force_evaluate_shortrange (gravlist.cpp:216-338).  The
// pair law is the reference's: minimum-image separation, cut at r^2 > rcut^2,
// 1/r^2 outside the spline softening length h and GADGET's spline inside,
// times the nearest-bin erfc split factor T[(int)(asmthfac*r)] (NTAB = 1000).
//
// Work layout (GB300-first rather than one thread per particle over a full
// cube of cells):
//   * a segment is S consecutive cells along z (ix, iy, iz0..iz0+S-1); its
//     targets are one contiguous range of the cell order.  A unit of work is a
//     slice of a segment's targets; a plan kernel lists the units, the short
//     slices of dense segments first, and the warps of a persistent grid pull
//     them from a counter, each on its own (no CTA barrier anywhere);
//   * a warp takes its unit's targets in groups of at most 16 (a dense unit:
//     one group of up to 32).  The sources a group needs lie in the neighbour
//     columns (dx, dy) within rcut of it in xy: lane k culls column k against
//     the group's bounding box and narrows it to the z range
//     sqrt(rcut^2 - d_xy^2) reaches, trimmed in the two end cells to the z
//     slices it reaches (the cells' particles are ordered by slice, with
//     per-cell slice counts).  A column's cells are consecutive keys, so that
//     is one contiguous run of the cell order (two when the z range wraps);
//   * the runs, concatenated by a warp scan, are walked 32 sources at a time;
//     each lane loads one, moves it relative to an integer origin at the
//     segment corner (with the run's periodic image shift) and tests it
//     against the group's bounding box; the sources within rcut of the box are
//     appended to the warp's list in shared memory;
//   * a full list is evaluated with a target per lane: 16 targets x 2 list
//     slots (fewer targets: more slots), each lane on four consecutive sources
//     of the list per iteration, two at a time in packed FP32 (float2
//     add/mul/fma, one instruction for two sources);
//   * the pair law runs without branches on the common path and flags the
//     rest (bin-edge and cut-edge pairs decided in double, the spline), which
//     is done per lane after every eight iterations;
//   * partial sums are folded every eight iterations (the precision form:
//     compensated), the slots' sums added by xor shuffles, and the warp's
//     lanes scatter the unit's forces to original particle order and, in the
//     engine's step, kick the velocities (timestep.c:56-59,86-91).
//
// What bounds it: instruction issue (about 300 warp instructions per target at
// z = 49, a third of them the pair law), then the latency of the window loads
// at 32 warps an SM.  The layout before it staged a segment's whole
// neighbourhood per CTA and put a source on each lane for two targets at a
// time: 274 candidates a target of which 84 are in range, and 578
// instructions, the list mapping and the cull paid per two targets and the CTA
// barriers and 45 KB of staging per unit.  The box test leaves 172 candidates
// for eight targets, 242 for sixteen, and a lane that keeps its target needs
// no reduction per pair.  128^3, L = 256, G = 64, one launch: 1.24 -> 0.69 ms
// at z = 49, 2.73 -> 1.59 ms in a clustered box (362 pairs a target); the
// reference's device calls on 64^3 cells with 32^3 particles 0.91 -> 0.20 ms.  Groups of 8
// instead of 16: 0.80 ms early, 1.76 ms clustered.  Loading the next window
// pair while this one is tested costs more registers than it hides (0.82 ms).
//
// Precision of the plain path.  A float computation of asmthfac*r lands in the
// neighbouring table bin for ~3e-5 of the pairs, and at high redshift (net
// force a small residual of cancelling pair terms) that alone costs ~1.6e-4
// rms against the reference's double path.  Coordinates relative to an integer
// origin make the image shift exact (origin -/+ L is an exact float for
// L < 2^23) and dx exact for ~97% of pairs; pairs whose r^2 lies within
// 8e-7 (relative) of rcut^2 or whose asmthfac*r lies within 4e-7 (relative)
// of a bin edge are decided in double as gravlist.cpp:298-320 does.
#include <algorithm>
#include <cmath>
#include <cstring>

#include "common.cuh"
#include "shortrange_plan.cuh"

namespace cuco {

namespace {


constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kMaxR = 8;         // neighbour reach in cells (the reference's G = PMGRID needs 6)
constexpr int kMaxCols = (2 * kMaxR + 1) * (2 * kMaxR + 1);
constexpr int kMaxSeg = 8;
// targets of a group (a warp's lanes are kGroup targets x 32 / kGroup list
// slots, or fewer targets and more slots)
constexpr int kGroup = 16;
// A warp's list is evaluated when it holds kListFull sources; one more window
// pair (64) may be appended before that is seen, and the last evaluation pads
// it to whole iterations.
constexpr uint32_t kListFull = 192, kListCap = 256;
static_assert(kUnitMax <= 32 && kUnitMax <= 2 * kGroup, "a unit is at most two groups");
static_assert(kListFull + 64 <= kListCap && kListCap % 128 == 0 && kListFull >= 128, "list sizes");
// list iterations between two folds of the partial sums (four flag bits each)
constexpr uint32_t kFold = 8;
// the split table in shared memory, padded to a power of two
constexpr int kTabPad = 1024;
static_assert(kTabPad >= kNTab && (kTabPad & (kTabPad - 1)) == 0, "table padding");
constexpr unsigned kFull = 0xffffffffu;
// CTAs per SM the register allocation is sized for (65536 / (256 * 4) = 64
// registers a thread at 4)
#ifndef CUCO_SR_MIN_BLOCKS
#define CUCO_SR_MIN_BLOCKS 4
#endif
constexpr int kMinBlocks = CUCO_SR_MIN_BLOCKS;

struct ColumnSet {
    int ncols;
    int R;
    int S;
    float margin;  // culling slack for the float cell assignment (length units)
    signed char dx[kMaxCols];
    signed char dy[kMaxCols];
};

// One box of a multi-box launch.
struct SRBoxDesc {
    ShortRangeParams p;
    ColumnSet cs;
    uint32_t slice;  // unit_slice of the box's own particles
};

// One warp's shared memory: the source list (origin-relative), the runs of
// the columns being walked (list position -> sorted index, and the periodic
// shift's subtrahend), the unit's forces.
struct WarpMem {
    float x[kListCap], y[kListCap], z[kListCap];
    uint32_t delta[32];
    float4 shift[32];
    float4 box[2];  // the group's bounding box
    float tx[kUnitMax], ty[kUnitMax], tz[kUnitMax];  // the lanes' targets
    float acc[3][kUnitMax];
};

// A list entry this far away is beyond any cut.
constexpr float kSentinel = 1e15f;

// s + e = a + b exactly (Knuth's two-sum; the intrinsics keep the compiler
// from contracting or reordering it).
__device__ __forceinline__ void two_sum(float a, float b, float &s, float &e) {
    s = __fadd_rn(a, b);
    const float bb = __fsub_rn(s, a);
    e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
}

// 1 << k for k < 32, else 0: PTX clamps a shift count above the width, so
// this is one shift with no compare and select.
__device__ __forceinline__ uint32_t bit_at(uint32_t k) {
    uint32_t b;
    asm("shl.b32 %0, %1, %2;" : "=r"(b) : "r"(1u), "r"(k));
    return b;
}

// The hardware reciprocal square root, flushing subnormal inputs (the fast
// path only sees r^2 well above them; without the flush the compiler wraps
// the instruction in a subnormal rescale).
__device__ __forceinline__ float rsqrt_ftz(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// r^2 with a fixed operation order: the candidate test and the force pass
// must agree on it bit for bit.
__device__ __forceinline__ float dist2(float dx, float dy, float dz) {
    return __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmul_rn(dx, dx)));
}

// max(a, b, 0), one instruction
__device__ __forceinline__ float max0(float a, float b) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(0.f));
    return r;
}

// the warp's smallest and largest value, in every lane
__device__ __forceinline__ float warp_min(float v) {
    float r;
    asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ float warp_max(float v) {
    float r;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}

// ---- The timeout word's self-test: one CTA waits, bounded, on a barrier that
// never completes.
__shared__ __align__(8) uint64_t g_probe_bar;

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void bar_init(uint64_t *bar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(bar)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// one arrival that also expects `bytes` of copies in this phase
__device__ __forceinline__ void bar_arrive_expect(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ bool bar_try_wait(uint64_t *bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}"
        : "=r"(done)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return done != 0;
}

// Wait for the phase with parity `parity` to complete, at most `limit`
// clock cycles.
__device__ __forceinline__ bool bar_wait_bounded(uint64_t *bar, uint32_t parity, long long limit) {
    const long long t0 = clock64();
    for (;;) {
        if (bar_try_wait(bar, parity)) return true;
        if (clock64() - t0 > limit) return false;
    }
}

// The timeout word's path on its own: one CTA arms the barrier for 16 bytes of
// copies that are never issued, waits at most `limit` cycles, and reports
// through the short range's timeout word.  No copy is in flight when it gives
// up.  (The short range itself waits on nothing.)
__global__ void k_timeout_probe(uint32_t *__restrict__ err, long long limit) {
    if (threadIdx.x == 0) bar_init(&g_probe_bar);
    __syncthreads();
    if (threadIdx.x == 0) bar_arrive_expect(&g_probe_bar, 16u);
    __syncthreads();
    const bool ok = bar_wait_bounded(&g_probe_bar, 0u, limit);
    if (__syncthreads_or(!ok) && threadIdx.x == 0) atomicOr(err, 1u);
}

// One unit (its record: plan_segment) of one box (p; ncols, R, S, margin of its
// column set, dxdy(col) its columns' offsets); dense: its targets are one
// group.  kick_pp/kick_pm are that
// box's kick factors.  Every lane of the warp calls it together; wm is the
// warp's shared memory, tab the split table.
// `law`: the pair law's constants (rc2_lo, rc2_hi, hmin2, alo, ahi, rcut2_d,
// asmthfac_d, h, hinv, h3inv): the box's own (p), or the launch's when every
// box of a many-box launch has the same (read from the kernel's parameters).
// PIN_LAW: the law lives in global memory (a many-box launch's descriptor):
// its three range bounds are held in registers, where the compiler would
// otherwise reload them in every iteration.
template <bool KICK, bool COUNT, bool FIXED, bool PIN_LAW, typename Columns>
__device__ __forceinline__ void shortrange_unit(
    const ShortRangeParams &p, const ShortRangeParams &law, const int ncols, const int R, const int S,
    const float margin, Columns dxdy, const uint4 unit, const bool dense,
    const double kick_pp, const double kick_pm, const float4 *__restrict__ spos, const uint32_t *__restrict__ perm,
    const uint32_t *__restrict__ cell_off, float4 *__restrict__ acc_out, const KickArgs &kick, WarpMem &wm,
    const float *tab, uint32_t &npairs) {
    const int lane = threadIdx.x & 31;
    const uint32_t lt_mask = (1u << lane) - 1u, le_mask = lt_mask | (1u << lane);
    const int G = p.grid, nz = S + 2 * R;
    const int ix = unit.z & 0xffff, iy = unit.z >> 16, iz0 = unit.w;
    const uint32_t t_begin = unit.x, len = unit.y & 255u;
    const float L = p.boxsize, w = p.cellw, winv = 1.0f / w, fs = p.fscale;
    const bool ZS = p.slices != nullptr;  // sources in z-slice order within cells, with slice counts

    // integer origin at the segment corner (see the file comment), and the
    // corner's offset from it
    const float ox = floorf(ix * w), oy = floorf(iy * w), oz = floorf(iz0 * w);
    const float fx = FIXED ? 0.f : ix * w - ox, fy = FIXED ? 0.f : iy * w - oy, fz = FIXED ? 0.f : iz0 * w - oz;
    // Fixed-point positions: the origin is the segment corner on the 2^32
    // grid, and an int32 difference from it is the periodic image for free
    // (every source lies within S + R < G/2 cells of it).
    // floor(i 2^32 / G) = i q + floor(i r / G), 2^32 = q G + r (i r < 2^20: the
    // float quotient of the odd numerator is never a whole number off)
    auto corner = [&](int i) { return (uint32_t)i * p.grid_q + (uint32_t)(((float)(i * (int)p.grid_r) + 0.5f) * p.grid_inv); };
    const uint32_t oxu = FIXED ? corner(ix) : 0u, oyu = FIXED ? corner(iy) : 0u, ozu = FIXED ? corner(iz0) : 0u;
    // __fmul_rn: a target's coordinates must equal its own list entry bit
    // for bit (the self pair then has r = 0 exactly), so the product may not
    // be contracted into the later subtraction
    auto rel = [&](float4 a) {
        return make_float4(__fmul_rn((float)(int32_t)(__float_as_uint(a.x) - oxu), fs),
                           __fmul_rn((float)(int32_t)(__float_as_uint(a.y) - oyu), fs),
                           __fmul_rn((float)(int32_t)(__float_as_uint(a.z) - ozu), fs), 0.f);
    };
    // the z range of the segment's stencil wraps below 0 or past G - 1 (never
    // both: S + 2R <= G), or an xy column does
    const bool z_below = iz0 < R, z_above = iz0 + S + R > G;
    const bool wrap = z_below || z_above || ix < R || ix + R >= G || iy < R || iy + R >= G;
    const int parts = z_below || z_above ? 2 : 1;
    const int batches = parts * ((ncols + 31) >> 5);

    const float rc2m = (p.rcut + margin) * (p.rcut + margin);
    float rc2_lo = law.rc2_lo, hmin2 = law.hmin2, r_hi = law.r_hi;
    if (PIN_LAW) asm volatile("" : "+f"(rc2_lo), "+f"(hmin2), "+f"(r_hi));
    const float2 alo2 = make_float2(law.alo, law.alo), ahi2 = make_float2(law.ahi, law.ahi);
    const float2 magic2 = make_float2(8388608.0f, 8388608.0f);

    // The pair law, in two parts.  pair_fast2 takes the common case - inside
    // the cut, away from a table-bin edge and from the cut, outside the
    // softening length - without a branch, for two sources at once in packed
    // FP32, and reports the rest (its contribution there is zero): a
    // candidate whose bin or cut decision is made in double and the spline
    // inside h (the self pair, r = 0, adds nothing and is skipped).
    // pair_slow applies the full law to those.
    // bin = floor(asmthfac * r): a round-toward-zero fma onto 2^23 leaves the
    // floor in the mantissa, with no conversion instruction.  Plain: the bins
    // of r * asmthfac * (1 -/+ kEdge) differ when r lies within kEdge
    // (relative) of a bin edge, and such a pair is decided in double.  The
    // table is padded to kTabPad entries with its last value, so a bin index
    // masked to the padding is the clamped one (fast pairs have bins below
    // kNTab; others read a padding value they do not use).
    auto pair_fast2 = [&](float2 sx, float2 sy, float2 sz, float2 ntx, float2 nty, float2 ntz, float2 &ax, float2 &ay,
                          float2 &az, bool &slow_a, bool &slow_b) {
        const float2 dx = __fadd2_rn(sx, ntx), dy = __fadd2_rn(sy, nty), dz = __fadd2_rn(sz, ntz);
        // dist2's order: dz^2 + (dy^2 + dx^2)
        const float2 r2 = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __fmul2_rn(dx, dx)));
        // r2 = 0 gives rinv = inf and r = NaN: not fast (r2 < hmin2), not flagged
        const float2 rinv = make_float2(rsqrt_ftz(r2.x), rsqrt_ftz(r2.y));
        const float2 r = __fmul2_rn(r2, rinv);
        const float2 xl = __ffma2_rz(r, alo2, magic2);
        bool edge_a = false, edge_b = false;
        if (!FIXED) {
            const float2 xh = __ffma2_rz(r, ahi2, magic2);
            edge_a = xl.x != xh.x;
            edge_b = xl.y != xh.y;
        }
        // the bin is the mantissa's low bits (2^23's own are zero)
        const float2 t = make_float2(tab[__float_as_uint(xl.x) & (kTabPad - 1)],
                                     tab[__float_as_uint(xl.y) & (kTabPad - 1)]);
        const bool fast_a = r2.x <= rc2_lo && r2.x >= hmin2 && !edge_a;
        const bool fast_b = r2.y <= rc2_lo && r2.y >= hmin2 && !edge_b;
        const float2 f = __fmul2_rn(__fmul2_rn(__fmul2_rn(rinv, rinv), rinv), t);
        const float2 fac = make_float2(fast_a ? f.x : 0.f, fast_b ? f.y : 0.f);
        ax = __ffma2_rn(dx, fac, ax);
        ay = __ffma2_rn(dy, fac, ay);
        az = __ffma2_rn(dz, fac, az);
        if (COUNT) npairs += fast_a + fast_b;
        // r2 == 0 (the self pair, or a coincident source): r is NaN, not
        // flagged, and it adds dx*fac = 0.  r_hi is a little above the flag
        // cut; pair_slow tests r2 against the cut itself.
        slow_a = r.x <= r_hi && !fast_a;
        slow_b = r.y <= r_hi && !fast_b;
    };
    auto pair_slow = [&](float sx, float sy, float sz, float tx, float ty, float tz, float &ax, float &ay, float &az) {
        const float dx = sx - tx, dy = sy - ty, dz = sz - tz;
        const float r2 = dist2(dx, dy, dz);
        bool ok = r2 <= law.rc2_hi && r2 != 0.f;
        const float rinv = rsqrtf(ok ? r2 : 1.f);
        const float r = r2 * rinv;
        const float xl = __fmaf_rz(r, law.alo, 8388608.0f);
        int ti = __float_as_int(xl) - 0x4B000000;
        float fac = rinv * rinv * rinv;
        if (!FIXED && (xl != __fmaf_rz(r, law.ahi, 8388608.0f) || r2 > law.rc2_lo)) {
            // decided in double as the reference's CPU path computes it
            const double dd = (double)dx * dx + (double)dy * dy + (double)dz * dz;
            ok = ok && dd <= law.rcut2_d;
            ti = (int)(law.asmthfac_d * sqrt(dd));
        }
        if (r < law.h) {
            const float u = r * law.hinv;
            const float h3inv = law.h3inv;
            if (u < 0.5f)
                fac = __fmul_rn(h3inv, __fmaf_rn(__fmul_rn(u, u), __fmaf_rn(32.0f, u, -38.4f), 10.66667f));
            else
                fac = __fmul_rn(h3inv, __fsub_rn(__fmaf_rn(u, __fmaf_rn(u, __fmaf_rn(-10.66667f, u, 38.4f), -48.0f),
                                                           21.33333f),
                                                 __fdiv_rn(0.06667f, __fmul_rn(__fmul_rn(u, u), u))));
        }
        fac = ok ? fac * tab[min(ti, kNTab - 1)] : 0.f;
        ax = __fmaf_rn(dx, fac, ax);
        ay = __fmaf_rn(dy, fac, ay);
        az = __fmaf_rn(dz, fac, az);
        if (COUNT) npairs += ok;
    };

    // the unit's targets split evenly into groups
    const bool two = !dense && len > (uint32_t)kGroup;
    for (uint32_t t0 = 0; t0 < len;) {
        // the group [t0, t0 + gs) on 1 << lg lanes, the other lanes repeating
        // it for their list slots
        const uint32_t gs = two && t0 == 0 ? len >> 1 : len - t0;
        const uint32_t lg = 32u - __clz(gs - 1u);  // (gs = 1: __clz(0) = 32)
        const uint32_t tl = lane & ((1u << lg) - 1u), slot = (uint32_t)lane >> lg;
        const uint32_t stride = 128u >> lg;  // list sources per iteration
        const bool has = tl < gs;
        const float4 praw = spos[t_begin + t0 + min(tl, gs - 1u)];
        float4 ta = FIXED ? rel(praw) : make_float4(praw.x - ox, praw.y - oy, praw.z - oz, 0.f);
        // the group's bounding box
        {
            const float4 lo = make_float4(warp_min(ta.x), warp_min(ta.y), warp_min(ta.z), 0.f);
            const float4 hi = make_float4(warp_max(ta.x), warp_max(ta.y), warp_max(ta.z), 0.f);
            if (!has) ta = make_float4(kSentinel, kSentinel, kSentinel, 0.f);
            if (lane == 0) wm.box[0] = lo, wm.box[1] = hi;
            wm.tx[lane] = ta.x, wm.ty[lane] = ta.y, wm.tz[lane] = ta.z;
        }

        // the lane's sums (two halves), their error terms (FIXED)
        float2 sx = make_float2(0.f, 0.f), sy = sx, sz = sx, ex = sx, ey = sx, ez = sx;
        uint32_t cnt = 0;                      // list entries
        uint32_t T = 0, base = 0, before = 0;  // the batch's run list: length, window, runs started before it
        uint32_t ps = kFull;                   // this lane's run start in it
        int batch = 0;
        bool more = true;
        do {
            __syncwarp();
            // fill the list
            const float4 lo = wm.box[0], hi = wm.box[1];
            while (cnt < kListFull) {
                if (base >= T) {
                    if (batch == batches) {
                        more = false;
                        break;
                    }
                    // the next 32 columns (of the part of their z range in
                    // the box, then the wrapped part): lane k narrows column k
                    const int part = parts == 2 ? batch & 1 : 0, col = ((parts == 2 ? batch >> 1 : batch) << 5) + lane;
                    ++batch;
                    uint32_t b = 0, e = 0;
                    float cx = ox, cy = oy, cz = oz;
                    if (col < ncols) {
                        const char2 d = dxdy(col);
                        const float x0 = fmaf((float)d.x, w, fx), y0 = fmaf((float)d.y, w, fy);
                        const float ddx = fmaxf(fmaxf(x0 - hi.x, lo.x - (x0 + w)), 0.f);
                        const float ddy = fmaxf(fmaxf(y0 - hi.y, lo.y - (y0 + w)), 0.f);
                        const float q = rc2m - (ddx * ddx + ddy * ddy);
                        if (q >= 0.f) {
                            // half-height of the cut disc over this column (an
                            // approximate square root: the margin covers it), in
                            // cells from the column's first z-cell
                            const float hz = q * rsqrt_ftz(fmaxf(q, 1e-30f));
                            const float ul = (lo.z - hz - fz) * winv + (float)R, uh = (hi.z + hz - fz) * winv + (float)R;
                            const int fl = __float2int_rd(ul), fh = __float2int_rd(uh);
                            const int za = iz0 - R + max(fl, 0), zb = iz0 - R + min(fh, nz - 1);
                            // this part's z-cells [z0, z1], and what brings them into the box
                            int z0 = max(za, 0), z1 = min(zb, G - 1), off = 0;
                            if (part) {
                                if (z_below)
                                    z0 = za, z1 = min(zb, -1), off = G;
                                else
                                    z0 = max(za, G), z1 = zb, off = -G;
                            }
                            if (z0 <= z1) {
                                const int cxu = ix + d.x, cyu = iy + d.y;
                                const int gx = cxu < 0 ? cxu + G : (cxu >= G ? cxu - G : cxu);
                                const int gy = cyu < 0 ? cyu + G : (cyu >= G ? cyu - G : cyu);
                                const uint32_t row = p.cell_base + ((uint32_t)gx * G + gy) * G;
                                const uint32_t c0 = row + (uint32_t)(z0 + off), c1 = row + (uint32_t)(z1 + off);
                                b = cell_off[c0];
                                e = cell_off[c1 + 1];
                                if (ZS) {
                                    // the end cells hold their sources by z slice: drop
                                    // the slices below ul and above uh (a cell whose
                                    // counts saturated, 0xffff, is kept whole)
                                    const uint16_t *sl16 = reinterpret_cast<const uint16_t *>(p.slices);
                                    if (fl >= 0 && z0 == za) {
                                        const int kl = __float2int_rd((ul - (float)fl) * (float)kZSub);
                                        if (kl > 0) {
                                            const uint32_t o = sl16[(size_t)c0 * kZSub + min(kl, kZSub) - 1];
                                            if (o != 0xffffu) b += o;
                                        }
                                    }
                                    if (fh <= nz - 1 && z1 == zb) {
                                        const int kh = __float2int_rd((uh - (float)fh) * (float)kZSub);
                                        if (kh < kZSub - 1) {
                                            const uint32_t o = sl16[(size_t)c1 * kZSub + max(kh, 0)];
                                            if (o != 0xffffu) e = cell_off[c1] + o;
                                        }
                                    }
                                }
                                if (!FIXED && wrap) {
                                    cx = ox - (cxu < 0 ? -L : (cxu >= G ? L : 0.0f));
                                    cy = oy - (cyu < 0 ? -L : (cyu >= G ? L : 0.0f));
                                    cz = oz - (off > 0 ? -L : (off < 0 ? L : 0.0f));
                                }
                            }
                        }
                    }
                    // The runs, concatenated, form one list of length T; ps is
                    // this lane's run start in it.
                    const uint32_t rl = b < e ? e - b : 0u;
                    ps = rl;
#pragma unroll
                    for (int off = 1; off < 32; off <<= 1) {
                        const uint32_t v = __shfl_up_sync(kFull, ps, off);
                        if (lane >= off) ps += v;
                    }
                    T = __shfl_sync(kFull, ps, 31);
                    ps -= rl;
                    // the k-th non-empty run's shift from list position to sorted index
                    const uint32_t nonempty = __ballot_sync(kFull, rl > 0);
                    if (rl > 0) {
                        const uint32_t k = __popc(nonempty & lt_mask);
                        wm.delta[k] = b - ps;
                        if (!FIXED && wrap) wm.shift[k] = make_float4(cx, cy, cz, 0.f);
                    } else {
                        ps = kFull;  // marks no start
                    }
                    base = before = 0;
                    __syncwarp();
                    continue;
                }
                // Two windows of 32 run-list positions: one bit per run start,
                // so a lane's run is (runs started before the window) +
                // (starts at or below its position) - 1.
                uint32_t run[2], at[2];
                bool in[2];
                float4 s[2];
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const uint32_t m0 = __reduce_or_sync(kFull, bit_at(ps - base));
                    run[u] = before + __popc(m0 & le_mask) - 1u;
                    before += __popc(m0);
                    in[u] = base + lane < T;
                    at[u] = min(base + lane, T - 1u) + wm.delta[run[u]];
                    base += 32;
                }
#pragma unroll
                for (int u = 0; u < 2; ++u) s[u] = spos[at[u]];
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    float4 a;
                    if (FIXED) {
                        a = rel(s[u]);
                    } else if (wrap) {
                        const float4 c = wm.shift[run[u]];
                        a = make_float4(s[u].x - c.x, s[u].y - c.y, s[u].z - c.z, 0.f);
                    } else {
                        a = make_float4(s[u].x - ox, s[u].y - oy, s[u].z - oz, 0.f);
                    }
                    // within rcut of the group's bounding box
                    const float ddx = max0(lo.x - a.x, a.x - hi.x);
                    const float ddy = max0(lo.y - a.y, a.y - hi.y);
                    const float ddz = max0(lo.z - a.z, a.z - hi.z);
                    const bool keep = in[u] && fmaf(ddz, ddz, fmaf(ddy, ddy, ddx * ddx)) <= rc2m;
                    const uint32_t kept = __ballot_sync(kFull, keep);
                    const uint32_t k = cnt + __popc(kept & lt_mask);
                    if (keep) {
                        wm.x[CUCO_IDX(k, kListCap)] = a.x;
                        wm.y[CUCO_IDX(k, kListCap)] = a.y;
                        wm.z[CUCO_IDX(k, kListCap)] = a.z;
                    }
                    cnt += __popc(kept);
                }
            }
            // whole iterations; the last list is padded with sources beyond any cut
            const uint32_t n_eval = (more ? cnt : cnt + stride - 1u) & ~(stride - 1u);
            for (uint32_t k = cnt + lane; k < n_eval; k += 32) wm.x[k] = wm.y[k] = wm.z[k] = kSentinel;
            __syncwarp();
            const float3 ta = make_float3(wm.tx[lane], wm.ty[lane], wm.tz[lane]);
            const float2 ntx = make_float2(-ta.x, -ta.x), nty = make_float2(-ta.y, -ta.y),
                         ntz = make_float2(-ta.z, -ta.z);
            uint32_t at = slot * 4u;
            for (uint32_t left = n_eval >> (7 - lg); left;) {
                // up to kFold iterations into fresh partial sums
                const uint32_t its = min(kFold, left);
                left -= its;
                float2 ax = make_float2(0.f, 0.f), ay = ax, az = ax;
                uint32_t m = 0;
#pragma unroll 2
                for (uint32_t k = 0; k < its; ++k) {
                    const float4 X = *reinterpret_cast<const float4 *>(wm.x + at);
                    const float4 Y = *reinterpret_cast<const float4 *>(wm.y + at);
                    const float4 Z = *reinterpret_cast<const float4 *>(wm.z + at);
                    bool s0, s1, s2, s3;
                    pair_fast2(make_float2(X.x, X.y), make_float2(Y.x, Y.y), make_float2(Z.x, Z.y), ntx, nty, ntz, ax,
                               ay, az, s0, s1);
                    pair_fast2(make_float2(X.z, X.w), make_float2(Y.z, Y.w), make_float2(Z.z, Z.w), ntx, nty, ntz, ax,
                               ay, az, s2, s3);
                    m <<= 4;
                    if (s0) m |= 1u;
                    if (s1) m |= 2u;
                    if (s2) m |= 4u;
                    if (s3) m |= 8u;
                    at += stride;
                }
                // the rare-case pairs, one per lane at a time
                while (__any_sync(kFull, m != 0)) {
                    if (m) {
                        const uint32_t bit = __ffs(m) - 1;
                        m &= m - 1;
                        const uint32_t k = at - stride * (1u + (bit >> 2)) + (bit & 3u);
                        pair_slow(wm.x[k], wm.y[k], wm.z[k], ta.x, ta.y, ta.z, ax.x, ay.x, az.x);
                    }
                }
                if (FIXED) {
                    // compensated: the sums' rounding goes to the error terms
                    // (two_sum of both halves at once; x - y as -1 y + x: at 256^3,
                    // fixed, the kernel took 5.26 ms with two scalar ones, 5.19 so)
                    auto add = [](float2 &s, float2 &e, float2 v) {
                        const float2 neg = make_float2(-1.f, -1.f), t = __fadd2_rn(s, v);
                        const float2 bb = __ffma2_rn(neg, s, t);
                        const float2 err = __fadd2_rn(__ffma2_rn(neg, __ffma2_rn(neg, bb, t), s), __ffma2_rn(neg, bb, v));
                        e = __fadd2_rn(e, err);
                        s = t;
                    };
                    add(sx, ex, ax);
                    add(sy, ey, ay);
                    add(sz, ez, az);
                } else {
                    sx = __fadd2_rn(sx, ax);
                    sy = __fadd2_rn(sy, ay);
                    sz = __fadd2_rn(sz, az);
                }
            }
            // what is left of the list (less than one iteration) moves to its front
            if (more) {
                __syncwarp();  // (the rare-case pairs have read the list)
                const uint32_t rest = cnt - n_eval;
                // (forward, 32 at a time: n_eval >= rest, so nothing is overwritten before it is read)
                for (uint32_t k = lane; k < rest; k += 32) {
                    const float x = wm.x[n_eval + k], y = wm.y[n_eval + k], z = wm.z[n_eval + k];
                    wm.x[k] = x, wm.y[k] = y, wm.z[k] = z;
                }
                cnt = rest;
            }
        } while (more);

        // the halves, then the slots
        float3 f;
        if (FIXED) {
            auto total = [&](float2 s, float2 e) {
                float h, l, t;
                two_sum(s.x, s.y, h, l);
                l = __fadd_rn(l, __fadd_rn(e.x, e.y));
                for (uint32_t off = 16; off >> lg; off >>= 1) {
                    const float oh = __shfl_xor_sync(kFull, h, off), ol = __shfl_xor_sync(kFull, l, off);
                    two_sum(h, oh, h, t);
                    l = __fadd_rn(__fadd_rn(l, ol), t);
                }
                return __fadd_rn(h, l);
            };
            f = make_float3(total(sx, ex), total(sy, ey), total(sz, ez));
        } else {
            f = make_float3(sx.x + sx.y, sy.x + sy.y, sz.x + sz.y);
            for (uint32_t off = 16; off >> lg; off >>= 1) {
                f.x += __shfl_xor_sync(kFull, f.x, off);
                f.y += __shfl_xor_sync(kFull, f.y, off);
                f.z += __shfl_xor_sync(kFull, f.z, off);
            }
        }
        const float mg = p.mass * p.G;
        if (slot == 0 && has) {
            wm.acc[0][t0 + tl] = f.x * mg;
            wm.acc[1][t0 + tl] = f.y * mg;
            wm.acc[2][t0 + tl] = f.z * mg;
        }
        t0 += gs;
    }
    __syncwarp();

    // the forces (already scaled by m G) to original order, PM scatter and kick
    if (lane < len) {
        const uint32_t i = t_begin + lane;
        const float4 a = make_float4(wm.acc[0][lane], wm.acc[1][lane], wm.acc[2][lane], 0.f);
        const uint32_t o = perm[i];
        acc_out[o] = a;
        float4 gpm = make_float4(0.f, 0.f, 0.f, 0.f);
        const bool with_pm = kick.acc_pm_s || kick.acc_pm_o;
        if (kick.acc_pm_s) {
            gpm = kick.acc_pm_s[i];
            if (kick.acc_pm_out) kick.acc_pm_out[o] = gpm;
        } else if (kick.acc_pm_o) {
            gpm = kick.acc_pm_o[o];
        }
        if (KICK) {
            float4 v = kick.vel[o];
            // vel += GravAccel*dt; vel += GravPM*dt (timestep.c:57-58,88), in
            // float (the reference rounds each product to float first)
            const float kp = (float)kick_pp, km = (float)kick_pm;
            v.x += __fmul_rn(a.x, kp);
            v.y += __fmul_rn(a.y, kp);
            v.z += __fmul_rn(a.z, kp);
            if (with_pm) {
                v.x = __fmaf_rn(gpm.x, km, v.x);
                v.y = __fmaf_rn(gpm.y, km, v.y);
                v.z = __fmaf_rn(gpm.z, km, v.z);
            }
            kick.vel[o] = v;
        }
    }
    __syncwarp();
}

__global__ void k_sr_plan(const __grid_constant__ SRPlan plan, const uint32_t *__restrict__ cell_off,
                          const uint32_t *__restrict__ hold, const __grid_constant__ SRWork w) {
    plan_box_segment(plan, blockIdx.x * blockDim.x + threadIdx.x, cell_off, 0u, 0u, w, hold);
}

// The next unit for a warp: the dense slices first (the longest work).  Takes
// the item fetched before and fetches the one after it, so that the counter's
// latency is behind a unit's work.
struct UnitQueue {
    const SRWork &w;
    uint32_t dense, total, item;
    uint32_t fixed;
    // The first `fixed` units go to the warps of the launch's first part by
    // their number (no counter); `late`: a warp of the second part.
    __device__ __forceinline__ UnitQueue(const SRWork &w_, uint32_t fixed_, bool late) : w(w_), fixed(fixed_) {
        dense = w.ctl[0];
        total = dense + w.ctl[2];
        item = late ? fetch() : blockIdx.x * kWarps + (threadIdx.x >> 5);
    }
    __device__ __forceinline__ uint32_t fetch() const {
        uint32_t i = 0;
        if ((threadIdx.x & 31) == 0 && total > fixed) i = atomicAdd(&w.ctl[1], 1u);
        return i + fixed;
    }
    // false when none is left; dense_unit: a slice of a dense segment
    __device__ __forceinline__ bool next(uint4 *unit, bool *dense_unit) {
        const uint32_t i = __shfl_sync(kFull, item, 0);
        if (i >= total) return false;
        item = fetch();
        *dense_unit = i < dense;
        *unit = w.units[i < dense ? i : w.cap - 1u - (i - dense)];
        return true;
    }
};

// The split table, once per CTA.
__device__ __forceinline__ void load_table(const float *__restrict__ table_g, float *tab) {
    for (int i = threadIdx.x; i < kTabPad; i += kThreads) tab[i] = table_g[min(i, kNTab - 1)];
}

__device__ __forceinline__ void add_pairs(uint32_t npairs, unsigned long long *pair_counter) {
    const uint32_t wsum = __reduce_add_sync(kFull, npairs);
    if ((threadIdx.x & 31) == 0 && wsum) atomicAdd(pair_counter, (unsigned long long)wsum);
}

// Persistent: as many CTAs as fit on the GPU, each warp taking units until
// none is left.
template <bool KICK, bool COUNT, bool FIXED>
__global__ void __launch_bounds__(kThreads, kMinBlocks)
    k_shortrange(const __grid_constant__ ShortRangeParams p, const __grid_constant__ ColumnSet cs,
                 uint32_t fixed, int late, const __grid_constant__ SRWork w, const float4 *__restrict__ spos,
                 const uint32_t *__restrict__ perm, const uint32_t *__restrict__ cell_off,
                 const float *__restrict__ table_g, float4 *__restrict__ acc_out,
                 const __grid_constant__ KickArgs kick, unsigned long long *__restrict__ pair_counter) {
    __shared__ WarpMem s_warp[kWarps];
    __shared__ float s_tab[kTabPad];
    __shared__ char2 s_col[kMaxCols];
    chain_next();  // (the next step's drift; its blocks start in the places this grid's leave)
    load_table(table_g, s_tab);
    for (int i = threadIdx.x; i < cs.ncols; i += kThreads) s_col[i] = make_char2(cs.dx[i], cs.dy[i]);
    __syncthreads();
    WarpMem &wm = s_warp[threadIdx.x >> 5];
    UnitQueue q(w, fixed, late != 0);
    uint4 u;
    bool dense;
    while (q.next(&u, &dense)) {
        uint32_t npairs = 0;
        shortrange_unit<KICK, COUNT, FIXED, false>(p, p, cs.ncols, cs.R, cs.S, cs.margin,
                                                   [&](int col) { return s_col[col]; }, u, dense, kick.kick_pp,
                                                   kick.kick_pm, spos, perm, cell_off, acc_out, kick, wm, s_tab,
                                                   npairs);
        if (COUNT) add_pairs(npairs, pair_counter);
    }
}

// Many boxes in one launch: segments numbered box after box (seg_base, nbox+1
// entries); particles, cells (p.cell_base) and outputs are the concatenated
// arrays of all boxes.
__global__ void k_sr_plan_multi(const SRBoxDesc *__restrict__ boxes, const uint32_t *__restrict__ seg_base,
                                int nbox, uint32_t nseg, const uint32_t *__restrict__ cell_off,
                                const __grid_constant__ SRWork w) {
    const uint32_t gseg = blockIdx.x * blockDim.x + threadIdx.x;
    SRPlan plan{1, 1, 0u, (uint32_t)kUnitMax};
    uint32_t b = 0, seg = 0, base = 0;
    if (gseg < nseg) {
        b = find_box(seg_base, nbox, gseg);
        const SRBoxDesc &d = boxes[b];
        seg = gseg - seg_base[b];
        plan = SRPlan{d.cs.S, d.p.grid, 0xffffffffu, d.slice};
        base = d.p.cell_base;
    }
    plan_box_segment(plan, seg, cell_off, base, b, w);
}

// UNIFORM: every box has the pair law of `law` (a kernel parameter, read as
// constant-bank operands); else each box's own from its descriptor.
template <bool KICK, bool COUNT, bool FIXED, bool UNIFORM>
__global__ void __launch_bounds__(kThreads, kMinBlocks)
    k_shortrange_multi(const SRBoxDesc *__restrict__ boxes, const double2 *__restrict__ kicks,
                       uint32_t fixed, const __grid_constant__ SRWork w, const float4 *__restrict__ spos,
                       const uint32_t *__restrict__ perm, const uint32_t *__restrict__ cell_off,
                       const float *__restrict__ table_g, float4 *__restrict__ acc_out,
                       const __grid_constant__ KickArgs kick, unsigned long long *__restrict__ pair_counter,
                       const __grid_constant__ ShortRangeParams law) {
    __shared__ WarpMem s_warp[kWarps];
    __shared__ float s_tab[kTabPad];
    load_table(table_g, s_tab);
    __syncthreads();
    WarpMem &wm = s_warp[threadIdx.x >> 5];
    UnitQueue q(w, fixed, false);
    uint4 u;
    bool dense;
    while (q.next(&u, &dense)) {
        const uint32_t b = u.y >> 8;
        const SRBoxDesc &d = boxes[b];
        const double2 k = KICK ? kicks[b] : make_double2(0.0, 0.0);
        uint32_t npairs = 0;
        shortrange_unit<KICK, COUNT, FIXED, !UNIFORM>(
            d.p, UNIFORM ? law : d.p, d.cs.ncols, d.cs.R, d.cs.S, d.cs.margin,
            [&](int col) { return make_char2(d.cs.dx[col], d.cs.dy[col]); }, u, dense, k.x, k.y, spos, perm, cell_off, acc_out, kick, wm, s_tab, npairs);
        if (COUNT) add_pairs(npairs, pair_counter);
    }
}

// The persistent grid of a kernel: SMs x its resident CTAs per SM.
struct PersistentGrid {
    unsigned sms, per;
};
template <typename K>
PersistentGrid persistent_grid(K kernel) {
    int dev = 0, sms = 0, per = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, kThreads, 0) != cudaSuccess || per < 1) per = 1;
    return {(unsigned)std::max(sms, 1), (unsigned)per};
}

// Targets of a unit: kUnitMax, halved while the launch would have fewer than
// two units for each of the GPU's resident warps (about 32 on each of ~150
// SMs), down to kUnitMin: a box of 32^3 then still gives every warp a unit.
// n is the box's own count, in a many-box launch too: the unit decides which
// targets share a list, and so the order of the sums, and a box's forces must
// not depend on the boxes beside it.
uint32_t unit_slice(uint32_t n) {
    uint32_t s = kUnitMax;
    while (s > (uint32_t)kUnitMin && n / s < 2u * 4864u) s >>= 1;
    return s;
}

// Neighbour columns (dx, dy) whose xy cell distance is within rcut (+margin).
bool build_columns(const ShortRangeParams &p, ColumnSet *cs) {
    const double w = (double)p.boxsize / p.grid;
    const double margin = 1e-5 * (double)p.boxsize + 1e-4 * w;
    const double rc = (double)p.rcut + margin;
    int R = (int)ceil(rc / w);
    if (R > kMaxR) return false;
    if (2.0 * p.rcut >= p.boxsize) return false;
    // segment length: a power of two dividing G, with the S + 2R z-cells of a
    // column at most G (so a column's z range wraps at most once)
    int S = kMaxSeg;
    // fixed point also needs every source within G/2 cells of the
    // segment corner (the int32 difference is the periodic image)
    auto bad = [&](int s) { return p.grid % s || p.grid < s + 2 * R || (p.fixed && 2 * (s + R) >= p.grid); };
    while (S > 1 && bad(S)) S >>= 1;
    if (bad(S)) return false;
    cs->R = R;
    cs->S = S;
    cs->margin = (float)margin;
    int n = 0;
    for (int dx = -R; dx <= R; ++dx)
        for (int dy = -R; dy <= R; ++dy) {
            double ex = fmax(abs(dx) - 1, 0) * w, ey = fmax(abs(dy) - 1, 0) * w;
            if (ex * ex + ey * ey > rc * rc) continue;
            cs->dx[n] = (signed char)dx;
            cs->dy[n] = (signed char)dy;
            n++;
        }
    cs->ncols = n;
    return true;
}

}  // namespace

template <bool KICK, bool FIXED>
void launch_kick(cudaStream_t stream, cudaStream_t late_stream, const ShortRangeParams &p, const ColumnSet &cs,
                 const SRWork &work, const float4 *sorted_pos, const uint32_t *perm, const uint32_t *cell_off,
                 const float *table, float4 *acc_out, const KickArgs &kick, unsigned long long *counter) {
    auto launch = [&](auto kernel) {
        const PersistentGrid g = persistent_grid(kernel);
        const unsigned late = late_stream && g.per > 1 ? g.sms : 0u;
        const unsigned first = g.sms * g.per - late;
        kernel<<<first, kThreads, 0, stream>>>(p, cs, first * kWarps, 0, work, sorted_pos, perm, cell_off,
                                               table, acc_out, kick, counter);
        if (late)
            kernel<<<late, kThreads, 0, late_stream>>>(p, cs, first * kWarps, 1, work, sorted_pos, perm,
                                                       cell_off, table, acc_out, kick, counter);
    };
    if (counter)
        launch(k_shortrange<KICK, true, FIXED>);
    else
        launch(k_shortrange<KICK, false, FIXED>);
}

uint32_t shortrange_unit_cap(uint32_t n, uint64_t segments) {
    // a dense segment: ceil(nt / slice) <= nt / slice + nt / kDense; another:
    // at most nt / slice + 1
    return n / unit_slice(n) + n / kDense + (uint32_t)std::min<uint64_t>(n, segments) + 16u;
}

cuco_status_t shortrange_timeout_probe(uint32_t *ctl, long long limit_cycles, cudaStream_t stream) {
    k_timeout_probe<<<1, kThreads, 0, stream>>>(ctl + 3, limit_cycles);
    CUCO_TRY_CUDA(cudaGetLastError());
    return shortrange_check(ctl, stream);
}

cuco_status_t shortrange_check(uint32_t *ctl, cudaStream_t stream) {
    uint32_t flag = 0;
    CUCO_TRY_CUDA(cudaMemcpyAsync(&flag, ctl + 3, sizeof flag, cudaMemcpyDeviceToHost, stream));
    CUCO_TRY_CUDA(cudaStreamSynchronize(stream));
    if (flag) {
        CUCO_TRY_CUDA(cudaMemsetAsync(ctl + 3, 0, sizeof(uint32_t), stream));
        set_error("short range: a bounded wait gave up; forces are invalid");
        return CUCO_ERR_TIMEOUT;
    }
    return CUCO_OK;
}

// The pair-law bounds the kernel reads from its parameters.
static void finish_pair_law(ShortRangeParams &p) {
    const float kEdge = 4e-7f;
    // plain: cut-edge band decided in double; fixed: the float cut
    p.rc2_lo = p.fixed ? p.rcut2 : p.rcut2 * (1.f - 2.f * kEdge);
    p.rc2_hi = p.fixed ? p.rcut2 : p.rcut2 * (1.f + 2.f * kEdge);
    const float hmin = std::max(p.h, 1e-9f);
    p.hmin2 = hmin * hmin;
    p.alo = p.fixed ? p.asmthfac : p.asmthfac * (1.f - kEdge);
    p.ahi = p.fixed ? p.asmthfac : p.asmthfac * (1.f + kEdge);
    p.rcut2_d = (double)p.rcut * (double)p.rcut;
    p.grid_q = (uint32_t)((1ull << 32) / (uint32_t)p.grid);
    p.grid_r = (uint32_t)((1ull << 32) % (uint32_t)p.grid);
    p.grid_inv = 1.0f / (float)p.grid;
    p.r_hi = (float)(sqrt((double)p.rc2_hi) * (1.0 + 1e-6));
}

namespace {
cuco_status_t columns_of(const ShortRangeParams &p, ColumnSet *cs) {
    if (build_columns(p, cs)) return CUCO_OK;
    set_error("short range: cell grid does not fit rcut (need rcut <= 8 cell widths, "
              "rcut < L/2 and at least S+2R cells per dimension)");
    return CUCO_ERR_UNSUPPORTED;
}
}  // namespace

cuco_status_t shortrange_plan(const ShortRangeParams &p, SRPlan *plan) {
    ColumnSet cs;
    CUCO_TRY(columns_of(p, &cs));
    *plan = SRPlan{cs.S, p.grid, (uint32_t)p.grid * p.grid * (p.grid / cs.S), unit_slice(p.n)};
    return CUCO_OK;
}

cuco_status_t launch_shortrange(const ShortRangeParams &p_in, const float4 *sorted_pos, const uint32_t *perm,
                                const uint32_t *cell_off, const float *table, float4 *acc_out, const KickArgs &kick,
                                const SRWork &work, bool planned, cudaStream_t stream,
                                unsigned long long *pair_counter, cudaStream_t late_stream, cudaEvent_t plan_done,
                                const uint32_t *hold) {
    ColumnSet cs;
    ShortRangeParams p = p_in;
    finish_pair_law(p);
    CUCO_TRY(columns_of(p, &cs));
    if (p.n == 0) return CUCO_OK;
    SRPlan plan;
    CUCO_TRY(shortrange_plan(p, &plan));
    if (work.cap < shortrange_unit_cap(p.n, plan.nseg)) {
        set_error("short range: work-plan scratch too small for this grid or particle count");
        return CUCO_ERR_INVALID;
    }
    const bool kick_on = kick.vel != nullptr;
    if (!planned) {
        CUCO_TRY_CUDA(cudaMemsetAsync(work.ctl, 0, 3 * sizeof(uint32_t), stream));
        k_sr_plan<<<(plan.nseg + 255) / 256, 256, 0, stream>>>(plan, cell_off, hold, work);
    }
    if (late_stream) {
        if (!plan_done) {
            set_error("short range: a split launch needs the caller's plan event");
            return CUCO_ERR_INVALID;
        }
        CUCO_TRY_CUDA(cudaEventRecord(plan_done, stream));
        CUCO_TRY_CUDA(cudaStreamWaitEvent(late_stream, plan_done, 0));
    }
    auto launch = p.fixed ? (kick_on ? launch_kick<true, true> : launch_kick<false, true>)
                          : (kick_on ? launch_kick<true, false> : launch_kick<false, false>);
    launch(stream, late_stream, p, cs, work, sorted_pos, perm, cell_off, table, acc_out, kick, pair_counter);
    CUCO_TRY_CUDA(cudaGetLastError());
    return CUCO_OK;
}

size_t shortrange_desc_bytes() { return sizeof(SRBoxDesc); }

cuco_status_t shortrange_desc_fill(const ShortRangeParams &p, void *desc, uint32_t *segments, uint32_t *units) {
    SRBoxDesc d{};
    d.p = p;
    finish_pair_law(d.p);
    CUCO_TRY(columns_of(p, &d.cs));
    d.slice = unit_slice(p.n);
    memcpy(desc, &d, sizeof d);
    *segments = (uint32_t)p.grid * p.grid * (p.grid / d.cs.S);
    *units = shortrange_unit_cap(p.n, *segments);
    return CUCO_OK;
}

bool shortrange_descs_uniform_law(const void *host_descs, int nbox) {
    const SRBoxDesc *d = static_cast<const SRBoxDesc *>(host_descs);
    for (int b = 1; b < nbox; ++b) {
        const ShortRangeParams &x = d[0].p, &y = d[b].p;
        if (x.rc2_lo != y.rc2_lo || x.rc2_hi != y.rc2_hi || x.hmin2 != y.hmin2 || x.alo != y.alo ||
            x.ahi != y.ahi || x.rcut2_d != y.rcut2_d || x.asmthfac_d != y.asmthfac_d || x.h != y.h ||
            x.hinv != y.hinv || x.h3inv != y.h3inv)
            return false;
    }
    return nbox > 0;
}

cuco_status_t launch_shortrange_multi(const void *descs, const double2 *kicks, const uint32_t *seg_base,
                                      int nbox, uint32_t segments, uint32_t units, uint32_t n, bool fixed,
                                      const float4 *sorted_pos, const uint32_t *perm, const uint32_t *cell_off,
                                      const float *table, float4 *acc_out, const KickArgs &kick,
                                      const SRWork &work, cudaStream_t stream, unsigned long long *pair_counter,
                                      const void *uniform_law_desc) {
    if (!segments || !n) return CUCO_OK;
    if (work.cap < units) {
        set_error("short range: work-plan scratch too small for the ensemble's units");
        return CUCO_ERR_INVALID;
    }
    const SRBoxDesc *d = static_cast<const SRBoxDesc *>(descs);
    const bool kick_on = kick.vel != nullptr;
    CUCO_TRY_CUDA(cudaMemsetAsync(work.ctl, 0, 3 * sizeof(uint32_t), stream));
    k_sr_plan_multi<<<(segments + 255) / 256, 256, 0, stream>>>(d, seg_base, nbox, segments, cell_off, work);
    // the shared law (any box's, all being equal) or, unused, box 0's shape
    ShortRangeParams law{};
    const bool uniform = uniform_law_desc != nullptr;
    if (uniform) law = static_cast<const SRBoxDesc *>(uniform_law_desc)->p;
#define CUCO_SR_MULTI_U(K, C, F, U)                                                                     \
    do {                                                                                                \
        const PersistentGrid g = persistent_grid(k_shortrange_multi<K, C, F, U>);                        \
        k_shortrange_multi<K, C, F, U><<<g.sms * g.per, kThreads, 0, stream>>>(                          \
            d, kicks, g.sms * g.per * kWarps, work, sorted_pos, perm, cell_off, table, acc_out, kick,        \
            pair_counter, law);                                                                         \
    } while (0)
#define CUCO_SR_MULTI(K, C, F)                 \
    do {                                       \
        if (uniform)                           \
            CUCO_SR_MULTI_U(K, C, F, true);    \
        else                                   \
            CUCO_SR_MULTI_U(K, C, F, false);   \
    } while (0)
    if (fixed) {
        if (kick_on) {
            if (pair_counter) CUCO_SR_MULTI(true, true, true); else CUCO_SR_MULTI(true, false, true);
        } else {
            if (pair_counter) CUCO_SR_MULTI(false, true, true); else CUCO_SR_MULTI(false, false, true);
        }
    } else {
        if (kick_on) {
            if (pair_counter) CUCO_SR_MULTI(true, true, false); else CUCO_SR_MULTI(true, false, false);
        } else {
            if (pair_counter) CUCO_SR_MULTI(false, true, false); else CUCO_SR_MULTI(false, false, false);
        }
    }
#undef CUCO_SR_MULTI
#undef CUCO_SR_MULTI_U
    CUCO_TRY_CUDA(cudaGetLastError());
    return CUCO_OK;
}

uint32_t bounds_violations_shortrange() { return bounds_violations_take(); }

}  // namespace cuco
