// Shared declarations of the GB300 force engine (sm_103a).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <cstdio>
#include <string>

#include "../../include/cuco_gb300.h"

namespace cuco {

struct SRPlan;
struct SRWork;

constexpr uint32_t kEmptyCell = 0xffffffffu;
constexpr int kNTab = CUCO_NTAB;

// ---------------------------------------------------------------- errors

void set_error(const std::string &msg);
const char *last_error();

#define CUCO_TRY_CUDA(expr)                                                         \
    do {                                                                            \
        cudaError_t _e = (expr);                                                    \
        if (_e != cudaSuccess) {                                                    \
            ::cuco::set_error(std::string(#expr) + ": " + cudaGetErrorString(_e));  \
            return CUCO_ERR_CUDA;                                                   \
        }                                                                           \
    } while (0)

#define CUCO_TRY(expr)                         \
    do {                                       \
        cuco_status_t _s = (expr);             \
        if (_s != CUCO_OK) return _s;          \
    } while (0)

// ---------------------------------------------------- debug bounds checks

// Debug builds (compiled with -DCUCO_BOUNDS_CHECK) check the index of the
// main global and shared memory accesses of the kernels against its bound.  A
// failed check adds one to this translation unit's violation counter and the
// access goes to the last in-bounds element instead, so the kernel keeps
// running and the host reads the count afterwards
// (cuco_debug_bounds_violations).  Release builds compile the checks away.
#ifdef CUCO_BOUNDS_CHECK
static __device__ unsigned int g_bounds_violations;
__device__ __forceinline__ uint32_t bounds_checked(uint32_t i, uint32_t limit) {
    if (i >= limit) {
        atomicAdd(&g_bounds_violations, 1u);
        return limit ? limit - 1u : 0u;
    }
    return i;
}
#define CUCO_IDX(i, limit) ::cuco::bounds_checked((uint32_t)(i), (uint32_t)(limit))
// this translation unit's count, read and reset (host)
static inline uint32_t bounds_violations_take() {
    unsigned int v = 0, zero = 0;
    cudaMemcpyFromSymbol(&v, g_bounds_violations, sizeof v);
    cudaMemcpyToSymbol(g_bounds_violations, &zero, sizeof zero);
    return v;
}
#else
#define CUCO_IDX(i, limit) (i)
static inline uint32_t bounds_violations_take() { return 0; }
#endif
uint32_t bounds_violations_sort();
uint32_t bounds_violations_pm();
uint32_t bounds_violations_shortrange();

// A kernel's dynamic shared-memory limit belongs to the device that is current
// when it is raised.  run(set) calls `set` (which raises limits and returns a
// cudaError_t) where it has not succeeded yet on the current device; a failure
// is returned and not kept.
class OncePerDevice {
    static constexpr int kDevices = 64;  // (a device beyond them: each time)
    std::atomic<bool> done_[kDevices] = {};

  public:
    template <typename F>
    cudaError_t run(F set) {
        int dev = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e != cudaSuccess) return e;
        const bool known = dev >= 0 && dev < kDevices;
        if (known && done_[dev].load(std::memory_order_acquire)) return cudaSuccess;
        e = set();
        if (e != cudaSuccess)
            cudaGetLastError();  // (reported by the value alone)
        else if (known)
            done_[dev].store(true, std::memory_order_release);
        return e;
    }
};

template <typename... P>
cudaError_t raise_smem_limit(void (*kernel)(P...), size_t bytes) {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

// ------------------------------------------------------- chained launches

// A kernel launched by launch_chained may start while the kernel before it on
// the stream still runs, once every block of that one has called chain_next()
// or ended: its launch and its constant tables' loads then cost nothing.  It
// calls chain_wait(), in every block, before it touches anything another kernel
// writes or reads; that returns when the kernel before it (and so, as that one
// waited too, every kernel before) has completed.  Both do nothing in a plain
// launch (`chain` false).
__device__ __forceinline__ void chain_wait() { cudaGridDependencySynchronize(); }
__device__ __forceinline__ void chain_next() { cudaTriggerProgrammaticLaunchCompletion(); }

template <typename... P, typename... A>
cudaError_t launch_chained(bool chain, void (*kernel)(P...), dim3 grid, unsigned threads, size_t smem, cudaStream_t stream,
                           A... args) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = &attr;
    cfg.numAttrs = chain ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// -------------------------------------------------------------- sorting

// Scratch a sort of n keys needs: alternate key/value buffers and the per-tile
// digit histogram (this many words for the tile size the sort prefers; a
// smaller one, of at least radix * ceil(n / 4096) words, makes it take larger
// tiles).
size_t sort_hist_entries(uint32_t n, int key_bits, int max_radix_bits);

// Stable LSD radix sort of (keys, vals) by the low key_bits bits.  vals_in may
// be null: the values are then the input positions 0..n-1.  The sorted data
// ends in (keys, vals) when `result_in_alt` comes back false, else in
// (keys_alt, vals_alt).  max_radix_bits bounds the digit width (4..8).
// offsets_done (or null): a sort that is one launch also writes cell_off (as
// launch_reorder_offsets) and says so.
cuco_status_t sort_pairs(uint32_t *keys, uint32_t *vals, const uint32_t *vals_in,
                         uint32_t *keys_alt, uint32_t *vals_alt, uint32_t *hist, size_t hist_words,
                         uint32_t n, int key_bits, int max_radix_bits, cudaStream_t stream,
                         bool *result_in_alt, int *launches, uint32_t *cell_off = nullptr, uint32_t ncells = 0,
                         bool *offsets_done = nullptr, uint32_t *plan_ctl = nullptr);

// Cell keys of float4 positions (calcHashD rule); idx gets 0..n-1 when non-null.
cuco_status_t launch_cell_keys(const float4 *pos, uint32_t *keys, uint32_t *idx, uint32_t n,
                               float gridfac, int G, cudaStream_t stream);

// Reference cell-bound format (cellStart/cellEnd, empty start = 0xffffffff) and
// the sorted-position gather.
cuco_status_t launch_reorder_start_end(uint32_t *cell_start, uint32_t *cell_end,
                                       float4 *sorted_pos, const uint32_t *sorted_keys,
                                       const uint32_t *perm, const float4 *pos, uint32_t n,
                                       uint32_t ncells, cudaStream_t stream);

// Engine cell-bound format: cell_off[c] = first sorted index with key >= c,
// for c in [0, ncells].  plan_ctl (or null): the first three words are cleared.
cuco_status_t launch_reorder_offsets(uint32_t *cell_off, const uint32_t *sorted_keys, uint32_t n, uint32_t ncells,
                                     cudaStream_t stream, uint32_t *plan_ctl = nullptr);

// The reference's cell bounds (cell_end is read where cell_start is not
// empty) -> the engine's offsets (ncells + 1), where the cells' ranges follow
// one another; gap_bit is set in *gap where they do not.  scratch:
// offsets_scratch(ncells) words; finished: a word that is 0 and is 0 again
// afterwards.
size_t offsets_scratch(uint32_t ncells);
cuco_status_t launch_start_end_offsets(const uint32_t *cell_start, const uint32_t *cell_end, uint32_t *cell_off,
                                       uint32_t ncells, uint32_t *scratch, uint32_t *finished, uint32_t *gap,
                                       uint32_t gap_bit, cudaStream_t stream);

// The same for ranges with gaps: the offsets that the cells' particles have
// when they are laid one after the other, and that layout of them.
cuco_status_t launch_start_end_counts(const uint32_t *cell_start, const uint32_t *cell_end, uint32_t *cell_off,
                                      uint32_t ncells, uint32_t *scratch, uint32_t *finished, cudaStream_t stream);
cuco_status_t launch_gather_cells(const uint32_t *cell_start, const uint32_t *cell_end, const uint32_t *cell_off,
                                  uint32_t ncells, const float4 *pos, const uint32_t *perm, float4 *pos_out,
                                  uint32_t *perm_out, cudaStream_t stream);

// A box's cell grid within a concatenated cell numbering (cells
// cell_base .. cell_base + G^3 - 1).
struct CellBox {
    uint32_t G, cell_base;
    float boxsize, gridfac;  // gridfac = (float)G / L, the key rule's factor
};

// Each cell's particles ordered by z slice: kZSub slices of the cell along z,
// stable within a slice.  From the cell-sorted permutation `perm` (cell_off:
// the cells' first sorted indices) it gathers sorted_pos in that order, with
// w = the slice as a float, and perm_s = its map to original indices.
// slices[c] holds eight u16: entry j = the cell's particles in slices 0..j
// (all 0xffff for a cell of 65535 or more).  Boxes: one (boxes null, `one`)
// or nbox descriptors sorted by cell_base.  fixed: positions are 32-bit fixed
// point.  plan, work (one box): the launch also writes the short range's work
// plan (its counters cleared by the kernel that wrote cell_off: plan_ctl).
constexpr int kZSubBits = 3;
constexpr int kZSub = 1 << kZSubBits;
cuco_status_t launch_cell_subsort(const uint32_t *cell_off, const uint32_t *perm, const float4 *pos,
                                  float4 *sorted_pos, uint32_t *perm_s, uint4 *slices, uint32_t ncells,
                                  const CellBox &one, const CellBox *boxes, int nbox, bool fixed,
                                  cudaStream_t stream, const SRPlan *plan = nullptr, const SRWork *work = nullptr);

// ----------------------------------------------------------- short range

struct ShortRangeParams {
    float boxsize;
    float gridfac;   // G / L in float, the key rule's factor
    float cellw;     // L / G
    float rcut, rcut2;
    float asmthfac;  // 0.5 / asmth * NTAB / 3
    double asmthfac_d;  // the same in double (gravlist.cpp:67), for bin-edge pairs
    float mass;      // source mass
    float G;         // gravitational constant (applied once per target)
    float h, hinv, h3inv;
    int grid;        // G
    uint32_t n;
    bool fixed;      // positions are 32-bit fixed point (bit patterns in the float4s)
    float fscale;    // L / 2^32
    uint32_t cell_base;  // first cell of this box in a multi-box cell array (0 otherwise)
    // pair-law bounds, filled in by the short-range launch from the above:
    // fast-path cut and flag cut (plain: a band around rcut^2 decided in
    // double), the softening bound below which the spline applies, the bin
    // factor scaled down and up by the bin-edge band, a radius just above the
    // flag cut, rcut^2 in double
    float rc2_lo, rc2_hi, hmin2, alo, ahi, r_hi;
    double rcut2_d;
    // the 2^32 grid's cell corners: 2^32 = grid_q * grid + grid_r
    uint32_t grid_q, grid_r;
    float grid_inv;
    // the z-slice counts of the cells (launch_cell_subsort), indexed by cell
    // id; null when the sources are not in slice order
    const uint4 *slices;
};

// Kick applied in the short-range epilogue (null vel: no kick).
struct KickArgs {
    float4 *vel;              // original order
    const float4 *acc_pm_s;   // PM acceleration in sorted order (may be null)
    float4 *acc_pm_out;       // PM acceleration scattered to original order (may be null)
    double kick_pp, kick_pm;
    const float4 *acc_pm_o;   // PM acceleration in original order (used when acc_pm_s is null)
};

// Device scratch of a launch's work plan: the units (shortrange_plan.cuh) and
// the control words.  cap must be at least shortrange_unit_cap(n, segments)
// of the launch (G^3 bounds a box's segments).
struct SRWork {
    uint4 *units;
    uint32_t cap;
    uint32_t *ctl;  // kSRCtlWords: [0] dense slices listed, [1] next unit, [2] other units listed
                    // (reset per launch), [3] timeout word (kept until read), the rest spare
};
uint32_t shortrange_unit_cap(uint32_t n, uint64_t segments);
// What a box's plan needs: cells a segment, the cell grid, segments, targets a
// unit.
struct SRPlan {
    int S, G;
    uint32_t nseg, slice;
};
cuco_status_t shortrange_plan(const ShortRangeParams &p, SRPlan *plan);
constexpr int kSRCtlWords = 8;
// Reads and clears the short range's timeout word (ctl[3]) after the work on
// `stream` is done: CUCO_ERR_TIMEOUT when a bounded wait gave up.
cuco_status_t shortrange_check(uint32_t *ctl, cudaStream_t stream);
// Runs a bounded wait on a barrier that never completes, with a limit of
// `limit_cycles`: returns what shortrange_check then reports.
cuco_status_t shortrange_timeout_probe(uint32_t *ctl, long long limit_cycles, cudaStream_t stream);

// planned: the work plan is in `work` already (launch_cell_subsort wrote it).
// hold (not planned, or null): a word in device memory; where it is not 0 when
// the plan is written, the plan stays empty and the launch does nothing.
// pair_counter: when non-null, the launch adds its in-range pair count to it.
// late_stream (with plan_done, an event of the caller's): the persistent grid
// is split, one CTA per SM fewer on `stream` and the rest queued on
// late_stream behind whatever that stream runs first (the PM).  The first
// part's warps start on units given by their number (every warp asking the
// counter at once cost 10 us of a small box's launch); the rest, for both
// parts, come from one counter, so work left when the late part starts
// spreads over both.  The launch is complete when both streams have run it.
cuco_status_t launch_shortrange(const ShortRangeParams &p, const float4 *sorted_pos,
                                const uint32_t *perm, const uint32_t *cell_off, const float *table,
                                float4 *acc_out, const KickArgs &kick, const SRWork &work, bool planned,
                                cudaStream_t stream, unsigned long long *pair_counter = nullptr, cudaStream_t late_stream = nullptr,
                                cudaEvent_t plan_done = nullptr, const uint32_t *hold = nullptr);

// Many boxes in one launch (the batched form).  A box's descriptor holds its
// parameters and neighbour-column set; shortrange_desc_fill writes one (in
// host memory, shortrange_desc_bytes() long) and returns the box's segment
// count and the units its plan takes at most; the launch's `units` is their sum
// over the boxes.  kicks[b] = (kick_pp, kick_pm) of box b.
size_t shortrange_desc_bytes();
cuco_status_t shortrange_desc_fill(const ShortRangeParams &p, void *desc, uint32_t *segments, uint32_t *units);
// uniform_law_desc (host memory, or null): a descriptor whose pair law every
// box shares (shortrange_descs_uniform_law said so); the launch then reads
// the law from its parameters instead of each box's descriptor.
bool shortrange_descs_uniform_law(const void *host_descs, int nbox);
cuco_status_t launch_shortrange_multi(const void *descs, const double2 *kicks, const uint32_t *seg_base,
                                      int nbox, uint32_t segments, uint32_t units, uint32_t n, bool fixed,
                                      const float4 *sorted_pos, const uint32_t *perm, const uint32_t *cell_off,
                                      const float *table, float4 *acc_out, const KickArgs &kick,
                                      const SRWork &work, cudaStream_t stream, unsigned long long *pair_counter,
                                      const void *uniform_law_desc = nullptr);

// ------------------------------------------------------------------- PM

struct PMPlan {
    int M;
    uint32_t stages;    // the Stockham transform's radices (meshes without register transforms)
    bool fixed;         // positions are 32-bit fixed point (units of L / 2^32)
    float boxsize;
    float to_slab_fac;  // M / L in float (pm_periodic.c:42)
    float mass;
    float fd_fac;       // G/(pi L) * M/(2L) (pm_periodic.c:85-86)
    float *rho;         // M^3 real grid: the potential
    unsigned long long *rho64;  // M^3 deposited mass in units of m / 2^32
    bool rho64_dirty;   // rho64 may hold sums (the z pass clears what it reads)
    float2 *spec;       // half spectrum, pm_spec_points(M)
    float *green1d;     // M/2+1: exp(-k^2 a) / sinc(pi k/M)^4
    float2 *twiddle;    // M: exp(-2 pi i t / M)
};

// Meshes the FFT supports: even, 8..1024, no prime factor above 5.
bool pm_mesh_supported(int M);
cuco_status_t pm_plan_create(PMPlan *plan, int M, float boxsize, float asmth, float mass,
                             double G, bool fixed = false);
void pm_plan_destroy(PMPlan *plan);
// Long-range acceleration of n positions (any order) into acc, in the same
// order or, with perm, of position i into acc[perm[i]].
cuco_status_t pm_forces(PMPlan &plan, const float4 *pos, const uint32_t *perm, uint32_t n, float4 *acc,
                        cudaStream_t stream, cudaEvent_t *ev_deposit_done,
                        cudaEvent_t *ev_fft_done, int *launches);

// Many boxes' meshes in one launch per PM phase (the batched form).
struct PMBoxDesc {
    int M, P, B;         // mesh; z-pass row pairs and axis-pass columns per CTA
    uint32_t stages;     // pm_stage_plan(M)
    float to_slab_fac, mass, fd_fac;
    float *rho;          // this box's M^3 real grid (the potential)
    unsigned long long *rho64;  // its deposited mass, units of m / 2^32
    float mscale;        // m / 2^32
    float2 *spec;        // its half spectrum, pm_spec_points(M)
    const float *green1d;
    const float2 *twiddle;
};
struct PMMulti {
    int nbox;
    bool fixed;
    const PMBoxDesc *boxes;   // device
    const uint32_t *pbeg;     // device, nbox+1: each box's first particle
    const uint2 *map_z;       // device: (box, block) per CTA of the z passes
    const uint2 *map_axis;    // device: (box, block) per CTA of the y/x passes
    uint32_t nz_blocks, naxis_blocks;
    size_t smz, sma;          // dynamic shared memory of the z and axis passes
    unsigned long long *rho64_all;  // all boxes' deposit grids, contiguous (one memset)
    size_t rho_all_count;
    bool big;  // some box's transforms need the large register kernels (pm_big_fft)
    bool wide; // some box's stages are wide (pm_wide_stages)
};
// Whether a box of mesh M with transform batches P, B takes the large (32-point)
// register transforms, which run in kernels of their own.
bool pm_big_fft(int M, int P, int B);
bool pm_fft_batches_ok(int M, int P, int B);
// Radices of a mesh's Stockham transform, five bits each.
uint32_t pm_stage_plan(int M);
// Whether they need the transforms with radices above 16 (more registers).
bool pm_wide_stages(uint32_t stages);
// Points of a mesh's half-spectrum array.
size_t pm_spec_points(int M);
int pm_batch_z(int M);
int pm_batch_axis(int M);
size_t pm_smem_z(int M, int P);
size_t pm_smem_axis(int M, int B);
void pm_tables(int M, float boxsize, float asmth, float *green1d, float2 *twiddle);
float pm_fd_fac(int M, float boxsize, double G);
// PM accelerations of n positions laid out box after box (pbeg), into acc.
cuco_status_t pm_forces_multi(const PMMulti &m, const float4 *pos, uint32_t n, float4 *acc,
                              cudaStream_t stream, int *launches);

// Index of the box whose range [pbeg[b], pbeg[b+1]) holds i (pbeg[0] = 0).
__device__ __forceinline__ int find_box(const uint32_t *__restrict__ pbeg, int nbox, uint32_t i) {
    int lo = 0, hi = nbox;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(&pbeg[mid]) <= i)
            lo = mid;
        else
            hi = mid;
    }
    return lo;
}

// ------------------------------------------------------------ integrator

cuco_status_t launch_drift_keys(float4 *pos, const float4 *vel, double drift, float boxsize,
                                bool do_drift, uint32_t *keys, uint32_t n, float gridfac, int G,
                                cudaStream_t stream);

// Fixed-point positions (uint32 per axis, units of L / 2^32, bit patterns in
// the float4 slots) from and to float triplets; float triplets <-> float4.
cuco_status_t to_fixed(const float *a, float4 *b, uint32_t n, float boxsize, cudaStream_t stream);
cuco_status_t from_fixed(const float4 *b, float *a, uint32_t n, float boxsize, cudaStream_t stream);
cuco_status_t pack3to4(const float *a, float4 *b, uint32_t n, cudaStream_t stream);
cuco_status_t unpack4to3(const float4 *b, float *a, uint32_t n, cudaStream_t stream);

// The reference's erfc split table T[i] (gravlist.cpp:56-67), FP64 -> float.
void shortrange_table(float *t);

// Host FP64 cosmological integrals.
double cosmo_integral(double a0, double a1, double omega0, double omega_lambda, double hubble,
                      int power);

}  // namespace cuco
