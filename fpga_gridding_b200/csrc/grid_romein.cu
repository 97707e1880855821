// Romein-style W-projection scatter kernel for sm_100a.
//
// Work arrives as tasks: runs of <= kTaskRaw sorted visibilities that share a
// support S (hence a footprint width W = 2S+1) and a coarse grid tile; with
// staging on, runs of <= kTaskMax that share a w-plane.  A persistent CTA pulls
// tasks from a device work queue.  For a task, in batches of kTaskMax, it
//   0. gathers the batch's placement records and visibilities through the
//      sort's index array (sorted position -> point),
//   1. orders the batch's visibilities by cell (and kernel row offset) and
//      turns each into a small tap record in shared memory, merging records
//      whose taps are identical,
//   2. reads kernel values through L1 (default) or, with staging on, copies
//      the W-row block of each kernel row offset into shared memory with
//      TMA bulk copies (cp.async.bulk + mbarrier) before that offset's run,
//   3. lets each thread own "classes" (a, b) in [0, W)^2: for every
//      visibility, the class's grid point is the unique footprint cell
//      (u, v) with u = a (mod W) and v = b (mod W).  Consecutive (spatially
//      sorted) visibilities mostly map a class to the same cell, so the
//      thread accumulates vis * kernel in registers and issues one atomic
//      (red.global.add.v2.f32, or two red.f64) only when its cell changes.
// Each grid cell receives exactly the reference's terms
//   grid[v][u] += vis * (conj ? conj(K) : K)(|off_v + j*os|, |off_u + k*os|)
// (oskar_grid_wproj.c:104-123), summed in a different order.
#include <algorithm>
#include <mutex>
#include <type_traits>

#include "common.cuh"
#include "grid_romein.cuh"
#include "internal.h"
#include "prep.cuh"
#include "task_order.cuh"

namespace b200 {
namespace {

template <typename GT> struct Vec2;
template <> struct Vec2<float> { using type = float2; };
template <> struct Vec2<double> { using type = double2; };

// Per-visibility tap record.  For a class (a, b) of a task with footprint W:
//   ru = (a + mu) mod W, rv = (b + mv) mod W   (offsets inside the footprint)
//   column = ru >= tu ? cp + ru : cn - ru      (slab column, see PlaneDesc)
//   kernel index = base + column + rv * pitch
//   cell         = origin + ru + rv * grid_size
// base: L1 path, the address of the visibility's first slab row (the points
// of a task may lie on several planes of one support); staged path, the index
// of that row in the plane's slab.
template <typename GT>
struct __align__(16) TapVis
{
    unsigned origin;
    int mu, mv, tu;
    int cp, cn;
    long long base;
    // re += c0.x * Kre + c1.x * Kim;  im += c0.y * Kre + c1.y * Kim
    typename Vec2<GT>::type c0, c1;
};

// A visibility as gathered from the caller's order: its placement record and
// its visibility (times its weight when asked for).
template <typename GT>
struct RawVis
{
    uint2 rec;
    typename Vec2<GT>::type vis;
};

// acc += c0 * k.x + c1 * k.y, component-wise, one rounding per product
// added (fma), in that order.  FP32: two packed fma.rn.f32x2 instead of
// four scalar fma, the same roundings.
__device__ __forceinline__ void cmac(float2& acc, const float2 c0,
                                     const float2 c1, const float2 k)
{
    acc = __ffma2_rn(c0, make_float2(k.x, k.x), acc);
    acc = __ffma2_rn(c1, make_float2(k.y, k.y), acc);
}

__device__ __forceinline__ void cmac(double2& acc, const double2 c0,
                                     const double2 c1, const double2 k)
{
    acc.x = fma(c0.x, k.x, acc.x);
    acc.x = fma(c1.x, k.y, acc.x);
    acc.y = fma(c0.y, k.x, acc.y);
    acc.y = fma(c1.y, k.y, acc.y);
}

// FP32 terms onto FP64 sums: each tap's two products are rounded to FP32
// (relative error 2^-23 of the tap, no larger than an FP32 running sum's
// rounding), their sum over the taps is not.
__device__ __forceinline__ void cmac(double2& acc, const float2 c0,
                                     const float2 c1, const float2 k)
{
    acc.x += (double)fmaf(c1.x, k.y, c0.x * k.x);
    acc.y += (double)fmaf(c1.y, k.y, c0.y * k.x);
}

// slabs: the cube's slab array (L1 path), or null (staged path).
template <typename GT, typename KT>
__device__ __forceinline__ TapVis<GT> derive(const int4 rec,
                                             const typename Vec2<GT>::type vis,
                                             const PlaneDesc& d,
                                             const KT* slabs, int grid_size,
                                             int oversample, int half,
                                             unsigned long long* status)
{
    TapVis<GT> t;
    const int s = d.support, w = 2 * s + 1, os = oversample;
    const int conj = rec.z < 0 ? -1 : 1;
    // Offsets lie in [-half, half] by construction; the clamp only guards
    // the slab bounds against a corrupted record.
    const int off_u = min(max((rec.w & 0xffff) - half, -half), half);
    const int off_v = min(max((rec.w >> 16) - half, -half), half);
    const int u0 = rec.x - s, v0 = rec.y - s;
    t.origin = (unsigned)u0 + (unsigned)v0 * (unsigned)grid_size;
    t.mu = (w - u0 % w) % w;
    t.mv = (w - v0 % w) % w;
    // Column taps k >= 0 (k >= 1 when off_u < 0) have off_u + k*os >= 0:
    // the ascending run of slab columns.
    t.tu = s + (off_u < 0 ? 1 : 0);
    const int rpu = ((off_u % os) + os) % os, rnu = ((-off_u % os) + os) % os;
    t.cp = rpu * d.L + (off_u - rpu) / os - s;
    t.cn = rnu * d.L + (-off_u - rnu) / os + s;
    // First of the W slab rows holding this row offset's taps.
    const int row = (off_v + half) * w * d.pitch;
    t.base = slabs ? (long long)(slabs + d.offset + row) : (long long)row;
    GT sc = (GT)d.scale;
    // The prep kernel only keeps points whose footprint lies inside the
    // grid; a record that breaks this is reported and neutralised (zero
    // weight at cell 0) so no flush can leave the grid.
    if (u0 < 0 || v0 < 0 || u0 + w > grid_size || v0 + w > grid_size)
    {
        atomicOr(status, (unsigned long long)DEV_ERR_GRID_INDEX);
        t.origin = 0;
        t.mu = t.mv = 0;
        sc = GT(0);
    }
    const GT vr = vis.x * sc, vi = vis.y * sc;
    t.c0.x = vr;
    t.c0.y = vi;
    t.c1.x = -(conj * vi);
    t.c1.y = conj * vr;
    return t;
}

// Predicated complex flush: one vector reduction when `pred` holds, no
// branch (the flush decision differs from lane to lane on most taps).
__device__ __forceinline__ void red_add_c_if(bool pred, float* addr, float re,
                                             float im)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %3, 0;\n\t"
                 "@p red.relaxed.gpu.global.add.v2.f32 [%0], {%1, %2};\n\t}"
                 :: "l"(addr), "f"(re), "f"(im), "r"((int)pred) : "memory");
}

__device__ __forceinline__ void red_add_c_if(bool pred, double* addr,
                                             double re, double im)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %3, 0;\n\t"
                 "@p red.relaxed.gpu.global.add.f64 [%0], %1;\n\t"
                 "@p red.relaxed.gpu.global.add.f64 [%4], %2;\n\t}"
                 :: "l"(addr), "d"(re), "d"(im), "r"((int)pred), "l"(addr + 1)
                 : "memory");
}

// Thread layout of one task.  The W x W classes are split into W columns
// (a) and ceil(W / CPT) row groups of CPT consecutive rows; a work item is
// one (column, row group) pair, so the column arithmetic of a tap is done
// once per visibility and shared by the item's CPT classes, and the 32
// lanes of a warp hold consecutive columns (contiguous kernel reads,
// coalesced flushes).  The last row group of a column is moved up to rows
// W - CPT .. W - 1 and its first slots, which repeat rows of the group
// before, are masked, so every slot reads an in-bounds kernel row.  When
// the items fit the CTA several times, `slices` copies of the layout split
// the task's visibilities between them; otherwise the CTA's threads take
// the items in passes of kGridThreads.  Against one column per thread with
// rows strided by the number of threads per column (the thread count per
// column capped at 256 / W, so wide footprints left up to a third of the
// CTA idle in their last pass), the plain_large gridding kernel went from
// 15.3 to 14.4 ms: fewer idle thread slots, and no per-slot row registers.
struct TaskLayout
{
    int items, slices, per_slice;
};

template <int CPT>
__device__ __forceinline__ TaskLayout task_layout(int w)
{
    TaskLayout t;
    t.items = w * ((w + CPT - 1) / CPT);
    if (t.items <= kGridThreads)
    {
        t.slices = kGridThreads / t.items;
        t.per_slice = t.items;
    }
    else
    {
        t.slices = 1;
        t.per_slice = kGridThreads;
    }
    return t;
}

// Grid flush policies.  PlainFlush: one predicated vector reduction.
// CompensatedFlush (FP32 grids): the running sums are FP64 and go to FP64
// planes of sums, one of the real and one of the imaginary parts, which are
// rounded to FP32 once, at the end of the job, and added to the grid's value in
// FP32.  Two fire-and-forget reductions of consecutive lanes replace the
// returning FP32 atomic whose rounding error (Knuth's TwoSum) was collected in
// an error grid: 3.4 M points on 4096^2, oversample 8, gridding 10.6 ->
// 5.1 ms, error against FP64 5.3e-8 -> 3.3e-8 (FP32 running sums with these
// reductions: 8e-8; 3 CTAs per SM instead of 4: 5.2 ms).  The sums take 16
// bytes per cell, the error grid took 8: where that much does not fit, the
// tasks run twice with one plane of sums (see pipeline.cu).
template <typename GT>
struct PlainFlush
{
    using Acc = typename Vec2<GT>::type;
    GT* grid;
    // FP32: the compare, the predicated reduction and the reset of the
    // running sum in one block of PTX.  When `valid` and cell != cur, the
    // sum goes to cur's grid cell and restarts from zero.
    __device__ __forceinline__ void flush_reset(int valid, unsigned cell,
                                                unsigned cur, float& ax,
                                                float& ay) const
    {
        asm volatile("{\n\t.reg .pred v, p;\n\t"
                     "setp.ne.s32 v, %5, 0;\n\t"
                     "setp.ne.and.u32 p, %2, %3, v;\n\t"
                     "@p red.relaxed.gpu.global.add.v2.f32 [%4], {%0, %1};\n\t"
                     "@p mov.f32 %0, 0f00000000;\n\t"
                     "@p mov.f32 %1, 0f00000000;\n\t}"
                     : "+f"(ax), "+f"(ay)
                     : "r"(cell), "r"(cur),
                       "l"(reinterpret_cast<float*>(grid) + 2 * (size_t)cur),
                       "r"(valid));
    }
    __device__ __forceinline__ void operator()(bool pred, unsigned cell, GT re,
                                               GT im) const
    {
        red_add_c_if(pred, grid + 2 * (size_t)cell, re, im);
    }
};

struct CompensatedFlush
{
    using Acc = double2;
    float* grid;
    double* re;    // sums of this pass, or null
    double* im;
    bool active;   // false: this task's cells are not compensated
    __device__ __forceinline__ void operator()(bool pred, unsigned cell,
                                               double x, double y) const
    {
        if (!pred) return;
        if (active)
        {
            if (re) red_add(re + cell, x);
            if (im) red_add(im + cell, y);
        }
        else if (re)
        {
            red_add_c(grid + 2 * (size_t)cell, (float)x, (float)y);
        }
    }
};

// One task: every class of the W x W footprint over the task's visibilities.
// Each class keeps a running sum for its current cell and flushes it when
// the cell changes (and at the end).  Every cell a class visits lies inside
// the grid: the prep kernel keeps only footprints inside the grid, derive()
// moves a record that breaks this to cell 0 with zero weight, and tasks
// whose footprint is wider than the grid are rejected before this point.
// Kernel values: read-only global memory (the L1 path, through the
// non-coherent load) or the staged shared-memory block.
template <bool GMEM, typename KT>
__device__ __forceinline__ KT load_kernel(const KT* p)
{
    if constexpr (GMEM) return __ldg(p);
    else return *p;
}

template <typename GT, typename KT, int CPT, bool STRAIGHT, bool COUNT,
          bool GMEM, typename FL>
__device__ __forceinline__ void process_task(const TapVis<GT>* __restrict__ s_vis,
                                             int m, int w, int pitch,
                                             int row_shift,
                                             const KT* __restrict__ slab,
                                             const FL& flush,
                                             int grid_size, unsigned& flushes)
{
    const TaskLayout lay = task_layout<CPT>(w);
    int slices = lay.slices < m ? lay.slices : m;
    const int r = threadIdx.x / lay.per_slice;
    if (r >= slices) return;
    const int l = threadIdx.x - r * lay.per_slice;
    const int i0 = (r * m) / slices, i1 = ((r + 1) * m) / slices;
    const unsigned pitch_b = (unsigned)pitch * (unsigned)sizeof(KT);
    for (int it = l; it < lay.items; it += kGridThreads)
    {
        const int a = it % w;
        // Rows b0 .. b0 + CPT - 1; slots q < skip repeat the previous
        // group's rows and never flush (CPT <= W).
        int b0 = (it / w) * CPT, skip = 0;
        if (b0 + CPT > w)
        {
            skip = b0 + CPT - w;
            b0 = w - CPT;
        }
        // Every slot runs the same straight-line code (a per-slot `break`
        // cost a branch and convergence barriers per tap: 19.9 -> 16.8 ms
        // at plain_large without it); masked slots never flush.
        using Acc = typename FL::Acc;
        Acc acc[CPT];                       // (re, im) of each row's cell
        // Of each slot: its footprint row, or (STRAIGHT) its cell.
        unsigned at[CPT];
        constexpr bool kFused =
            std::is_same<FL, PlainFlush<float>>::value && !COUNT;
        // In dense tasks most visibilities have the cell of the one before
        // (tasks hold all planes of a support, in cell order): their classes
        // stay where they are, and a branch the whole warp takes skips the row
        // wrap, the cell arithmetic and the flush.  What counts is that the
        // loads still come before the flush (after it, 39.2 M points 15.6 ->
        // 17.7 ms).  STRAIGHT has no such branch and takes two visibilities
        // per iteration.
        unsigned origin = s_vis[i0].origin, ru, cell0;
        {
            const unsigned mu = s_vis[i0].mu, xb = (unsigned)(b0 + s_vis[i0].mv);
            ru = min((unsigned)a + mu, (unsigned)a + mu - (unsigned)w);
            cell0 = origin + ru;
#pragma unroll
            for (int q = 0; q < CPT; ++q)
            {
                at[q] = min(xb + q, xb + q - (unsigned)w);
                if (STRAIGHT) at[q] = cell0 + at[q] * (unsigned)grid_size;
                acc[q].x = acc[q].y = 0;
            }
        }
#pragma unroll (STRAIGHT ? 2 : 1)
        for (int i = i0; i < i1; ++i)
        {
            const TapVis<GT> v = s_vis[i];
            // (a + mu) mod W for a + mu in [0, 2W): min over unsigned wraps
            const bool moved = STRAIGHT || v.origin != origin;
            unsigned rvn[CPT];
            if (moved)
            {
                ru = min((unsigned)(a + v.mu), (unsigned)(a + v.mu - w));
                const unsigned xb = (unsigned)(b0 + v.mv);
#pragma unroll
                for (int q = 0; q < CPT; ++q)
                    rvn[q] = min(xb + q, xb + q - (unsigned)w);
            }
            else
            {
#pragma unroll
                for (int q = 0; q < CPT; ++q) rvn[q] = at[q];
            }
            const int col = (int)ru >= v.tu ? v.cp + (int)ru : v.cn - (int)ru;
            // The kernel row base of this visibility's column, as a byte
            // address: each tap's address is then one wide multiply-add of
            // its row by the row pitch in bytes.
            const char* __restrict__ kp =
                (GMEM ? reinterpret_cast<const char*>(v.base)
                      : reinterpret_cast<const char*>(
                            slab + ((int)v.base - row_shift))) +
                (size_t)(unsigned)col * sizeof(KT);
            // All of this visibility's kernel values for the thread's rows
            // are requested before any is used.
            typename KernelLoad<KT>::Wide kv[CPT];
#pragma unroll
            for (int q = 0; q < CPT; ++q)
                kv[q] = KernelLoad<KT>::get(load_kernel<GMEM>(
                    reinterpret_cast<const KT*>(kp + (size_t)rvn[q] * pitch_b)));
            if (moved)
            {
                origin = v.origin;
                const unsigned cell1 = origin + ru;
#pragma unroll
                for (int q = 0; q < CPT; ++q)
                {
                    const unsigned cur =
                        STRAIGHT ? at[q] : cell0 + at[q] * (unsigned)grid_size;
                    const unsigned cell = cell1 + rvn[q] * (unsigned)grid_size;
                    if constexpr (kFused)
                        flush.flush_reset(q >= skip, cell, cur, acc[q].x,
                                          acc[q].y);
                    else
                    {
                        const bool change = q >= skip && cell != cur;
                        flush(change, cur, acc[q].x, acc[q].y);
                        if (COUNT) flushes += change;
                        acc[q].x = change ? 0 : acc[q].x;
                        acc[q].y = change ? 0 : acc[q].y;
                    }
                    at[q] = STRAIGHT ? cell : rvn[q];
                }
                cell0 = cell1;
            }
#pragma unroll
            for (int q = 0; q < CPT; ++q)
            {
                typename Vec2<GT>::type kk;
                kk.x = (GT)kv[q].x;
                kk.y = (GT)kv[q].y;
                cmac(acc[q], v.c0, v.c1, kk);
            }
        }
#pragma unroll
        for (int q = 0; q < CPT; ++q)
            flush(q >= skip,
                  STRAIGHT ? at[q] : cell0 + at[q] * (unsigned)grid_size,
                  acc[q].x, acc[q].y);
        if (COUNT) flushes += CPT - skip;
    }
}

template <typename GT, typename KT, bool STRAIGHT, bool COUNT, bool GMEM,
          typename FL>
__device__ __forceinline__ void dispatch_cpt(int cpt, const TapVis<GT>* s_vis,
                                             int m, int w, int pitch,
                                             int row_shift, const KT* slab,
                                             const FL& fl, int grid_size,
                                             unsigned& flushes)
{
#define B200_CPT(C)                                                         \
    process_task<GT, KT, C, STRAIGHT, COUNT, GMEM, FL>(                     \
        s_vis, m, w, pitch, row_shift, slab, fl, grid_size, flushes)
    // A row group never has more rows than the footprint (W = 1, 3, 5
    // take CPT = W).
    if (cpt > w) cpt = w;
    switch (cpt)
    {
    case 1: B200_CPT(1); break;
    case 2: B200_CPT(2); break;
    case 3: B200_CPT(3); break;
    case 4: B200_CPT(4); break;
    case 6: B200_CPT(6); break;
    default: B200_CPT(5); break;
    }
#undef B200_CPT
}

// moving: most tap records of the task lie at another cell than the one before.
// FP32 sums of FP32 data then take the straight-line code, else the code with
// the branch (see process_task).  Gridding with the branch everywhere, moving
// above a half, straight-line code everywhere:
//   39.2 M points on 8192^2, dense core        12.2, 12.0, 12.7 ms
//   24 channels on 2048^2                      2.27, 2.27, 2.35 ms
//   1.2 M spread over 3682^2, FP16, S 6..34    1.71, 1.46, 1.46 ms
//   20 x 0.42 M spread over 2048^2, S 6..34    5.63, 5.26, 5.35 ms
// A quarter or 0.7 instead of a half: 12.1 and 12.1 ms in the first, 5.31 and
// 5.30 in the last.  FP64 data always has the branch: it gains in dense tasks
// (1.9 M points 1799 -> 1631 us) and loses nothing in spread ones.  FP64 sums of
// FP32 data need more registers than it leaves (5.06 -> 7.8 ms).
// BOTH false: the branch only, in a kernel half as long, for calls of so few
// points that its start counts (10 thousand: 17.0 us against 17.9 with both).
template <typename GT, typename KT, bool BOTH, bool COUNT, bool GMEM,
          typename FL>
__device__ __forceinline__ void dispatch_task(bool moving, int cpt,
                                              const TapVis<GT>* s_vis, int m,
                                              int w, int pitch, int row_shift,
                                              const KT* slab, const FL& fl,
                                              int grid_size, unsigned& flushes)
{
    constexpr bool kFp64Data = std::is_same<GT, double>::value;
    constexpr bool kFp64Sums = std::is_same<typename FL::Acc, double2>::value;
    if constexpr (!kFp64Data && (kFp64Sums || BOTH))
        if (kFp64Sums || moving)
            return dispatch_cpt<GT, KT, true, COUNT, GMEM>(
                cpt, s_vis, m, w, pitch, row_shift, slab, fl, grid_size,
                flushes);
    if constexpr (kFp64Data || !kFp64Sums)
        dispatch_cpt<GT, KT, false, COUNT, GMEM>(cpt, s_vis, m, w, pitch,
                                                 row_shift, slab, fl,
                                                 grid_size, flushes);
}

template <typename GT, bool COMP> struct FlushFor { using type = PlainFlush<GT>; };
template <> struct FlushFor<float, true> { using type = CompensatedFlush; };

template <typename GT, bool COMP>
__device__ __forceinline__ typename FlushFor<GT, COMP>::type
make_flush(const JobDesc& jd, int comp_part, bool active)
{
    if constexpr (COMP)
        return CompensatedFlush{static_cast<float*>(jd.grid),
                                comp_part ? nullptr : jd.comp[0],
                                jd.comp[comp_part ? 0 : 1], active};
    else
        return PlainFlush<GT>{static_cast<GT*>(jd.grid)};
}

// At least grid_ctas_per_sm<GT>() CTAs per SM, with at most 6 rows per thread.
// 39.2 M FP32 points: 4 CTAs (64 registers) 15.6 ms, 3 16.6, 5 16.2.  1.9 M
// FP64 points: 3 CTAs (80 registers) 1692 us, 2 1860, 4 2406 (spills).
template <typename GT, typename KT, bool STAGED, bool COMP, bool COUNT,
          bool BOTH>
__global__ void __launch_bounds__(kGridThreads, grid_ctas_per_sm<GT>())
romein_grid_kernel(const GridArgs a)
{
    using V2 = typename Vec2<GT>::type;
    extern __shared__ __align__(128) unsigned char smem[];
    // [row block of the current run (STAGED)][tap records]
    KT* s_block = reinterpret_cast<KT*>(smem);
    TapVis<GT>* s_vis = reinterpret_cast<TapVis<GT>*>(
        smem + (STAGED ? a.block_smem_bytes : 0));
    // A batch's raw points lie at the end of the tap records, behind the
    // first kKeep (a place of their own cost 4 KB of L1 per CTA, 8 in FP64).
    constexpr int kKeep = kTaskMax - (int)((kTaskMax * sizeof(RawVis<GT>) +
                                            sizeof(TapVis<GT>) - 1) /
                                           sizeof(TapVis<GT>));
    RawVis<GT>* s_raw = reinterpret_cast<RawVis<GT>*>(s_vis + kKeep);
    // (see dispatch_task; the others have one loop, and nothing to count for it)
    constexpr bool kBoth = BOTH && sizeof(GT) == 4 && !COMP;
    __shared__ uint64_t s_bar;
    // The CTA's task: what is left of it when the classes run (kept here and
    // not in registers, which the tap loop needs).
    __shared__ struct
    {
        const JobDesc* job;
        uint32_t begin;   // its first sorted position
        int total;        // its points; -1: no task is left
        int done;         // points gathered
        int pending;      // merged points of the batch in s_raw
        int moves;        // tap records at another cell than the one before
        uint2 point;      // record of one of its points
    } s_task;
    __shared__ uint32_t s_order[kGridThreads];
    __shared__ int s_run_begin[kMaxOffsets], s_run_end[kMaxOffsets];
    __shared__ bool s_head[kTaskMax + 1];
    __shared__ int4 s_box[kGridThreads / 32];
    __shared__ int s_warp_heads[kGridThreads / 32];
    __shared__ int s_warp_moves[kGridThreads / 32];

    unsigned long long* status = &a.counters[CNT_STATUS];
    const unsigned num_tasks = tasks_listed(a.counters);
    unsigned long long first = 0, end = num_tasks;
    unsigned long long* queue = &a.counters[CNT_TASK_NEXT];
    if (a.range)
    {
        first = a.range[0];
        end = min((unsigned long long)a.range[1], end);
        queue = a.queue;
    }

    if (STAGED && threadIdx.x == 0)
    {
        mbar_init(&s_bar, 1);
        mbar_fence_init();
    }
    __syncthreads();

    uint32_t phase = 0;
    unsigned flushes = 0;
    const int t = threadIdx.x;
    if (t == 0) s_task.total = s_task.done = s_task.pending = 0;
    for (;;)
    {
        // Every thread has finished with the records, the row block and the
        // task before they are overwritten below.
        __syncthreads();
        if (kBoth && t == 0) s_task.moves = 0;
        if (t == 0 && s_task.pending == 0 && s_task.done == s_task.total)
        {
            const unsigned long long task = first + atomicAdd(queue, 1ull);
            s_task.done = 0;
            if (task >= end)
                s_task.total = -1;
            else
            {
                const uint32_t begin = a.task_start[task];
                const int total = (int)(a.task_start[task + 1] - begin);
                s_task.begin = begin;
                s_task.job = a.jobs + a.task_job[task];
                s_task.total = total;
                if (total <= 0 || total > (STAGED ? kTaskMax : kTaskRaw))
                {
                    atomicOr(status, (unsigned long long)DEV_ERR_TASK);
                    s_task.total = 0;
                }
            }
        }
        if (t < kMaxOffsets)
        {
            s_run_begin[t] = 0;
            s_run_end[t] = 0;
        }
        __syncthreads();
        const int total = s_task.total;
        if (total < 0) break;
        if (total == 0) continue;
        // The task's job: its cube, grid and geometry.
        const JobDesc& jd = *s_task.job;
        const uint32_t begin = s_task.begin;
        const KT* __restrict__ slabs = static_cast<const KT*>(jd.slabs);
        const PlaneDesc* __restrict__ planes = jd.planes;
        const int grid_size = jd.grid_size;
        // The task's points come in batches of at most kTaskMax.  A batch is
        // ordered, its points with identical placements are merged, and the
        // merged ones are appended to the tap records; the classes run when
        // the next batch does not fit any more.  Where many points share
        // their placement (dense cells near the uv origin) one run then
        // serves several batches: a quarter of the flushes into the densest
        // cells, whose FP32 sums are rounded that much less often (2.2 M
        // points on 3000^2: error against FP64 1.5e-6 -> 0.65e-6, gridding
        // 518 -> 508 us; one batch per task was 1 % faster on 39.2 M points,
        // 3 % on 24 channels).
        int done = s_task.done, pending = s_task.pending;
        int count = 0;     // tap records
        for (;;)
        {
            if (pending == 0)
            {
                if (done == total || count > kKeep) break;
                // Gather the batch (sorted positions begin + done ...)
                // straight from the caller's arrays: record, visibility
                // and weight of each point.  Against a separate pass that
                // permuted records and visibilities into sorted order:
                // plain_large step 19.15 -> 18.25 ms (the 1.6 ms pass
                // gone, the gridding kernel 0.7 ms slower; prefetching
                // the next task's points into L2 cost more than it hid).
                const int m = min(total - done, kTaskMax);
                int4 rec = make_int4(0, 0, 0, 0);
                if (t < m)
                {
                    const uint32_t i = a.order[begin + done + t];
                    RawVis<GT> rv;
                    rv.rec = a.rec[i];
                    const size_t local = i - jd.first;
                    const GT* __restrict__ vis =
                        static_cast<const GT*>(jd.vis);
                    GT re = vis[2 * local], im = vis[2 * local + 1];
                    if (a.apply_weight)
                    {
                        const GT wt =
                            static_cast<const GT*>(jd.weight)[local];
                        re *= wt;
                        im *= wt;
                    }
                    rv.vis.x = re;
                    rv.vis.y = im;
                    s_raw[t] = rv;
                    if (t == 0) s_task.point = rv.rec;
                    rec = unpack_record(rv.rec);
                }
                const TaskKey tk(jd.half, task_box(t < m, rec, s_box),
                                 sizeof(GT) == 8 ? m : 0);
                uint32_t key = 0xffffffffu;
                if (t < m) key = tk.template make<!STAGED>(rec, t);
                // Order the batch (see TaskKey): consecutive points are
                // neighbours.  (Its block barriers also publish the raw
                // records.)
                static_assert(kGridThreads >= 64,
                              "task_order has a block barrier");
                key = task_order(key, s_order);
                s_order[t] = key;
                __syncthreads();
                // Points with the same record read the same kernel values
                // into the same cells: the first of each run stands for
                // it with the sum of their visibilities.
                bool head = false, move = false;
                if (t < m)
                {
                    const uint2 r = s_raw[key & 0xffu].rec;
                    const uint2 q =
                        s_raw[s_order[t ? t - 1 : 0] & 0xffu].rec;
                    move = t == 0 || r.x != q.x;
                    head = move || r.y != q.y;
                }
                // (the end of the batch ends its last run)
                s_head[t] = head || t >= m;
                if (t == 0) s_head[kTaskMax] = true;
                const unsigned ball = __ballot_sync(0xffffffffu, head);
                if ((t & 31) == 0) s_warp_heads[t >> 5] = __popc(ball);
                if (kBoth)
                {
                    const unsigned moved = __ballot_sync(0xffffffffu, move);
                    if ((t & 31) == 0) s_warp_moves[t >> 5] = __popc(moved);
                }
                __syncthreads();
                for (int wi = 0; wi < kGridThreads / 32; ++wi)
                    pending += s_warp_heads[wi];
                done += m;
            }
            if (count + pending > kTaskMax) break;
            // Append the batch's merged points.
            const int batch = done - (done - 1) / kTaskMax * kTaskMax;
            const bool head = t < batch && s_head[t];
            const unsigned ball = __ballot_sync(0xffffffffu, head);
            int pos = count + __popc(ball & ((1u << (t & 31)) - 1u));
            for (int wi = 0; wi < (t >> 5); ++wi) pos += s_warp_heads[wi];
            TapVis<GT> tv;
            if (head)
            {
                RawVis<GT> rv = s_raw[s_order[t] & 0xffu];
                for (int q = t + 1; !s_head[q]; ++q)
                {
                    const RawVis<GT>& o = s_raw[s_order[q] & 0xffu];
                    rv.vis.x += o.vis.x;
                    rv.vis.y += o.vis.y;
                }
                const int4 rec = unpack_record(rv.rec);
                tv = derive<GT, KT>(rec, rv.vis,
                                    planes[rec.z & 0x7fffffff],
                                    STAGED ? nullptr : slabs, grid_size,
                                    jd.oversample, jd.half, status);
            }
            const uint32_t key = s_order[t];
            if (kBoth && t == 0)
                for (int wi = 0; wi < kGridThreads / 32; ++wi)
                    s_task.moves += s_warp_moves[wi];
            __syncthreads();   // the raw batch is read
            if (head) s_vis[pos] = tv;
            if (STAGED)
            {
                // The runs of each row offset in the merged order.
                if (head) s_order[pos] = key;
                __syncthreads();
                if (t < pending)
                {
                    const TaskKey tk(jd.half, make_int4(0, 0, 0, 0));
                    const int ov = tk.row_offset(s_order[t]);
                    if (t == 0 || tk.row_offset(s_order[t - 1]) != ov)
                        s_run_begin[ov] = t;
                    if (t == pending - 1 ||
                        tk.row_offset(s_order[t + 1]) != ov)
                        s_run_end[ov] = t + 1;
                }
            }
            __syncthreads();
            count += pending;
            pending = 0;
        }
        // Any point of the task tells its geometry (its planes share it).
        const uint2 r0 = s_task.point;
        const PlaneDesc d = planes[r0.y & 0x7fffu];
        const int w = 2 * d.support + 1, offsets = 2 * jd.half + 1;
        if (t == 0)
        {
            s_task.done = done;
            s_task.pending = pending;
        }
        // No kept footprint is wider than its grid; a task that says
        // otherwise is malformed (and its cells could leave the grid).
        if (w > grid_size)
        {
            if (t == 0) atomicOr(status, (unsigned long long)DEV_ERR_TASK);
            continue;
        }
        const int cpt = d.support < kTuneMax ? a.cpt[d.support] : 5;
        // Compensation is limited to tasks near the grid centre when a radius
        // is set (a task is a compact run of one coarse tile).
        bool comp_here = true;
        if (COMP && a.comp_radius > 0)
        {
            const int c = grid_size / 2;
            comp_here = abs((int)(r0.x & 0xffffu) - c) <= a.comp_radius &&
                        abs((int)(r0.x >> 16) - c) <= a.comp_radius;
        }
        const auto fl = make_flush<GT, COMP>(jd, a.comp_part, comp_here);
        if (!STAGED)
        {
            dispatch_task<GT, KT, kBoth, COUNT, true>(
                kBoth && 2 * s_task.moves > count, cpt, s_vis, count, w, d.pitch, 0,
                slabs, fl, grid_size, flushes);
            continue;
        }
        const unsigned block_elems = (unsigned)w * (unsigned)d.pitch;
        const unsigned block_bytes = block_elems * (unsigned)sizeof(KT);
        for (int ov = 0; ov < offsets; ++ov)
        {
            const int rb = s_run_begin[ov], re = s_run_end[ov];
            if (re <= rb) continue;
            if (threadIdx.x == 0)
            {
                // Every thread finished reading the previous block (barrier
                // below / above); order that before the async-proxy write.
                fence_proxy_async_shared();
                mbar_arrive_expect_tx(&s_bar, block_bytes);
                const unsigned char* src = reinterpret_cast<const unsigned char*>(
                    slabs + d.offset + (long long)ov * block_elems);
                for (unsigned off = 0; off < block_bytes; off += kBulkChunk)
                    bulk_copy_g2s(reinterpret_cast<unsigned char*>(s_block) + off,
                                  src + off, min(kBulkChunk, block_bytes - off),
                                  &s_bar);
            }
            const bool ok = mbar_wait_bounded(&s_bar, phase);
            if (!__syncthreads_and(ok))
            {
                // Record the failure, let the copy drain (bounded), leave.
                if (threadIdx.x == 0)
                    atomicOr(status, (unsigned long long)DEV_ERR_TIMEOUT);
                mbar_wait_bounded(&s_bar, phase);
                return;
            }
            phase ^= 1u;
            dispatch_task<GT, KT, kBoth, COUNT, false>(
                kBoth && 2 * s_task.moves > count, cpt, s_vis + rb, re - rb, w, d.pitch,
                ov * (int)block_elems, s_block, fl, grid_size, flushes);
            __syncthreads();
        }
    }
    if (COUNT)
    {
        const unsigned long long f = warp_sum((unsigned long long)flushes);
        if ((threadIdx.x & 31) == 0 && f)
            atomicAdd(&a.counters[CNT_FLUSHES], f);
    }
}

template <typename GT, typename KT, bool STAGED, bool COMP = false,
          bool COUNT = false, bool BOTH = true>
cudaError_t launch_variant(const GridArgs& a, int num_sms, size_t smem,
                           cudaStream_t st, int* ctas_out)
{
    auto fn = romein_grid_kernel<GT, KT, STAGED, COMP, COUNT, BOTH>;
    // Function attributes and occupancy are looked up once per (variant,
    // device, shared-memory size), not on every launch.
    static std::mutex mu;
    static int cached_dev = -1;
    static size_t cached_smem = 0;
    static int cached_per_sm = 0;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    {
        std::lock_guard<std::mutex> lock(mu);
        if (dev == cached_dev && smem == cached_smem)
        {
            per_sm = cached_per_sm;
        }
        else
        {
            e = cudaFuncSetAttribute(
                fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            if (e != cudaSuccess) return e;
            if (!STAGED)
            {
                // Only the shared memory grid_ctas_per_sm CTAs need; the
                // rest of the SM's unified L1/shared storage caches kernel
                // values (measured 19.88 -> 19.66 ms at plain_large against
                // the default carveout).
                cudaFuncAttributes fa{};
                e = cudaFuncGetAttributes(&fa, fn);
                if (e != cudaSuccess) return e;
                const size_t per = smem + fa.sharedSizeBytes + 1024;
                int pct = (int)((100 * grid_ctas_per_sm<GT>() * per +
                                 228 * 1024 - 1) /
                                (228 * 1024));
                pct = pct > 100 ? 100 : pct;
                e = cudaFuncSetAttribute(
                    fn, cudaFuncAttributePreferredSharedMemoryCarveout, pct);
                if (e != cudaSuccess) return e;
            }
            e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                &per_sm, fn, kGridThreads, smem);
            if (e != cudaSuccess) return e;
            cached_dev = dev;
            cached_smem = smem;
            cached_per_sm = per_sm;
        }
    }
    if (per_sm < 1) return cudaErrorInvalidConfiguration;
    const int ctas = num_sms * per_sm;
    if (ctas_out) *ctas_out = ctas;
    fn<<<ctas, kGridThreads, smem, st>>>(a);
    return cudaGetLastError();
}

}  // namespace

// Rows-per-thread (CPT) for each support, from a cost model of
// process_task: per visibility a thread does ~12 instructions of shared
// column work plus ~20 per class, so the cost of a tap is
// (12 / CPT + 20) / utilisation, utilisation being the fraction of the
// CTA's thread slots (threads x CPT x passes) holding a live class under
// the (column, row group) layout of process_task.  (Modelled on FP32 sums; FP64
// data and FP64 sums, twice as wide in registers, take the same table.)
void default_tune_table(unsigned char* cpt)
{
    const int choices[] = {1, 2, 3, 4, 5, 6};
    for (int s = 0; s < kTuneMax; ++s)
    {
        const int w = 2 * s + 1;
        double best = 1e30;
        int pick = 1;
        for (int c : choices)
        {
            if (c > w) continue;
            const int items = w * ((w + c - 1) / c);
            const int slices = items <= kGridThreads ? kGridThreads / items : 1;
            const int passes = (items + kGridThreads - 1) / kGridThreads;
            const double util = (double)w * w * slices /
                                ((double)kGridThreads * c * passes);
            const double cost = (12.0 / c + 20.0) / util;
            if (cost < best - 1e-9)
            {
                best = cost;
                pick = c;
            }
        }
        cpt[s] = (unsigned char)pick;
    }
}

namespace {

// Block (x, j) adds part of job j's FP64 sums to its grid (jobs of a batch
// may share a grid: a reduction per cell).
__global__ void fold_kernel(const JobDesc* __restrict__ jobs, int comp_part)
{
    const JobDesc& jd = jobs[blockIdx.y];
    const double* re = comp_part ? nullptr : jd.comp[0];
    const double* im = jd.comp[comp_part ? 0 : 1];
    float* grid = static_cast<float*>(jd.grid);
    const size_t cells = (size_t)jd.grid_size * (size_t)jd.grid_size;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < cells;
         i += (size_t)gridDim.x * blockDim.x)
    {
        const float x = re ? (float)re[i] : 0.f, y = im ? (float)im[i] : 0.f;
        if (x != 0.f || y != 0.f) red_add_c(grid + 2 * i, x, y);
    }
}

}  // namespace

cudaError_t launch_fold_jobs(const JobDesc* jobs, int num_jobs, int comp_part,
                             int num_sms, cudaStream_t st)
{
    int bx = num_sms * 8 / (num_jobs > 0 ? num_jobs : 1);
    if (bx < 4) bx = 4;
    fold_kernel<<<dim3(bx, num_jobs), 256, 0, st>>>(jobs, comp_part);
    return cudaGetLastError();
}

size_t grid_smem_bytes(int data_is_double, unsigned max_block_bytes,
                       bool staged)
{
    const size_t rec = data_is_double ? sizeof(TapVis<double>)
                                      : sizeof(TapVis<float>);
    const size_t block = staged ? ((max_block_bytes + 127) / 128) * 128 : 0;
    return block + rec * kTaskMax;
}

cudaError_t launch_grid(const GridArgs& a, int data_is_double,
                        int kernel_type, unsigned max_block_bytes, bool staged,
                        bool compensated, int num_sms, cudaStream_t st,
                        int* ctas_out)
{
    const size_t smem = grid_smem_bytes(data_is_double, max_block_bytes,
                                        staged);
    GridArgs args = a;
    args.block_smem_bytes = staged ? (unsigned)(((max_block_bytes + 127) /
                                                  128) * 128)
                                    : 0u;
    if (compensated)
    {
        // FP32 grids only; kernel values read through L1.
        if (data_is_double || staged) return cudaErrorInvalidValue;
        switch (kernel_type)
        {
        case OSKAR_B200_KERNEL_F16:
            return a.count_flushes
                ? launch_variant<float, __half2, false, true, true>(args, num_sms, smem, st, ctas_out)
                : launch_variant<float, __half2, false, true>(args, num_sms, smem, st, ctas_out);
        case OSKAR_B200_KERNEL_BF16:
            return a.count_flushes
                ? launch_variant<float, __nv_bfloat162, false, true, true>(args, num_sms, smem, st, ctas_out)
                : launch_variant<float, __nv_bfloat162, false, true>(args, num_sms, smem, st, ctas_out);
        default:
            return a.count_flushes
                ? launch_variant<float, float2, false, true, true>(args, num_sms, smem, st, ctas_out)
                : launch_variant<float, float2, false, true>(args, num_sms, smem, st, ctas_out);
        }
    }
    // Flushes are counted (statistics) on the L1 path only.
    const bool count = a.count_flushes && !staged;
    if (data_is_double)
    {
        if (kernel_type != OSKAR_B200_KERNEL_NATIVE)
            return cudaErrorInvalidValue;
        if (staged) return launch_variant<double, double2, true>(args, num_sms, smem, st, ctas_out);
        return count ? launch_variant<double, double2, false, false, true>(args, num_sms, smem, st, ctas_out)
                     : launch_variant<double, double2, false>(args, num_sms, smem, st, ctas_out);
    }
    if (a.few_points && !staged && !count)
        switch (kernel_type)
        {
        case OSKAR_B200_KERNEL_F16:
            return launch_variant<float, __half2, false, false, false, false>(args, num_sms, smem, st, ctas_out);
        case OSKAR_B200_KERNEL_BF16:
            return launch_variant<float, __nv_bfloat162, false, false, false, false>(args, num_sms, smem, st, ctas_out);
        default:
            return launch_variant<float, float2, false, false, false, false>(args, num_sms, smem, st, ctas_out);
        }
    switch (kernel_type)
    {
    case OSKAR_B200_KERNEL_F16:
        if (staged) return launch_variant<float, __half2, true>(args, num_sms, smem, st, ctas_out);
        return count ? launch_variant<float, __half2, false, false, true>(args, num_sms, smem, st, ctas_out)
                     : launch_variant<float, __half2, false>(args, num_sms, smem, st, ctas_out);
    case OSKAR_B200_KERNEL_BF16:
        if (staged) return launch_variant<float, __nv_bfloat162, true>(args, num_sms, smem, st, ctas_out);
        return count ? launch_variant<float, __nv_bfloat162, false, false, true>(args, num_sms, smem, st, ctas_out)
                     : launch_variant<float, __nv_bfloat162, false>(args, num_sms, smem, st, ctas_out);
    default:
        if (staged) return launch_variant<float, float2, true>(args, num_sms, smem, st, ctas_out);
        return count ? launch_variant<float, float2, false, false, true>(args, num_sms, smem, st, ctas_out)
                     : launch_variant<float, float2, false>(args, num_sms, smem, st, ctas_out);
    }
}

}  // namespace b200
