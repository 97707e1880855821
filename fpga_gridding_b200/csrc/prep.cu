// Per-visibility preparation of a batch of jobs: placement (grid cell,
// w-plane, oversample offsets, conjugation, skip test) exactly as
// oskar_grid_wproj.c:70-101 computes it, the sort key, the skip counts, the
// norms and the grid updates; then, after the sort, the gridding work
// list (tasks).
#include <algorithm>
#include <vector>

#include "common.cuh"
#include "internal.h"
#include "prep.cuh"

namespace b200 {

// Sort key bits (skip flag included) that the fine cell index may fill: whole
// passes of the sort.  Fewer bits put points of a wider block into a task in
// arrival order, which its own sort cannot undo: its columns are then swept
// again and again, and the densest cells take more roundings.  One B200, 16 /
// 24 / 32 bits: 10 thousand points, sort 30 / 38 / 38 us, gridding 16 us each;
// 0.24 M, 32 / 46 / 57 and 68 / 45 / 45 us; 2.2 M, 77 / 108 / 136 and 703 /
// 541 / 508 us, error against FP64 1.5e-6 with 24 bits, 0.65e-6 with 32;
// 39.2 M, 0.70 / 1.04 / 1.36 and 29.4 / 18.8 / 16.2 ms.  (Single jobs.  The job
// field of a batch comes out of the same bits: against the build before, which
// always had 31, batches of 16 to 200 jobs of 1 to 60 thousand points take 0.74
// to 0.92 of the time, with errors of 0.70 to 1.03; the lines were not measured
// for batches by themselves.)
static int key_bits(size_t num_points)
{
    return num_points <= (size_t(1) << 14)   ? 16
           : num_points <= (size_t(1) << 18) ? 24
                                             : 32;
}

std::vector<int> assign_groups(PlaneDesc* planes, int num_planes)
{
    std::vector<int> s((size_t)num_planes);
    for (int p = 0; p < num_planes; ++p) s[p] = planes[p].support;
    std::sort(s.begin(), s.end());
    s.erase(std::unique(s.begin(), s.end()), s.end());
    for (int p = 0; p < num_planes; ++p)
        planes[p].group = (int)(std::lower_bound(s.begin(), s.end(),
                                                 planes[p].support) -
                                s.begin());
    return s;
}

bool make_key_layout(int grid_size, int num_planes, int num_jobs,
                     size_t num_points, KeyLayout* out, int tile_shift,
                     int num_groups)
{
    KeyLayout k{};
    int gbits = 0;
    while ((1 << gbits) < grid_size) ++gbits;
    // Coarse tiles: at most 16 per axis and at least 64 cells wide, so the
    // visibilities in flight at any time touch a few coarse tiles of grid
    // (or the width asked for, within 64 cells and the grid).
    k.coarse_shift = gbits - 4 > 6 ? gbits - 4 : 6;
    if (tile_shift > 0)
        k.coarse_shift = std::max(6, std::min(tile_shift, std::max(gbits, 6)));
    const int ctiles = (grid_size + (1 << k.coarse_shift) - 1) >> k.coarse_shift;
    while ((1 << k.coarse_bits) < ctiles) ++k.coarse_bits;
    int plane_bits = 0;
    while ((1 << plane_bits) < num_planes) ++plane_bits;
    k.by_plane = num_groups == 0;
    if (k.by_plane) num_groups = num_planes;
    while ((1 << k.group_bits) < num_groups) ++k.group_bits;
    while ((1 << k.job_bits) < num_jobs) ++k.job_bits;
    k.fine_shift = 0;
    k.fine_bits = k.coarse_shift;
    // (The same jobs are refused whatever the grouping.)
    if (k.job_bits + 2 * k.coarse_bits + plane_bits + 1 > 32) return false;
    const int fixed = k.job_bits + 2 * k.coarse_bits + k.group_bits + 1;
    const int bits = key_bits(num_points);
    while (fixed + 2 * k.fine_bits > bits && k.fine_bits > 0)
    {
        ++k.fine_shift;
        --k.fine_bits;
    }
    k.job_shift = 2 * k.coarse_bits + k.group_bits + 2 * k.fine_bits;
    k.total_bits = k.job_shift + k.job_bits;
    *out = k;
    return true;
}

int prep_blocks_per_job(size_t max_points, int num_jobs, int num_sms)
{
    const size_t need = (max_points + 255) / 256;
    size_t want = (size_t)num_sms * 8 / (size_t)(num_jobs > 0 ? num_jobs : 1);
    if (want < 1) want = 1;
    if (want > need) want = need > 0 ? need : 1;
    return (int)want;
}

namespace {

constexpr int kPrepThreads = 256;

// Spreads the low 16 bits of x to the even bit positions.
__device__ __forceinline__ uint32_t spread_bits(uint32_t x)
{
    x &= 0xffffu;
    x = (x | (x << 8)) & 0x00ff00ffu;
    x = (x | (x << 4)) & 0x0f0f0f0fu;
    x = (x | (x << 2)) & 0x33333333u;
    x = (x | (x << 1)) & 0x55555555u;
    return x;
}

__device__ __forceinline__ uint32_t make_key(const KeyLayout& k, int job,
                                             int gu, int gv, int group)
{
    const uint32_t cu = (uint32_t)gu >> k.coarse_shift;
    const uint32_t cv = (uint32_t)gv >> k.coarse_shift;
    const uint32_t in_mask = (1u << k.coarse_shift) - 1u;
    const uint32_t fu = ((uint32_t)gu & in_mask) >> k.fine_shift;
    const uint32_t fv = ((uint32_t)gv & in_mask) >> k.fine_shift;
    // Coarse tiles in row-major order: tasks of one row of tiles are
    // contiguous, so a band of grid rows is complete once its tasks and its
    // neighbours' are (the drop-in streams such bands back to the host).
    const uint32_t coarse = (cv << k.coarse_bits) | cu;
    const uint32_t fine = spread_bits(fu) | (spread_bits(fv) << 1);
    return ((uint32_t)job << k.job_shift) |
           (coarse << (k.group_bits + 2 * k.fine_bits)) |
           ((uint32_t)group << (2 * k.fine_bits)) | fine;
}

__device__ __forceinline__ PlaceConsts place_consts(const JobDesc& jd)
{
    PlaceConsts pc;
    pc.grid_scale = jd.grid_scale;
    pc.w_scale = jd.w_scale;
    pc.grid_scale_f = jd.grid_scale_f;
    pc.w_scale_f = jd.w_scale_f;
    pc.grid_size = jd.grid_size;
    pc.centre = jd.grid_size / 2;
    pc.num_planes = jd.num_planes;
    pc.oversample = jd.oversample;
    return pc;
}

// One point per thread and step.  The grid updates are summed per thread from
// the supports; a histogram of planes by __match_any_sync and 16 KB of shared
// counters, summed at the end, cost a tenth: 39.2 M FP32 points 441 -> 395 us,
// 15.7 M 187 -> 168.  Bounded to 5, 6, 8 blocks per SM (48, 40, 32 registers):
// 474, 467, 438 us against 395 unbounded (60 registers).  What must be moved
// takes 144 us; the FP64 placement has the rest.
template <typename T, int MODE>
__global__ void __launch_bounds__(kPrepThreads)
prep_kernel(const __grid_constant__ PrepArgs a)
{
    const int job = blockIdx.y;
    const JobDesc& jd = a.job_out ? a.job : a.jobs[job];
    static_assert(sizeof(JobDesc) % 4 == 0 &&
                  sizeof(JobDesc) / 4 <= kPrepThreads, "a word per thread");
    if (a.job_out && blockIdx.x == 0 && threadIdx.x < sizeof(JobDesc) / 4)
        reinterpret_cast<uint32_t*>(a.job_out)[threadIdx.x] =
            reinterpret_cast<const uint32_t*>(&a.job)[threadIdx.x];
    const T* __restrict__ uu = static_cast<const T*>(jd.uu);
    const T* __restrict__ vv = static_cast<const T*>(jd.vv);
    const T* __restrict__ ww = static_cast<const T*>(jd.ww);
    const T* __restrict__ wt = static_cast<const T*>(jd.weight);
    const PlaceConsts pc = place_consts(jd);
    const PlaneDesc* __restrict__ planes = jd.planes;
    const double* __restrict__ norm_table = jd.norm_table;
    const int* __restrict__ support = jd.support;
    const CoordScale scale = coord_scale(jd);
    const int half = jd.half;
    const unsigned long long first = jd.first, n = jd.n;
    __shared__ double s_norm[kPrepThreads / 32];
    __shared__ unsigned s_skip[kPrepThreads / 32];
    __shared__ unsigned long long s_updates[kPrepThreads / 32];

    const int span = 2 * half + 1;
    const uint32_t skip_key = 1u << a.key.total_bits;
    const int lane = threadIdx.x & 31;
    double norm = 0.0;
    unsigned skipped = 0;
    unsigned long long updates = 0;   // taps of the kept points
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t base = (size_t)blockIdx.x * blockDim.x; base < n;
         base += stride)
    {
        const size_t i = base + threadIdx.x;
        const bool in_range = i < n;
        const size_t g = first + i;
        Placed p{};
        if (in_range)
            p = place_one<T, MODE>(scale_coord(uu[i], scale),
                                   scale_coord(vv[i], scale),
                                   scale_coord(ww[i], scale), pc, support);
        const bool keep = in_range && !p.skipped;
        if (in_range)
        {
            if (keep)
            {
                a.rec[g] = pack_record(p, half);
                a.keys[g] = make_key(a.key, job, p.gu, p.gv,
                                     a.key.by_plane
                                         ? p.plane : planes[p.plane].group);
                double s = norm_table[((size_t)p.plane * span +
                                          (p.off_v + half)) * span +
                                         (p.off_u + half)];
                if (a.apply_weight) s *= (double)wt[i];
                norm += s;
                const unsigned w = 2u * (unsigned)p.support + 1u;
                updates += w * w;
            }
            else
            {
                a.keys[g] = skip_key;
            }
        }
        skipped += in_range && !keep;
    }
    norm = warp_sum(norm);
    skipped = warp_sum(skipped);
    updates = warp_sum(updates);
    if (lane == 0)
    {
        s_norm[threadIdx.x >> 5] = norm;
        s_skip[threadIdx.x >> 5] = skipped;
        s_updates[threadIdx.x >> 5] = updates;
    }
    __syncthreads();
    if (threadIdx.x == 0)
    {
        double t = 0.0;
        unsigned long long k = 0, u = 0;
        for (int w = 0; w < kPrepThreads / 32; ++w)
        {
            t += s_norm[w];
            k += s_skip[w];
            u += s_updates[w];
        }
        if (u) atomicAdd(&a.counters[CNT_UPDATES], u);
        a.norm_partials[(size_t)job * gridDim.x + blockIdx.x] = t;
        if (k)
        {
            atomicAdd(&a.job_skipped[job], k);
            atomicAdd(&a.counters[CNT_SKIPPED], k);
        }
    }
    // The job's last block sums its norm partials in a fixed order
    // (deterministic), adds them to the caller's norm and publishes the skip
    // count.  (As a kernel of its own this took a launch and 4 us.)
    __shared__ bool s_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0)
        s_last = atomicAdd(&a.job_tickets[job], 1u) == gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    norm = 0.0;
    for (unsigned k = threadIdx.x; k < gridDim.x; k += kPrepThreads)
        norm += __ldcg(&a.norm_partials[(size_t)job * gridDim.x + k]);
    norm = warp_sum(norm);
    if (lane == 0) s_norm[threadIdx.x >> 5] = norm;
    __syncthreads();
    if (threadIdx.x == 0)
    {
        double t = 0.0;
        for (int w = 0; w < kPrepThreads / 32; ++w) t += s_norm[w];
        if (jd.d_norm) *jd.d_norm += t;
        if (jd.d_skipped) *jd.d_skipped = __ldcg(&a.job_skipped[job]);
    }
}

// Task list in one pass over the sorted keys, in tiles of kTaskTile positions:
// each tile counts its task starts, finds the starts of the tiles before it by
// chained scan (a tile's word holds its own count until it knows the sum up to
// it; 32 earlier words are read at once) and writes its starts.  A task starts
// at sorted position s < valid when s == 0, at every multiple of its group's
// task size, or where the key above the fine cell bits changes.  (Counting,
// a three-launch scan and writing took 34 us for 10 thousand points and 260 us
// for 39 M.)
constexpr int kTaskTile = 4096;
constexpr int kTaskThreads = 256;
constexpr int kTaskRounds = kTaskTile / kTaskThreads;
constexpr int kTaskWarps = kTaskThreads / 32;

// Sum of tile words [0, tile) by one warp; false when the bounded wait
// expired.  Word: flag (1: the tile's count, 2: all tiles up to it) << 62 |
// count.
__device__ __forceinline__ bool tasks_before(const unsigned long long* state,
                                             unsigned tile, unsigned* sum)
{
    const int lane = threadIdx.x & 31;
    unsigned total = 0, end = tile, spins = 0;
    while (end > 0)
    {
        const unsigned long long w =
            (unsigned)lane < end
                ? *((const volatile unsigned long long*)state + (end - 1 - lane))
                : 2ull << 62;
        const unsigned pending = __ballot_sync(0xffffffffu, (w >> 62) == 0);
        const unsigned prefix = __ballot_sync(0xffffffffu, (w >> 62) == 2);
        // words before the first pending one, up to the first prefix
        const int usable = min(pending ? __ffs(pending) - 1 : 32,
                               prefix ? __ffs(prefix) : 32);
        total += __reduce_add_sync(
            0xffffffffu, lane < usable ? (unsigned)(w & 0xffffffffull) : 0u);
        if (prefix && __ffs(prefix) <= usable) break;
        end -= (unsigned)usable;
        if (usable == 0 && ++spins > kSpinLimit) return false;
    }
    *sum = total;
    return true;
}

__global__ void __launch_bounds__(kTaskThreads)
task_list_kernel(const uint32_t* __restrict__ keys, size_t n,
                 unsigned long long* __restrict__ counters, int fine_key_bits,
                 const TaskSizes sizes, int job_shift,
                 unsigned long long* state, unsigned expired_tile,
                 uint32_t* __restrict__ task_start,
                 uint32_t* __restrict__ task_job)
{
    __shared__ unsigned s_tile, s_base;
    __shared__ unsigned s_w[kTaskRounds][kTaskWarps];
    // A sort that gave up leaves no tasks (counters[CNT_TASKS] stays zero).
    if (threadIdx.x == 0)
        s_tile = counters[CNT_STATUS] & DEV_ERR_TIMEOUT
                     ? 0xffffffffu
                     : (unsigned)atomicAdd(&counters[CNT_TASK_TILE], 1ull);
    __syncthreads();
    const unsigned tile = s_tile;
    if (tile == 0xffffffffu) return;
    const size_t valid = n - counters[CNT_SKIPPED];
    const size_t tile0 = (size_t)tile * kTaskTile;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // rounds of kTaskThreads consecutive positions, in order
    unsigned ball[kTaskRounds];
    uint32_t key[kTaskRounds], edge[kTaskRounds];
#pragma unroll
    for (int r = 0; r < kTaskRounds; ++r)
    {
        const size_t s = tile0 + (size_t)r * kTaskThreads + threadIdx.x;
        key[r] = s < valid ? keys[s] : 0u;
        edge[r] = lane == 0 && s > 0 && s < valid ? keys[s - 1] : 0u;
    }
#pragma unroll
    for (int r = 0; r < kTaskRounds; ++r)
    {
        const size_t s = tile0 + (size_t)r * kTaskThreads + threadIdx.x;
        const uint32_t up = __shfl_up_sync(0xffffffffu, key[r], 1);
        const uint32_t prev = (lane ? up : edge[r]) >> fine_key_bits;
        const uint32_t k = key[r] >> fine_key_bits;
        const uint32_t low =
            (1u << sizes.log2_max[k & sizes.group_mask]) - 1u;
        ball[r] = __ballot_sync(0xffffffffu, s < valid &&
                                (s == 0 || k != prev ||
                                 ((uint32_t)s & low) == 0));
        if (lane == 0) s_w[r][warp] = __popc(ball[r]);
    }
    __syncthreads();
    if (warp == 0)
    {
        // Exclusive scan of the tile's warp counts, 4 per lane.
        static_assert(kTaskRounds * kTaskWarps == 128, "4 counts per lane");
        unsigned* w = &s_w[0][0] + 4 * lane;
        const unsigned c0 = w[0], c1 = w[1], c2 = w[2], c3 = w[3];
        unsigned inc = c0 + c1 + c2 + c3;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
        {
            const unsigned t = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += t;
        }
        const unsigned ex = inc - (c0 + c1 + c2 + c3);
        w[0] = ex;
        w[1] = ex + c0;
        w[2] = ex + c0 + c1;
        w[3] = ex + c0 + c1 + c2;
        const unsigned total = __shfl_sync(0xffffffffu, inc, 31);
        volatile unsigned long long* word = state + tile;
        if (lane == 0) *word = (tile ? 1ull : 2ull) << 62 | total;
        unsigned before = 0;
        const bool ok = tile != expired_tile &&
                        tasks_before(state, tile, &before);
        if (lane == 0)
        {
            if (ok)
                *word = 2ull << 62 | (before + total);
            else
                atomicOr(&counters[CNT_STATUS],
                         (unsigned long long)DEV_ERR_TIMEOUT);
            s_base = ok ? before : 0xffffffffu;
            if (ok && tile == gridDim.x - 1)
            {
                counters[CNT_TASKS] = before + total;
                task_start[before + total] = (uint32_t)valid;
            }
        }
    }
    __syncthreads();
    const unsigned base = s_base;
    if (base == 0xffffffffu) return;
#pragma unroll
    for (int r = 0; r < kTaskRounds; ++r)
        if ((ball[r] >> lane) & 1u)
        {
            const size_t pos = tile0 + (size_t)r * kTaskThreads + threadIdx.x;
            const uint32_t t = base + s_w[r][warp] +
                               __popc(ball[r] & ((1u << lane) - 1u));
            task_start[t] = (uint32_t)pos;
            task_job[t] = key[r] >> job_shift;
        }
}

// Placement only, for inspection (oskar_b200_place).
template <typename T, int MODE>
__global__ void place_kernel(const T* __restrict__ uu, const T* __restrict__ vv,
                             const T* __restrict__ ww, size_t n,
                             PlaceConsts pc, const int* __restrict__ support,
                             int32_t* gu, int32_t* gv, int32_t* plane,
                             int32_t* off_u, int32_t* off_v, int32_t* conj,
                             int32_t* skipped)
{
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x)
    {
        const Placed p = place_one<T, MODE>(uu[i], vv[i], ww[i], pc, support);
        if (gu) gu[i] = p.gu_report;
        if (gv) gv[i] = p.gv_report;
        if (plane) plane[i] = p.plane;
        if (off_u) off_u[i] = p.off_u;
        if (off_v) off_v[i] = p.off_v;
        if (conj) conj[i] = p.conj;
        if (skipped) skipped[i] = p.skipped;
    }
}

unsigned grid_blocks(size_t n, int num_sms, int per_sm, int threads)
{
    const size_t need = (n + threads - 1) / threads;
    const size_t cap = (size_t)num_sms * per_sm;
    return (unsigned)(need < cap ? (need > 0 ? need : 1) : cap);
}

}  // namespace

cudaError_t launch_prep(const PrepArgs& a, int data_is_double, int coord_mode,
                        cudaStream_t st)
{
    const dim3 grid(a.blocks_per_job, a.num_jobs);
    if (data_is_double)
        prep_kernel<double, COORD_F64><<<grid, kPrepThreads, 0, st>>>(a);
    else if (coord_mode == OSKAR_B200_COORDS_REFERENCE_F32)
        prep_kernel<float, COORD_REF_F32><<<grid, kPrepThreads, 0, st>>>(a);
    else
        prep_kernel<float, COORD_F64><<<grid, kPrepThreads, 0, st>>>(a);
    return cudaGetLastError();
}

size_t task_tiles(size_t n) { return (n + kTaskTile - 1) / kTaskTile; }

cudaError_t launch_tasks(const uint32_t* sorted_keys, size_t n,
                         unsigned long long* counters, int fine_key_bits,
                         int job_shift, const TaskSizes& sizes,
                         unsigned long long* tile_state, uint32_t* task_start,
                         uint32_t* task_job, cudaStream_t st, int* launches,
                         unsigned expired_tile)
{
    const size_t tiles = task_tiles(n);
    if (tiles == 0) return cudaSuccess;
    if (launches) *launches += 1;
    task_list_kernel<<<(unsigned)tiles, kTaskThreads, 0, st>>>(
        sorted_keys, n, counters, fine_key_bits, sizes, job_shift, tile_state,
        expired_tile, task_start, task_job);
    return cudaGetLastError();
}

namespace {

__device__ __forceinline__ int band_of_task(const uint32_t* keys,
                                            const uint32_t* task_start,
                                            unsigned t, int band_shift,
                                            uint32_t band_mask)
{
    return (int)((keys[task_start[t]] >> band_shift) & band_mask);
}

// band_first[b] = first task whose band is >= b, for b in [0, num_bands];
// tasks are in key order, so bands are non-decreasing along the list.
__global__ void band_first_kernel(const uint32_t* __restrict__ sorted_keys,
                                  const uint32_t* __restrict__ task_start,
                                  const unsigned long long* __restrict__ counters,
                                  int band_shift, uint32_t band_mask,
                                  int num_bands, uint32_t* __restrict__ band_first)
{
    const unsigned nt = tasks_listed(counters);
    for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t <= nt;
         t += (size_t)gridDim.x * blockDim.x)
    {
        int b = t < nt ? band_of_task(sorted_keys, task_start, (unsigned)t,
                                      band_shift, band_mask)
                       : num_bands;
        b = b < num_bands ? b : num_bands;
        int prev = t > 0 ? band_of_task(sorted_keys, task_start,
                                        (unsigned)t - 1, band_shift, band_mask)
                         : -1;
        prev = prev < num_bands ? prev : num_bands;
        for (int c = prev + 1; c <= b; ++c) band_first[c] = (uint32_t)t;
    }
}

}  // namespace

cudaError_t launch_band_first(const uint32_t* sorted_keys,
                              const uint32_t* task_start, size_t n,
                              const unsigned long long* counters,
                              const KeyLayout& kl, int num_bands,
                              uint32_t* band_first, int num_sms,
                              cudaStream_t st)
{
    const int shift = kl.group_bits + 2 * kl.fine_bits + kl.coarse_bits;
    const uint32_t mask = (1u << kl.coarse_bits) - 1u;
    const unsigned blocks = grid_blocks(n + 1, num_sms, 8, 256);
    band_first_kernel<<<blocks, 256, 0, st>>>(sorted_keys, task_start,
                                              counters, shift, mask, num_bands,
                                              band_first);
    return cudaGetLastError();
}

cudaError_t launch_place(int data_is_double, int coord_mode, const void* uu,
                         const void* vv, const void* ww, size_t n,
                         const PlaceConsts& pc, const int* support,
                         int32_t* gu, int32_t* gv, int32_t* plane,
                         int32_t* off_u, int32_t* off_v, int32_t* conj,
                         int32_t* skipped, int num_sms, cudaStream_t st)
{
    const unsigned blocks = grid_blocks(n, num_sms, 8, 256);
    if (data_is_double)
        place_kernel<double, COORD_F64><<<blocks, 256, 0, st>>>(
            static_cast<const double*>(uu), static_cast<const double*>(vv),
            static_cast<const double*>(ww), n, pc, support, gu, gv, plane,
            off_u, off_v, conj, skipped);
    else if (coord_mode == OSKAR_B200_COORDS_REFERENCE_F32)
        place_kernel<float, COORD_REF_F32><<<blocks, 256, 0, st>>>(
            static_cast<const float*>(uu), static_cast<const float*>(vv),
            static_cast<const float*>(ww), n, pc, support, gu, gv, plane,
            off_u, off_v, conj, skipped);
    else
        place_kernel<float, COORD_F64><<<blocks, 256, 0, st>>>(
            static_cast<const float*>(uu), static_cast<const float*>(vv),
            static_cast<const float*>(ww), n, pc, support, gu, gv, plane,
            off_u, off_v, conj, skipped);
    return cudaGetLastError();
}

}  // namespace b200
