// Degridding: the adjoint of the W-projection gridder.  The reference has
// no degridder (Defines.h:48 only reserves the switch); this one is defined
// as the exact adjoint of the gridding path of this library: with the
// gridder's placement, skip test and tap kernel value
//   Kt = conj?(K[plane][|off_v + j*os|][|off_u + k*os|])
// (conjugated for w > 0, oskar_grid_wproj.c:70-122), each kept visibility
// becomes
//   vis = sum over the (2S+1)^2 taps of grid[(gv+j)*G + gu+k] * conj(Kt).
//
// The visibilities arrive in the gridder's sort order (coarse tile, support,
// fine cell); each CTA takes chunks of 256 consecutive ones from a work queue,
// so its warps read neighbouring grid rows and the same kernel slab rows
// from L1.  The kernel is bound by L1 (two loads per tap; data pipe 76 % busy
// at 16 taps per clock and SM), so a chunk is first ordered by cell as a
// gridding task is, and then
//   - visibilities with the same placement are gathered once and written to
//     each of them,
//   - two different ones of the same cell and support are gathered together,
//     sharing the grid loads.
// 15.7 M points on 8192^2 (8.0e9 taps): 8.60 -> 7.17 ms, without pairs 8.7,
// chunks in Morton order instead of column by column 7.4; 0.24 M points in dense
// cells 119 -> 48 us.
// A group of 16 lanes takes one or two visibilities (two groups per warp): its
// lanes walk the footprint's taps in row-major order, 16 at a time (busy
// whatever the support; the per-visibility set-up and reduction serve both
// groups at once), and the lane sums are reduced within the group.
// Measured at plain_large: 16 lanes 28.5 ms, 8 lanes 30.2, 4 lanes 33.8,
// 32 lanes 40.9.
// The result goes to the visibility's own slot (the sort's values are the
// original indices).
#include <atomic>

#include "common.cuh"
#include "degrid_plan.h"
#include "internal.h"
#include "prep.cuh"
#include "task_order.cuh"

namespace b200 {
namespace {

template <typename GT> struct Cplx;
template <> struct Cplx<float> { using type = float2; };
template <> struct Cplx<double> { using type = double2; };

constexpr int kDegridWarps = 8;     // warps per CTA
constexpr int kGroup = 16;          // lanes per visibility
constexpr int kGroups = 32 / kGroup;
constexpr int kDegridMaxW = 255;   // footprint width for support <= 127
// Widest footprint gathered in pairs: in wider ones the two walks' kernel rows
// crowd each other out of L1 where points are spread.  Pairs to a width of 24,
// 32, 40, 48 (no pairs), FP32: 15.7 million points on 8192^2, oversample 4, 6.84,
// 6.65, 6.71, 6.77 ms (7.52); 3.9 million spread over 4096^2, oversample 8, 4.12,
// 4.05, 4.24, 4.45 (4.24), FP64 8.57, 8.59, 9.01, 9.15 (8.23).  33 is as good as
// 32 (6.66 and 4.09 ms) and the first width with three columns per lane: without
// that walk for pairs the compiled kernel takes 7.19 and 4.31 ms.
constexpr int kPairMaxW = 33;

// Sum over taps of grid * conj(Kt), Kt = (kr, sgn * ki).  FP32: two packed
// FMAs per tap, A += g * kr and B += g * ki, with the sign applied once at
// the end (re = A.x + sgn B.y, im = A.y - sgn B.x).  FP64: four FMAs per
// tap in the order of the definition.
template <typename GT> struct DegridAcc;
template <> struct DegridAcc<float>
{
    float2 a = make_float2(0.f, 0.f), b = make_float2(0.f, 0.f);
    float sgn;
    __device__ __forceinline__ explicit DegridAcc(float s = 1.f) : sgn(s) {}
    __device__ __forceinline__ void add(const float2 g, float kr, float ki)
    {
        a = __ffma2_rn(g, make_float2(kr, kr), a);
        b = __ffma2_rn(g, make_float2(ki, ki), b);
    }
    __device__ __forceinline__ void finish(float& re, float& im) const
    {
        re = fmaf(sgn, b.y, a.x);
        im = fmaf(-sgn, b.x, a.y);
    }
};
template <> struct DegridAcc<double>
{
    double re = 0.0, im = 0.0, sgn;
    __device__ __forceinline__ explicit DegridAcc(double s = 1.0) : sgn(s) {}
    __device__ __forceinline__ void add(const double2 g, double kr, double ki)
    {
        ki *= sgn;
        re = fma(g.x, kr, fma(g.y, ki, re));
        im = fma(g.y, kr, fma(-g.x, ki, im));
    }
    __device__ __forceinline__ void finish(double& r, double& i) const
    {
        r = re;
        i = im;
    }
};

// Slab column of footprint column k: the quadrant column |off_u + (k - S) os|
// in the phase-major layout, (x mod os) * L + x / os.  For k >= tu the
// argument is non-negative and the column is cp + k; below, cn - k.  With
// |off_u| <= os the remainders and quotients need no division.
struct ColumnMap
{
    int tu, cp, cn;
    ColumnMap() = default;
    __device__ __forceinline__ ColumnMap(int off_u, int S, int os, int L)
    {
        const int rp = off_u < 0 ? off_u + os : (off_u >= os ? off_u - os : off_u);
        const int qp = off_u < 0 ? -1 : (off_u >= os ? 1 : 0);
        const int on = -off_u;
        const int rn = on < 0 ? on + os : (on >= os ? on - os : on);
        const int qn = on < 0 ? -1 : (on >= os ? 1 : 0);
        tu = S + (off_u < 0 ? 1 : 0);
        cp = rp * L + qp - S;
        cn = rn * L + qn + S;
    }
    __device__ __forceinline__ int operator()(int k) const
    {
        return k >= tu ? cp + k : cn - k;
    }
};

// Rows in the outer loop, each lane of a group owning the footprint columns
// k = gl + kGroup * m, m < M: the byte addresses of each column's kernel
// value and grid cell in the first row are registers, so a tap costs two
// wide multiply-adds (row times the row pitch in bytes), two loads and the
// packed multiply-adds.  Used for footprints kGroup to 5 * kGroup wide
// (narrower ones would leave lanes idle; wider ones take the flattened
// walk).  The slab and the grid are read-only here: non-coherent loads.
// P visibilities of one cell and support at a time.
template <int M, int P, typename GT, typename KT, typename C2>
__device__ __forceinline__ void degrid_rows(const KT* const (&slab)[P],
                                            const C2* __restrict__ grid,
                                            int W, int pitch, int G,
                                            const ColumnMap (&cm)[P], int gl,
                                            DegridAcc<GT> (&acc)[P])
{
    const char* kc[P][M];
    const char* gc[M];
    bool ok[M];
#pragma unroll
    for (int m = 0; m < M; ++m)
    {
        const int k = gl + kGroup * m;
        ok[m] = k < W;
#pragma unroll
        for (int p = 0; p < P; ++p)
            kc[p][m] = reinterpret_cast<const char*>(
                slab[p] + (ok[m] ? cm[p](k) : 0));
        gc[m] = reinterpret_cast<const char*>(grid + (ok[m] ? k : 0));
    }
    const unsigned kb = (unsigned)pitch * (unsigned)sizeof(KT);
    const unsigned gb = (unsigned)G * (unsigned)sizeof(C2);
    // (rows in flight: 1 at a time 2.48, 2: 2.35, 4: 2.27 ms, 3.9 M points)
#pragma unroll 4
    for (int j = 0; j < W; ++j)
    {
#pragma unroll
        for (int m = 0; m < M; ++m)
        {
            if (!ok[m]) continue;
            typename KernelLoad<KT>::Wide kv[P];
#pragma unroll
            for (int p = 0; p < P; ++p)
                kv[p] = KernelLoad<KT>::get(__ldg(
                    reinterpret_cast<const KT*>(kc[p][m] + (size_t)j * kb)));
            const C2 g = __ldg(
                reinterpret_cast<const C2*>(gc[m] + (size_t)j * gb));
#pragma unroll
            for (int p = 0; p < P; ++p)
                acc[p].add(g, (GT)kv[p].x, (GT)kv[p].y);
        }
    }
}

// The lane's tap (j, k) as 32-bit running offsets (grid cell j * G + k, kernel
// row j * pitch), stepped kGroup taps at a time with k wrapping past W: the
// 64-bit index arithmetic per tap cost 28.4 -> 26.5 ms at plain_large.
template <int P, typename GT, typename KT, typename C2>
__device__ __forceinline__ void degrid_taps(const KT* const (&slab)[P],
                                            const C2* __restrict__ grid,
                                            int W, int pitch, int G,
                                            const ColumnMap (&cm)[P], int gl,
                                            DegridAcc<GT> (&acc)[P])
{
    const int taps = W * W, dj = kGroup / W, dk = kGroup % W;
    const int j0 = gl / W;
    int k = gl - j0 * W;
    unsigned goff = (unsigned)j0 * (unsigned)G + (unsigned)k;
    unsigned krow = (unsigned)j0 * (unsigned)pitch;
    const unsigned gstep = (unsigned)dj * (unsigned)G + (unsigned)dk;
    const unsigned kstep = (unsigned)dj * (unsigned)pitch;
    const unsigned gwrap = (unsigned)G - (unsigned)W;
    const unsigned kwrap = (unsigned)pitch;
#pragma unroll 4
    for (int t = gl; t < taps; t += kGroup)
    {
        typename KernelLoad<KT>::Wide kv[P];
#pragma unroll
        for (int p = 0; p < P; ++p)
            kv[p] = KernelLoad<KT>::get(__ldg(slab[p] + krow + cm[p](k)));
        const C2 g = __ldg(grid + goff);
#pragma unroll
        for (int p = 0; p < P; ++p)
            acc[p].add(g, (GT)kv[p].x, (GT)kv[p].y);
        k += dk;
        goff += gstep;
        krow += kstep;
        const bool wrap = k >= W;
        k = wrap ? k - W : k;
        goff += wrap ? gwrap : 0u;
        krow += wrap ? kwrap : 0u;
    }
}

// The lane's part of the sums of P visibilities of one job, cell and support.
// False when the footprint would leave the grid: the prep kernel keeps only
// footprints inside it, and a record that says otherwise is reported and left
// out.
template <int P, typename GT, typename KT, typename C2>
__device__ __forceinline__ bool degrid_unit(const JobDesc& jd,
                                            const uint2 (&rec)[P], int gl,
                                            unsigned long long* status,
                                            C2 (&sum)[P])
{
    const int half = jd.half, os = jd.oversample, G = jd.grid_size;
    const KT* slab[P];
    ColumnMap cm[P];
    DegridAcc<GT> acc[P];
    int u0 = 0, v0 = 0, W = 0, pitch = 0;
#pragma unroll
    for (int p = 0; p < P; ++p)
    {
        const int4 r = unpack_record(rec[p]);
        const PlaneDesc& d = jd.planes[r.z & 0x7fffffff];
        const int off_u = min(max((r.w & 0xffff) - half, -half), half);
        const int off_v = min(max((r.w >> 16) - half, -half), half);
        W = 2 * d.support + 1;
        pitch = d.pitch;
        u0 = r.x - d.support;
        v0 = r.y - d.support;
        slab[p] = static_cast<const KT*>(jd.slabs) + d.offset +
                  (long long)(off_v + half) * W * pitch;
        cm[p] = ColumnMap(off_u, d.support, os, d.L);
        acc[p] = DegridAcc<GT>(r.z < 0 ? GT(-1) : GT(1));
    }
    if (u0 < 0 || v0 < 0 || u0 + W > G || v0 + W > G || W > kDegridMaxW)
    {
        if (gl == 0)
            atomicOr(status, (unsigned long long)DEV_ERR_GRID_INDEX);
        return false;
    }
    const C2* __restrict__ grid =
        static_cast<const C2*>(jd.grid) + (size_t)v0 * G + u0;
    // rows outer, columns per lane (plain_large degrid 26.5 -> 25.2 ms)
    const int mc = W < kGroup ? 0 : (W + kGroup - 1) / kGroup;
    switch (mc)
    {
    case 1: degrid_rows<1, P, GT>(slab, grid, W, pitch, G, cm, gl, acc); break;
    case 2: degrid_rows<2, P, GT>(slab, grid, W, pitch, G, cm, gl, acc); break;
    case 3: degrid_rows<3, P, GT>(slab, grid, W, pitch, G, cm, gl, acc); break;
    // (pairs are no wider: kPairMaxW)
    case 4:
        if constexpr (P == 1)
        {
            degrid_rows<4, P, GT>(slab, grid, W, pitch, G, cm, gl, acc);
            break;
        }
    case 5:
        if constexpr (P == 1)
        {
            degrid_rows<5, P, GT>(slab, grid, W, pitch, G, cm, gl, acc);
            break;
        }
    default: degrid_taps<P, GT>(slab, grid, W, pitch, G, cm, gl, acc); break;
    }
#pragma unroll
    for (int p = 0; p < P; ++p)
    {
        GT x, y;
        acc[p].finish(x, y);
        sum[p].x = x;
        sum[p].y = y;
    }
    return true;
}

// apply_weight: the adjoint of gridding weight * vis, i.e. the degridded
// value times the visibility's weight.
// Registers bounded for 4 resident CTAs (32 warps) per SM.  FP32 at
// plain_large: 2 CTAs 30.3 ms, 3: 23.2, 4: 20.8, 5: 22.1, 6: 23.3 (more
// warps share the same L1 for their kernel rows and grid lines).
template <typename GT, typename KT>
__global__ void __launch_bounds__(kDegridWarps * 32, kDegridResident)
degrid_kernel(const uint32_t* __restrict__ order,
              const uint32_t* __restrict__ sorted_keys,
              const uint2* __restrict__ rec, const JobDesc* __restrict__ jobs,
              int job_shift, int apply_weight,
              unsigned long long* __restrict__ counters, size_t n, int chunk)
{
    using C2 = typename Cplx<GT>::type;
    static_assert(kDegridChunk == kDegridWarps * 32 &&
                  kDegridChunk == kGridThreads, "one visibility per thread");
    __shared__ unsigned long long s_chunk;
    __shared__ uint2 s_rec[kDegridChunk];        // as gathered
    __shared__ uint32_t s_order[kDegridChunk];   // gathered slot, in cell order
    __shared__ uint8_t s_first[kDegridChunk];    // slot of each distinct one
    __shared__ uint16_t s_unit[kDegridChunk];    // distinct one | pair << 8
    __shared__ C2 s_sum[kDegridChunk];
    __shared__ bool s_ok[kDegridChunk];
    __shared__ int4 s_box[kDegridWarps];
    __shared__ int s_count[3][kDegridWarps];
    __shared__ int s_next;                       // next unit to take
    // A sort that gave up leaves nothing to do.
    const size_t valid = counters[CNT_STATUS] & DEV_ERR_TIMEOUT
                             ? 0 : n - counters[CNT_SKIPPED];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int group = lane / kGroup, gl = lane % kGroup;
    const unsigned below = (1u << lane) - 1u;
    // A CTA takes chunks of `chunk` consecutive sorted visibilities
    // from a work queue: its warps work on neighbouring footprints and share
    // grid lines and kernel rows in L1, and the uneven cost of the chunks
    // (footprints of 81 to 5329 taps) balances across CTAs.
    for (;;)
    {
        if (t == 0) s_chunk = atomicAdd(&counters[CNT_TASK_NEXT], 1ull);
        __syncthreads();
        const size_t begin = (size_t)s_chunk * chunk;
        if (begin >= valid) break;
        const int m = (int)min(valid - begin, (size_t)chunk);
        // The visibility with sorted position begin + t, in cell order.
        const JobDesc* const jd0 = &jobs[sorted_keys[begin] >> job_shift];
        uint32_t i = 0;
        uint2 r = make_uint2(0, 0);
        if (t < m)
        {
            i = order[begin + t];
            r = rec[i];
            s_rec[t] = r;
        }
        const int4 r4 = unpack_record(r);
        const TaskKey tk(jd0->half, task_box(t < m, r4, s_box));
        uint32_t key = 0xffffffffu;
        if (t < m) key = tk.template make<true>(r4, t);
        key = task_order(key, s_order);
        const unsigned slot = key & 0xffu;
        s_order[t] = slot;
        __syncthreads();
        auto job_of = [&](unsigned k) {
            return sorted_keys[begin + k] >> job_shift;
        };
        // First of each run of equal placements.
        bool head = false;
        if (t < m)
        {
            r = s_rec[slot];
            const unsigned p = s_order[t ? t - 1 : 0];
            const uint2 q = s_rec[p];
            head = t == 0 || r.x != q.x || r.y != q.y ||
                   job_of(slot) != job_of(p);
        }
        const unsigned ball = __ballot_sync(0xffffffffu, head);
        if (lane == 0) s_count[0][warp] = __popc(ball);
        if (t == 0) s_next = 0;
        __syncthreads();
        int rank = __popc(ball & (below | (1u << lane))) - 1, distinct = 0;
        for (int w = 0; w < kDegridWarps; ++w)
        {
            rank += w < warp ? s_count[0][w] : 0;
            distinct += s_count[0][w];
        }
        if (head) s_first[rank] = (uint8_t)slot;
        __syncthreads();
        // Units: pairs of neighbours in one cell with one support (within a
        // warp's 32), then what is left one by one, so that the two groups
        // of a warp mostly run the same code.
        bool same = false;
        if (t < distinct)
        {
            const unsigned a = s_first[t], b = s_first[t ? t - 1 : 0];
            r = s_rec[a];
            const uint2 q = s_rec[b];
            const JobDesc& jd = jobs[job_of(a)];
            const int w = jd.planes[r.y & 0x7fffu].support;
            same = lane != 0 && r.x == q.x && job_of(a) == job_of(b) &&
                   jd.planes[q.y & 0x7fffu].support == w &&
                   2 * w + 1 <= kPairMaxW;
        }
        const unsigned joined = __ballot_sync(0xffffffffu, same);
        // position in the run of joined ones: odd ones belong to a pair
        const int back = __clz(~(joined << (31 - lane)));
        const bool second = same && (back & 1);
        const unsigned seconds = __ballot_sync(0xffffffffu, second);
        const bool pair = t < distinct && !second &&
                          lane < 31 && ((seconds >> (lane + 1)) & 1u);
        const bool single = t < distinct && !second && !pair;
        const unsigned pairs = __ballot_sync(0xffffffffu, pair);
        const unsigned singles = __ballot_sync(0xffffffffu, single);
        if (lane == 0)
        {
            s_count[1][warp] = __popc(pairs);
            s_count[2][warp] = __popc(singles);
        }
        __syncthreads();
        int np = 0, units = 0, at = pair ? __popc(pairs & below)
                                         : __popc(singles & below);
        for (int w = 0; w < kDegridWarps; ++w)
        {
            np += s_count[1][w];
            units += s_count[1][w] + s_count[2][w];
            if (w < warp) at += s_count[pair ? 1 : 2][w];
        }
        if (pair) s_unit[at] = (uint16_t)(t | 256);
        if (single) s_unit[np + at] = (uint16_t)t;
        __syncthreads();
        // Each warp takes the next kGroups units, one per group of kGroup
        // lanes (the loop bounds are the same for the whole warp).
        for (;;)
        {
            int base = 0;
            if (lane == 0) base = atomicAdd(&s_next, kGroups);
            base = __shfl_sync(0xffffffffu, base, 0);
            if (base >= units) break;
            const int u = base + group;
            const uint32_t unit = u < units ? s_unit[u] : 0u;
            const int q = (int)(unit & 0xffu);
            C2 sum[2];
            sum[0].x = sum[0].y = sum[1].x = sum[1].y = GT(0);
            bool ok = false;
            if (u < units)
            {
                const unsigned a = s_first[q];
                const JobDesc& jd = jobs[job_of(a)];
                unsigned long long* status = &counters[CNT_STATUS];
                if (unit & 256u)
                {
                    const uint2 two[2] = {s_rec[a], s_rec[s_first[q + 1]]};
                    ok = degrid_unit<2, GT, KT>(jd, two, gl, status, sum);
                }
                else
                {
                    const uint2 one[1] = {s_rec[a]};
                    C2 x[1];
                    x[0] = sum[0];
                    ok = degrid_unit<1, GT, KT>(jd, one, gl, status, x);
                    sum[0] = x[0];
                }
            }
#pragma unroll
            for (int o = kGroup / 2; o > 0; o >>= 1)
            {
#pragma unroll
                for (int p = 0; p < 2; ++p)
                {
                    sum[p].x += __shfl_xor_sync(0xffffffffu, sum[p].x, o);
                    sum[p].y += __shfl_xor_sync(0xffffffffu, sum[p].y, o);
                }
            }
            if (u < units && gl < 1 + (int)(unit >> 8))
            {
                s_sum[q + gl] = gl ? sum[1] : sum[0];
                s_ok[q + gl] = ok;
            }
        }
        __syncthreads();
        if (t < m && s_ok[rank])
        {
            // (thread t's own visibility has slot `slot`)
            const uint32_t point = order[begin + slot];
            const JobDesc& jd = jobs[job_of(slot)];
            const size_t local = point - jd.first;
            GT sc = (GT)jd.planes[s_rec[slot].y & 0x7fffu].scale;
            if (apply_weight)
                sc *= static_cast<const GT*>(jd.weight)[local];
            GT* out = static_cast<GT*>(const_cast<void*>(jd.vis));
            out[2 * local] = s_sum[rank].x * sc;
            out[2 * local + 1] = s_sum[rank].y * sc;
        }
        // (the next chunk's arrays are written behind the next barriers; the
        // sums behind many)
    }
}

}  // namespace

namespace {

template <typename GT, typename KT>
cudaError_t launch_variant(const uint32_t* order, const uint32_t* sorted_keys,
                           const uint2* rec, const JobDesc* jobs,
                           int job_shift, int apply_weight,
                           unsigned long long* counters, size_t n,
                           int chunk, unsigned blocks, cudaStream_t st)
{
    auto fn = degrid_kernel<GT, KT>;
    // Only the shared memory 4 CTAs need: the rest of the SM's unified storage
    // is L1, which is what the kernel lives on.
    // (Asked for once per device; a hint, so a lost race does no harm.)
    static std::atomic<unsigned long long> asked{0};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const unsigned long long bit = 1ull << (dev & 63);
    if (!(asked.load() & bit))
    {
        cudaFuncAttributes a{};
        e = cudaFuncGetAttributes(&a, fn);
        if (e != cudaSuccess) return e;
        const size_t need = 4 * (a.sharedSizeBytes + 1024);
        e = cudaFuncSetAttribute(
            fn, cudaFuncAttributePreferredSharedMemoryCarveout,
            (int)((100 * need + 228 * 1024 - 1) / (228 * 1024)));
        if (e != cudaSuccess) return e;
        asked.fetch_or(bit);
    }
    fn<<<blocks, kDegridWarps * 32, 0, st>>>(order, sorted_keys, rec, jobs,
                                             job_shift, apply_weight, counters,
                                             n, chunk);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_degrid(const uint32_t* order, const uint32_t* sorted_keys,
                          const uint2* rec, const JobDesc* jobs, int job_shift,
                          int apply_weight, unsigned long long* counters,
                          size_t n, int max_support,
                          int data_is_double, int kernel_type, int num_sms,
                          cudaStream_t st)
{
    const int chunk = degrid_chunk(n, max_support, data_is_double, num_sms);
    // up to 8 CTAs of 8 warps per SM, persistent over the work queue
    const size_t want = (n + chunk - 1) / chunk;
    const size_t cap = (size_t)num_sms * 8;
    const unsigned blocks = (unsigned)(want < cap ? (want ? want : 1) : cap);
    auto run = [&](auto launch) {
        return launch(order, sorted_keys, rec, jobs, job_shift, apply_weight,
                      counters, n, chunk, blocks, st);
    };
    if (data_is_double)
        return kernel_type == OSKAR_B200_KERNEL_NATIVE
                   ? run(launch_variant<double, double2>)
                   : cudaErrorInvalidValue;
    switch (kernel_type)
    {
    case OSKAR_B200_KERNEL_F16: return run(launch_variant<float, __half2>);
    case OSKAR_B200_KERNEL_BF16:
        return run(launch_variant<float, __nv_bfloat162>);
    default: return run(launch_variant<float, float2>);
    }
}

}  // namespace b200
