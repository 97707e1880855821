// Uniform weighting on the device: the weights-grid histogram ("write") and
// the density lookup ("read") of utils/oskar_grid_weights.c:38-172.
//
// Both steps place a point at the cell
//   grid_u = (int)round(-u * grid_size * cell) + grid_size / 2,
//   grid_v = (int)round( v * grid_size * cell) + grid_size / 2
// (u, v first scaled from metres to wavelengths as scale_coords does, when a
// frequency is given)
// and skip it when the cell is outside the grid.  The weights grid is real
// (one value per cell), row-major in v.
//
// write, ordered (the default, bit-exact): the reference adds the weights of
//   a cell in point order, so a stable radix sort of (cell, weight), or of
//   (cell, point index) in FP64, gathers each cell's points in that order, and
//   they are added one after the other onto the cell's previous value (by one
//   thread, or by one warp for a cell with many points).  The sums are the
//   reference's to the bit for any weights.
// write, atomic: one fire-and-forget reduction per point.  Cell sums then
//   depend on the order the reductions land in; they are exact whenever the
//   partial sums are (e.g. unit weights below 2^24 per cell in FP32).
// read: one thread per point; out = in / grid[cell] (IEEE division), 0 where
//   the cell is empty, and skipped points keep their previous output value.
#include <algorithm>
#include <climits>

#include "common.cuh"
#include "internal.h"

namespace b200 {
namespace {

struct WeightConsts
{
    double grid_scale;   // grid_size * cell_size_rad, FP64
    float grid_scale_f;  // the same product in float arithmetic
    double coord_scale;  // metres to wavelengths (scale_coords), or 1
    float coord_scale_f;
    int grid_size;
    int centre;
};

// Cell index of a point, or -1 when it is skipped.  A rounded coordinate
// outside the int range (or NaN) converts to INT_MIN, as x86-64's truncating
// conversion does, and is therefore skipped.
template <typename T>
__device__ __forceinline__ long long weight_cell(T u, T v,
                                                 const WeightConsts& c)
{
    long long gu, gv;
    if (sizeof(T) == sizeof(double))
    {
        const double us = __dmul_rn((double)u, c.coord_scale);
        const double vs = __dmul_rn((double)v, c.coord_scale);
        const double ru = round(__dmul_rn(-us, c.grid_scale));
        const double rv = round(__dmul_rn(vs, c.grid_scale));
        gu = (ru > -2147483649.0 && ru < 2147483648.0 ? (long long)ru
                                                        : (long long)INT_MIN);
        gv = (rv > -2147483649.0 && rv < 2147483648.0 ? (long long)rv
                                                        : (long long)INT_MIN);
    }
    else
    {
        const float us = __fmul_rn((float)u, c.coord_scale_f);
        const float vs = __fmul_rn((float)v, c.coord_scale_f);
        const float ru = roundf(__fmul_rn(-us, c.grid_scale_f));
        const float rv = roundf(__fmul_rn(vs, c.grid_scale_f));
        gu = (ru > -2147483649.0f && ru < 2147483648.0f ? (long long)ru
                                                          : (long long)INT_MIN);
        gv = (rv > -2147483649.0f && rv < 2147483648.0f ? (long long)rv
                                                          : (long long)INT_MIN);
    }
    gu += c.centre;
    gv += c.centre;
    if (gu < 0 || gu >= c.grid_size || gv < 0 || gv >= c.grid_size) return -1;
    return gv * c.grid_size + gu;
}

__device__ __forceinline__ double add_rn(double a, double b)
{
    return __dadd_rn(a, b);
}
__device__ __forceinline__ float add_rn(float a, float b)
{
    return __fadd_rn(a, b);
}
__device__ __forceinline__ double div_rn(double a, double b)
{
    return __ddiv_rn(a, b);
}
__device__ __forceinline__ float div_rn(float a, float b)
{
    return __fdiv_rn(a, b);
}

__device__ __forceinline__ void count_skipped(unsigned local,
                                              unsigned long long* skipped)
{
    local = warp_sum(local);
    if ((threadIdx.x & 31) == 0 && local)
        atomicAdd(skipped, (unsigned long long)local);
}

template <typename T>
__global__ void __launch_bounds__(256)
weights_write_atomic_kernel(size_t n, const T* __restrict__ uu,
                            const T* __restrict__ vv,
                            const T* __restrict__ weight, WeightConsts c,
                            T* __restrict__ grid,
                            unsigned long long* __restrict__ skipped)
{
    unsigned local = 0;
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += stride)
    {
        const long long t = weight_cell(uu[i], vv[i], c);
        if (t < 0)
            ++local;
        else
            atomicAdd(grid + t, weight[i]);
    }
    count_skipped(local, skipped);
}

// Sort keys for the ordered write: the cell, or `sentinel` (= grid_size^2,
// above every cell) for a skipped point.
template <typename T>
__global__ void __launch_bounds__(256)
weights_key_kernel(size_t n, const T* __restrict__ uu,
                   const T* __restrict__ vv, WeightConsts c,
                   uint32_t sentinel, uint32_t* __restrict__ keys,
                   unsigned long long* __restrict__ skipped)
{
    unsigned local = 0;
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += stride)
    {
        const long long t = weight_cell(uu[i], vv[i], c);
        local += t < 0;
        keys[i] = t < 0 ? sentinel : (uint32_t)t;
    }
    count_skipped(local, skipped);
}

// Sums each run of equal keys (one cell's points, in point order) onto the
// cell's previous value: the reference's additions, in its order.
//
// FP32 weights are the sort's values, so they lie in that order already; FP64
// ones are gathered by the sorted point indices.  A warp takes kSpan sorted
// positions at a time from a queue and goes through them in windows of 32
// with the next 32 at hand: a run that ends inside the two is summed by the
// lane holding its first element, from shared memory.  A longer one (the
// dense cells near the grid centre, up to ~10^5 points) is summed by the
// whole warp, kSpan weights at a time with the next kSpan in flight, every
// lane keeping the same sum of what it reads as broadcasts.  A long run is a
// chain of dependent additions, which nothing shortens; so spans are handed
// out from the middle of the order outwards, where the densest cells lie.
//
// 39.2 M FP32 points, densest cells near 10^5 points: 307 us, against 2357
// with point indices as values, 32 weights gathered one step ahead and the
// windows dealt out in order; reading keys and weights once takes 48 us, the
// rest is the longest chain.
constexpr int kSpan = 256;
constexpr int kSumThreads = 256;
constexpr int kSumCtasPerSm = 4;

template <typename T>
__device__ __forceinline__ T sorted_weight(const uint32_t* __restrict__ vals,
                                           const T* __restrict__ weight,
                                           size_t j)
{
    if constexpr (sizeof(T) == sizeof(uint32_t))
        return __uint_as_float(vals[j]);
    else
        return weight[vals[j]];
}

template <typename T> struct __align__(16) Four { T e[4]; };

template <typename T>
__global__ void __launch_bounds__(kSumThreads, kSumCtasPerSm)
weights_run_sum_kernel(size_t n, const uint32_t* __restrict__ keys,
                       const uint32_t* __restrict__ vals,
                       const T* __restrict__ weight, uint32_t sentinel,
                       T* __restrict__ grid,
                       const unsigned long long* __restrict__ status,
                       unsigned long long* __restrict__ host_status,
                       unsigned long long* __restrict__ queue,
                       unsigned long long* __restrict__ skipped)
{
    constexpr unsigned kAll = 0xffffffffu;
    // (four more: a lane reads its run four values at a time)
    __shared__ __align__(16) T s_v[kSumThreads / 32][kSpan + 4];
    // The status goes to the host from here (pinned memory; a copy of its own
    // would cost a launch).
    const bool reports = blockIdx.x == 0 && threadIdx.x == 0;
    if (reports) *host_status = *status;
    if (*status)   // the sort gave up: its pairs are not to be used
    {
        if (reports) *skipped = kSortFailed;
        return;
    }
    const int lane = threadIdx.x & 31;
    T* sv = s_v[threadIdx.x >> 5];
    const size_t spans = (n + kSpan - 1) / kSpan, mid = spans / 2;
    for (;;)
    {
        unsigned long long g = 0;
        if (lane == 0) g = atomicAdd(queue, 1ull);
        g = __shfl_sync(kAll, g, 0);
        if (g >= spans) return;
        // mid, mid - 1, mid + 1, mid - 2, ...: every span once
        const size_t base =
            ((g & 1) ? mid - (g + 1) / 2 : mid + g / 2) * kSpan;
        size_t i = base + lane;
        uint32_t k = i < n ? keys[i] : sentinel;
        T v = i < n ? sorted_weight(vals, weight, i) : T(0);
        uint32_t before = base ? keys[base - 1] : sentinel;
        for (int w = 0; w < kSpan && base + w < n; w += 32, i += 32)
        {
            // Where the key changes, in this window (m0) and the next (m1);
            // positions from n on hold the sentinel.
            const uint32_t kn = i + 32 < n ? keys[i + 32] : sentinel;
            T vn = T(0);
            if (sizeof(T) == sizeof(uint32_t) && i + 32 < n)
                vn = sorted_weight(vals, weight, i + 32);
            uint32_t up = __shfl_up_sync(kAll, k, 1);
            if (lane == 0) up = before;
            before = __shfl_sync(kAll, k, 31);
            uint32_t up_next = __shfl_up_sync(kAll, kn, 1);
            if (lane == 0) up_next = before;
            const bool change = k != up || i == 0;
            const unsigned m0 = __ballot_sync(kAll, change);
            const unsigned m1 = __ballot_sync(kAll, kn != up_next);
            // (without a change in the next window only a long run, which
            // reads its weights itself, reaches into it)
            if (sizeof(T) != sizeof(uint32_t) && m1 && i + 32 < n)
                vn = sorted_weight(vals, weight, i + 32);
            // Changes behind this lane's position: the first ends its run.
            const unsigned long long rest =
                (m0 | (unsigned long long)m1 << 32) >> 1 >> lane;
            const bool head = change && k != sentinel;
            sv[lane] = v;
            sv[32 + lane] = vn;
            __syncwarp();
            if (head && rest)
            {
                const int len = __ffsll(rest);
                T acc = grid[k];
                for (int t = 0; t < len; t += 4)
                {
                    T x[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) x[q] = sv[lane + t + q];
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        if (t + q < len) acc = add_rn(acc, x[q]);
                }
                grid[k] = acc;
            }
            __syncwarp();
            const unsigned longrun = __ballot_sync(kAll, head && !rest);
            if (longrun)   // one at most: the window's last head
            {
                const int src = __ffs(longrun) - 1;
                const uint32_t key = __shfl_sync(kAll, k, src);
                T acc = grid[key];
                size_t j = base + w + src + lane;
                uint32_t kk[kSpan / 32];
                T x[kSpan / 32];
                auto load = [&]() {
#pragma unroll
                    for (int q = 0; q < kSpan / 32; ++q)
                    {
                        const size_t p = j + q * 32;
                        kk[q] = p < n ? keys[p] : sentinel;
                        x[q] = T(0);
                        if (p < n && (sizeof(T) == sizeof(uint32_t) ||
                                      kk[q] == key))
                            x[q] = sorted_weight(vals, weight, p);
                    }
                };
                load();
                int cnt;
                do
                {
                    cnt = 0;
#pragma unroll
                    for (int q = 0; q < kSpan / 32; ++q)
                    {
                        cnt += __popc(__ballot_sync(kAll, kk[q] == key));
                        sv[q * 32 + lane] = x[q];
                    }
                    __syncwarp();
                    if (cnt == kSpan)
                    {
                        j += kSpan;
                        load();
#pragma unroll 4
                        for (int t = 0; t < kSpan; t += 4)
                        {
                            const Four<T> y =
                                *reinterpret_cast<const Four<T>*>(sv + t);
#pragma unroll
                            for (int q = 0; q < 4; ++q)
                                acc = add_rn(acc, y.e[q]);
                        }
                    }
                    else
                        for (int t = 0; t < cnt; t += 4)
                        {
                            const Four<T> y =
                                *reinterpret_cast<const Four<T>*>(sv + t);
#pragma unroll
                            for (int q = 0; q < 4; ++q)
                                if (t + q < cnt) acc = add_rn(acc, y.e[q]);
                        }
                    __syncwarp();
                } while (cnt == kSpan);
                if (lane == 0) grid[key] = acc;
            }
            k = kn;
            v = vn;
        }
    }
}

template <typename T>
__global__ void __launch_bounds__(256)
weights_read_kernel(size_t n, const T* __restrict__ uu,
                    const T* __restrict__ vv,
                    const T* __restrict__ weight_in,
                    T* __restrict__ weight_out, WeightConsts c,
                    const T* __restrict__ grid,
                    unsigned long long* __restrict__ skipped)
{
    unsigned local = 0;
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += stride)
    {
        const long long t = weight_cell(uu[i], vv[i], c);
        if (t < 0)
        {
            ++local;
            continue;
        }
        const T g = grid[t];
        weight_out[i] = g != T(0) ? div_rn(weight_in[i], g) : T(0);
    }
    count_skipped(local, skipped);
}

WeightConsts make_consts(int data_is_double, double cell_size_rad,
                         int grid_size, double frequency_hz)
{
    WeightConsts c;
    c.grid_scale = grid_size * cell_size_rad;
    // C evaluates int * float in float (FLT_EVAL_METHOD 0 on x86-64).
    c.grid_scale_f = (float)grid_size * (float)cell_size_rad;
    c.coord_scale = coord_scale_of(frequency_hz);
    c.coord_scale_f = (float)c.coord_scale;
    (void)data_is_double;
    c.grid_size = grid_size;
    c.centre = grid_size / 2;
    return c;
}

int bit_length(unsigned long long x)
{
    int b = 0;
    while (x) { ++b; x >>= 1; }
    return b;
}

int launch_blocks(const oskar_B200Workspace* ws, size_t n)
{
    const size_t want = (n + 255) / 256;
    const size_t cap = (size_t)ws->num_sms * 8;
    return (int)(want < cap ? (want ? want : 1) : cap);
}

#define B200_TRY(expr)                                      \
    do {                                                    \
        const cudaError_t e_ = (expr);                      \
        if (e_ != cudaSuccess) return status_from_cuda(e_); \
    } while (0)

unsigned long long* skip_counter(oskar_B200Workspace* ws,
                                 unsigned long long* d_num_skipped)
{
    if (d_num_skipped) return d_num_skipped;
    return static_cast<unsigned long long*>(ws->counters.ptr) + CNT_SKIPPED;
}

}  // namespace

int run_weights_write(oskar_B200Workspace* ws, int data_is_double,
                      int ordered, size_t n, const void* uu, const void* vv,
                      const void* weight, double cell_size_rad,
                      int grid_size, void* grid,
                      unsigned long long* d_num_skipped, double frequency_hz,
                      cudaStream_t st)
{
    // The counters and, behind them, the sort's scratch start from zero.
    const size_t zero_bytes = sizeof(unsigned long long) * CNT_COUNT +
                              (ordered && n ? radix_sort_temp_bytes(n) : 0);
    B200_TRY(ws->counters.ensure(zero_bytes));
    unsigned long long* skipped = skip_counter(ws, d_num_skipped);
    B200_TRY(cudaMemsetAsync(skipped, 0, sizeof(unsigned long long), st));
    int launches = 0;
    if (n == 0)
    {
        ws->last_launches = 0;
        return OSKAR_B200_OK;
    }
    const WeightConsts c = make_consts(data_is_double, cell_size_rad,
                                       grid_size, frequency_hz);
    const int blocks = launch_blocks(ws, n);
    if (!ordered)
    {
        if (data_is_double)
            weights_write_atomic_kernel<double><<<blocks, 256, 0, st>>>(
                n, (const double*)uu, (const double*)vv,
                (const double*)weight, c, (double*)grid, skipped);
        else
            weights_write_atomic_kernel<float><<<blocks, 256, 0, st>>>(
                n, (const float*)uu, (const float*)vv, (const float*)weight,
                c, (float*)grid, skipped);
        B200_TRY(cudaGetLastError());
        ws->last_launches = 1;
        return OSKAR_B200_OK;
    }
    B200_TRY(ws->keys[0].ensure(4 * n));
    B200_TRY(ws->keys[1].ensure(4 * n));
    B200_TRY(ws->vals[0].ensure(4 * n));
    B200_TRY(ws->vals[1].ensure(4 * n));
    unsigned long long* counters =
        static_cast<unsigned long long*>(ws->counters.ptr);
    B200_TRY(cudaMemsetAsync(counters, 0, zero_bytes, st));
    unsigned long long* status = counters + CNT_STATUS;
    uint32_t* keys[2] = {static_cast<uint32_t*>(ws->keys[0].ptr),
                         static_cast<uint32_t*>(ws->keys[1].ptr)};
    uint32_t* vals[2] = {static_cast<uint32_t*>(ws->vals[0].ptr),
                         static_cast<uint32_t*>(ws->vals[1].ptr)};
    const unsigned long long cells =
        (unsigned long long)grid_size * (unsigned long long)grid_size;
    const uint32_t sentinel = (uint32_t)cells;
    if (data_is_double)
        weights_key_kernel<double><<<blocks, 256, 0, st>>>(
            n, (const double*)uu, (const double*)vv, c, sentinel, keys[0],
            skipped);
    else
        weights_key_kernel<float><<<blocks, 256, 0, st>>>(
            n, (const float*)uu, (const float*)vv, c, sentinel, keys[0],
            skipped);
    B200_TRY(cudaGetLastError());
    ++launches;
    int which = 0;
    B200_TRY(radix_sort_pairs(keys, vals, n, bit_length(cells),
                              counters + CNT_COUNT, status, ws->num_sms, st,
                              &which, &launches,
                              data_is_double
                                  ? nullptr
                                  : static_cast<const uint32_t*>(weight),
                              ws->expired.sort_tile));
    const size_t sum_want = (n + kSumThreads / 32 * kSpan - 1) /
                            (kSumThreads / 32 * kSpan);
    unsigned long long* host_status =
        static_cast<unsigned long long*>(ws->h_counters) + CNT_WEIGHTS_STATUS;
    const int sum_blocks = (int)std::min<size_t>(
        sum_want, (size_t)ws->num_sms * kSumCtasPerSm);
    if (data_is_double)
        weights_run_sum_kernel<double><<<sum_blocks, kSumThreads, 0, st>>>(
            n, keys[which], vals[which], (const double*)weight, sentinel,
            (double*)grid, status, host_status, counters + CNT_TASK_NEXT,
            skipped);
    else
        weights_run_sum_kernel<float><<<sum_blocks, kSumThreads, 0, st>>>(
            n, keys[which], vals[which], (const float*)weight, sentinel,
            (float*)grid, status, host_status, counters + CNT_TASK_NEXT,
            skipped);
    B200_TRY(cudaGetLastError());
    ++launches;
    ws->last_launches = launches;
    return OSKAR_B200_OK;
}

int run_weights_read(oskar_B200Workspace* ws, int data_is_double, size_t n,
                     const void* uu, const void* vv, const void* weight_in,
                     void* weight_out, double cell_size_rad, int grid_size,
                     const void* grid, unsigned long long* d_num_skipped,
                     double frequency_hz, cudaStream_t st)
{
    B200_TRY(ws->counters.ensure(sizeof(unsigned long long) * CNT_COUNT));
    unsigned long long* skipped = skip_counter(ws, d_num_skipped);
    B200_TRY(cudaMemsetAsync(skipped, 0, sizeof(unsigned long long), st));
    ws->last_launches = 0;
    if (n == 0) return OSKAR_B200_OK;
    const WeightConsts c = make_consts(data_is_double, cell_size_rad,
                                       grid_size, frequency_hz);
    const int blocks = launch_blocks(ws, n);
    if (data_is_double)
        weights_read_kernel<double><<<blocks, 256, 0, st>>>(
            n, (const double*)uu, (const double*)vv,
            (const double*)weight_in, (double*)weight_out, c,
            (const double*)grid, skipped);
    else
        weights_read_kernel<float><<<blocks, 256, 0, st>>>(
            n, (const float*)uu, (const float*)vv, (const float*)weight_in,
            (float*)weight_out, c, (const float*)grid, skipped);
    B200_TRY(cudaGetLastError());
    ws->last_launches = 1;
    return OSKAR_B200_OK;
}

}  // namespace b200
