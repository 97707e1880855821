// Ordering of up to 256 points by one CTA (gridding tasks, degridding chunks).
#pragma once

#include <climits>

#include "common.cuh"
#include "grid_romein.cuh"

namespace b200 {

// Spreads the low 9 bits of x to the even bit positions.
__device__ __forceinline__ uint32_t spread9(uint32_t x)
{
    x &= 0x1ffu;
    x = (x | (x << 8)) & 0x00ff00ffu;
    x = (x | (x << 4)) & 0x0f0f0f0fu;
    x = (x | (x << 2)) & 0x33333333u;
    x = (x | (x << 1)) & 0x55555555u;
    return x;
}

// In-task order key, most significant first:
//   row-offset major (staged kernel values: each row offset's run reads one
//   W-row block):  (off_v + H) | Morton(gu, gv) | (off_u + H) | index
//   cell major (kernel values through L1):  column gu | row gv (up and down
//   in turn) | low bits of the w-plane | (off_v + H) | (off_u + H) | index.
//   Neighbours then mostly differ in gv: what leaves their shared footprint
//   is whole rows, which a warp adds to the grid as contiguous lanes, while a
//   step in gu flushes one lane of every row.  Against Morton order of the
//   same tasks: plain_large gridding 16.6 -> 16.3 ms, a 10x thinner one
//   2.15 -> 2.12 ms.
//   strips: strips of columns (up and down in turn) instead of single ones,
//   the wider the fewer points the task has for its box, so that neighbours
//   stay close in spread-out tasks too.  For FP64 data, whose flush is two
//   reductions and the most of such a task: 0.22 million points over 2580^2,
//   supports 5 to 33, gridding 699 -> 559 us (Morton order 576), 1.3 million
//   over 4096^2 1161 -> 1042; dense tasks within 1 %.  (Half and twice the
//   width within 2 %.)  FP32 data gains nothing (1710 -> 1732 us, 5.67 -> 5.79
//   ms in two such jobs), nor does compensation over all (0.54 million over
//   4096^2 1025 -> 914 us, 2.7 million over 2628^2 2380 -> 2440).
// The offsets take `ob` bits each (the bit width of 2H, H = ceil(os / 2)),
// the index the low 8 bits.  Cell major: column and row are counted from the
// task's smallest ones, so they need only the bits of its extent; what is
// left over tells planes apart (at least 3 bits; the low bits of the place are
// dropped where they do not fit).  Records with identical taps are adjacent,
// except where more planes meet in a cell than those bits can tell apart, or
// both signs of w (which the key leaves out).
struct TaskKey
{
    int ob, mb;           // row-offset major
    int u0, v0, bv, pb, shift, strip;
    // box: smallest and largest gu (x, y) and gv (z, w) of the task; strips: its
    // points where the columns are to be taken in strips, or 0
    __device__ __forceinline__ TaskKey(int half, const int4 box, int strips = 0)
    {
        ob = 32 - __clz(2 * half);
        const int avail = 32 - 8 - 2 * ob;
        mb = min(9, avail / 2);
        u0 = box.x;
        v0 = box.z;
        bv = 32 - __clz(box.w - box.z);
        const int bu = 32 - __clz(box.y - box.x), bits = bu + bv;
        // width 2^strip, its square at most twice the cells per point
        strip = 0;
        if (strips)
        {
            const float cells = (float)(box.y - box.x + 1) *
                                (float)(box.w - box.z + 1);
            const unsigned twice = (unsigned)(2.0f * cells / (float)strips);
            strip = min(max((31 - __clz(twice)) >> 1, 0), bu);
        }
        pb = min(max(avail - bits, 3), 15);
        shift = max(bits + pb - avail, 0);
    }
    template <bool CELL_MAJOR>
    __device__ __forceinline__ uint32_t make(const int4 r, unsigned t) const
    {
        const uint32_t ov = (uint32_t)(r.w >> 16), ou = (uint32_t)(r.w & 0xffff);
        if constexpr (CELL_MAJOR)
        {
            const uint32_t du = (uint32_t)(r.x - u0);
            uint32_t dv = (uint32_t)(r.y - v0);
            const uint32_t su = du >> strip;
            if (su & 1u) dv = (1u << bv) - 1u - dv;
            const uint32_t plane = (uint32_t)r.z & ((1u << pb) - 1u);
            const uint32_t place = (su << bv | dv) << strip |
                                   (du & ((1u << strip) - 1u));
            return (((((place >> shift) << pb | plane) << ob | ov) << ob | ou)
                    << 8) | t;
        }
        else
        {
            const uint32_t mask = (1u << mb) - 1u;
            const uint32_t morton = spread9((uint32_t)r.x & mask) |
                                    (spread9((uint32_t)r.y & mask) << 1);
            return (ov << (32 - ob)) | (morton << (8 + ob)) | (ou << 8) | t;
        }
    }
    __device__ __forceinline__ int row_offset(uint32_t key) const
    {
        return (int)(key >> (32 - ob));
    }
};

// Smallest and largest gu (x, y) and gv (z, w) of a task's records (`in`:
// this thread holds one).  All threads of the CTA must call it.
__device__ __forceinline__ int4 task_box(bool in, const int4 rec, int4* s_box)
{
    const int x0 = __reduce_min_sync(0xffffffffu, in ? rec.x : INT_MAX);
    const int x1 = __reduce_max_sync(0xffffffffu, in ? rec.x : INT_MIN);
    const int y0 = __reduce_min_sync(0xffffffffu, in ? rec.y : INT_MAX);
    const int y1 = __reduce_max_sync(0xffffffffu, in ? rec.y : INT_MIN);
    if ((threadIdx.x & 31) == 0)
        s_box[threadIdx.x >> 5] = make_int4(x0, x1, y0, y1);
    __syncthreads();
    int4 b = s_box[0];
#pragma unroll
    for (int q = 1; q < kGridThreads / 32; ++q)
    {
        const int4 c = s_box[q];
        b.x = min(b.x, c.x);
        b.y = max(b.y, c.y);
        b.z = min(b.z, c.z);
        b.w = max(b.w, c.w);
    }
    return b;
}

// Returns, for thread t < m, the key of the t-th visibility of the task in
// TaskKey order; its low 8 bits are the task-relative index of that
// visibility.  Bitonic sort of one key
// per thread (m <= 256); strides below 32 use warp shuffles, larger ones go
// through shared memory.  All threads of the CTA must call it.
__device__ __forceinline__ uint32_t task_order(uint32_t key,
                                               uint32_t* s_order)
{
    static_assert(kTaskMax == kGridThreads, "one key per thread");
    const unsigned t = threadIdx.x;
#pragma unroll
    for (unsigned k = 2; k <= (unsigned)kGridThreads; k <<= 1)
    {
#pragma unroll
        for (unsigned j = k >> 1; j > 0; j >>= 1)
        {
            uint32_t other;
            if (j >= 32)
            {
                s_order[t] = key;
                __syncthreads();
                other = s_order[t ^ j];
                __syncthreads();
            }
            else
            {
                other = __shfl_xor_sync(0xffffffffu, key, j);
            }
            const bool ascending = (t & k) == 0;
            const bool take_min = ((t & j) == 0) == ascending;
            key = take_min ? min(key, other) : max(key, other);
        }
    }
    return key;
}

}  // namespace b200
