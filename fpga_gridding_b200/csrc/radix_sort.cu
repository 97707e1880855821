// Stable LSD radix sort of (uint32 key, uint32 value) pairs, written for this
// project (no CUB).
//
// One-sweep form: rs_histogram counts the digits of every pass in one read of
// the keys; then each 8-bit digit takes one launch, in which a tile of 4096
// pairs ranks its keys, publishes its digit counts, finds the counts of the
// tiles before it by decoupled look-back (Merrill and Garland's chained scan:
// a tile's word holds its own count until it knows the sum of all tiles up to
// it) and writes its pairs.  What a pass must move is 16 bytes per pair; a
// histogram, a three-launch scan and a scatter per digit (20 launches for 32
// bits) took 2.16 ms for 39 M pairs and 80 us for 10 thousand.
//
// Inside a tile each of 16 warps owns a contiguous run of 256 keys, read as 8
// coalesced rows of 32.  Lanes with equal digits find each other through a
// mask word per digit in shared memory; the running counts are private to the
// warp, so ranks need no block barrier.  The tile's pairs are put in digit
// order in shared memory and leave as one contiguous run per digit.  A pass is
// bound by the latency of that chain, so what counts is warps in flight: 39 M
// pairs, 4 passes, 8 warps of 16 rows (126 registers) 2.21 ms, 16 warps of 8
// rows at 3 blocks per SM 1.36 (1.46 at 2 blocks, 1.34 at 4 with spills);
// __match_any_sync instead of the mask words 2.35 against 2.21 ms.
//
// A look-back waits only for tiles with smaller tickets, which are running
// already.  The wait is bounded all the same: when it expires the sort sets
// DEV_ERR_TIMEOUT in the status word and writes nothing more, and the kernels
// that read the sorted pairs do nothing when that bit is set.
#include "common.cuh"
#include "internal.h"

namespace b200 {
namespace {

constexpr int kSortThreads = 512;
constexpr int kSortWarps = kSortThreads / 32;
constexpr int kSortItems = 8;
constexpr int kSortTile = kSortThreads * kSortItems;  // 4096
constexpr int kRadix = 256;
constexpr int kHistThreads = 256;
constexpr int kMaxPasses = 4;
constexpr int kLookback = 8;   // tiles read at once

// Scratch: tile words of one pass (see look_back), then the digit counts of
// every pass, turned into the digits' first positions by the histogram's last
// block, then one ticket per pass and the histogram's.
struct SortTemp
{
    unsigned long long* state;
    uint32_t* digits;     // [kMaxPasses][kRadix]
    uint32_t* tickets;    // [kMaxPasses + 1]
};

size_t sort_tiles(size_t n) { return (n + kSortTile - 1) / kSortTile; }

SortTemp sort_temp(void* temp, size_t n)
{
    SortTemp t;
    t.state = static_cast<unsigned long long*>(temp);
    t.digits = reinterpret_cast<uint32_t*>(t.state + sort_tiles(n) * kRadix);
    t.tickets = t.digits + kMaxPasses * kRadix;
    return t;
}

// Exclusive scan of one value per thread over the block's first kRadix
// threads (all threads call it).
__device__ __forceinline__ uint32_t digit_exclusive_scan(uint32_t v,
                                                         uint32_t* s_warp)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
        const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
    }
    if (lane == 31 && warp < kRadix / 32) s_warp[warp] = inc;
    __syncthreads();
    uint32_t before = 0;
#pragma unroll
    for (int w = 0; w < kRadix / 32; ++w) before += w < warp ? s_warp[w] : 0u;
    __syncthreads();
    return before + inc - v;
}

// Digit counts of every pass; the last block turns them into the digits'
// first positions.
__global__ void __launch_bounds__(kHistThreads)
rs_histogram_kernel(const uint32_t* __restrict__ keys, size_t n, int num_bits,
                    SortTemp t)
{
    __shared__ uint32_t s_count[kMaxPasses][kRadix];
    __shared__ uint32_t s_warp[kRadix / 32];
    __shared__ unsigned s_last;
    const int passes = (num_bits + 7) / 8;
    for (int i = threadIdx.x; i < kMaxPasses * kRadix; i += kHistThreads)
        (&s_count[0][0])[i] = 0;
    __syncthreads();
    const uint32_t top = (1u << (num_bits - 8 * (passes - 1))) - 1u;
    auto count = [&](uint32_t k) {
#pragma unroll
        for (int p = 0; p < kMaxPasses; ++p)
            if (p < passes)
                atomicAdd(&s_count[p][(k >> (8 * p)) &
                                      (p == passes - 1 ? top : 0xffu)], 1u);
    };
    // (the key buffers are at least 16-byte aligned)
    const uint4* keys4 = reinterpret_cast<const uint4*>(keys);
    const size_t stride = (size_t)gridDim.x * kHistThreads;
    const size_t first = (size_t)blockIdx.x * kHistThreads + threadIdx.x;
    size_t i = first;
    for (; i + stride < n / 4; i += 2 * stride)
    {
        const uint4 a = keys4[i], b = keys4[i + stride];
        count(a.x); count(a.y); count(a.z); count(a.w);
        count(b.x); count(b.y); count(b.z); count(b.w);
    }
    for (; i < n / 4; i += stride)
    {
        const uint4 a = keys4[i];
        count(a.x); count(a.y); count(a.z); count(a.w);
    }
    if (first < n % 4) count(keys[n - 1 - first]);
    __syncthreads();
    static_assert(kRadix == kHistThreads, "one digit per thread");
    for (int p = 0; p < passes; ++p)
    {
        const uint32_t c = s_count[p][threadIdx.x];
        if (c) atomicAdd(&t.digits[p * kRadix + threadIdx.x], c);
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0)
        s_last = atomicAdd(&t.tickets[kMaxPasses], 1u) == gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    for (int p = 0; p < passes; ++p)
    {
        uint32_t* d = t.digits + p * kRadix + threadIdx.x;
        *d = digit_exclusive_scan(__ldcg(d), s_warp);
    }
}

// Tile words: flag (2 bits) | pass + 1 (8 bits) | count.  The pass tells the
// words of this pass from those left by the one before.
constexpr unsigned long long kTileSum = 1ull << 62;        // this tile's count
constexpr unsigned long long kTilePrefix = 2ull << 62;     // all tiles up to it
constexpr unsigned long long kTileCount = (1ull << 40) - 1;

__device__ __forceinline__ unsigned long long load_word(
    const unsigned long long* p)
{
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p)
                 : "memory");
    return v;
}

__device__ __forceinline__ void store_word(unsigned long long* p,
                                           unsigned long long v)
{
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" :: "l"(p), "l"(v)
                 : "memory");
}

// Sum of the counts of tiles [0, tile), for the word column `col` (stride
// words per tile); false when the bounded wait expired.
__device__ __forceinline__ bool look_back(const unsigned long long* col,
                                          size_t stride, size_t tile,
                                          unsigned tag, uint32_t* sum)
{
    uint32_t s = 0;
    size_t end = tile;   // tiles [0, end) are still to be added
    unsigned spins = 0;
    bool done = tile == 0;
    while (!done)
    {
        unsigned long long w[kLookback];
#pragma unroll
        for (int j = 0; j < kLookback; ++j)
            w[j] = end > (size_t)j ? load_word(col + (end - 1 - j) * stride)
                                   : 0ull;
        int used = 0;
        bool ready = true;
#pragma unroll
        for (int j = 0; j < kLookback; ++j)
        {
            ready = ready && !done && (w[j] >> 62) != 0 &&
                    ((w[j] >> 40) & 0xffu) == tag;
            if (ready)
            {
                s += (uint32_t)(w[j] & kTileCount);
                ++used;
                done = (w[j] >> 62) == 2;
            }
        }
        end -= used;
        if (used == 0 && ++spins > kSpinLimit) return false;
    }
    *sum = s;
    return true;
}

// One pass.  vals_in null: the values are the positions 0 .. n - 1.
__global__ void __launch_bounds__(kSortThreads, 3)
rs_pass_kernel(const uint32_t* __restrict__ keys_in,
               const uint32_t* __restrict__ vals_in, size_t n, int pass,
               uint32_t mask, SortTemp t, unsigned long long* status,
               unsigned expired_tile, uint32_t* __restrict__ keys_out,
               uint32_t* __restrict__ vals_out)
{
    __shared__ uint16_t s_count[kSortWarps][kRadix];
    // The tile's pairs in digit order; before that, the lanes of each warp
    // that hold a digit.
    __shared__ uint32_t s_keys[kSortTile], s_vals[kSortTile];
    uint32_t (*s_peers)[kRadix] = reinterpret_cast<uint32_t (*)[kRadix]>(s_keys);
    static_assert(kSortWarps * kRadix <= kSortTile, "peer masks fit");
    __shared__ uint32_t s_out[kRadix];   // global minus in-tile position
    __shared__ uint32_t s_warp[kRadix / 32];
    __shared__ unsigned s_tile;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int shift = 8 * pass;
    if (threadIdx.x == 0)
        s_tile = (load_word(status) & DEV_ERR_TIMEOUT)
                     ? 0xffffffffu : atomicAdd(&t.tickets[pass], 1u);
    for (int i = threadIdx.x; i < kSortWarps * kRadix; i += kSortThreads)
    {
        (&s_count[0][0])[i] = 0;
        (&s_peers[0][0])[i] = 0;
    }
    __syncthreads();
    if (s_tile == 0xffffffffu) return;   // an earlier pass gave up
    const size_t tile = s_tile, tile0 = tile * kSortTile;
    const int tile_n = (int)min((size_t)kSortTile, n - tile0);
    const int base = warp * (32 * kSortItems) + lane;
    uint32_t key[kSortItems], rank[kSortItems];
    keys_in += tile0 + base;
#pragma unroll
    for (int i = 0; i < kSortItems; ++i)
        key[i] = base + i * 32 < tile_n ? keys_in[i * 32] : 0u;
#pragma unroll
    for (int i = 0; i < kSortItems; ++i)
    {
        const bool ok = base + i * 32 < tile_n;
        const unsigned d = (key[i] >> shift) & mask;
        if (ok) atomicOr(&s_peers[warp][d], 1u << lane);
        __syncwarp();
        const unsigned peers = ok ? s_peers[warp][d] : 0u;
        const uint32_t before = ok ? s_count[warp][d] : 0u;
        __syncwarp();
        if (ok && (peers >> lane) == 1u)   // the last of them
        {
            s_count[warp][d] = (uint16_t)(before + __popc(peers));
            s_peers[warp][d] = 0;
        }
        __syncwarp();
        rank[i] = before + __popc(peers & ((1u << lane) - 1u));
    }
    __syncthreads();
    // Digit d of the tile: its count, and the warps' starts inside the tile.
    const int d = threadIdx.x;
    const unsigned tag = (unsigned)pass + 1u;
    const unsigned long long tag_bits = (unsigned long long)tag << 40;
    unsigned long long* col = t.state + d;
    uint32_t total = 0;
    if (d < kRadix)
    {
#pragma unroll
        for (int w = 0; w < kSortWarps; ++w) total += s_count[w][d];
        store_word(col + tile * kRadix,
                   (tile == 0 ? kTilePrefix : kTileSum) | tag_bits | total);
    }
    const uint32_t start = digit_exclusive_scan(total, s_warp);
    if (d < kRadix)
    {
        uint32_t run = start;
#pragma unroll
        for (int w = 0; w < kSortWarps; ++w)
        {
            const uint32_t c = s_count[w][d];
            s_count[w][d] = (uint16_t)run;
            run += c;
        }
    }
    // (read only now: eight more registers through the ranking cost a third of
    // the warps in flight)
    uint32_t val[kSortItems];
    const uint32_t* vp = vals_in + tile0 + base;
#pragma unroll
    for (int i = 0; i < kSortItems; ++i)
        val[i] = vals_in && base + i * 32 < tile_n
                     ? vp[i * 32] : (uint32_t)tile0 + (uint32_t)(base + i * 32);
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kSortItems; ++i)
        if (base + i * 32 < tile_n)
        {
            const uint32_t local =
                s_count[warp][(key[i] >> shift) & mask] + rank[i];
            s_keys[local] = key[i];
            s_vals[local] = val[i];
        }
    bool ok = true;
    if (d < kRadix)
    {
        uint32_t before = 0;
        ok = s_tile != expired_tile &&
             look_back(col, kRadix, tile, tag, &before);
        if (ok && tile != 0)
            store_word(col + tile * kRadix,
                       kTilePrefix | tag_bits | (before + total));
        s_out[d] = t.digits[pass * kRadix + d] + before - start;
    }
    if (!__syncthreads_and(ok))
    {
        if (threadIdx.x == 0)
            atomicOr(status, (unsigned long long)DEV_ERR_TIMEOUT);
        return;
    }
#pragma unroll
    for (int i = 0; i < kSortItems; ++i)
    {
        const int q = i * kSortThreads + threadIdx.x;
        if (q < tile_n)
        {
            const uint32_t k = s_keys[q];
            const uint32_t dst = s_out[(k >> shift) & mask] + (uint32_t)q;
            if (dst < n)
            {
                keys_out[dst] = k;
                vals_out[dst] = s_vals[q];
            }
        }
    }
}

}  // namespace

size_t radix_sort_temp_bytes(size_t n)
{
    return sort_tiles(n) * kRadix * sizeof(unsigned long long) +
           (kMaxPasses * kRadix + kMaxPasses + 1) * sizeof(uint32_t);
}

cudaError_t radix_sort_pairs(uint32_t* keys[2], uint32_t* vals[2], size_t n,
                             int num_bits, void* temp,
                             unsigned long long* status, int num_sms,
                             cudaStream_t st, int* which, int* launches,
                             const uint32_t* first_vals,
                             unsigned expired_tile)
{
    *which = 0;
    if (n == 0) return cudaSuccess;
    const size_t tiles = sort_tiles(n);
    const SortTemp t = sort_temp(temp, n);
    const unsigned cap = (unsigned)num_sms * 4u;
    const size_t want = (n + 8 * kHistThreads - 1) / (8 * kHistThreads);
    const unsigned blocks = want < cap ? (unsigned)want : cap;
    if (num_bits < 1) num_bits = 1;
    rs_histogram_kernel<<<blocks, kHistThreads, 0, st>>>(keys[0], n, num_bits,
                                                         t);
    if (launches) *launches += 1;
    int cur = 0;
    for (int pass = 0; 8 * pass < num_bits; ++pass)
    {
        const int bits = num_bits - 8 * pass < 8 ? num_bits - 8 * pass : 8;
        rs_pass_kernel<<<(unsigned)tiles, kSortThreads, 0, st>>>(
            keys[cur], pass ? vals[cur] : first_vals, n, pass, (1u << bits) - 1u,
            t, status, expired_tile, keys[cur ^ 1], vals[cur ^ 1]);
        if (launches) *launches += 1;
        cur ^= 1;
    }
    *which = cur;
    return cudaGetLastError();
}

}  // namespace b200
