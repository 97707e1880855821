// How many visibilities a CTA of the degridding kernel takes at a time (host
// code, no CUDA).
#pragma once

#include <algorithm>
#include <cstddef>

namespace b200 {

constexpr int kDegridChunk = 256;      // at most: one per thread
constexpr int kDegridChunkMin = 32;
constexpr int kDegridResident = 4;     // CTAs per SM that run at once

// Chunks of kDegridChunk share most.  They are halved
//   - while there are fewer of them than resident CTAs, which leaves SMs idle:
//     23 thousand FP64 points, supports 5 to 30, 450 -> 213 us a call;
//   - while the taps of one chunk at the widest support exceed a share of the
//     call that goes with its points: such chunks, last in the queue, are
//     waited for.  Three quarters of a tap per point, 0.6 in FP64, on 148 SMs,
//     and never below 300 thousand taps.
// Chunks of 256 / 128 / 64 / 32 (the rule's in brackets):
//   FP32, 242 thousand points, supports 4 to 16   [112] 115 us (a call)
//   FP32, 301 thousand points, supports 4 to 36    387  293  286 [325] us
//   FP32, 1.0 M, supports 4 to 36                  550 [518] 600  758 us
//   FP32, 1.0 M, supports 4 to 24                 [409] 409  473  615 us
//   FP32, 1.3 M, supports 4 to 127                6.19 5.03 4.73 [4.89] ms
//   FP64, 601 thousand, supports 4 to 36           766  609 [596] 695 us
//   FP64, 2.5 M, supports 4 to 127                16.7 14.3 13.1 [13.0] ms
// A fixed bound of 300 thousand taps in calls of up to 1.2 million points, and
// none above, took 32 and 256 at 1.0 M and 1.3 M: 760 us and 6.17 ms.
inline int degrid_chunk(size_t n, int max_support, bool is_double, int num_sms)
{
    const double w = 2.0 * max_support + 1.0;
    const double most = std::max(300000.0, (is_double ? 0.6 : 0.75) * (double)n);
    const size_t resident = (size_t)num_sms * kDegridResident;
    int chunk = kDegridChunk;
    while (chunk > kDegridChunkMin &&
           (n < resident * (size_t)chunk || chunk * w * w > most))
        chunk /= 2;
    return chunk;
}

}  // namespace b200
