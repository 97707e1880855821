// Checks b200::degrid_chunk (fpga_gridding_b200/csrc/degrid_plan.h): a power of
// two from 32 to 256, never larger for fewer points or wider supports, enough
// chunks to give every resident CTA one where that is possible, and within a
// seventh of the fastest of 32, 64, 128, 256 at the points where all four were
// measured (microseconds a call on 148 SMs, log-radial and disk layouts of 128
// and 400 stations).  Prints "ok" and exits 0, or prints the first violation
// and exits 1.
#include <cstdio>

#include "degrid_plan.h"

using namespace b200;

struct Measured
{
    bool f64;
    int support;
    size_t n;
    double us[4];   // 32, 64, 128, 256
};

static const Measured kMeasured[] = {
    {false, 24, 999744, {615.4, 473.4, 409.1, 409.2}},
    {false, 36, 300736, {325.2, 285.7, 293.4, 386.7}},
    {false, 36, 601472, {515.7, 431.0, 393.0, 452.8}},
    {false, 36, 999744, {757.7, 599.7, 517.6, 549.7}},
    {false, 36, 601472, {926.9, 816.4, 814.4, 946.5}},
    {false, 36, 999744, {1430.0, 1235.2, 1210.5, 1316.6}},
    {false, 36, 1037400, {904.4, 778.2, 782.8, 855.0}},
    {false, 30, 999744, {741.8, 573.7, 504.8, 508.3}},
    {false, 48, 999744, {1803.2, 1671.7, 1644.4, 1758.4}},
    {false, 64, 1300480, {3489.4, 3291.1, 3280.7, 3656.8}},
    {false, 127, 1300480, {4891.3, 4732.3, 5025.1, 6193.7}},
    {false, 127, 97536, {1141.7, 1664.4, 2272.2, 3076.2}},
    {true, 36, 601472, {695.2, 596.0, 609.0, 766.2}},
    {true, 36, 999744, {1039.5, 834.4, 792.4, 899.8}},
    {true, 30, 97536, {358.5, 404.7, 493.0, 777.6}},
    {true, 127, 1300480, {21366.2, 23642.1, 26480.4, 30565.4}},
    {true, 127, 2503424, {38597.7, 41059.0, 45399.6, 49682.1}},
};

int main()
{
    for (const Measured& m : kMeasured)
    {
        const int c = degrid_chunk(m.n, m.support, m.f64, 148);
        double best = m.us[0], got = -1.0;
        for (int i = 0; i < 4; ++i)
        {
            best = m.us[i] < best ? m.us[i] : best;
            if (c == 32 << i) got = m.us[i];
        }
        if (got < 0 || got > (1.0 + 1.0 / 7.0) * best)
        {
            std::printf("f64=%d support=%d n=%zu: chunk %d\n", m.f64,
                        m.support, m.n, c);
            return 1;
        }
    }
    // 242 thousand points of supports to 16: 112 us with 256, 115 with 128
    if (degrid_chunk(241920, 16, false, 148) != 256)
    {
        std::printf("short chunks of narrow footprints\n");
        return 1;
    }
    const size_t ns[] = {0, 1, 31, 18943, 18944, 37887, 37888, 75776, 151551,
                         151552, 300000, 1000000, 1300000, 5000000, 39000000,
                         4000000000ull};
    for (int sms : {1, 100, 148})
        for (int f64 = 0; f64 < 2; ++f64)
            for (int s = 0; s <= 127; ++s)
            {
                int last = 0;
                for (size_t n : ns)
                {
                    const int c = degrid_chunk(n, s, f64, sms);
                    const bool ok =
                        (c == 32 || c == 64 || c == 128 || c == 256) &&
                        c >= last &&
                        (s == 0 || c <= degrid_chunk(n, s - 1, f64, sms)) &&
                        (c == 32 || n / c >= (size_t)sms * kDegridResident);
                    if (!ok)
                    {
                        std::printf("n=%zu support=%d f64=%d sms=%d: %d\n", n,
                                    s, f64, sms, c);
                        return 1;
                    }
                    last = c;
                }
            }
    std::printf("ok\n");
    return 0;
}
