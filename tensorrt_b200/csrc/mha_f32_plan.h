// Which form of the FP32 attention a launch takes (plain C++).
#pragma once
#include <stdint.h>

namespace b200
{

struct AttPlan
{
    int32_t rows;  // query rows of a CTA: 64 or 32
    int32_t perSm; // CTAs that may share an SM, 0: as many as fit
    bool async;    // keys and values by asynchronous copies (always with 32 rows)
    bool skip;     // keys beyond a sequence are left out
};

// FP32, heads of up to 64 channels (headSize: 32 or 64).
//
// How many CTAs share an SM. A launch whose CTAs are no more than one or two per SM (32 rows: three) is spread over all of them by the shared memory that it asks for:
// left to the placement of CTAs, three go to the first SM that the kernel before leaves. 64 rows, 12 heads, behind a fully connected layer of 4.7 us and with it,
// as placed / spread: 8 x 128 tokens 32.1 / 24.8 us, 4 x 256 55.4 / 41.6 us, 2 x 512 103 / 75 us; launch after launch 24.3 / 19.6, 44.7 / 36.4, 85.7 / 69.3 us; alone
// on the GPU there is no difference.
// Rows. 32 of them where twice as many CTAs still take a round of 64-row ones less, since the last CTAs of a launch that is a little more than one, two ...
// per SM cost as much as all before them. Alone on the GPU, 32 / 64 rows: 5 x 65 tokens, 16 heads 13.0 / 17 us, 7 x 200, 12 heads 37 / 47 us. Elsewhere 32 rows
// are slower (8 x 128, 12 heads 22.4 / 21.1 us, 2 x 512 78 / 71 us). From six rounds on it evens out, but for sequences of up to 32 tokens, where
// half of 64 rows would be empty.
// Copies. With one or two blocks of keys asynchronous ones hide most of the loads (4 x 64 tokens, 16 heads 9.2 us instead of 10.1 us). With more, the two
// barriers that they need on top cost 1 ... 2 % more than they bring (16 x 256, 12 heads 100.8 us instead of 99.6 us), since other CTAs' work hides the loads; with
// 32 channels, whose products are half as long, from one block on (12 heads, 8 x 384 7 %).
// Keys beyond a sequence. The loop that leaves them out is 1 ... 1.5 % slower (64 channels, 16 x 256, 12 heads), so it is not taken where there are none (`full`: all
// sequences have S tokens).
inline AttPlan planAtt(int32_t B, int32_t N, int32_t S, int32_t headSize, bool full, int64_t sms)
{
    int64_t const pairs = static_cast<int64_t>(B) * N;
    int64_t const n64 = (pairs * ((S - 1) / 64 + 1) + sms - 1) / sms, n32 = (pairs * ((S - 1) / 32 + 1) + sms - 1) / sms;
    if (n32 <= 2 * (n64 - 1) && (n64 <= 6 || S <= 32))
        return {32, n32 <= 3 ? static_cast<int32_t>(n32) : 0, true, true};
    bool const async = headSize == 64 && S <= 128;
    return {64, n64 <= 2 ? static_cast<int32_t>(n64) : 0, async, async || headSize != 64 || !full || S % 64 != 0};
}

} // namespace b200
