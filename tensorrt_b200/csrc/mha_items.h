// How the INT8 attention divides its work into items and deals them to persistent CTAs (plain C++, host and device).
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define B200_HOST_DEVICE __host__ __device__
#else
#define B200_HOST_DEVICE
#endif

namespace b200
{

constexpr int32_t kItemTile = 128;   // query rows per tile
constexpr int32_t kItemOrder = 256;  // sequences that a CTA can put in order
constexpr int32_t kItemRounds = 64;  // items per CTA that it can list

struct ItemPlan
{
    int32_t tilesPerItem, chunks; // an item = some (or all) query tiles of a (sequence, head) pair; chunks = items per pair
    bool longestFirst;            // the sequences are dealt in the order of their lengths, else as they come
};

// All tiles of a pair share one load of K and V, which an item waits for at about a third of a tile's time; items are cut smaller only
// when that shortens the longest CTA's list. Measured in an earlier form of the kernel, 8 % slower (16 heads; whole pairs in brackets): 2 x 512 tokens 9.4 us (30.2 us), 3 x 384 7.8 us (17.5
// us), 4 x 256 6.5 us (10.2 us), 12 x 384 22.5 us (31.8 us); 8 x 384 whole, 16.7 us.
// The lengths are on the device; what the host knows is how many tokens the batch has less than B * S (`missing`; INT64_MAX: unknown).
// With no more pairs than CTAs a cut into equal items is never the longer way, whatever they are. With more, pairs are cut only when every sequence is
// known to have the same number of tiles: whether halves or whole pairs even out better depends on where the long ones lie. Ragged
// batches keep whole pairs, and every CTA puts the sequences in the order of their lengths first (0.3 us) and takes a long pair, then a
// short one. Measured, packed, longest first / halves as they come / whole pairs as they come: 14 sequences of 87 ... 338 tokens, 12
// heads 17.6 / 21.3 / 30.9 us, others of these lengths 17.6 / 20.5 / 17.2 us, 16 of 67 ... 283 17.6 / 20.5 / 24.3 us, 47 of up to 422, 16 heads
// 95 / 137 / 121 us, 37 interleaved of 100 ... 256 whole either way: 41.0 us in order and as they come.
inline ItemPlan planItems(int32_t B, int32_t N, int32_t S, int64_t missing, int64_t ctas)
{
    int64_t const pairs = static_cast<int64_t>(B) * N;
    int32_t const nq = (S + kItemTile - 1) / kItemTile;
    ItemPlan plan{nq, 1, false};
    if (pairs > ctas && missing >= S - static_cast<int64_t>(nq - 1) * kItemTile) // a sequence may lack a whole tile
    {
        plan.longestFirst = B <= kItemOrder && pairs <= kItemRounds * ctas;
        return plan;
    }
    int64_t best = 0;
    for (int32_t tiles = nq; tiles >= 1; --tiles)
    {
        int32_t const chunks = (nq + tiles - 1) / tiles;
        int64_t const cost = (pairs * chunks + ctas - 1) / ctas * (3 * tiles + 1);
        if (tiles == nq || (cost < best && pairs * chunks <= INT32_MAX))
        {
            best = cost;
            plan.tilesPerItem = tiles;
            plan.chunks = chunks;
        }
    }
    return plan;
}

// Ragged packed batches of no more pairs than CTAs, which planItems leaves whole because full sequences would be: their tiles, one by one, in the order
// of the sequences' lengths. The longest pair then no longer holds up the launch, at the price of K and V for each tile. In the units above a tile
// costs up to four per key block and a whole pair 3 tiles + 1, so the cut is shorter while the rounds of tiles are fewer than that over four.
// The host knows the tokens only and guesses, half a tile per sequence for its last one and a sixteenth on top, whether that can be; then the CTAs, which
// put the lengths in order anyway, count the tiles and decide (cutIsShorter). The cut alone by the guess was up to 1.2 times as long (lengths just beyond a multiple
// of 128), and wherever S is far above the lengths. Measured (whole pairs / cut by the guess / as it is): 8 sequences of 90 ... 384 tokens, 16 heads
// 17.0 / 11.7 / 11.6 us, 12 of 32 ... 384, 12 heads 17.0 / 12.1 / 11.8 us; 5 of 133 ... 160, 16 heads 9.9 / 10.3 / 9.8 us (a launch that the host keeps whole
// 9.3 us), 92 of 129, one of 256, one head 9.9 / 15.9 / 10.8 us, 12 of up to 128 with S = 512, 12 heads 5.2 / 6.4 / 5.8 us (5.0 us).
// Returns the most tiles that there can be, or 0: not cut. tokens: of the batch.
inline int64_t cutTiles(int32_t B, int32_t N, int32_t S, int64_t tokens, int64_t ctas)
{
    int64_t const pairs = static_cast<int64_t>(B) * N, nq = (S + kItemTile - 1) / kItemTile;
    if (pairs > ctas || B > kItemOrder || tokens > pairs / N * S - (S - (nq - 1) * kItemTile))
        return 0;
    int64_t const about = N * (tokens / kItemTile + (B + 1) / 2), rounds = (about + about / 16 + ctas - 1) / ctas;
    int64_t const most = N * (tokens / kItemTile + B);
    return 4 * rounds < 3 * nq + 1 && most <= kItemRounds * ctas ? (most < pairs * nq ? most : pairs * nq) : 0;
}

// Whether `tiles` tiles, dealt one by one to `ctas` CTAs, are shorter than whole pairs, one to a CTA: 4 * rounds < 3 * longest + 1, so at most
// 3 / 4 * longest rounds. longest: tiles of the longest sequence.
B200_HOST_DEVICE inline bool cutIsShorter(int32_t tiles, int32_t longest, int32_t ctas)
{
    return tiles <= 3 * longest / 4 * ctas;
}

// The item that CTA `cta` takes in its `round`-th turn, the items being in the order of their lengths: every second round runs
// backwards, so that who had the longest of a round gets the shortest of the next. May lie beyond the last item in the last round.
B200_HOST_DEVICE inline int32_t itemOfRound(int32_t round, int32_t cta, int32_t ctas)
{
    return round * ctas + ((round & 1) != 0 ? ctas - 1 - cta : cta);
}

} // namespace b200
