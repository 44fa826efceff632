// How the FP16 attention kernel divides its work over persistent CTAs: the query tiles of all (sequence, head) pairs, in one
// list, cut at equal costs.
//
// The list counts the tiles (128 queries) of sequence 0, then those of sequence 1, ..., within a sequence head by head. A tile
// costs its key blocks (128 keys) and a fixed amount for what is done once per tile. Neighbours of the list share keys and
// values, so a CTA still loads most of them once; cutting by cost instead of dealing whole pairs round-robin keeps all SMs busy
// to the end when the sequences differ in length, and lets several SMs work on a pair when there are few pairs. Measured in
// mha_f16_online.cu. (The INT8 kernel divides its work in its own way, mha_items.h: it works on one tile at a time and waits for the keys of every pair
// it starts, so pairs cut at equal costs take longer there: 37 interleaved sequences of 100 ... 256 tokens 45 us, 41 us whole.)
#pragma once
#include "common.cuh"

namespace b200
{

constexpr int kShareTile = 128;       // query rows per tile = keys per block
constexpr int kShareGeoEntries = 128; // sequences whose lengths are kept in shared memory

struct ShareArgs
{
    int32_t B, S, N;
    int32_t const* cu;      // packed layout: row offsets of the sequences; null: fixed layout
    int32_t const* maskIdx; // fixed layout: valid keys per sequence, or null
    bool tilePerCta;        // a CTA for every tile that the longest sequence allows for
    bool fewSequences;      // one per lane of a warp, and their costs add up in 32 bits

    __device__ __forceinline__ bool fixedLayout() const
    {
        return cu == nullptr;
    }
};

// One sequence: its first row (packed layout), query rows and valid keys, and the tiles per head and key blocks these make.
struct Sequence
{
    int32_t rowBase, rows, len, nq, nb;
};

// What a CTA computes: the tiles from (b0, i0) up to, not including, (b1, i1); i = head * nq + tile.
struct Share
{
    int32_t b0, i0, b1, i1;
};

struct ShareSmem
{
    Share share;
    uint64_t sums[32];           // one per warp
    int2 geo[kShareGeoEntries]; // length words of sequences geoBase ...
};

__device__ __forceinline__ int2 fetchGeometry(ShareArgs const& a, int32_t b)
{
    if (a.fixedLayout())
        return make_int2(0, a.maskIdx ? __ldg(a.maskIdx + b) : a.S);
    return make_int2(__ldg(a.cu + b), __ldg(a.cu + b + 1));
}

__device__ __forceinline__ Sequence makeSequence(ShareArgs const& a, int2 w)
{
    Sequence q;
    if (a.fixedLayout())
    {
        q.rowBase = 0;
        q.rows = a.S;
        q.len = min(max(w.y, 0), a.S);
    }
    else
    {
        q.rowBase = w.x;
        q.len = min(max(w.y - w.x, 0), a.S);
        q.rows = q.len;
    }
    q.nb = (q.len + kShareTile - 1) / kShareTile;
    q.nq = q.len > 0 ? (q.rows + kShareTile - 1) / kShareTile : 0; // without a valid key there is nothing to multiply
    return q;
}

// The sums fit 32 bits in all but extreme launches.
__device__ __forceinline__ uint64_t divideCost(uint64_t x, uint32_t y)
{
    return (x >> 32) == 0 ? static_cast<uint32_t>(x) / y : x / y;
}

// Finds the CTA's share; called by all threads. Returns whether there may be a sequence without a valid key.
// Fewer tiles than SMs: the CTA's number says which tile is its own. Few sequences: one per lane of warp 0. In general every
// thread sums the costs of a run of sequences, a scan over the block places the runs, and the threads in whose runs the share's
// two ends fall write them down. That takes 1.2 us (code fetched for a single use, three barriers), which small launches would feel:
// a sequence of two key blocks takes some 6 us in all. Few sequences: 0.3 us.
template <int kThreads, uint32_t kTileCost>
__device__ __forceinline__ bool findShare(ShareArgs const& a, ShareSmem* sm)
{
    static_assert(kThreads % 32 == 0 && kThreads >= kShareGeoEntries, "block size");
    Share* const share = &sm->share;
    uint64_t* const sums = sm->sums;
    int2* const geo = sm->geo;
    int const t = static_cast<int>(threadIdx.x), lane = t & 31, warp = t >> 5;
    uint32_t const ctas = gridDim.x, c = blockIdx.x;
    if (a.tilePerCta)
    {
        if (t == 0)
        {
            int32_t const nqMax = (a.S + kShareTile - 1) / kShareTile, perSequence = nqMax * a.N;
            int32_t const b = static_cast<int32_t>(c) / perSequence, i = static_cast<int32_t>(c) - b * perSequence;
            int32_t const head = i / nqMax, tile = i - head * nqMax;
            int2 const w = fetchGeometry(a, b);
            Sequence const q = makeSequence(a, w);
            geo[a.B <= kShareGeoEntries ? b : 0] = w;
            int32_t const at = head * q.nq + min(tile, q.nq); // beyond a shorter sequence: nothing
            *share = Share{b, at, b, tile < q.nq ? at + 1 : at};
        }
        __syncthreads();
        return a.maskIdx != nullptr;
    }
    if (a.fewSequences)
    {
        bool empty = false;
        if (warp == 0)
        {
            Sequence q{};
            if (lane < a.B)
            {
                int2 const w = fetchGeometry(a, lane);
                geo[lane] = w;
                q = makeSequence(a, w);
                empty = q.len == 0;
            }
            uint32_t const cost = static_cast<uint32_t>(q.nb) + kTileCost;
            uint32_t const own = static_cast<uint32_t>(q.nq * a.N) * cost;
            uint32_t end = own;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1)
            {
                uint32_t const v = __shfl_up_sync(0xffffffffu, end, o);
                end += lane >= o ? v : 0;
            }
            uint32_t const total = __shfl_sync(0xffffffffu, end, 31), part = total / ctas, rest = total - part * ctas;
            int32_t* const ends = reinterpret_cast<int32_t*>(share);
#pragma unroll
            for (int k = 0; k < 2; ++k) // first tile that starts at or behind the cut; (B, 0) when there is none
            {
                uint32_t const at = c + k, cut = part * at + min(at, rest);
                uint32_t const behind = __ballot_sync(0xffffffffu, cut < end);
                int const owner = behind != 0 ? __ffs(static_cast<int>(behind)) - 1 : 0;
                if (lane == owner)
                {
                    ends[2 * k] = behind != 0 ? lane : a.B;
                    ends[2 * k + 1] = behind != 0 ? static_cast<int32_t>((cut - (end - own) + cost - 1) / cost) : 0;
                }
            }
        }
        return __syncthreads_or(empty) != 0;
    }
    uint32_t const batch = static_cast<uint32_t>(a.B), per = (batch + kThreads - 1) / kThreads;
    int32_t const first = static_cast<int32_t>(min(batch, t * per)), last = static_cast<int32_t>(min(batch, t * per + per));
    uint64_t own = 0;
    bool empty = false;
    for (int32_t b = first; b < last; ++b)
    {
        int2 const w = fetchGeometry(a, b);
        if (b < kShareGeoEntries && a.B <= kShareGeoEntries)
            geo[b] = w;
        Sequence const q = makeSequence(a, w);
        empty = empty || q.len == 0;
        own += static_cast<uint64_t>(static_cast<uint32_t>(q.nq) * static_cast<uint32_t>(a.N)) * (static_cast<uint32_t>(q.nb) + kTileCost);
    }
    uint64_t end = own; // inclusive sum over the warp
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
        uint64_t const v = __shfl_up_sync(0xffffffffu, end, o);
        end += lane >= o ? v : 0;
    }
    if (lane == 31)
        sums[warp] = end;
    if (t == 0)
        *share = Share{a.B, 0, a.B, 0};
    bool const anyEmpty = __syncthreads_or(empty) != 0;
    uint64_t total = 0, before = 0;
#pragma unroll
    for (int i = 0; i < kThreads / 32; ++i)
    {
        before += i < warp ? sums[i] : 0;
        total += sums[i];
    }
    end += before;
    uint64_t const part = divideCost(total, ctas);
    uint32_t const rest = static_cast<uint32_t>(total - part * ctas);
    uint64_t const cut[2] = {part * c + min(c, rest), part * (c + 1) + min(c + 1, rest)};
#pragma unroll
    for (int k = 0; k < 2; ++k) // first tile that starts at or behind the cut; (B, 0) when there is none
    {
        if (cut[k] < end - own || cut[k] >= end)
            continue;
        uint64_t at = end - own;
        for (int32_t b = first; b < last; ++b)
        {
            Sequence const q = makeSequence(a, a.B <= kShareGeoEntries ? geo[b] : fetchGeometry(a, b));
            uint32_t const cost = static_cast<uint32_t>(q.nb) + kTileCost;
            uint64_t const seq = static_cast<uint64_t>(static_cast<uint32_t>(q.nq) * static_cast<uint32_t>(a.N)) * cost;
            if (cut[k] < at + seq)
            {
                int32_t const i = static_cast<int32_t>(divideCost(cut[k] - at + cost - 1, cost));
                if (k == 0)
                {
                    share->b0 = b;
                    share->i0 = i;
                }
                else
                {
                    share->b1 = b;
                    share->i1 = i;
                }
                break;
            }
            at += seq;
        }
    }
    __syncthreads();
    if (a.B > kShareGeoEntries)
    {
        int32_t const b = share->b0 + t;
        if (t < kShareGeoEntries && b < a.B)
            geo[t] = fetchGeometry(a, b);
        __syncthreads();
    }
    return anyEmpty;
}

// The share as runs of consecutive tiles of one (sequence, head).
struct ShareWalker
{
    ShareArgs const* ap;
    ShareSmem const* sm;
    Sequence g;
    int32_t b, head;
    int32_t runBegin, runEnd; // tiles of the run inside the (sequence, head)
    int32_t left;             // tiles of the sequence behind the run that are in the share

    __device__ __forceinline__ ShareWalker(ShareArgs const& args, ShareSmem const* s)
        : ap(&args)
        , sm(s)
    {
    }

    __device__ __forceinline__ bool firstRun()
    {
        b = sm->share.b0;
        return seek(sm->share.i0);
    }

    __device__ __forceinline__ bool nextRun()
    {
        if (left > 0) // more heads of this sequence
        {
            ++head;
            setRun(0, left);
            return true;
        }
        if (b == sm->share.b1)
            return false;
        ++b;
        return seek(0);
    }

private:
    __device__ __forceinline__ void setRun(int32_t t, int32_t tiles)
    {
        runBegin = t;
        runEnd = min(g.nq, t + tiles);
        left = tiles - (runEnd - t);
    }

    // settles on tile i of sequence b or the first one behind it that is in the share
    __device__ __forceinline__ bool seek(int32_t i)
    {
        int32_t const geoBase = ap->B <= kShareGeoEntries ? 0 : sm->share.b0;
        for (; b < ap->B; ++b, i = 0)
        {
            int32_t const e = b - geoBase;
            g = makeSequence(*ap, e < kShareGeoEntries ? sm->geo[e] : fetchGeometry(*ap, b));
            int32_t const end = b == sm->share.b1 ? sm->share.i1 : g.nq * ap->N;
            if (i < end)
            {
                head = i / g.nq;
                setRun(i - head * g.nq, end - i);
                return true;
            }
            if (b == sm->share.b1)
                break;
        }
        return false;
    }
};

inline ShareArgs shareArgs(int32_t B, int32_t S, int32_t N, int32_t const* cu, int32_t const* maskIdx)
{
    int64_t const nb = (S + kShareTile - 1) / kShareTile;
    return ShareArgs{B, S, N, cu, maskIdx, nb * B * N <= smCount(), B <= 32 && nb * (nb + 8) < (int64_t{1} << 31) / 32 / N};
}

// One CTA per SM, or fewer when there are fewer tiles.
inline int shareGrid(ShareArgs const& a)
{
    int64_t const tiles = static_cast<int64_t>(a.B) * a.N * ((a.S + kShareTile - 1) / kShareTile);
    return static_cast<int>(tiles < smCount() ? tiles : smCount());
}

} // namespace b200
