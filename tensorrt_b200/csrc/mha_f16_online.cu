// FP16 fused multi-head attention on the sm_100a tensor cores with a key-block-wise online softmax
// (head sizes 16, 32, 48, 64; any sequence length), fixed [S,B,N,3,d], packed [total,N,3,d] and separate
// [B,N,S,d] layouts.
//
// Replaces, for FP16, the precompiled fused attention kernels the reference launches through
// FusedMHARunnerFP16[v2]::run (plugin/bertQKVToContextPlugin/mhaRunner.cu:835-860, 1127-1265) and its unfused
// cuBLAS + softmax path (mhaRunner.cu:533-601) for the sequence lengths those kernels do not cover.
//
// One persistent CTA per SM keeps TWO 128-query tiles in flight (streams 0 and 1). The tiles of the CTA's share of the
// work (mha_share.cuh) are dealt alternately to the two streams, across the boundaries of (sequence, head) pairs, so an
// odd number of tiles per pair (S = 384) leaves no stream idle. 12 warps:
//   warps 0-3 / 4-7 : softmax of stream 0 / 1, ONE THREAD PER QUERY ROW (the 32x32b TMEM load hands lane = row):
//                     no cross-thread reduction, no barrier among softmax threads. Per key block: load the 128
//                     scores into registers (their TMEM columns are then free for the next block's scores), block
//                     maximum, lazy rescale (below), p = exp2(x*scale*log2e - m), row sum, P as FP16 pairs into 64
//                     TMEM columns of its own. The normalising epilogue of a tile is deferred into the first block of
//                     the stream's next tile, so its wait for the last context product costs nothing.
//   warp 8          : loads the Q tiles (four slots, two per stream: with one, a tile's Q was requested only
//                     when the last scores of the tile before were done, which short sequences waited for).
//   warp 9          : loads K / V blocks (128 keys x 64 channels, 16 KB) into a ring of 10 stages. The
//                     blocks of a pair stay resident for all its query tiles when they fit (S <= 640); longer
//                     sequences stream their blocks once per two query tiles.
//   warps 10 / 11   : the MMA warp of stream 0 / 1 (an elected lane issues). It issues the stream's scores  S = Q K_j^T
//                     (128 x 128, FP32, TMEM columns 128*stream ..) as soon as the softmax threads hold the previous
//                     block in registers - the first block of the stream's NEXT tile right behind the last block of
//                     this one -, and the context products  O (+)= P_j V_j  (128 x 64, A operand = P straight from TMEM
//                     columns 256 + 64*stream .., accumulator in columns 384 + 64*stream ..) as soon as P_j is stored.
//                     (Every tcgen05.mma / commit keeps its issuing warp busy for 30-60 cycles: the twelve MMAs and
//                     four commits of a block are a warp's work of its own per stream.) A warp per stream may block
//                     on its stream's barriers; one warp serving both streams must not - an operand that a loader
//                     delivers only after the OTHER stream has been served would never arrive.
// Online softmax: the running maximum m only moves when the block maximum exceeds it by more than 8 in the log2
// domain (P then stays below 2^8, far inside FP16); when it moves, the softmax threads scale the row sum and the
// context accumulator in TMEM themselves (after the previous P V product has completed). The final context is
// O / rowsum. Compared with a softmax over the exact row maximum this changes nothing but the rounding of P.
// Measured (16 heads of 64; whole pairs dealt round-robin and one Q slot per stream before): 11 sequences of 200 ... 2000
// tokens 203 -> 113 us, 148 x 384 165 us, 37 x 1024 249 us; bound by the exponentials (a 128 x 128 block takes 1024
// cycles of the unit) at half of their rate: the two streams' other work is not hidden behind them completely.
// Every wait is bounded (sm100.cuh); on expiry the CTA drains, frees TMEM and reports through the status word.
#include "mha_share.cuh"
#include "sm100.cuh"

namespace b200
{

namespace
{

#ifdef MHA_TRACE
// timeline of CTA 0: (role, event code, cycle) triples, 512 events per role, roles 0/1 softmax, 2/3 MMA warps
#define TR_DECL(role) uint32_t trN = 0; uint32_t* const trBuf = (blockIdx.x == 0 && args.statusWord) ? args.statusWord + 16 + (role) * 1024 : nullptr
#define TR_EVT(code) do { if (trBuf && trN < 512) { trBuf[2 * trN] = (code); trBuf[2 * trN + 1] = static_cast<uint32_t>(clock64()); ++trN; } } while (0)
#else
#define TR_DECL(role)
#define TR_EVT(code)
#endif

constexpr int kTile = 128;       // query rows per tile = keys per block
constexpr int kHeadSize = 64;    // channels per tile row (smaller heads are zero-filled by the TMA unit)
constexpr int kStages = 10;      // K / V ring
constexpr int kQSlots = 4;       // Q tiles: two per stream, so that a tile's Q is on its way during the whole tile before it
constexpr int kStageBytes = kTile * kHeadSize * 2; // 16 KB: one Q tile, one K block, one V block
constexpr int kThreads = 384;    // 8 softmax warps, Q loader, K/V loader, two MMA issuers
constexpr uint32_t kTmemCols = 512;
constexpr uint32_t kPColumn = 256; // P blocks (FP16 pairs): 64 columns per stream
constexpr uint32_t kOColumn = 384; // context accumulators: 64 columns per stream
constexpr float kRescaleLog2 = 8.f;

struct OnlineArgs : ShareArgs
{
    int32_t d;
    void* out;
    float scaleBmm1;
    uint32_t* statusWord;
};

// [ Q slots ][ K/V stages ][ barriers ][ shares ]
constexpr int kSmemQ = 0;
constexpr int kSmemKv = kQSlots * kStageBytes;
constexpr int kSmemBars = kSmemKv + kStages * kStageBytes;
// full[kStages] empty[kStages] qFull[kQSlots] qFree[kQSlots] sFull[2] sFree[2] pReady[2] pvDone[2], tmem slot, abort flag
constexpr int kNumBars = 2 * kStages + 2 * kQSlots + 8;
constexpr int kSmemShare = kSmemBars + kNumBars * 8 + 16;
constexpr int kSmemBytes = kSmemShare + static_cast<int>(sizeof(ShareSmem)) + 1024;
// a query tile costs its key blocks and about one block more for what is done once per tile
constexpr uint32_t kTileCost = 1;

__device__ __forceinline__ float ex2Approx(float x)
{
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ float fmax3(float a, float b, float c)
{
    float y;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(y) : "f"(a), "f"(b), "f"(c));
    return y;
}

__device__ __forceinline__ uint32_t packHalf2(float lo, float hi)
{
    __half2 const h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t const*>(&h);
}

// The CTA's query tiles in processing order. Tile number n (counted per CTA) belongs to stream n & 1.
// A "sub-item" is the run of tiles that shares one load of the K / V blocks: all tiles of a (sequence, head) in the share
// when its blocks fit the ring, otherwise pairs of tiles (one per stream). `loadBase` is the number of K / V blocks loaded
// before it: block j of the sub-item is load number loadBase + 2j (K) and loadBase + 2j + 1 (V); a load number L lives in
// ring stage L % kStages and is the (L / kStages)-th fill of that stage.
struct Walker : ShareWalker
{
    int32_t t;        // query tile inside the (sequence, head)
    int32_t subEnd;   // one past the last tile of the sub-item
    int32_t subTiles; // tiles in the sub-item = uses of each of its stages
    uint32_t loadBase;
    uint32_t n;

    __device__ __forceinline__ Walker(OnlineArgs const& args, ShareSmem const* s)
        : ShareWalker(args, s)
    {
    }

    __device__ __forceinline__ bool resident() const
    {
        return 2 * g.nb <= kStages;
    }

    __device__ __forceinline__ void setSub()
    {
        subTiles = resident() ? runEnd - t : min(2, runEnd - t);
        subEnd = t + subTiles;
    }

    __device__ __forceinline__ bool begin()
    {
        n = 0;
        loadBase = 0;
        if (!firstRun())
            return false;
        t = runBegin;
        setSub();
        return true;
    }

    __device__ __forceinline__ bool next()
    {
        ++t;
        ++n;
        if (t == subEnd)
        {
            loadBase += 2u * static_cast<uint32_t>(g.nb);
            if (t == runEnd)
            {
                if (!nextRun())
                    return false;
                t = runBegin;
            }
            setSub();
        }
        return true;
    }

    __device__ __forceinline__ bool firstOfSub() const
    {
        return t == subEnd - subTiles;
    }
};

// The loads [first, last) of a ring of kStages stages, in load order, for a warp that reads none of them: wait until
// each block has landed, hand its stage back. Out of line: it runs once per tile at most and the kernel is sensitive to
// the size of its hot code.
static __device__ __noinline__ bool passThroughLoads(
    uint32_t fullAddr, uint32_t emptyAddr, uint32_t first, uint32_t last, volatile uint32_t* abortFlag)
{
    for (uint32_t L = first; L < last; ++L)
    {
        uint32_t const stage = L % kStages;
        if (!mbarWaitWarp(fullAddr + 8 * stage, (L / kStages) & 1u, abortFlag, kWaitTmaFull))
            return false;
        if (electOne())
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(emptyAddr + 8 * stage) : "memory");
        __syncwarp();
    }
    return true;
}

template <bool BNSD>
__global__ void __maxnreg__(168)
    mhaOnlineF16Kernel(const __grid_constant__ CUtensorMap mapQ, const __grid_constant__ CUtensorMap mapK,
        const __grid_constant__ CUtensorMap mapV, OnlineArgs const args)
{
    constexpr uint32_t kIdescQk = makeInstrDesc(1u, 0u, 0u, 0u, 128u, 128u);
    constexpr uint32_t kIdescPv = makeInstrDesc(1u, 0u, 0u, 1u, 128u, 64u);

    int const warp = threadIdx.x >> 5;
    int const lane = threadIdx.x & 31;

    extern __shared__ uint8_t smemRaw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smemRaw) + 1023) & ~static_cast<uintptr_t>(1023));
    uint8_t* sQ = smem + kSmemQ;
    uint8_t* sKv = smem + kSmemKv;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kSmemBars);
    uint64_t* full = bars;                    // [kStages] K / V block landed
    uint64_t* empty = bars + kStages;         // [kStages] every MMA that reads the stage has completed
    uint64_t* qFull = bars + 2 * kStages;     // [kQSlots] Q tile landed
    uint64_t* qFree = qFull + kQSlots;        // [kQSlots] all score MMAs of the slot's tile have completed
    uint64_t* sFull = qFree + kQSlots;        // [2]  scores of a key block complete               (once per block)
    uint64_t* sFree = sFull + 2;              // [2]  scores are in registers, 4 arrivals           (once per block)
    uint64_t* pReady = sFree + 2;             // [2]  P block written, 4 arrivals                   (once per block)
    uint64_t* pvDone = pReady + 2;            // [2]  context product of a block complete           (once per block)
    uint32_t* tmemSlot = reinterpret_cast<uint32_t*>(pvDone + 2);
    volatile uint32_t* abortFlag = tmemSlot + 1;
    ShareSmem* share = reinterpret_cast<ShareSmem*>(smem + kSmemShare);

    if (threadIdx.x == 0)
    {
        for (int i = 0; i < kStages; ++i)
        {
            mbarInit(&full[i], 1);
            mbarInit(&empty[i], 2); // one arrival per stream (see the MMA warps)
        }
        for (int i = 0; i < kQSlots; ++i)
        {
            mbarInit(&qFull[i], 1);
            mbarInit(&qFree[i], 1);
        }
        for (int i = 0; i < 2; ++i)
        {
            mbarInit(&sFull[i], 1);
            mbarInit(&sFree[i], 4); // one arrival per softmax warp of the stream
            mbarInit(&pReady[i], 4);
            mbarInit(&pvDone[i], 1);
        }
        *abortFlag = 0;
        fenceBarrierInit();
        prefetchTensorMap(&mapQ);
        if (BNSD)
        {
            prefetchTensorMap(&mapK);
            prefetchTensorMap(&mapV);
        }
    }
    if (warp == 8)
        tmemAlloc(tmemSlot, kTmemCols);
    tcFenceBefore();
    __syncthreads();
    tcFenceAfter();
    uint32_t const tmemBase = *tmemSlot;
    gridDependencyLaunch();
    gridDependencyWait();
    bool const anyEmpty = findShare<kThreads, kTileCost>(args, share);

    // which: 0 = Q, 1 = K, 2 = V; row = first token of the box inside the (packed or per-sequence) tensor
    auto load = [&](uint8_t* dst, uint64_t* bar, int which, Walker const& w, int32_t row) {
        if (BNSD) // (channel, position, head, sequence)
            tmaLoad4d(dst, which == 0 ? &mapQ : (which == 1 ? &mapK : &mapV), bar, 0, row, w.head, w.b);
        else // (channel, which of [N][3], batch, row)
            tmaLoad4d(dst, &mapQ, bar, 0, w.head * 3 + which, args.fixedLayout() ? w.b : 0, row);
    };

    if (warp == 8)
    {
        // ---- Q tiles: slot n % kQSlots, refilled when the score MMAs of the tile before in it have completed ----
        Walker w(args, share);
        bool ok = true;
        for (bool more = w.begin(); more && ok; more = w.next())
        {
            uint32_t const slot = w.n % kQSlots;
            if (w.n >= kQSlots)
                ok = mbarWaitWarp(smemAddr(&qFree[slot]), (w.n / kQSlots - 1) & 1u, abortFlag, kWaitStageFree);
            if (!ok)
                break;
            if (electOne())
            {
                mbarArriveExpectTx(&qFull[slot], kStageBytes);
                load(sQ + slot * kStageBytes, &qFull[slot], 0, w, (args.fixedLayout() ? 0 : w.g.rowBase) + w.t * kTile);
            }
            __syncwarp();
        }
    }
    else if (warp == 9)
    {
        // ---- K / V blocks of every sub-item, in the order the MMA warps consume them ----
        Walker w(args, share);
        bool ok = true;
        for (bool more = w.begin(); more && ok; more = w.next())
        {
            if (!w.firstOfSub())
                continue;
            int32_t const rowK = args.fixedLayout() ? 0 : w.g.rowBase;
            for (int j = 0; j < w.g.nb && ok; ++j)
            {
                for (int kv = 0; kv < 2 && ok; ++kv)
                {
                    uint32_t const L = w.loadBase + 2u * j + kv;
                    uint32_t const s = L % kStages;
                    uint32_t const fill = L / kStages;
                    if (fill > 0)
                        ok = mbarWaitWarp(smemAddr(&empty[s]), (fill - 1) & 1u, abortFlag, kWaitStageFree);
                    if (!ok)
                        break;
                    if (electOne())
                    {
                        mbarArriveExpectTx(&full[s], kStageBytes);
                        load(sKv + s * kStageBytes, &full[s], 1 + kv, w, rowK + j * kTile);
                    }
                    __syncwarp();
                }
            }
        }
    }
    else if (warp == 10 || warp == 11)
    {
        // ---- MMA issue: warp 10 owns stream 0, warp 11 stream 1 ----
        // The events of one stream come in a fixed order - scores of block j in registers (sFree), P_j written
        // (pReady), scores of block j+1 in registers, ... - so its thread simply waits for them in turn: after sFree it
        // issues the next scores (of this tile or of the stream's next one), after pReady the context product.
        uint32_t const s = static_cast<uint32_t>(warp - 10);
        // K-major Q / K tiles (128-byte rows, 128-byte swizzle): SBO = 8 rows = 1024 B. V is MN-major (the head
        // dimension contiguous): one MMA consumes 16 key rows = 2048 B.
        uint64_t const dQk = makeSmemDesc(0, 16, 1024, kSwizzle128B);
        uint64_t const dV = makeSmemDesc(0, 1024, 1024, kSwizzle128B);
        uint32_t const hiQk = static_cast<uint32_t>(dQk >> 32), hiV = static_cast<uint32_t>(dV >> 32);
        uint32_t const qLo = static_cast<uint32_t>(dQk) + (smemAddr(sQ) >> 4);
        uint32_t const kLo = static_cast<uint32_t>(dQk) + (smemAddr(sKv) >> 4);
        uint32_t const vLo = static_cast<uint32_t>(dV) + (smemAddr(sKv) >> 4);
        constexpr uint32_t kStage16 = kStageBytes >> 4;
        uint32_t const fullAddr = smemAddr(full), emptyAddr = smemAddr(empty);
        uint32_t const sFullAddr = smemAddr(&sFull[s]), sFreeAddr = smemAddr(&sFree[s]), pReadyAddr = smemAddr(&pReady[s]);
        uint32_t const pvDoneAddr = smemAddr(&pvDone[s]), qFullAddr = smemAddr(qFull), qFreeAddr = smemAddr(qFree);
        uint32_t const tS = tmemBase + s * kTile, tP = tmemBase + kPColumn + s * kHeadSize, tO = tmemBase + kOColumn + s * kHeadSize;
        bool ok = true;
        auto commitAddr = [](uint32_t barAddr) {
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(barAddr) : "memory");
        };
        // A ring stage goes back to the loader when BOTH streams' MMA warps are done with it: each commits once, with
        // its last tile of the sub-item. A sub-item of a single tile is read by one stream only; the other stream's
        // thread still takes part in every one of its loads (passThrough below).
        auto release = [&](uint32_t stage, Walker const& w) {
            if (w.t >= w.subEnd - 2)
                commitAddr(emptyAddr + 8 * stage);
        };
        // The loads of a single-tile sub-item of the OTHER stream, in load order: wait until the block has landed, hand
        // the stage back. A parity wait on an mbarrier is only valid for the barrier's NEXT phase, so a thread that
        // waits on the `full` barrier of a ring stage has to have seen every earlier fill of that stage - also the
        // fills whose data it never reads. (Skipping them - the other stream's thread adding the second arrival - let
        // a thread that came back to a stage two fills later see "complete" at once and multiply blocks that had not
        // landed: with many long sequences per CTA the attention hung until the waits expired.)
        auto passThrough = [&](Walker const& w) {
            ok = ok && passThroughLoads(fullAddr, emptyAddr, w.loadBase, w.loadBase + 2u * static_cast<uint32_t>(w.g.nb), abortFlag);
        };
        // scores of key block j of the tile `w` stands on
        auto issueQk = [&](Walker const& w, int32_t j) {
            uint32_t const L = w.loadBase + 2u * j;
            uint32_t const stage = L % kStages;
            ok = ok && mbarWaitWarp(fullAddr + 8 * stage, (L / kStages) & 1u, abortFlag, kWaitTmaFull);
            if (!ok)
                return;
            tcFenceAfter();
            uint32_t const b = kLo + stage * kStage16, slot = w.n % kQSlots, q = qLo + slot * kStage16;
            if (electOne())
            {
#pragma unroll
                for (int k = 0; k < 4; ++k) // head size 64 = 4 x 16
                    mmaLoHi<false>(tS, q + 2 * k, hiQk, b + 2 * k, hiQk, kIdescQk, k != 0);
                commitAddr(sFullAddr);
                release(stage, w);
                if (j == w.g.nb - 1)
                    commitAddr(qFreeAddr + 8 * slot);
            }
            __syncwarp();
        };
        auto issuePv = [&](Walker const& w, int32_t j) {
            uint32_t const L = w.loadBase + 2u * j + 1u;
            uint32_t const stage = L % kStages;
            ok = ok && mbarWaitWarp(fullAddr + 8 * stage, (L / kStages) & 1u, abortFlag, kWaitTmaFull);
            if (!ok)
                return;
            tcFenceAfter();
            uint32_t const b = vLo + stage * kStage16;
            if (electOne())
            {
#pragma unroll
                for (int k = 0; k < 8; ++k) // 128 keys = 8 x 16; P: 8 TMEM columns per 16 keys
                    mmaF16TmemA(tO, tP + 8 * k, b + k * 128u, hiV, kIdescPv, (j | k) != 0);
                commitAddr(pvDoneAddr);
                release(stage, w);
            }
            __syncwarp();
        };

        TR_DECL(2 + s);
        Walker cur(args, share);
        bool active = cur.begin();
        if (s == 1 && active)
        {
            // tile 0 is stream 0's
            if (cur.subTiles == 1)
                passThrough(cur);
            active = cur.next();
        }
        uint32_t qk = 0, pv = 0; // groups of score / context MMAs issued so far
        if (active && ok)
        {
            ok = mbarWaitWarp(qFullAddr + 8 * (cur.n % kQSlots), (cur.n / kQSlots) & 1u, abortFlag, kWaitTmaFull);
            if (ok)
                issueQk(cur, 0);
            qk = 1;
        }
        while (active && ok)
        {
            // the other stream's tile that follows this one, then this stream's next tile
            Walker nxt = cur;
            bool const hasMid = nxt.next();
            bool const midAlone = hasMid && nxt.subTiles == 1; // a sub-item this thread reads nothing of
            uint32_t const midFirst = nxt.loadBase, midBlocks = static_cast<uint32_t>(nxt.g.nb);
            bool const hasNext = hasMid && nxt.next();
            for (int j = 0; j < cur.g.nb && ok; ++j)
            {
                // Two things to issue per block: the scores that follow block j - block j + 1, or the first block of the
                // stream's next tile - and the context product of block j. The scores go first, so that the tensor pipe
                // has them done when the softmax threads come for them. Across a tile boundary the wait for their
                // operands then holds back the product whose completion frees this tile's last V stage, and the loader
                // works in load order: that is safe only while fewer than kStages - 1 loads lie between that V block and
                // the next tile's first K block (none when the tiles share sub-items; the 2 nb loads of the other stream's
                // tile when that is a sub-item of its own). With more, the loader would need the stage of that very V
                // block first - a cycle - and the product goes first. (One call site each for the two MMA groups: the
                // kernel is sensitive to the size of its code.)
                bool const lastBlock = j + 1 == cur.g.nb;
                bool qkPending = !lastBlock || hasNext, pvPending = true;
                bool const qkFirst = !lastBlock || !midAlone || midBlocks <= (kStages - 2) / 2;
                bool midPending = lastBlock && midAlone;
                if (qkPending)
                    ok = mbarWaitWarp(sFreeAddr, (qk - 1) & 1u, abortFlag, kWaitAccFree);
                TR_EVT(1);
#pragma unroll 1
                while ((qkPending || pvPending) && ok)
                {
                    if (qkPending && (qkFirst || !pvPending))
                    {
                        if (lastBlock)
                        {
                            if (midPending)
                                ok = passThroughLoads(fullAddr, emptyAddr, midFirst, midFirst + 2u * midBlocks, abortFlag);
                            midPending = false;
                            ok = ok && mbarWaitWarp(qFullAddr + 8 * (nxt.n % kQSlots), (nxt.n / kQSlots) & 1u, abortFlag, kWaitTmaFull);
                        }
                        if (ok)
                            issueQk(lastBlock ? nxt : cur, lastBlock ? 0 : j + 1);
                        TR_EVT(2);
                        ++qk;
                        qkPending = false;
                    }
                    else
                    {
                        ok = mbarWaitWarp(pReadyAddr, pv & 1u, abortFlag, kWaitSoftmax);
                        TR_EVT(3);
                        if (ok)
                            issuePv(cur, j);
                        TR_EVT(4);
                        ++pv;
                        pvPending = false;
                    }
                }
                // the other stream's last tile, when this stream has none after it
                if (midPending && ok)
                    ok = passThroughLoads(fullAddr, emptyAddr, midFirst, midFirst + 2u * midBlocks, abortFlag);
            }
            cur = nxt;
            active = hasNext;
        }
    }
    else
    {
        // ---- softmax: stream = warp / 4, query row = TMEM lane ----
        uint32_t const s = static_cast<uint32_t>(warp >> 2);
        int const r = (warp & 3) * 32 + lane;
        uint32_t const tRow = tmemBase + (static_cast<uint32_t>((warp & 3) * 32) << 16);
        uint32_t const tS = tRow + s * kTile;
        uint32_t const tP = tRow + kPColumn + s * kHeadSize;
        uint32_t const tO = tRow + kOColumn + s * kHeadSize;
        float const sl2 = args.scaleBmm1 * 1.4426950408889634f;
        float const thrRaw = kRescaleLog2 / sl2; // the same threshold on the unscaled scores
        bool ok = true;

        if (s == 0 && args.fixedLayout() && anyEmpty)
        {
            // sequences without a valid key: every probability is zero and so is the context row
            int const chunks16 = args.d / 8;
            for (int64_t u = blockIdx.x; u < static_cast<int64_t>(args.B) * args.N; u += gridDim.x)
            {
                int32_t const b = static_cast<int32_t>(u / args.N), head = static_cast<int32_t>(u % args.N);
                if (makeSequence(args, fetchGeometry(args, b)).len > 0)
                    continue;
                for (int i = threadIdx.x; i < args.S * chunks16; i += kTile)
                {
                    int const q = i / chunks16, c = i % chunks16;
                    __half* row = BNSD
                        ? static_cast<__half*>(args.out) + ((static_cast<int64_t>(b) * args.N + head) * args.S + q) * args.d
                        : static_cast<__half*>(args.out) + (static_cast<int64_t>(q) * args.B + b) * args.N * args.d + head * args.d;
                    reinterpret_cast<uint4*>(row)[c] = make_uint4(0, 0, 0, 0);
                }
            }
        }

        TR_DECL(lane == 0 && (warp & 3) == 0 ? s : 7);
        Walker w(args, share);
        bool active = w.begin() && (s == 0 || w.next());
        uint32_t blocks = 0; // key blocks this stream has completed: parity of sFull / pvDone
        // the tile whose context still has to be normalised and stored (null: none, or a row beyond the sequence)
        bool pending = false;
        __half* pendDst = nullptr;
        float pendInv = 0.f;
        // context of the stream's previous tile: wait for its last product, O / rowsum -> FP16
        auto epilogue = [&]() {
            ok = ok && mbarWait(&pvDone[s], (blocks - 1) & 1u, abortFlag, kWaitAccFull);
            tcFenceAfter();
#pragma unroll 1
            for (int c = 0; c < kHeadSize; c += 16) // 16 columns at a time: the block's scores stay in registers
            {
                uint32_t o[16];
                tmemLoad16(tO + c, o);
                tmemLoadWait16(o);
                if (pendDst != nullptr && ok && c < args.d)
                {
                    float f[8];
#pragma unroll
                    for (int h = 0; h < 2; ++h)
                    {
#pragma unroll
                        for (int i = 0; i < 8; ++i)
                            f[i] = __uint_as_float(o[8 * h + i]) * pendInv;
                        reinterpret_cast<uint4*>(pendDst + c)[h] = packHalf8(f);
                    }
                }
            }
            tcFenceBefore();
            pending = false;
        };
        // Keys at or beyond `limit` (counted from the chunk's first column) take no part: -inf scores, zero probabilities.
        auto maskChunk = [](uint32_t(&x)[32], int limit) {
            if (limit < 32)
            {
#pragma unroll
                for (int i = 0; i < 32; ++i)
                    if (i >= limit)
                        x[i] = 0xff800000u;
            }
        };
        while (active)
        {
            Sequence const g = w.g;
            float mRun = -INFINITY;
            uint64_t l01 = 0, l23 = 0; // row sums of every fourth key, two to a register pair
#pragma unroll 1
            for (int j = 0; j < g.nb; ++j)
            {
                TR_EVT(10);
                ok = ok && mbarWait(&sFull[s], blocks & 1u, abortFlag, kWaitSoftmax);
                tcFenceAfter();
                TR_EVT(11);
                int const limit = g.len - j * kTile;
                // All 128 scores of the row go to registers at once; their TMEM columns are free for the next block's
                // scores from here on, so the tensor pipe works on S_{j+1} during this block's exponentials.
                uint32_t x0[32], x1[32], x2[32], x3[32];
                tmemLoad32(tS, x0);
                tmemLoad32(tS + 32, x1);
                tmemLoad32(tS + 64, x2);
                tmemLoad32(tS + 96, x3);
                tmemLoadWait32(x0);
                tmemLoadWait32(x1);
                tmemLoadWait32(x2);
                tmemLoadWait32(x3);
                tcFenceBefore();
                __syncwarp();
                if (lane == 0)
                    mbarArrive(&sFree[s]);
                TR_EVT(12);
                // eight independent chains: the block maximum costs the latency of eight dependent maxima, not thirty-two
                float mA = -INFINITY, mB = -INFINITY, mC = -INFINITY, mD = -INFINITY;
                float mE = -INFINITY, mF = -INFINITY, mG = -INFINITY, mH = -INFINITY;
                maskChunk(x0, limit);
                maskChunk(x1, limit - 32);
                maskChunk(x2, limit - 64);
                maskChunk(x3, limit - 96);
#pragma unroll
                for (int i = 0; i < 32; i += 4)
                {
                    mA = fmax3(mA, __uint_as_float(x0[i]), __uint_as_float(x0[i + 1]));
                    mB = fmax3(mB, __uint_as_float(x0[i + 2]), __uint_as_float(x0[i + 3]));
                    mC = fmax3(mC, __uint_as_float(x1[i]), __uint_as_float(x1[i + 1]));
                    mD = fmax3(mD, __uint_as_float(x1[i + 2]), __uint_as_float(x1[i + 3]));
                    mE = fmax3(mE, __uint_as_float(x2[i]), __uint_as_float(x2[i + 1]));
                    mF = fmax3(mF, __uint_as_float(x2[i + 2]), __uint_as_float(x2[i + 3]));
                    mG = fmax3(mG, __uint_as_float(x3[i]), __uint_as_float(x3[i + 1]));
                    mH = fmax3(mH, __uint_as_float(x3[i + 2]), __uint_as_float(x3[i + 3]));
                }
                mA = fmax3(mA, mB, mC);
                mD = fmax3(mD, mE, mF);
                mG = fmaxf(mG, mH);
                float const mBlk = fmax3(mA, mD, mG);
                if (j == 0)
                    mRun = mBlk;
                else
                {
                    // The running maximum moves only when this block exceeds it by more than 2^8 after scaling.
                    bool const move = mBlk > mRun + thrRaw;
                    if (__any_sync(0xffffffffu, move))
                    {
                        float const f = move ? ex2Approx((mRun - mBlk) * sl2) : 1.f;
                        if (move)
                            mRun = mBlk;
                        uint64_t const ff = pack2(f, f);
                        l01 = mul2(l01, ff);
                        l23 = mul2(l23, ff);
                        // the context so far, once the previous block's product has completed
                        ok = ok && mbarWait(&pvDone[s], (blocks - 1) & 1u, abortFlag, kWaitAccFull);
                        tcFenceAfter();
#pragma unroll 1
                        for (int c = 0; c < kHeadSize; c += 16)
                        {
                            uint32_t o[16];
                            tmemLoad16(tO + c, o);
                            tmemLoadWait16(o);
#pragma unroll
                            for (int i = 0; i < 16; ++i)
                                o[i] = __float_as_uint(__uint_as_float(o[i]) * f);
                            tmemStore16(tO + c, o);
                        }
                    }
                }
                float const negM = -mRun * sl2;
                uint64_t const scale2 = pack2(sl2, sl2), negM2 = pack2(negM, negM);

                // p = exp2(x * scale * log2e - m), row sum, P as FP16 pairs (32 keys -> 16 columns)
                auto expChunk = [&](uint32_t(&x)[32], uint32_t(&p)[16]) {
#pragma unroll
                    for (int i = 0; i < 32; i += 4)
                    {
                        float e0, e1, e2, e3;
                        unpack2(fma2(pack2(__uint_as_float(x[i]), __uint_as_float(x[i + 1])), scale2, negM2), e0, e1);
                        unpack2(fma2(pack2(__uint_as_float(x[i + 2]), __uint_as_float(x[i + 3])), scale2, negM2), e2, e3);
                        e0 = ex2Approx(e0);
                        e1 = ex2Approx(e1);
                        e2 = ex2Approx(e2);
                        e3 = ex2Approx(e3);
                        l01 = add2(l01, pack2(e0, e1));
                        l23 = add2(l23, pack2(e2, e3));
                        p[i / 2] = packHalf2(e0, e1);
                        p[i / 2 + 1] = packHalf2(e2, e3);
                    }
                };
                {
                    uint32_t pa[16], pb[16];
                    TR_EVT(13);
                    expChunk(x0, pa);
                    expChunk(x1, pb);
                    TR_EVT(14);
                    // The P columns are read by the previous block's product and the context accumulator by the previous
                    // tile's epilogue: half a block of exponentials later both are long done.
                    if (pending)
                        epilogue();
                    else if (blocks > 0)
                        ok = ok && mbarWait(&pvDone[s], (blocks - 1) & 1u, abortFlag, kWaitAccFull);
                    TR_EVT(15);
                    tmemStore16(tP, pa);
                    tmemStore16(tP + 16, pb);
                    expChunk(x2, pa);
                    tmemStore16(tP + 32, pa);
                    expChunk(x3, pb);
                    tmemStore16(tP + 48, pb);
                    TR_EVT(16);
                }
                tmemStoreWait();
                tcFenceBefore();
                __syncwarp();
                if (lane == 0)
                    mbarArrive(&pReady[s]);
                TR_EVT(17);
                ++blocks;
            }
            int const q = w.t * kTile + r;
            pending = true;
            float l0, l1, l2, l3;
            unpack2(l01, l0, l1);
            unpack2(l23, l2, l3);
            asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(pendInv) : "f"((l0 + l1) + (l2 + l3)));
            pendDst = nullptr;
            if (q < g.rows)
            {
                if (BNSD)
                    pendDst = static_cast<__half*>(args.out) + ((static_cast<int64_t>(w.b) * args.N + w.head) * args.S + q) * args.d;
                else
                {
                    int64_t const rr = args.fixedLayout() ? static_cast<int64_t>(q) * args.B + w.b : static_cast<int64_t>(g.rowBase) + q;
                    pendDst = static_cast<__half*>(args.out) + rr * args.N * args.d + w.head * args.d;
                }
            }
            active = w.next() && w.next();
        }
        if (pending)
            epilogue();
        tcFenceBefore();
    }

    __syncthreads();
    uint32_t const aborted = *abortFlag;
    if (aborted != 0)
    {
        uint64_t const t0 = globalTimerNs();
        while (globalTimerNs() - t0 < 1000000ull)
            __nanosleep(1000);
        if (threadIdx.x == 0 && args.statusWord)
            atomicMax(args.statusWord, aborted);
        __syncthreads();
    }
    if (warp == 8)
    {
        __syncwarp();
        tcFenceAfter();
        tmemFree(tmemBase, kTmemCols);
    }
}

// Sequences of at most one key block: one CTA per (sequence, head), four warps that do everything in turn.
//
// A launch of few such tiles is a chain of latencies: lengths, loads, scores, softmax, product, store. The persistent kernel adds
// to them what its division of the work and the hand-overs between its twelve warps take, and the fetch of 80 KB of code, of
// which a tile runs through a small part: a forward's other kernels have replaced it in the instruction caches since the layer
// before. Here the code is a few KB, and a tile takes 50 KB of shared memory, 128 columns of tensor memory (P and the context lie where the scores
// were) and 150 registers a thread, so that three CTAs can share an SM. The arithmetic is that of the persistent kernel, to the bit. Measured, 16 heads
// (persistent kernel in brackets): 1 x 37 tokens 3.4 us (5.1 us), 8 x 128 4.4 us (6.4 us), 36 x 64 7.1 us (12.6 us), 148 x 128 34.0 us (42.8 us).
// Two or three: see launchOnline.
constexpr int kShortThreads = 128;
constexpr int kShortBars = 3 * kStageBytes; // after Q, K and V
constexpr int kShortSmemBytes = kShortBars + 64 + 1024;
constexpr int kShortSmemTwo = 80 * 1024; // asked for where two CTAs are to share an SM
constexpr uint32_t kShortTmemCols = 128; // scores; once they are in registers, P in the first 64 columns and the context in the others

// COLS: tensor memory of a CTA, 128 or 256 columns (an argument instead has to arrive before the allocation: 1 x 37 ... 8 x 128 tokens alone on the GPU 0.1 us)
template <bool BNSD, uint32_t COLS>
__global__ void __launch_bounds__(kShortThreads, 3) mhaShortF16Kernel(const __grid_constant__ CUtensorMap mapQ,
    const __grid_constant__ CUtensorMap mapK, const __grid_constant__ CUtensorMap mapV, OnlineArgs const args)
{
    constexpr uint32_t kIdescQk = makeInstrDesc(1u, 0u, 0u, 0u, 128u, 128u);
    constexpr uint32_t kIdescPv = makeInstrDesc(1u, 0u, 0u, 1u, 128u, 64u);
    int const warp = threadIdx.x >> 5;

    extern __shared__ uint8_t smemRaw[];
    uint8_t* const smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smemRaw) + 1023) & ~static_cast<uintptr_t>(1023));
    uint8_t* const sQ = smem;
    uint8_t* const sK = smem + kStageBytes;
    uint8_t* const sV = smem + 2 * kStageBytes;
    uint64_t* const qkFull = reinterpret_cast<uint64_t*>(smem + kShortBars);
    uint64_t* const vFull = qkFull + 1;
    uint64_t* const sFull = qkFull + 2;
    uint64_t* const oFull = qkFull + 3;
    uint32_t* const tmemSlot = reinterpret_cast<uint32_t*>(qkFull + 4);
    volatile uint32_t* const abortFlag = tmemSlot + 1;
    if (threadIdx.x == 0)
    {
        for (int i = 0; i < 4; ++i)
            mbarInit(&qkFull[i], 1);
        *abortFlag = 0;
        fenceBarrierInit();
        prefetchTensorMap(&mapQ);
        if (BNSD)
        {
            prefetchTensorMap(&mapK);
            prefetchTensorMap(&mapV);
        }
    }
    __syncwarp();
    if (warp == 0)
        tmemAlloc(tmemSlot, COLS);
    tcFenceBefore();
    __syncthreads();
    tcFenceAfter();
    uint32_t const tmemBase = *tmemSlot;
    gridDependencyLaunch();
    gridDependencyWait();

    int32_t const b = static_cast<int32_t>(blockIdx.x) / args.N, head = static_cast<int32_t>(blockIdx.x) - b * args.N;
    Sequence const g = makeSequence(args, fetchGeometry(args, b));
    int const q = static_cast<int>(threadIdx.x); // query row = TMEM lane
    __half* dst = nullptr;
    if (q < g.rows)
    {
        if (BNSD)
            dst = static_cast<__half*>(args.out) + ((static_cast<int64_t>(b) * args.N + head) * args.S + q) * args.d;
        else
        {
            int64_t const row = args.fixedLayout() ? static_cast<int64_t>(q) * args.B + b : static_cast<int64_t>(g.rowBase) + q;
            dst = static_cast<__half*>(args.out) + row * args.N * args.d + head * args.d;
        }
    }
    if (g.len > 0) // the same for all threads
    {
        auto load = [&](uint8_t* to, uint64_t* bar, int which) {
            if (BNSD) // (channel, position, head, sequence)
                tmaLoad4d(to, which == 0 ? &mapQ : (which == 1 ? &mapK : &mapV), bar, 0, 0, head, b);
            else // (channel, which of [N][3], batch, row)
                tmaLoad4d(to, &mapQ, bar, 0, head * 3 + which, args.fixedLayout() ? b : 0, g.rowBase);
        };
        bool ok = true;
        if (warp == 0)
        {
            if (electOne())
            {
                mbarArriveExpectTx(qkFull, 2 * kStageBytes);
                load(sQ, qkFull, 0);
                load(sK, qkFull, 1);
                mbarArriveExpectTx(vFull, kStageBytes);
                load(sV, vFull, 2);
            }
            __syncwarp();
            ok = mbarWaitWarp(smemAddr(qkFull), 0, abortFlag, kWaitTmaFull);
            tcFenceAfter();
            if (electOne() && ok)
            {
                uint64_t const d = makeSmemDesc(0, 16, 1024, kSwizzle128B);
                uint32_t const lo = static_cast<uint32_t>(d), hi = static_cast<uint32_t>(d >> 32);
#pragma unroll
                for (int k = 0; k < 4; ++k) // head size 64 = 4 x 16
                    mmaLoHi<false>(tmemBase, lo + (smemAddr(sQ) >> 4) + 2 * k, hi, lo + (smemAddr(sK) >> 4) + 2 * k, hi, kIdescQk, k != 0);
                tcCommit(sFull);
            }
            __syncwarp();
        }
        uint32_t const tRow = tmemBase + (static_cast<uint32_t>(warp * 32) << 16);
        uint32_t const tP = tRow, tO = tRow + 64;
        float const sl2 = args.scaleBmm1 * 1.4426950408889634f;
        ok = ok && mbarWait(sFull, 0, abortFlag, kWaitSoftmax);
        __syncwarp();
        tcFenceAfter();
        uint32_t x[4][32];
        float m = -INFINITY;
#pragma unroll
        for (int c = 0; c < 4; ++c)
        {
            int const limit = g.len - c * 32;
            if (limit <= 0) // nothing is done for chunks of keys beyond the sequence
                continue;
            tmemLoad32(tRow + c * 32, x[c]);
            tmemLoadWait32(x[c]);
            if (limit < 32)
            {
#pragma unroll
                for (int i = 0; i < 32; ++i)
                    if (i >= limit)
                        x[c][i] = 0xff800000u;
            }
#pragma unroll
            for (int i = 0; i < 32; i += 2)
                m = fmax3(m, __uint_as_float(x[c][i]), __uint_as_float(x[c][i + 1]));
        }
        float const negM = -m * sl2;
        uint64_t const scale2 = pack2(sl2, sl2), negM2 = pack2(negM, negM);
        uint64_t l01 = 0, l23 = 0;
#pragma unroll
        for (int c = 0; c < 4; ++c)
        {
            if (g.len <= c * 32)
                continue;
            uint32_t p[16];
#pragma unroll
            for (int i = 0; i < 32; i += 4)
            {
                float e0, e1, e2, e3;
                unpack2(fma2(pack2(__uint_as_float(x[c][i]), __uint_as_float(x[c][i + 1])), scale2, negM2), e0, e1);
                unpack2(fma2(pack2(__uint_as_float(x[c][i + 2]), __uint_as_float(x[c][i + 3])), scale2, negM2), e2, e3);
                e0 = ex2Approx(e0);
                e1 = ex2Approx(e1);
                e2 = ex2Approx(e2);
                e3 = ex2Approx(e3);
                l01 = add2(l01, pack2(e0, e1));
                l23 = add2(l23, pack2(e2, e3));
                p[i / 2] = packHalf2(e0, e1);
                p[i / 2 + 1] = packHalf2(e2, e3);
            }
            tmemStore16(tP + c * 16, p);
        }
        tmemStoreWait();
        tcFenceBefore();
        __syncthreads();
        if (warp == 0)
        {
            ok = ok && mbarWaitWarp(smemAddr(vFull), 0, abortFlag, kWaitTmaFull);
            tcFenceAfter();
            if (electOne() && ok)
            {
                // V is MN-major (the head dimension contiguous): one MMA consumes 16 key rows = 2048 bytes
                uint64_t const d = makeSmemDesc(0, 1024, 1024, kSwizzle128B);
                uint32_t const lo = static_cast<uint32_t>(d) + (smemAddr(sV) >> 4), hi = static_cast<uint32_t>(d >> 32);
#pragma unroll
                for (int k = 0; k < 8; ++k)
                    if (k * 16 < g.len)
                        mmaF16TmemA(tmemBase + 64, tmemBase + 8 * k, lo + k * 128u, hi, kIdescPv, k != 0);
                tcCommit(oFull);
            }
            __syncwarp();
        }
        float l0, l1, l2, l3, inv;
        unpack2(l01, l0, l1);
        unpack2(l23, l2, l3);
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(inv) : "f"((l0 + l1) + (l2 + l3)));
        ok = ok && mbarWait(oFull, 0, abortFlag, kWaitAccFull);
        __syncwarp();
        tcFenceAfter();
#pragma unroll
        for (int c = 0; c < kHeadSize; c += 32)
        {
            uint32_t o[32];
            tmemLoad32(tO + c, o);
            tmemLoadWait32(o);
            if (dst != nullptr && ok)
            {
#pragma unroll
                for (int h = 0; h < 4; ++h)
                {
                    float f[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        f[i] = __uint_as_float(o[8 * h + i]) * inv;
                    if (c + 8 * h < args.d)
                        reinterpret_cast<uint4*>(dst + c)[h] = packHalf8(f);
                }
            }
        }
        tcFenceBefore();
    }
    else if (dst != nullptr) // no valid key: every probability is zero and so is the context row
    {
        for (int c = 0; c < args.d / 8; ++c)
            reinterpret_cast<uint4*>(dst)[c] = make_uint4(0, 0, 0, 0);
    }

    __syncthreads();
    uint32_t const aborted = *abortFlag;
    if (aborted != 0)
    {
        uint64_t const t0 = globalTimerNs();
        while (globalTimerNs() - t0 < 1000000ull)
            __nanosleep(1000);
        if (threadIdx.x == 0 && args.statusWord)
            atomicMax(args.statusWord, aborted);
        __syncthreads();
    }
    if (warp == 0)
    {
        __syncwarp();
        tcFenceAfter();
        tmemFree(tmemBase, COLS);
    }
}

template <bool BNSD>
int32_t launchOnline(CUtensorMap const (&maps)[3], OnlineArgs args, cudaStream_t stream)
{
    int64_t const pairs = static_cast<int64_t>(args.B) * args.N;
    if (args.S <= kTile && pairs <= INT32_MAX) // one key block: the short kernel is ahead from one pair to thousands (see there)
    {
        // How many CTAs share an SM. Three where that takes fewer rounds than two: 32 x 64 ... 128 tokens, 12 heads 7.1 us (two: 8.9 us), 64 x 128, 16
        // heads 14.4 us (16.1 us), 1000 x 20 ... 60, 12 heads 107 us (121 us); in as many rounds they hinder each other: 40 x 64 ... 128, 12 heads
        // 9.4 us (9.0 us). Two by their tensor memory, which the placement of CTAs knows nothing of: a third one waits for it, but has been set up
        // when it gets it. That is ahead where attention follows attention and a CTA per SM does - 8 x 128, 16 heads 4.4 us, limited by shared memory
        // 5.3 us -, and behind where a round has more of them, as placement puts three on the SMs that the kernel before leaves first: behind a fully
        // connected layer of 4.7 us and with it, pairs of 128 tokens, by tensor memory / by shared memory: 149 12.6 / 9.8 us, 296 12.9 / 10.4 us; attention after
        // attention 149 5.4 / 5.6 us, 222 5.8 / 6.0 us, 240 7.5 / 5.9 us, 296 7.4 / 5.7 us.
        int64_t const sms = smCount(), two = (pairs + 2 * sms - 1) / (2 * sms), three = (pairs + 3 * sms - 1) / (3 * sms);
        bool const bySmem = three == two && pairs > sms && pairs <= 2 * sms, few = three < two || bySmem;
        int const smem = bySmem ? kShortSmemTwo : kShortSmemBytes;
        static SmemOptIn optIn[2];
        auto const kernel = few ? mhaShortF16Kernel<BNSD, kShortTmemCols> : mhaShortF16Kernel<BNSD, 2 * kShortTmemCols>;
        cudaError_t const e = launchDependentCluster(&optIn[few], kernel, dim3(static_cast<unsigned>(pairs)), dim3(kShortThreads),
            smem, stream, 1, maps[0], maps[1], maps[2], args);
        if (e != cudaSuccess)
            B200_FAIL(BERT_B200_CUDA_ERROR, "mhaShortF16Kernel: %s", cudaGetErrorString(e));
        return checkLaunch("mhaShortF16Kernel");
    }
    auto kernel = mhaOnlineF16Kernel<BNSD>;
    static SmemOptIn optIn;
    int const grid = shareGrid(args);
    cudaError_t const le = launchDependentCluster(&optIn, kernel, dim3(grid), dim3(kThreads), kSmemBytes, stream, 1, maps[0], maps[1], maps[2], args);
    if (le != cudaSuccess)
        B200_FAIL(BERT_B200_CUDA_ERROR, "mhaOnlineF16Kernel: %s", cudaGetErrorString(le));
    return checkLaunch("mhaOnlineF16Kernel");
}

} // namespace

// FP16, head sizes 16 / 32 / 48 / 64, fused [N][3][d] tensor in the fixed or the packed layout.
int32_t mhaOnlineF16(bert_b200_mha_params const& p, cudaStream_t stream)
{
    bool const fixedLayout = p.cu_seqlens == nullptr;
    uint64_t const d = static_cast<uint64_t>(p.head_size);
    uint64_t const rowElems = 3ull * static_cast<uint64_t>(p.num_heads) * d;
    // dim0: the d channels of one of Q, K, V of a head (the box is 64 wide: channels beyond d arrive as zeros);
    // dim1: which of [N][3]; dim2: batch (fixed layout only); dim3: sequence position / packed row
    uint64_t const dims[4] = {d, 3ull * static_cast<uint64_t>(p.num_heads), fixedLayout ? static_cast<uint64_t>(p.B) : 1ull,
        fixedLayout ? static_cast<uint64_t>(p.S) : static_cast<uint64_t>(p.total)};
    uint64_t const strides[3] = {d * 2, rowElems * 2, (fixedLayout ? static_cast<uint64_t>(p.B) : 1ull) * rowElems * 2};
    uint32_t const box[4] = {kHeadSize, 1, 1, kTile};
    CUtensorMap maps[3];
    int32_t const st = makeTensorMap(&maps[0], CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, p.qkv, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
    if (st != BERT_B200_OK)
        return st;
    maps[1] = maps[0];
    maps[2] = maps[0];
    OnlineArgs const args{shareArgs(p.B, p.S, p.num_heads, p.cu_seqlens, p.mask_idx), p.head_size, p.out, p.scale_bmm1, p.status_word};
    return launchOnline<false>(maps, args, stream);
}

// Separate Q, K, V tensors of shape [B][N][S][d] (the operand layout of TensorRT's attention layer), output
// [B][N][S][d]: three tensor maps, the same kernel.
int32_t mhaOnlineF16Bnsd(bert_b200_attention_bnsd_params const& p, cudaStream_t stream)
{
    uint64_t const d = static_cast<uint64_t>(p.head_size), S = static_cast<uint64_t>(p.S), N = static_cast<uint64_t>(p.num_heads);
    CUtensorMap maps[3];
    void const* const base[3] = {p.q, p.k, p.v};
    for (int i = 0; i < 3; ++i)
    {
        uint64_t const dims[4] = {d, S, N, static_cast<uint64_t>(p.B)};
        uint64_t const strides[3] = {d * 2, S * d * 2, N * S * d * 2};
        uint32_t const box[4] = {kHeadSize, kTile, 1, 1};
        int32_t const st = makeTensorMap(&maps[i], CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, base[i], dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
        if (st != BERT_B200_OK)
            return st;
    }
    OnlineArgs const args{shareArgs(p.B, p.S, p.num_heads, nullptr, p.kv_lengths), p.head_size, p.out, p.scale_bmm1, p.status_word};
    return launchOnline<true>(maps, args, stream);
}

} // namespace b200
