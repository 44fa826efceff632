// INT8 fused multi-head attention on the sm_100a tensor cores (head sizes 16, 32, 48, 64; sequence length <= 512),
// fixed [S,B,N,3,d], packed [total,N,3,d] and INT8 CHW32-interleaved layouts, and the C entry points of both
// attention kernels (FP16 runs the online-softmax kernel of mha_f16_online.cu).
//
// Replaces the precompiled fused INT8 attention kernels the reference launches through
// FusedMHARunnerInt8[v2]::run (plugin/bertQKVToContextPlugin/mhaRunner.cu:835-860, 1127-1265) and the head-size
// padding copies (zeroPadding2d.cu:190-204: here the TMA unit zero-fills the channels beyond the head size).
//
// The quantised probabilities P_q = rni(p / rowsum * scale_softmax) need the exact row maximum and the complete row
// sum before the first of them can be formed, so the whole score row lives in TMEM (<= 512 keys) and the softmax makes
// three sweeps over it; that is what keeps the result bit-identical with the reference's INT8 kernels.
//
// Sequences of one key block go through mhaShortInt8Kernel (see there), longer ones through the persistent kernel:
// Persistent CTAs (one per SM) take (sequence, head) work items, or parts of them where there are few, round-robin or, in
// ragged batches of many, each a long one, then a short one (mha_items.h). Per item a CTA loops over its 128-query tiles,
// so that K and V are loaded once and the tensor pipe works on the next tile (of this item or the next) while the
// softmax warps finish the current one. 19 warps:
//   warp 0    : TMA - the K / V blocks (128 keys each) of an item once, the Q tile of each iteration
//               (swizzled shared-memory tiles, one mbarrier each).
//   warp 1    : TMEM allocation (512 columns); issues the context products (an elected lane does)
//                 O  += P_j V_j           (128 x 64, accumulator in TMEM columns 384..447; for S > 384 it re-uses
//                                          the columns of S_0: the next tile's scores of that block wait for them)
//   warp 18   : issues the scores of the following tile, per key block as soon as the softmax warps hold
//               the current S_j in registers:
//                 S_j = Q K_j^T           (128 x 128 per key block, accumulators in TMEM columns 128j..)
//   warps 2-17: softmax, four threads per query row (each owns 32 of every 128 key columns):
//                 pass A  row maximum over all key blocks straight from TMEM (integer maximum, no conversions),
//                 pass B  p = exp2((x - max) * scale * log2e), row sum; the exponentials go back to TMEM,
//                 pass C  P_q = rni(p / sum * scale_softmax) -> INT8 P_j into swizzled shared memory for the PV product,
//                 epilogue O * scale_bmm2, round, saturate -> 128-bit global stores, deferred until after pass A of
//                         the next tile.
//               The passes loop over the key blocks (not unrolled): unrolled, the kernel was bound by instruction
//               fetch (122 KB of text, 77 % instruction-cache hits). For the same reason what differs at four key blocks (the context
//               shares columns with scores, blocks of P share slots), and the layout, is decided when the kernel is compiled: 64 x 384
//               tokens, 16 heads 101 -> 94 us, the layout too 93.5 us, 64 x 256 53.4 -> 49.2 -> 48.2 us, 64 x 512 180 -> 170 -> 168 us. Of these
//               first 10, 7 us come from the scores of key blocks 1 ... 3, which are formed while the context of the tile before is finished
//               and read: only those of block 0 wait for its columns.
// Every wait is bounded (sm100.cuh); on expiry the CTA drains, frees TMEM, reports through the status word.
#include "mha_items.h"
#include "sm100.cuh"

#include <cstdlib>
#include <type_traits>

namespace b200
{

int32_t mhaSimt(bert_b200_mha_params const& p, cudaStream_t stream);
int32_t mhaOnlineF16(bert_b200_mha_params const& p, cudaStream_t stream);
int32_t mhaOnlineF16Bnsd(bert_b200_attention_bnsd_params const& p, cudaStream_t stream);

namespace
{

constexpr int kQTile = 128;
constexpr int kKeyBlock = 128;
constexpr int kHeadSize = 64;
constexpr int kMaxBlocks = 4; // S <= 512
constexpr int kMhaThreads = 608;     // TMA warp, MMA warp, 16 softmax warps, second MMA warp
constexpr int kSoftmaxThreads = 512;
constexpr uint32_t kTmemCols = 512;
constexpr uint32_t kOColumn = 384;   // context accumulator when the scores need at most 384 columns

struct MhaArgs
{
    int32_t B, S, N, total;
    int32_t d; // head size: 16, 32, 48 or 64; the tiles are always 64 wide, TMA fills the missing channels with zeros
    int32_t fixedLayout;
    void* out;
    int32_t const* cu;
    int32_t const* maskIdx;
    float scaleBmm1, scaleSoftmax, scaleBmm2;
    uint32_t* statusWord;
    int32_t tilesPerItem, chunks; // a work item = (sequence, head, chunk of tilesPerItem query tiles)
    int32_t rounds;               // listed items per CTA, at most
};

enum class Order
{
    kNone,
    kPairs,
    kTiles,
};

// Sequences by length and the items of a CTA (see ORDER).
struct alignas(1024) ItemTable
{
    int4 ordered[kItemOrder]; // number, first row, length
    int4 items[kItemRounds];  // sequence (-1: none), head | first tile << 16 | tiles (at most) << 24, first row, length
    int32_t lengths[kItemOrder];
};

struct MhaSmem
{
    static constexpr int kTileBytes = kQTile * kHeadSize; // Q tile, one K block, one V block
    static constexpr int kPBytes = kQTile * kKeyBlock;    // one P block
    // [ Q ][ K blocks ][ V blocks ][ P slots ][ barriers, reduction scratch ]
    static __host__ __device__ constexpr int kOffset()
    {
        return kTileBytes;
    }
    static __host__ __device__ constexpr int vOffset(int nb)
    {
        return (1 + nb) * kTileBytes;
    }
    static __host__ __device__ constexpr int pOffset(int nb)
    {
        return (1 + 2 * nb) * kTileBytes;
    }
    // one P slot per key block up to three blocks; four blocks share two slots (shared memory is full then)
    static __host__ __device__ constexpr int pSlots(int nb)
    {
        return nb <= 3 ? nb : 2;
    }
    static __host__ __device__ constexpr int barrierOffset(int nb)
    {
        return pOffset(nb) + pSlots(nb) * kPBytes;
    }
    // kFull[4] vFull[4] sFull[4] pReady[4] pFree[4] sFree[4] qFull qFree oFull oFree vFree, tmem slot + abort flag, max / sum scratch
    static constexpr int kBarrierBytes = (6 * kMaxBlocks + 5) * 8 + 16 + 8 * kQTile * 4;
    static __host__ __device__ constexpr int dynamicBytes(int nb)
    {
        return barrierOffset(nb) + kBarrierBytes + 1024;
    }
};

__device__ __forceinline__ float ex2Approx(float x)
{
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Four non-negative values -> round-to-nearest-even integers saturated at 127, packed into one word.
// Adding 1.5 * 2^23 leaves the rounded integer in the low mantissa bits (the FP32 adder rounds to nearest even,
// like cvt.rni); the clamp at 127 is the saturation of the reference's conversion for scale_softmax > 127.
// kClamp = false: the caller knows that no value exceeds 127.49 (scale_softmax <= 127 and p <= 1).
template <bool kClamp>
__device__ __forceinline__ uint32_t packProb4(float a, float b, float c, float d)
{
    constexpr float kMagic = 12582912.f;
    if (kClamp)
    {
        a = fminf(a, 127.f);
        b = fminf(b, 127.f);
        c = fminf(c, 127.f);
        d = fminf(d, 127.f);
    }
    uint32_t const ua = __float_as_uint(a + kMagic), ub = __float_as_uint(b + kMagic);
    uint32_t const uc = __float_as_uint(c + kMagic), ud = __float_as_uint(d + kMagic);
    return __byte_perm(__byte_perm(ua, ub, 0x0040), __byte_perm(uc, ud, 0x0040), 0x5410);
}

// All sixteen softmax warps in step: the row reductions only join the four that own the columns of the same 32 query rows, but the
// per-key-block hand-overs to the MMA warps need every warp's arrival anyway (a barrier per four warps: -4 %).
__device__ __forceinline__ void softmaxBarrier()
{
    asm volatile("bar.sync 1, 512;" ::: "memory");
}

__device__ __forceinline__ void tmemStore32(uint32_t taddr, uint32_t const (&r)[32])
{
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
        "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]),
        "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]),
        "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}

// First row and valid keys of sequence b.
template <bool FIXED>
__device__ __forceinline__ void sequenceOf(
    int32_t const S, int32_t const* __restrict__ cu, int32_t const* __restrict__ maskIdx, int const b, int32_t& rowBase, int32_t& len)
{
    if (FIXED)
    {
        rowBase = 0;
        len = maskIdx ? min(max(__ldg(maskIdx + b), 0), S) : S;
    }
    else
    {
        rowBase = __ldg(cu + b);
        len = min(max(__ldg(cu + b + 1) - rowBase, 0), S);
    }
}

// IL: CHW32-interleaved tensors. Q, K and V tiles then arrive as two 32-channel sub-tiles of
// [128 tokens][32 B] (32-byte swizzle); the head dimension is covered by one MMA per sub-tile.
// BNSD: Q, K and V are three separate [B][N][S][d] tensors (mapQkv, mapK, mapV) and the output is [B][N][S][d];
// otherwise mapQkv covers the fused tensor and the other two maps are not used.
// ORDER: items as they come; or the CTA first puts the sequences in the order of their lengths and lists its items (see mha_items.h), whole pairs, or tiles where
// these, counted, are shorter. The last is a form of its own: with its code beside the other's, launches that deal pairs were 1 ... 2 % slower, and with it in a
// function of its own the launches that deal tiles 0.4 us.
// FIXED: the fixed layout (or separate tensors), not the packed one.
// FOUR: the longest sequence has four key blocks, not up to three. The context accumulator then has to share TMEM columns with the scores of key block 0, and four
// blocks of P share two slots.
// CLAMP: with FOUR, whether scale_softmax is above 127 (64 x 512 tokens, 16 heads 168.7 -> 165.1 us); the form for shorter sequences finds out (decided when it is
// compiled, it is 2 % slower).
template <bool IL, bool BNSD, bool FIXED, Order ORDER, bool FOUR, bool CLAMP>
__global__ void __launch_bounds__(kMhaThreads, 1)
    mhaTcgen05Kernel(const __grid_constant__ CUtensorMap mapQkv, const __grid_constant__ CUtensorMap mapK,
        const __grid_constant__ CUtensorMap mapV, MhaArgs const args)
{
    static_assert(!BNSD || !IL, "separate Q / K / V tensors: linear layout");
    static_assert(!FIXED || ORDER != Order::kTiles, "packed layout");
    constexpr bool ORDERED = ORDER != Order::kNone, kCut = ORDER == Order::kTiles;
    using L = MhaSmem;
    // Q, K, V rows are 64 B or 32 B (interleaved sub-tiles)
    constexpr uint64_t kSwz = IL ? kSwizzle32B : kSwizzle64B;
    constexpr uint32_t kAtomBytes = IL ? 256u : 8 * kHeadSize; // 8 rows of a swizzle atom: SBO
    constexpr uint32_t kSubTile = L::kTileBytes / 2;           // interleaved: bytes of one 32-channel sub-tile
    constexpr int kQkMmas = 2;                                 // head size 64 = 2 x 32
    constexpr int kPvMmas = 4;                                 // 128 keys = 4 x 32
    constexpr uint32_t kIdescQk = makeInstrDesc(2u, 1u, 0u, 0u, 128u, 128u);
    constexpr uint32_t kIdescPv = makeInstrDesc(2u, 1u, 0u, 1u, 128u, 64u);

    int const warp = threadIdx.x >> 5;
    int const lane = threadIdx.x & 31;

    extern __shared__ uint8_t smemRaw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smemRaw) + 1023) & ~static_cast<uintptr_t>(1023));
    ItemTable* const table = reinterpret_cast<ItemTable*>(smem);
    if (ORDERED)
        smem += sizeof(ItemTable);

    // ---- work items: some or all query tiles of a (sequence, head), item = (b * N + head) * chunks + chunk, dealt round-robin
    //      to the persistent CTAs; or whole (sequence, head) pairs, or single tiles, as the CTA has listed them ----
    struct Item
    {
        int32_t b, head, rowBase, rows, len, nb, tBegin, tEnd;
    };
    int const numItems = ORDERED ? args.rounds : args.B * args.N * args.chunks;
    int const firstItem = ORDERED ? 0 : static_cast<int>(blockIdx.x);
    int const itemStep = ORDERED ? 1 : static_cast<int>(gridDim.x);
    auto sequence = [&](int b, int32_t& rowBase, int32_t& len) { sequenceOf<FIXED>(args.S, args.cu, args.maskIdx, b, rowBase, len); };
    // Geometry of item i (uniform over the CTA; every role derives the same values). Returns whether the item has
    // work for the tensor pipeline (at least one query row and one valid key).
    auto getItem = [&](int i, Item& it) -> bool {
        int tiles = args.tilesPerItem;
        if (ORDERED)
        {
            int4 const q = table->items[i];
            it.b = q.x;
            it.head = q.y & 0xffff;
            it.tBegin = q.y >> 16 & 0xff;
            tiles = q.y >> 24;
            it.rowBase = q.z;
            it.len = q.w;
            it.rows = FIXED && q.x >= 0 ? args.S : it.len;
        }
        else
        {
            int const pair = i / args.chunks;
            it.b = pair / args.N;
            it.head = pair - it.b * args.N;
            it.tBegin = (i - pair * args.chunks) * args.tilesPerItem;
            sequence(it.b, it.rowBase, it.len);
            it.rows = FIXED ? args.S : it.len;
        }
        it.nb = (it.len + kKeyBlock - 1) / kKeyBlock; // key blocks
        it.tEnd = min((it.rows + kQTile - 1) / kQTile, it.tBegin + tiles);
        return it.len > 0 && it.tBegin < it.tEnd;
    };
    // first item >= i of this CTA's sequence that has pipeline work; numItems or more if there is none
    auto nextWork = [&](int i, Item& it) -> int {
        while (i < numItems && !getItem(i, it))
            i += itemStep;
        return i;
    };

    // The layout of shared memory and TMEM follows the longest sequence the launch admits.
    int const nbMax = (args.S + kKeyBlock - 1) / kKeyBlock;
    constexpr bool oAliasesScores = FOUR;
    constexpr uint32_t oCol = oAliasesScores ? 0u : kOColumn;
    auto slotOf = [&](int j) { return oAliasesScores ? (j & 1) : j; };

    uint8_t* sQ = smem;                          // kTileBytes
    uint8_t* sK = smem + L::kOffset();           // nbMax x kTileBytes
    uint8_t* sV = smem + L::vOffset(nbMax);      // nbMax x kTileBytes
    uint8_t* sP = smem + L::pOffset(nbMax);      // pSlots(nbMax) x kPBytes
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::barrierOffset(nbMax));
    uint64_t* kFull = bars;                      // [4] K_j landed                        (once per item using block j)
    uint64_t* vFull = bars + kMaxBlocks;         // [4] V_j landed                        (once per item using block j)
    uint64_t* sFull = bars + 2 * kMaxBlocks;     // [4] scores of block j complete        (once per tile using block j)
    uint64_t* pReady = bars + 3 * kMaxBlocks;    // [4] P_j written, 512 arrivals         (once per tile using block j)
    uint64_t* pFree = bars + 4 * kMaxBlocks;     // [4] PV product consumed P slot        (once per fill of the slot)
    uint64_t* sFree = bars + 5 * kMaxBlocks;     // [4] softmax holds S_j in registers, 512 arrivals (once per tile using block j)
    uint64_t* qFull = sFree + kMaxBlocks;        // Q tile landed                         (once per tile)
    uint64_t* qFree = qFull + 1;                 // all score MMAs of the tile done: Q slot (after an item's last tile: K) reusable
    uint64_t* oFull = qFree + 1;                 // context accumulator complete          (once per tile)
    uint64_t* oFree = oFull + 1;                 // epilogue has read it, 512 arrivals    (once per tile)
    uint64_t* vFree = oFree + 1;                 // all PV products of an item done: V reusable (once per item)
    uint32_t* tmemSlot = reinterpret_cast<uint32_t*>(vFree + 1);
    volatile uint32_t* abortFlag = tmemSlot + 1;
    float* rowRed = reinterpret_cast<float*>(tmemSlot + 4); // [2][4][128]: max then sum, per 32-column owner

    if (threadIdx.x == 0)
    {
        for (int i = 0; i < kMaxBlocks; ++i)
        {
            mbarInit(&kFull[i], 1);
            mbarInit(&vFull[i], 1);
            mbarInit(&sFull[i], 1);
            mbarInit(&pReady[i], kSoftmaxThreads);
        }
        for (int i = 0; i < kMaxBlocks; ++i)
        {
            mbarInit(&pFree[i], 1);
            mbarInit(&sFree[i], kSoftmaxThreads);
        }
        mbarInit(qFull, 1);
        mbarInit(qFree, 1);
        mbarInit(oFull, 1);
        mbarInit(oFree, kSoftmaxThreads);
        mbarInit(vFree, 1);
        *abortFlag = 0;
        fenceBarrierInit();
        prefetchTensorMap(&mapQkv);
        if (BNSD)
        {
            prefetchTensorMap(&mapK);
            prefetchTensorMap(&mapV);
        }
    }
    if (warp == 1)
        tmemAlloc(tmemSlot, kTmemCols);
    tcFenceBefore();
    __syncthreads();
    tcFenceAfter();
    uint32_t const tmemBase = *tmemSlot;
    // set-up done: the next kernel of the stream may start its own; the inputs of this one must be complete
    gridDependencyLaunch();
    gridDependencyWait();

    if (ORDERED)
    {
        // a sequence's place is the number of longer ones, and of equal ones before it (those beyond the batch count as -1)
        int const b = static_cast<int>(threadIdx.x);
        if (b < kItemOrder)
        {
            int32_t rowBase = 0, len = -1;
            if (b < args.B)
                sequence(b, rowBase, len);
            table->lengths[b] = len;
            asm volatile("bar.sync 8, %0;" ::"n"(kItemOrder) : "memory");
            [[maybe_unused]] int total = 0, most = 0; // tiles of the batch and of its longest sequence (threads with a sequence or an item)
            if (b < args.B || (kCut && b < args.rounds))
            {
                int place = 0;
                for (int u = 0; u < args.B; u += 4)
                {
                    int4 const v = *reinterpret_cast<int4 const*>(table->lengths + u);
                    place += (v.x > len || (v.x == len && u < b)) + (v.y > len || (v.y == len && u + 1 < b))
                        + (v.z > len || (v.z == len && u + 2 < b)) + (v.w > len || (v.w == len && u + 3 < b));
                    if (kCut)
                    {
                        total += (v.x + kQTile - 1) / kQTile + (v.y + kQTile - 1) / kQTile + (v.z + kQTile - 1) / kQTile + (v.w + kQTile - 1) / kQTile;
                        most = max(max(max(most, v.x), max(v.y, v.z)), v.w);
                    }
                }
                if (!kCut || b < args.B)
                    table->ordered[place] = make_int4(b, rowBase, len, 0);
            }
            asm volatile("bar.sync 8, %0;" ::"n"(kItemOrder) : "memory");
            if (b < args.rounds)
            {
                int const item = itemOfRound(b, static_cast<int>(blockIdx.x), static_cast<int>(gridDim.x));
                int place = item / args.N, what = (item - place * args.N) | kMaxBlocks << 24;
                if (kCut)
                {
                    if (cutIsShorter(total * args.N, (most + kQTile - 1) / kQTile, static_cast<int>(gridDim.x)))
                    {
                        // the tiles of a pair one by one: a longer sequence has more of them
                        int left = item;
                        for (place = 0; place < args.B; ++place)
                        {
                            int const tiles = (table->ordered[place].z + kQTile - 1) / kQTile;
                            if (left < tiles * args.N)
                            {
                                int const head = left / tiles;
                                what = head | (left - head * tiles) << 16 | 1 << 24;
                                break;
                            }
                            left -= tiles * args.N;
                        }
                    }
                    else if (b > 0)
                        place = args.B; // whole pairs: one round
                }
                int4 q = make_int4(-1, 0, 0, 0);
                if (place < args.B)
                {
                    int4 const o = table->ordered[place];
                    q = make_int4(o.x, what, o.y, o.z);
                }
                table->items[b] = q;
            }
        }
        __syncthreads();
    }

    // Barriers that complete once per tile (qFull, qFree, oFull, oFree) are waited on with the parity of the CTA's
    // running tile count; those that complete once per use of key block j keep one parity bit per block.
    if (warp == 0)
    {
        Item it;
        uint32_t tiles = 0;       // Q tiles requested so far
        uint32_t itemsLoaded = 0; // items whose K / V have been requested
        bool ok = true;
        for (int item = nextWork(firstItem, it); item < numItems && ok; item = nextWork(item + itemStep, it))
        {
            int32_t const rowK = FIXED ? 0 : it.rowBase;
            int32_t const rowKv = rowK; // first key of this item
            // linear: (channel, which of [N][3], batch, row). interleaved: (channel, row, 32-channel group, which of [3][N])
            auto load = [&](uint8_t* dst, uint64_t* bar, int which, int32_t row) {
                if (BNSD) // (channel, position, head, sequence) of the tensor `which` selects
                    tmaLoad4d(dst, which == 0 ? &mapQkv : (which == 1 ? &mapK : &mapV), bar, 0, row, it.head, it.b);
                else if (IL)
                    tmaLoad4d(dst, &mapQkv, bar, 0, row, 0, which * args.N + it.head);
                else
                    tmaLoad4d(dst, &mapQkv, bar, 0, it.head * 3 + which, FIXED ? it.b : 0, row);
            };
            for (int t = it.tBegin; t < it.tEnd && ok; ++t)
            {
                // the score MMAs of the previous tile have read Q (and, across items, K)
                if (tiles > 0)
                    ok = mbarWaitWarp(qFree, (tiles - 1) & 1, abortFlag, kWaitStageFree);
                if (!ok)
                    break;
                if (electOne())
                {
                    mbarArriveExpectTx(qFull, L::kTileBytes);
                    load(sQ, qFull, 0, rowK + t * kQTile);
                }
                __syncwarp();
                if (t == it.tBegin)
                {
                    for (int j = 0; j < it.nb; ++j)
                    {
                        if (electOne())
                        {
                            mbarArriveExpectTx(&kFull[j], L::kTileBytes);
                            load(sK + j * L::kTileBytes, &kFull[j], 1, rowKv + j * kKeyBlock);
                        }
                        __syncwarp();
                    }
                    // The PV products of the previous item have read V. (Not oFull: this thread may run ahead of
                    // or behind the per-tile barriers by more than one phase, and a parity wait is only meaningful
                    // for the very next phase; vFree completes once per item, in step with this loop.)
                    if (itemsLoaded > 0)
                        ok = mbarWaitWarp(vFree, (itemsLoaded - 1) & 1, abortFlag, kWaitStageFree);
                    if (!ok)
                        break;
                    for (int j = 0; j < it.nb; ++j)
                    {
                        if (electOne())
                        {
                            mbarArriveExpectTx(&vFull[j], L::kTileBytes);
                            load(sV + j * L::kTileBytes, &vFull[j], 2, rowKv + j * kKeyBlock);
                        }
                        __syncwarp();
                    }
                }
                ++tiles;
            }
            ++itemsLoaded;
        }
    }
    else if (warp == 1 || warp == kMhaThreads / 32 - 1)
    {
        // ---- MMA issue: scores S_j = Q K_j^T of the tile after the one the softmax warps work on, and
        //      context_t += P_j V_j as they hand over P_j ----
        // Every tcgen05.mma / tcgen05.commit keeps its issuing warp busy for 30-60 cycles (measured), and one
        // warp issuing both products of a tile was the slowest link of the tile pipeline: the scores are issued by
        // a second one, the last warp (+11 % at S = 384).
        // Operand descriptors are formed arithmetically: one low word per operand tile (+ bytes >> 4 per key block
        // and MMA step, compile-time constants of the unrolled loops) and one high word per operand kind (mmaLoHi).
        auto issuer = [&](auto doScoresTag, auto doContextTag) {
            constexpr bool kDoScores = decltype(doScoresTag)::value;
            constexpr bool kDoContext = decltype(doContextTag)::value;
            bool ok = true;
            uint64_t const dQk = makeSmemDesc(0, 16, kAtomBytes, kSwz);
            // P: K-major, 128-byte rows, 128-byte swizzle.
            uint64_t const dP = makeSmemDesc(0, 16, 1024, kSwizzle128B);
            // V: MN-major (head dimension contiguous), one MMA consumes 32 key rows.
            // Interleaved: the two 32-channel sub-tiles are LBO apart, 32 key rows are 1024 bytes.
            uint64_t const dV = IL ? makeSmemDesc(0, kSubTile, kAtomBytes, kSwz) : makeSmemDesc(0, kAtomBytes, kAtomBytes, kSwz);
            uint32_t const hiQk = static_cast<uint32_t>(dQk >> 32), hiP = static_cast<uint32_t>(dP >> 32),
                           hiV = static_cast<uint32_t>(dV >> 32);
            uint32_t const qLo = static_cast<uint32_t>(dQk) + (smemAddr(sQ) >> 4);
            uint32_t const kLo = static_cast<uint32_t>(dQk) + (smemAddr(sK) >> 4);
            uint32_t const vLo = static_cast<uint32_t>(dV) + (smemAddr(sV) >> 4);
            uint32_t const pLo = static_cast<uint32_t>(dP) + (smemAddr(sP) >> 4);
            constexpr uint32_t pPairStep = oAliasesScores ? 0u : 2u * (L::kPBytes >> 4); // slotOf(j) = (j & 1) + (j >> 1) * (2 or 0)
            constexpr uint32_t kTile16 = L::kTileBytes >> 4;
            uint32_t qkTiles = 0;  // tiles whose scores have been issued
            uint32_t pvTiles = 0;  // tiles of this CTA that the loop below has passed (= whose context has been issued)
            uint32_t kBits = 0, vBits = 0, pBits = 0, fBits = 0; // parity per key block: K landed, V landed, P written, S read
            // scores of key block j for the query tile whose Q is in shared memory; last: of that tile's, Q is free after them
            auto issueScores = [&](int j, bool last) {
                if (electOne())
                {
#pragma unroll
                    for (int k = 0; k < kQkMmas; ++k)
                    {
                        uint32_t const off = (IL ? k * kSubTile : k * 32) >> 4; // next 32 bytes of the head dimension
                        mmaLoHi<true>(tmemBase + j * kKeyBlock, qLo + off, hiQk, kLo + j * kTile16 + off, hiQk, kIdescQk, k != 0);
                    }
                    tcCommit(&sFull[j]);
                    if (last)
                        tcCommit(qFree);
                }
                __syncwarp();
            };
            // first use of K_j by an item: wait for it to land
            auto waitK = [&](int j) -> bool {
                bool const got = mbarWaitWarp(&kFull[j], (kBits >> j) & 1u, abortFlag, kWaitTmaFull);
                kBits ^= 1u << j;
                return got;
            };
            constexpr int firstBlock = oAliasesScores ? 1 : 0; // key blocks whose scores do not wait for the context
            Item cur, nxt;
            int item = nextWork(firstItem, cur);
            if (kDoScores && item < numItems)
            {
                ok = mbarWaitWarp(qFull, 0, abortFlag, kWaitTmaFull);
#pragma unroll 1
                for (int j = 0; j < kMaxBlocks; ++j)
                {
                    if (j < cur.nb && ok)
                    {
                        ok = waitK(j);
                        if (ok)
                        {
                            tcFenceAfter();
                            issueScores(j, j == cur.nb - 1);
                        }
                    }
                }
                qkTiles = 1;
            }
            while (item < numItems && ok)
            {
                // only the scores look one item ahead (its geometry comes from global memory: not in the way of a
                // warp that only issues context products)
                int const nextItem = kDoScores ? nextWork(item + itemStep, nxt) : numItems;
                for (int t = cur.tBegin; t < cur.tEnd && ok; ++t)
                {
                    bool const lastT = t + 1 == cur.tEnd;
                    // the scores issued while this tile's context is formed: the item's next tile, or the first tile
                    // of the CTA's next item (whose K then has to have landed), or none
                    int const nbFollow = !lastT ? cur.nb : (nextItem < numItems ? nxt.nb : 0);
#pragma unroll 1
                    for (int j = 0; j < kMaxBlocks; ++j)
                    {
                        if (j < cur.nb && ok)
                        {
                            // Scores of the following tile for this key block first: they only need the softmax warps
                            // to hold this tile's S_j in registers (sFree), not the finished P_j, and the next pass A
                            // waits for them, while this tile's context is not read before the pass after.
                            if (kDoScores && j == 0 && nbFollow > 0)
                                ok = mbarWaitWarp(qFull, qkTiles & 1, abortFlag, kWaitTmaFull);
                            if (kDoScores && j < nbFollow && j >= firstBlock)
                            {
                                if (ok && lastT)
                                    ok = waitK(j);
                                ok = ok && mbarWaitWarp(&sFree[j], (fBits >> j) & 1u, abortFlag, kWaitSoftmax);
                                if (ok)
                                {
                                    tcFenceAfter();
                                    issueScores(j, j == nbFollow - 1 && !oAliasesScores);
                                }
                            }
                            fBits ^= 1u << j; // the softmax warps complete this phase in every tile that uses block j
                            if (kDoContext)
                            {
                                if (ok && t == cur.tBegin)
                                {
                                    ok = mbarWaitWarp(&vFull[j], (vBits >> j) & 1u, abortFlag, kWaitTmaFull);
                                    vBits ^= 1u << j;
                                }
                                if (ok && j == 0 && pvTiles > 0) // the previous tile's context must have been read out
                                    ok = mbarWaitWarp(oFree, (pvTiles - 1) & 1, abortFlag, kWaitAccFree);
                                ok = ok && mbarWaitWarp(&pReady[j], (pBits >> j) & 1u, abortFlag, kWaitSoftmax);
                                pBits ^= 1u << j;
                                if (ok)
                                {
                                    tcFenceAfter();
                                    uint32_t const a = pLo + (j & 1) * (L::kPBytes >> 4) + (j >> 1) * pPairStep;
                                    uint32_t const b = vLo + j * kTile16;
                                    if (electOne())
                                    {
#pragma unroll
                                        for (int k = 0; k < kPvMmas; ++k)
                                        {
                                            constexpr uint32_t kVStep = (IL ? 1024u : 2048u) >> 4;
                                            mmaLoHi<true>(tmemBase + oCol, a + k * 2, hiP, b + k * kVStep, hiV, kIdescPv, (j | k) != 0);
                                        }
                                        if (oAliasesScores) // otherwise every tile has its own P slots, released with oFull
                                            tcCommit(&pFree[slotOf(j)]);
                                        if (j == cur.nb - 1)
                                        {
                                            tcCommit(oFull);
                                            if (lastT)
                                                tcCommit(vFree);
                                        }
                                    }
                                    __syncwarp();
                                }
                            }
                        }
                    }
                    if (kDoScores && ok)
                    {
                        // key blocks the next item has beyond this one's: their score columns are idle, since all softmax threads are done with the
                        // tile before, the last that can have used them. Up to three key blocks: they have arrived at sFree[0] for this tile. Four:
                        // at oFree for the tile before, which this tile's scores of block 0 waited for
#pragma unroll 1
                        for (int j = 1; j < kMaxBlocks; ++j)
                        {
                            if (j >= cur.nb && j < nbFollow && ok)
                            {
                                ok = waitK(j);
                                if (ok)
                                {
                                    tcFenceAfter();
                                    issueScores(j, j == nbFollow - 1 && !oAliasesScores);
                                }
                            }
                        }
                    }
                    if (kDoScores && ok && nbFollow > 0 && oAliasesScores)
                    {
                        // the context accumulator occupies the columns of key block 0: wait until the epilogue has read it
                        ok = (!lastT || waitK(0)) && mbarWaitWarp(oFree, pvTiles & 1, abortFlag, kWaitAccFree);
                        if (ok)
                        {
                            tcFenceAfter();
                            issueScores(0, true);
                        }
                    }
                    if (nbFollow > 0)
                        ++qkTiles;
                    ++pvTiles;
                }
                if (kDoScores)
                {
                    cur = nxt;
                    item = nextItem;
                }
                else
                    item = nextWork(item + itemStep, cur);
            }
        };
        if (warp == 1)
            issuer(std::false_type{}, std::true_type{});
        else
            issuer(std::true_type{}, std::false_type{});
    }
    else if (warp < 2 + kSoftmaxThreads / 32)
    {
        int const quad = warp & 3;        // TMEM lanes [32*quad, 32*quad+32) are the ones this warp may touch
        int const sub = (warp - 2) >> 2;  // which 32 of every 128 key columns this thread owns (4 warps per quadrant)
        int const r = quad * 32 + lane;   // query row inside the tile = TMEM lane
        uint32_t const tRow = tmemBase + (static_cast<uint32_t>(quad * 32) << 16);
        float const sl2 = args.scaleBmm1 * 1.4426950408889634f;
        constexpr float kMagic = 12582912.f;       // 1.5 * 2^23: as_float(0x4B400000 + v) == kMagic + v for |v| < 2^22
        constexpr uint32_t kMagicBits = 0x4B400000u;
        bool ok = true;
        auto colOf = [&](int j) { return j * kKeyBlock + sub * 32; };
        uint32_t tiles = 0;       // tiles this CTA has started
        uint32_t sBits = 0;       // parity per key block of sFull (and of this thread's arrivals on pReady)
        uint32_t slotFilled = 0;  // per P slot: has it been filled before ...
        uint32_t slotParity = 0;  // ... and the parity of the pFree phase that ends its latest fill
        // Before a P slot is refilled, the PV product that read its previous contents must have completed (pFree is only
        // signalled when four key blocks share two slots).
        auto acquireP = [&](int j) -> bool {
            // One slot per key block (up to three blocks): a slot is refilled one tile later, after this thread has
            // waited for the previous tile's complete context in its (deferred) epilogue - nothing to wait for.
            if (!oAliasesScores)
                return true;
            int const slot = slotOf(j);
            bool got = true;
            if ((slotFilled >> slot) & 1u)
            {
                got = mbarWait(&pFree[slot], (slotParity >> slot) & 1u, abortFlag, kWaitSoftmax);
                slotParity ^= 1u << slot;
            }
            slotFilled |= 1u << slot;
            return got;
        };
        // Reads 16 of the 64 context values of this row (tile number `tileNo` of the CTA), requantises
        // and stores them to `pendDst` (null: row beyond the sequence).
        bool pending = false;
        int8_t* pendDst = nullptr;
        auto epilogue = [&](uint32_t tileNo) {
            pending = false;
            if (ok)
                ok = mbarWait(oFull, tileNo & 1, abortFlag, kWaitAccFull);
            if (!ok)
                return;
            tcFenceAfter();
            uint32_t x[16];
            tmemLoad16(tRow + oCol + sub * 16, x);
            tmemLoadWait16(x);
            tcFenceBefore();
            mbarArrive(oFree);
            if (pendDst == nullptr)
                return;
            float const s2 = args.scaleBmm2;
            uint4 o;
            uint32_t* w = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
            for (int i = 0; i < 4; ++i)
                w[i] = packChar4(static_cast<float>(static_cast<int32_t>(x[4 * i])) * s2,
                    static_cast<float>(static_cast<int32_t>(x[4 * i + 1])) * s2,
                    static_cast<float>(static_cast<int32_t>(x[4 * i + 2])) * s2,
                    static_cast<float>(static_cast<int32_t>(x[4 * i + 3])) * s2);
            *reinterpret_cast<uint4*>(pendDst) = o;
        };

        // The epilogue of a tile runs after pass A of the CTA's next tile (of the same or the next item): the last PV product then completes
        // under useful work instead of a stall. Where the context accumulator shares columns with the scores of key block 0, it runs
        // before the maximum over that block, which comes last then (not in a CTA's first tile, where block 0 is there
        // first: 2 x 512 tokens, 16 heads 9.0 -> 8.8 us, 1 x 400, 12 heads 9.1 -> 9.0 us).

        Item it;
        for (int item = firstItem; item < numItems; item += itemStep)
        {
            bool const work = getItem(item, it);
            int64_t const outRowStride = static_cast<int64_t>(args.N) * args.d; // elements
            int8_t* const out = static_cast<int8_t*>(args.out);
            int8_t* const outBase = out + static_cast<int64_t>(it.head) * args.d;
            // linear layouts: the d values of (token, head) are contiguous
            auto outRow = [&](int q) -> int8_t* {
                if (BNSD)
                    return out + ((static_cast<int64_t>(it.b) * args.N + it.head) * args.S + q) * args.d;
                int64_t const rr = FIXED ? static_cast<int64_t>(q) * args.B + it.b : static_cast<int64_t>(it.rowBase) + q;
                return outBase + rr * outRowStride;
            };
            // interleaved output [N][d/32][total][32]: 32-channel group `grp` of (token, head)
            auto outPtrIl = [&](int q, int grp) -> int8_t* {
                return out + ((static_cast<int64_t>(it.head) * (args.d / 32) + grp) * args.total + it.rowBase + q) * 32;
            };
            if (!work)
            {
                // no valid key: every probability is zero and so is the context row
                int const kChunks = args.d / 16;
                int const q0 = it.tBegin * kQTile, q1 = min(it.rows, it.tEnd * kQTile);
                for (int i = threadIdx.x - 64; i < (q1 - q0) * kChunks; i += kSoftmaxThreads)
                {
                    int const q = q0 + i / kChunks;
                    int const c = i % kChunks;
                    if (IL)
                        reinterpret_cast<uint4*>(outPtrIl(q, c / 2))[c % 2] = make_uint4(0, 0, 0, 0);
                    else
                        reinterpret_cast<uint4*>(outRow(q))[c] = make_uint4(0, 0, 0, 0);
                }
                continue;
            }
            int const nb = it.nb;
            int const len = it.len;
            for (int t = it.tBegin; t < it.tEnd; ++t)
            {
                uint32_t x[32];

                // ---- pass A: row maximum (integers, no conversions) ----
                int32_t mxi = INT32_MIN;
                // the block whose columns hold the context of the tile before comes last
                int const firstBlock = oAliasesScores && pending ? 1 : 0;
#pragma unroll 1
                for (int i = firstBlock; i < nb + firstBlock; ++i)
                {
                    int const j = i < nb ? i : 0;
                    if constexpr (FOUR)
                    {
                        if (pending && j == 0)
                            epilogue(tiles - 1);
                    }
                    ok = ok && mbarWait(&sFull[j], (sBits >> j) & 1u, abortFlag, kWaitSoftmax);
                    tcFenceAfter();
                    tmemLoad32(tRow + colOf(j), x);
                    tmemLoadWait32(x);
                    int const limit = len - colOf(j);
                    if (limit >= 32)
                    {
#pragma unroll
                        for (int k = 0; k < 32; ++k)
                            mxi = max(mxi, static_cast<int32_t>(x[k]));
                    }
                    else
                    {
#pragma unroll
                        for (int k = 0; k < 32; ++k)
                            if (k < limit)
                                mxi = max(mxi, static_cast<int32_t>(x[k]));
                    }
                }
                float mx = mxi == INT32_MIN ? -INFINITY : static_cast<float>(mxi);
                if constexpr (!FOUR)
                {
                    if (pending)
                        epilogue(tiles - 1);
                }
                rowRed[sub * kQTile + r] = mx;
                softmaxBarrier();
                mx = fmaxf(fmaxf(rowRed[r], rowRed[kQTile + r]), fmaxf(rowRed[2 * kQTile + r], rowRed[3 * kQTile + r]));
                float const mxMagic = kMagic + mx; // exact: both are integers below 2^24

                // ---- pass B: exponentials, back to where the scores were, and the row sum ----
                float sum = 0.f;
#pragma unroll 1
                for (int j = 0; j < nb; ++j)
                {
                    tmemLoad32(tRow + colOf(j), x);
                    tmemLoadWait32(x);
                    int const limit = len - colOf(j);
                    // (acc - max) is formed exactly (integers through the 2^23 trick, no conversion unit), so the exponent carries a
                    // single rounding
                    auto expOf = [&](uint32_t v) { return ex2Approx((__uint_as_float(v + kMagicBits) - mxMagic) * sl2); };
                    if (limit >= 32) // all 32 keys valid: no per-element select
                    {
#pragma unroll
                        for (int i = 0; i < 32; ++i)
                        {
                            float const e = expOf(x[i]);
                            sum += e;
                            x[i] = __float_as_uint(e);
                        }
                    }
                    else
                    {
#pragma unroll
                        for (int i = 0; i < 32; ++i)
                        {
                            float const e = i < limit ? expOf(x[i]) : 0.f;
                            sum += e;
                            x[i] = __float_as_uint(e);
                        }
                    }
                    tmemStore32(tRow + colOf(j), x);
                }
                tmemStoreWait();
                rowRed[4 * kQTile + sub * kQTile + r] = sum;
                softmaxBarrier();
                sum = (rowRed[4 * kQTile + r] + rowRed[5 * kQTile + r]) + (rowRed[6 * kQTile + r] + rowRed[7 * kQTile + r]);
                float const inv = 1.f / sum;

                // ---- pass C: P_q = rni(p / sum * scale_softmax) ----
                float const pq = inv * args.scaleSoftmax;
#pragma unroll 1
                for (int j = 0; j < nb; ++j)
                {
                    tmemLoad32(tRow + colOf(j), x);
                    tmemLoadWait32(x);
                    tcFenceBefore();
                    mbarArrive(&sFree[j]); // the parked exponentials are in registers: columns free for new scores
                    ok = acquireP(j) && ok;
                    uint8_t* pRow = sP + slotOf(j) * L::kPBytes + r * 128; // P block: [128 rows][128 keys]
#pragma unroll
                    for (int g = 0; g < 2; ++g)
                    {
                        uint4 o;
                        uint32_t* w = reinterpret_cast<uint32_t*>(&o);
                        // p / sum <= 1 (the sum contains p; a rounded-up reciprocal adds a few ulp at most), so
                        // with scale_softmax <= 127 nothing can round beyond 127 and the clamp is left out
                        if (FOUR ? !CLAMP : args.scaleSoftmax <= 127.f)
                        {
#pragma unroll
                            for (int i = 0; i < 4; ++i)
                                w[i] = packProb4<false>(__uint_as_float(x[g * 16 + 4 * i]) * pq,
                                    __uint_as_float(x[g * 16 + 4 * i + 1]) * pq, __uint_as_float(x[g * 16 + 4 * i + 2]) * pq,
                                    __uint_as_float(x[g * 16 + 4 * i + 3]) * pq);
                        }
                        else
                        {
#pragma unroll
                            for (int i = 0; i < 4; ++i)
                                w[i] = packProb4<true>(__uint_as_float(x[g * 16 + 4 * i]) * pq,
                                    __uint_as_float(x[g * 16 + 4 * i + 1]) * pq, __uint_as_float(x[g * 16 + 4 * i + 2]) * pq,
                                    __uint_as_float(x[g * 16 + 4 * i + 3]) * pq);
                        }
                        int const chunk = sub * 2 + g; // 16 keys per 16-byte chunk
                        *reinterpret_cast<uint4*>(pRow + ((chunk ^ (r & 7)) << 4)) = o;
                    }
                    fenceProxyAsync();
                    tcFenceBefore();
                    mbarArrive(&pReady[j]);
                }
                sBits ^= (1u << nb) - 1u; // every block of this tile used its sFull / pReady phase
                int const q = t * kQTile + r;
                // this thread's 16 of the 64 context columns; columns >= d are the zero padding
                int8_t* const dst = q >= it.rows || sub * 16 >= args.d
                    ? nullptr
                    : (IL ? outPtrIl(q, sub >> 1) + (sub & 1) * 16 : outRow(q) + sub * 16);
                ++tiles;
                pending = true;
                pendDst = dst;
            }
        }
        if (pending)
            epilogue(tiles - 1);
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
    if (warp == 1)
    {
        __syncwarp();
        tcFenceAfter();
        tmemFree(tmemBase, kTmemCols);
    }
}

// Sequences of at most one key block: one CTA per (sequence, head), four warps that do everything in turn, a thread per query row.
//
// Bound by a pair's chain of latencies (lengths, loads, scores, softmax, product, store), with many pairs too: 64 x 128 tokens, 16 heads take 13.3
// us, the exponentials' unit (1024 cycles per pair, 3.7 us) is busy for 27 % of it and the issue slots for 40 %, with 16 warps on an SM. The persistent
// kernel works on one tile at a time: its sixteen warps pass through the same phase together, so one unit after the other waits, and two
// barriers per tile keep them in step. Here four CTAs share an SM (128 columns of tensor memory each, the context in the first ones once
// the exponentials there have been read), each in a phase of its own, no row is shared between threads, and the code is small: loops over
// pieces of 32 columns. The arithmetic is that of the persistent kernel, to the bit, the row sum's order included.
// Measured, GPU time (persistent kernel in brackets): 1 x 37 tokens, 12 heads 4.1 us (4.9 us), 32 x 64 ... 128, 12 heads 8.3 us (10.9 us), 64 x 128,
// 16 heads 13.3 us (21.2 us), 128 x 16, 16 heads 15.9 us (39.5 us), 1024 x 128, 16 heads 172 us (307 us). Two threads per row are 0 ... 20 % slower. The
// same for two key blocks (256 columns, two CTAs per SM) is no clear gain: 9 x 256, 16 heads 8.3 us (10.0 us), 64 x 256 49.5 us (53.4 us),
// but 2 x 256 7.1 us (6.3 us), 37 interleaved sequences of 100 ... 256 28.4 us (26.5 us).
constexpr int kShortThreads = 128;
constexpr int kShortTile = kQTile * kHeadSize;  // bytes of the Q, K or V tile
constexpr int kShortP = 3 * kShortTile;         // after Q, K and V
constexpr int kShortBars = kShortP + kQTile * kKeyBlock;
constexpr int kShortSmemBytes = kShortBars + 64 + 1024;
constexpr uint32_t kShortTmemCols = kKeyBlock;

template <bool IL, bool BNSD>
__global__ void __launch_bounds__(kShortThreads, 4) mhaShortInt8Kernel(const __grid_constant__ CUtensorMap mapQkv,
    const __grid_constant__ CUtensorMap mapK, const __grid_constant__ CUtensorMap mapV, MhaArgs const args)
{
    constexpr uint64_t kSwz = IL ? kSwizzle32B : kSwizzle64B;
    constexpr uint32_t kAtomBytes = IL ? 256u : 512u;
    constexpr uint32_t kSubTile = kShortTile / 2; // interleaved: bytes of one 32-channel sub-tile
    constexpr uint32_t kIdescQk = makeInstrDesc(2u, 1u, 0u, 0u, 128u, 128u);
    constexpr uint32_t kIdescPv = makeInstrDesc(2u, 1u, 0u, 1u, 128u, 64u);
    int const warp = threadIdx.x >> 5;

    extern __shared__ uint8_t smemRaw[];
    uint8_t* const smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smemRaw) + 1023) & ~static_cast<uintptr_t>(1023));
    uint8_t* const sK = smem + kShortTile;
    uint8_t* const sV = smem + 2 * kShortTile;
    uint8_t* const sP = smem + kShortP;
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
        prefetchTensorMap(&mapQkv);
        if (BNSD)
        {
            prefetchTensorMap(&mapK);
            prefetchTensorMap(&mapV);
        }
    }
    __syncwarp();
    if (warp == 0)
        tmemAlloc(tmemSlot, kShortTmemCols);
    tcFenceBefore();
    __syncthreads();
    tcFenceAfter();
    uint32_t const tmemBase = *tmemSlot;
    gridDependencyLaunch();
    gridDependencyWait();

    int32_t const b = static_cast<int32_t>(blockIdx.x) / args.N, head = static_cast<int32_t>(blockIdx.x) - b * args.N;
    int32_t rowBase, len;
    if (args.fixedLayout)
    {
        rowBase = 0;
        len = args.maskIdx ? min(max(__ldg(args.maskIdx + b), 0), args.S) : args.S;
    }
    else
    {
        rowBase = __ldg(args.cu + b);
        len = min(max(__ldg(args.cu + b + 1) - rowBase, 0), args.S);
    }
    int32_t const rows = args.fixedLayout ? args.S : len;
    int const q = static_cast<int>(threadIdx.x); // query row = TMEM lane
    // the 16 context channels from c on of this thread's row
    auto outPtr = [&](int c) -> uint4* {
        int8_t* const out = static_cast<int8_t*>(args.out);
        if (BNSD)
            return reinterpret_cast<uint4*>(out + ((static_cast<int64_t>(b) * args.N + head) * args.S + q) * args.d + c);
        if (IL)
            return reinterpret_cast<uint4*>(
                out + ((static_cast<int64_t>(head) * (args.d / 32) + c / 32) * args.total + rowBase + q) * 32 + c % 32);
        int64_t const row = args.fixedLayout ? static_cast<int64_t>(q) * args.B + b : static_cast<int64_t>(rowBase) + q;
        return reinterpret_cast<uint4*>(out + (row * args.N + head) * args.d + c);
    };
    if (len > 0) // the same for all threads
    {
        // linear: (channel, which of [N][3], batch, row). interleaved: (channel, row, 32-channel group, which of [3][N])
        auto load = [&](uint8_t* dst, uint64_t* bar, int which) {
            if (BNSD) // (channel, position, head, sequence) of the tensor `which` selects
                tmaLoad4d(dst, which == 0 ? &mapQkv : (which == 1 ? &mapK : &mapV), bar, 0, 0, head, b);
            else if (IL)
                tmaLoad4d(dst, &mapQkv, bar, 0, rowBase, 0, which * args.N + head);
            else
                tmaLoad4d(dst, &mapQkv, bar, 0, head * 3 + which, args.fixedLayout ? b : 0, rowBase);
        };
        bool ok = true;
        if (warp == 0)
        {
            if (electOne())
            {
                mbarArriveExpectTx(qkFull, 2 * kShortTile);
                load(smem, qkFull, 0);
                load(sK, qkFull, 1);
                mbarArriveExpectTx(vFull, kShortTile);
                load(sV, vFull, 2);
            }
            __syncwarp();
            ok = mbarWaitWarp(smemAddr(qkFull), 0, abortFlag, kWaitTmaFull);
            tcFenceAfter();
            if (electOne() && ok)
            {
                uint64_t const dQk = makeSmemDesc(0, 16, kAtomBytes, kSwz);
                uint32_t const lo = static_cast<uint32_t>(dQk), hi = static_cast<uint32_t>(dQk >> 32);
#pragma unroll
                for (int k = 0; k < 2; ++k) // head size 64 = 2 x 32
                {
                    uint32_t const off = (IL ? k * kSubTile : k * 32) >> 4;
                    mmaLoHi<true>(tmemBase, lo + (smemAddr(smem) >> 4) + off, hi, lo + (smemAddr(sK) >> 4) + off, hi, kIdescQk, k != 0);
                }
                tcCommit(sFull);
            }
            __syncwarp();
        }
        uint32_t const tRow = tmemBase + (static_cast<uint32_t>(warp * 32) << 16);
        float const sl2 = args.scaleBmm1 * 1.4426950408889634f;
        constexpr float kMagic = 12582912.f; // 1.5 * 2^23: as_float(0x4B400000 + v) == kMagic + v for |v| < 2^22
        constexpr uint32_t kMagicBits = 0x4B400000u;
        ok = ok && mbarWait(sFull, 0, abortFlag, kWaitSoftmax);
        __syncwarp();
        tcFenceAfter();

        // row maximum (integers, no conversions); pieces of keys beyond the sequence are left out of all passes
        int const pieces = (len + 31) / 32;
        int32_t m0 = INT32_MIN, m1 = INT32_MIN, m2 = INT32_MIN, m3 = INT32_MIN;
#pragma unroll 1
        for (int p = 0; p < pieces; ++p)
        {
            uint32_t x[32];
            tmemLoad32(tRow + p * 32, x);
            tmemLoadWait32(x);
            int const limit = len - p * 32;
            if (limit < 32)
            {
#pragma unroll
                for (int i = 0; i < 32; ++i)
                    x[i] = i < limit ? x[i] : 0x80000000u;
            }
#pragma unroll
            for (int i = 0; i < 32; i += 8)
            {
                m0 = max(max(m0, static_cast<int32_t>(x[i])), static_cast<int32_t>(x[i + 1]));
                m1 = max(max(m1, static_cast<int32_t>(x[i + 2])), static_cast<int32_t>(x[i + 3]));
                m2 = max(max(m2, static_cast<int32_t>(x[i + 4])), static_cast<int32_t>(x[i + 5]));
                m3 = max(max(m3, static_cast<int32_t>(x[i + 6])), static_cast<int32_t>(x[i + 7]));
            }
        }
        float const mxMagic = kMagic + static_cast<float>(max(max(m0, m1), max(m2, m3))); // exact: both are integers below 2^24

        // exponentials, back to where the scores were, and the row sum: (p0 + p1) + (p2 + p3) of the pieces' sums
        float total = 0.f, before = 0.f;
#pragma unroll 1
        for (int p = 0; p < pieces; ++p)
        {
            uint32_t x[32];
            tmemLoad32(tRow + p * 32, x);
            tmemLoadWait32(x);
            int const limit = len - p * 32;
#pragma unroll
            for (int i = 0; i < 32; ++i)
                x[i] = __float_as_uint(ex2Approx((__uint_as_float(x[i] + kMagicBits) - mxMagic) * sl2));
            if (limit < 32)
            {
#pragma unroll
                for (int i = 0; i < 32; ++i)
                    x[i] = i < limit ? x[i] : 0u;
            }
            float sum = 0.f;
#pragma unroll
            for (int i = 0; i < 32; ++i)
                sum += __uint_as_float(x[i]);
            tmemStore32(tRow + p * 32, x);
            if ((p & 1) == 0)
                before = sum;
            else
                total += before + sum;
        }
        if ((pieces & 1) != 0)
            total += before;
        tmemStoreWait();
        float const inv = 1.f / total;
        float const pq = inv * args.scaleSoftmax;

        // P_q = rni(p / sum * scale_softmax); see the persistent kernel for the clamp
        bool const noClamp = args.scaleSoftmax <= 127.f;
#pragma unroll 1
        for (int p = 0; p < 4; ++p)
        {
            uint4 w[2] = {make_uint4(0, 0, 0, 0), make_uint4(0, 0, 0, 0)};
            if (p < pieces)
            {
                uint32_t x[32];
                tmemLoad32(tRow + p * 32, x);
                tmemLoadWait32(x);
                uint32_t* const o = reinterpret_cast<uint32_t*>(w);
#pragma unroll
                for (int i = 0; i < 8; ++i)
                {
                    float f[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        f[j] = __uint_as_float(x[4 * i + j]) * pq;
                    if (!noClamp)
                    {
#pragma unroll
                        for (int j = 0; j < 4; ++j)
                            f[j] = fminf(f[j], 127.f);
                    }
                    o[i] = packProb4<false>(f[0], f[1], f[2], f[3]);
                }
            }
            uint8_t* const pRow = sP + q * 128; // P: [128 rows][128 keys]
#pragma unroll
            for (int g = 0; g < 2; ++g)
                *reinterpret_cast<uint4*>(pRow + (((p * 2 + g) ^ (q & 7)) << 4)) = w[g];
        }
        fenceProxyAsync();
        tcFenceBefore();
        __syncthreads();
        if (warp == 0)
        {
            ok = ok && mbarWaitWarp(smemAddr(vFull), 0, abortFlag, kWaitTmaFull);
            tcFenceAfter();
            if (electOne() && ok)
            {
                uint64_t const dP = makeSmemDesc(0, 16, 1024, kSwizzle128B);
                uint64_t const dV = IL ? makeSmemDesc(0, kSubTile, kAtomBytes, kSwz) : makeSmemDesc(0, kAtomBytes, kAtomBytes, kSwz);
#pragma unroll
                for (int k = 0; k < 4; ++k) // 128 keys = 4 x 32
                    mmaLoHi<true>(tmemBase, static_cast<uint32_t>(dP) + (smemAddr(sP) >> 4) + k * 2, static_cast<uint32_t>(dP >> 32),
                        static_cast<uint32_t>(dV) + (smemAddr(sV) >> 4) + k * ((IL ? 1024u : 2048u) >> 4), static_cast<uint32_t>(dV >> 32), kIdescPv, k != 0);
                tcCommit(oFull);
            }
            __syncwarp();
        }
        ok = ok && mbarWait(oFull, 0, abortFlag, kWaitAccFull);
        __syncwarp();
        tcFenceAfter();
        float const s2 = args.scaleBmm2;
#pragma unroll 1
        for (int c = 0; c < args.d; c += 16)
        {
            uint32_t x[16];
            tmemLoad16(tRow + c, x);
            tmemLoadWait16(x);
            float v[16];
            if (noClamp) // |context| <= (127 + 256 / 2) * 128 < 2^22: the integer becomes a number without the conversion unit
            {
#pragma unroll
                for (int i = 0; i < 16; ++i)
                    v[i] = __uint_as_float(x[i] + kMagicBits) - kMagic;
            }
            else
            {
#pragma unroll
                for (int i = 0; i < 16; ++i)
                    v[i] = static_cast<float>(static_cast<int32_t>(x[i]));
            }
            if (q < rows && ok)
            {
                uint32_t w[4];
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    w[i] = packChar4(v[4 * i] * s2, v[4 * i + 1] * s2, v[4 * i + 2] * s2, v[4 * i + 3] * s2);
                *outPtr(c) = make_uint4(w[0], w[1], w[2], w[3]);
            }
            __syncwarp();
        }
        tcFenceBefore();
    }
    else if (q < rows) // no valid key: every probability is zero and so is the context row
    {
        for (int c = 0; c < args.d; c += 16)
            *outPtr(c) = make_uint4(0, 0, 0, 0);
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
        tmemFree(tmemBase, kShortTmemCols);
    }
}

using MhaKernel = void (*)(CUtensorMap, CUtensorMap, CUtensorMap, MhaArgs);

// form: up to three key blocks; four; four with the clamp of the probabilities
template <bool IL, bool BNSD, bool FIXED, Order ORDER>
MhaKernel mhaForm(int form)
{
    static constexpr MhaKernel kForms[3] = {mhaTcgen05Kernel<IL, BNSD, FIXED, ORDER, false, false>, mhaTcgen05Kernel<IL, BNSD, FIXED, ORDER, true, false>,
        mhaTcgen05Kernel<IL, BNSD, FIXED, ORDER, true, true>};
    return kForms[form];
}

// Sets the work items and launches: one persistent CTA per SM (512 TMEM columns and most of the shared memory each).
template <bool IL, bool BNSD>
int32_t launchItems(MhaArgs& args, CUtensorMap const (&maps)[3], cudaStream_t stream)
{
    static_assert(kItemTile == kQTile, "tiles of the plan");
    int64_t const pairs = static_cast<int64_t>(args.B) * args.N;
    if (args.S <= kKeyBlock && pairs <= INT32_MAX) // one key block: the short kernel is ahead from one pair to thousands (see there)
    {
        static SmemOptIn optIn;
        cudaError_t const e = launchDependentCluster(&optIn, mhaShortInt8Kernel<IL, BNSD>, dim3(static_cast<unsigned>(pairs)), dim3(kShortThreads),
            kShortSmemBytes, stream, 1, maps[0], maps[1], maps[2], args);
        if (e != cudaSuccess)
            B200_FAIL(BERT_B200_CUDA_ERROR, "mhaShortInt8Kernel: %s", cudaGetErrorString(e));
        return checkLaunch("mhaShortInt8Kernel");
    }
    int64_t const missing = !args.fixedLayout ? static_cast<int64_t>(args.B) * args.S - args.total : (args.maskIdx ? INT64_MAX : 0);
    ItemPlan const plan = planItems(args.B, args.N, args.S, missing, smCount());
    int64_t const cut = args.fixedLayout || plan.chunks > 1 ? 0 : cutTiles(args.B, args.N, args.S, args.total, smCount());
    args.tilesPerItem = plan.tilesPerItem;
    args.chunks = plan.chunks;
    int64_t const items = cut > 0 ? cut : static_cast<int64_t>(args.B) * args.N * plan.chunks;
    Order const order = cut > 0 ? Order::kTiles : plan.longestFirst ? Order::kPairs : Order::kNone;
    int const grid = static_cast<int>(items < smCount() ? items : smCount());
    args.rounds = cut > 0 ? 3 * plan.tilesPerItem / 4 : static_cast<int32_t>((items + grid - 1) / grid); // cut: see cutIsShorter
    int const smem = MhaSmem::dynamicBytes((args.S + kKeyBlock - 1) / kKeyBlock) + (order != Order::kNone ? static_cast<int>(sizeof(ItemTable)) : 0);
    int const form = args.S <= 3 * kKeyBlock ? 0 : args.scaleSoftmax <= 127.f ? 1 : 2;
    MhaKernel kernel;
    if constexpr (BNSD) // always fixed
        kernel = order == Order::kPairs ? mhaForm<IL, BNSD, true, Order::kPairs>(form) : mhaForm<IL, BNSD, true, Order::kNone>(form);
    else
    {
        kernel = order == Order::kTiles ? mhaForm<IL, BNSD, false, Order::kTiles>(form)
            : order == Order::kPairs    ? mhaForm<IL, BNSD, false, Order::kPairs>(form)
                                        : mhaForm<IL, BNSD, false, Order::kNone>(form);
        if constexpr (!IL) // interleaved: always packed
            if (args.fixedLayout)
                kernel = order == Order::kPairs ? mhaForm<IL, BNSD, true, Order::kPairs>(form) : mhaForm<IL, BNSD, true, Order::kNone>(form);
    }
    static SmemOptIn optIn[2][3][3];
    cudaError_t const e = launchDependentCluster(&optIn[args.fixedLayout ? 1 : 0][static_cast<int>(order)][form], kernel, dim3(grid), dim3(kMhaThreads), smem,
        stream, 1, maps[0], maps[1], maps[2], args);
    if (e != cudaSuccess)
        B200_FAIL(BERT_B200_CUDA_ERROR, "mhaTcgen05Kernel: %s", cudaGetErrorString(e));
    return checkLaunch("mhaTcgen05Kernel");
}

template <bool IL>
int32_t launchMha(bert_b200_mha_params const& p, cudaStream_t stream)
{
    bool const fixedLayout = p.cu_seqlens == nullptr;
    uint64_t const d = static_cast<uint64_t>(p.head_size);
    uint64_t const rowElems = 3ull * static_cast<uint64_t>(p.num_heads) * d;
    // The boxes are always 64 channels wide (two 32-channel groups when interleaved); for a smaller head the channels
    // beyond d lie outside the tensor's channel dimension and arrive as zeros, which change neither Q.K nor P.V.
    CUtensorMap maps[3];
    CUtensorMap& map = maps[0];
    if (IL)
    {
        // [3][N][d/32][total][32]: dim0 the 32 channels of a group, dim1 the token, dim2 the group, dim3 which of [3][N]
        uint64_t const dims[4] = {32, static_cast<uint64_t>(p.total), d / 32, 3ull * static_cast<uint64_t>(p.num_heads)};
        uint64_t const strides[3] = {32, static_cast<uint64_t>(p.total) * 32, (d / 32) * static_cast<uint64_t>(p.total) * 32};
        uint32_t const box[4] = {32, kKeyBlock, 2, 1};
        int32_t const st = makeTensorMap(&map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, p.qkv, dims, strides, box,
            CU_TENSOR_MAP_SWIZZLE_32B);
        if (st != BERT_B200_OK)
            return st;
    }
    else
    {
        // dim0: the d channels of one of Q, K, V of a head; dim1: which of [N][3]; dim2: batch (fixed layout only);
        // dim3: sequence position / packed row
        uint64_t const dims[4] = {d, 3ull * static_cast<uint64_t>(p.num_heads), fixedLayout ? static_cast<uint64_t>(p.B) : 1ull,
            fixedLayout ? static_cast<uint64_t>(p.S) : static_cast<uint64_t>(p.total)};
        uint64_t const strides[3] = {d, rowElems, (fixedLayout ? static_cast<uint64_t>(p.B) : 1ull) * rowElems};
        uint32_t const box[4] = {kHeadSize, 1, 1, kKeyBlock};
        int32_t const st = makeTensorMap(&map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, p.qkv, dims, strides, box,
            CU_TENSOR_MAP_SWIZZLE_64B);
        if (st != BERT_B200_OK)
            return st;
    }
    maps[1] = map;
    maps[2] = map;
    MhaArgs args{p.B, p.S, p.num_heads, p.total, p.head_size, fixedLayout ? 1 : 0, p.out, p.cu_seqlens, p.mask_idx, p.scale_bmm1,
        p.scale_softmax, p.scale_bmm2, p.status_word, 1, 1, 1};
    return launchItems<IL, false>(args, maps, stream);
}

// Separate Q, K, V tensors of shape [B][N][S][d] (the operand layout of TensorRT's attention layer), output
// [B][N][S][d]: three tensor maps, the same kernel.
int32_t launchMhaBnsd(bert_b200_attention_bnsd_params const& p, cudaStream_t stream)
{
    uint64_t const d = static_cast<uint64_t>(p.head_size), S = static_cast<uint64_t>(p.S), N = static_cast<uint64_t>(p.num_heads);
    CUtensorMap maps[3];
    void const* const base[3] = {p.q, p.k, p.v};
    for (int i = 0; i < 3; ++i)
    {
        // dim0: channel (box 64 wide, zero-filled beyond d); dim1: position; dim2: head; dim3: sequence
        uint64_t const dims[4] = {d, S, N, static_cast<uint64_t>(p.B)};
        uint64_t const strides[3] = {d, S * d, N * S * d};
        uint32_t const box[4] = {kHeadSize, kKeyBlock, 1, 1};
        int32_t const st = makeTensorMap(&maps[i], CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, base[i], dims, strides, box,
            CU_TENSOR_MAP_SWIZZLE_64B);
        if (st != BERT_B200_OK)
            return st;
    }
    MhaArgs args{p.B, p.S, p.num_heads, 0, p.head_size, 1, p.out, nullptr, p.kv_lengths, p.scale_bmm1, p.scale_softmax,
        p.scale_bmm2, p.status_word, 1, 1, 1};
    return launchItems<false, true>(args, maps, stream);
}

} // namespace

} // namespace b200

using namespace b200;

extern "C" int32_t bert_b200_attention_bnsd(bert_b200_attention_bnsd_params const* params, void* stream)
{
    B200_REQUIRE(params != nullptr, "attention_bnsd: null params");
    bert_b200_attention_bnsd_params const& p = *params;
    B200_REQUIRE(p.B >= 0 && p.S > 0 && p.num_heads > 0 && p.head_size > 0, "attention_bnsd: bad sizes B=%d S=%d N=%d d=%d", p.B,
        p.S, p.num_heads, p.head_size);
    B200_REQUIRE(p.q && p.k && p.v && p.out, "attention_bnsd: null pointer");
    if (p.B == 0)
        return BERT_B200_OK;
    B200_REQUIRE(p.B <= 65535 && p.num_heads <= 65535, "attention_bnsd: B and num_heads are limited to 65535");
    B200_REQUIRE(p.type_id == BERT_B200_FP16 || p.type_id == BERT_B200_INT8, "attention_bnsd: type_id %d", p.type_id);
    if (p.head_size > kHeadSize || p.head_size % 16 != 0)
        B200_FAIL(BERT_B200_NOT_SUPPORTED, "attention_bnsd: head sizes 16, 32, 48 and 64, got %d", p.head_size);
    if (p.S > kMaxBlocks * kKeyBlock && p.type_id == BERT_B200_INT8)
        B200_FAIL(BERT_B200_NOT_SUPPORTED, "attention_bnsd: INT8 takes S <= %d, got %d", kMaxBlocks * kKeyBlock, p.S);
    B200_REQUIRE(aligned16(p.q) && aligned16(p.k) && aligned16(p.v) && aligned16(p.out),
        "attention_bnsd: q, k, v and out must be 16-byte aligned");
    auto s = static_cast<cudaStream_t>(stream);
    if (p.type_id == BERT_B200_FP16)
    {
        B200_REQUIRE(p.scale_bmm1 > 0.f, "attention_bnsd: scale_bmm1 must be positive");
        return mhaOnlineF16Bnsd(p, s);
    }
    return launchMhaBnsd(p, s);
}

extern "C" int32_t bert_b200_mha(bert_b200_mha_params const* params, void* stream)
{
    B200_REQUIRE(params != nullptr, "mha: null params");
    bert_b200_mha_params const& p = *params;
    B200_REQUIRE(p.B >= 0 && p.S > 0 && p.num_heads > 0 && p.head_size > 0, "mha: bad sizes B=%d S=%d N=%d d=%d", p.B, p.S,
        p.num_heads, p.head_size);
    B200_REQUIRE(p.qkv && p.out, "mha: null pointer");
    B200_REQUIRE(p.cu_seqlens == nullptr || p.total >= 0, "mha: packed layout needs total >= 0");
    if (p.B == 0 || (p.cu_seqlens && p.total == 0))
        return BERT_B200_OK;
    B200_REQUIRE(p.B <= 65535 && p.num_heads <= 65535, "mha: B and num_heads are limited to 65535");
    auto s = static_cast<cudaStream_t>(stream);
    if (p.type_id == BERT_B200_FP32)
        return mhaSimt(p, s);
    B200_REQUIRE(p.type_id == BERT_B200_FP16 || p.type_id == BERT_B200_INT8, "mha: type_id %d", p.type_id);
    B200_REQUIRE(!p.interleaved || (p.type_id == BERT_B200_INT8 && p.cu_seqlens != nullptr),
        "mha: the interleaved (CHW32) layout needs INT8 and the packed (cu_seqlens) form");
    bool const headOk = p.head_size <= kHeadSize && p.head_size % 16 == 0 && (!p.interleaved || p.head_size % 32 == 0);
    bool const lengthOk = p.S <= kMaxBlocks * kKeyBlock;
    if (headOk && p.type_id == BERT_B200_FP16 && !p.interleaved && p.scale_bmm1 > 0.f)
    {
        B200_REQUIRE(aligned16(p.qkv) && aligned16(p.out), "mha: qkv and out must be 16-byte aligned");
        return mhaOnlineF16(p, s);
    }
    // Outside the tensor-core kernel's shapes FP16 takes the SIMT kernel, like the reference's unfused runner
    // (qkvToContextPlugin.cpp:335-341, 522-531); INT8 has no such path there either (qkvToContextPlugin.cpp:530).
    if (p.type_id == BERT_B200_FP16) // heads wider than 64 or not a multiple of 16 (or a non-positive scale)
        return mhaSimt(p, s);
    if (!headOk)
        B200_FAIL(BERT_B200_NOT_SUPPORTED,
            "mha: INT8 takes head sizes 16, 32, 48 and 64 (32 and 64 when interleaved), got %d", p.head_size);
    if (!lengthOk)
        B200_FAIL(BERT_B200_NOT_SUPPORTED, "mha: INT8 takes S <= %d, got %d", kMaxBlocks * kKeyBlock, p.S);
    B200_REQUIRE(aligned16(p.qkv) && aligned16(p.out), "mha: qkv and out must be 16-byte aligned");
    if (p.interleaved)
        return launchMha<true>(p, s);
    return launchMha<false>(p, s);
}

extern "C" int64_t bert_b200_mha_workspace_size(bert_b200_mha_params const* params)
{
    (void) params; // no attention kernel of this library needs scratch memory
    return 0;
}
