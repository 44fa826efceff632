// FP32 (type_id 0) fully connected layer on the sm_100a tensor cores: C = act(alpha * A * Wt^T + bias) at full FP32 precision.
//
// Replaces the FP32 cublasLtMatmul of the FC plugin (plugin/fcPlugin/fcPlugin.cpp:551-610). TF32 would break the 1e-5 tolerance
// that the reference configuration states for FP32 (plugin/bertQKVToContextPlugin/CustomQKVToContextPluginDynamic_PluginConfig.yaml:72-76),
// so every operand is cut into three BF16 numbers, x = h + m + l (the split of Henry, Tang and Heinecke, "Leveraging the bfloat16 artificial
// intelligence datatype for higher-precision computations", 2019). h and m are rounded to nearest, which is exact: |m| <= 2^-8, |l| <= 2^-17 of the
// largest number of x's exponent. Six products are formed: h h + (h m + m h) + (h l + m m + l h). The three that are left out are below
// 2^-24 of a product in sum and have either sign.
//
// The tensor core cuts off what does not fit its FP32 accumulator, always towards zero, so nothing is summed there for long, and what is lost on
// the way up is lost again on the way down: of a chunk of 64 products per output, the first half of h h goes into one accumulator, P; the other gets
// the five small products (from zero, so that their additions lose little), minus that first half and plus the second one, Q. The sum is 2 P + Q,
// and on products of one sign Q ends near zero. Chunks are added in registers, rounded to nearest. Error against 64 bits: see fcF32.
#include "sm100.cuh"

namespace b200
{

int32_t fcF32Simt(bert_b200_fc_params const& p, cudaStream_t stream);

namespace
{

constexpr int kTileM = 128;
constexpr int kChunk = 64;      // of K: one 128-byte row of a BF16 operand tile, two of the FP32 tiles
constexpr int kWorkers = 16;    // warps, in two groups of eight
constexpr int kThreadsF32 = 64 + kWorkers * 32;
constexpr int kMaxSegments = 8; // portable cluster size
constexpr int kParts = 2;       // chunks whose parts are in place

struct FcF32TcArgs
{
    int64_t M, N, K, lda, ldc;
    float const* A;
    float const* Wt;
    float* C;
    float const* bias;
    int32_t act;
    float alpha;
    int32_t nTiles;   // tiles along N
    int32_t segments; // of K
    int32_t ctas;     // per tile: 1 or `segments`
    int32_t wide;     // rows of C may be stored in 16-byte pieces
    uint32_t* statusWord;
};

template <int BN>
struct FcF32Smem
{
    static constexpr int kStages = BN >= 96 ? 2 : 3; // FP32 tiles
    static constexpr int kABytes = kTileM * kChunk * 4;
    static constexpr int kWBytes = BN * kChunk * 4;
    static constexpr int kStageBytes = kABytes + kWBytes;
    static constexpr int kPlaneBytes = BN * kChunk * 2; // one BF16 part of the Wt tile
    static constexpr int kPlanesOff = kStages * kStageBytes;
    static constexpr int kBarrierOff = kPlanesOff + kParts * 3 * kPlaneBytes;
    static constexpr int kAccs = BN <= 64 ? 2 : 1;      // chunks whose sums are in tensor memory, two accumulators each
    static constexpr int kHalves = kAccs == 1 ? 2 : 1; // of the columns, whose products are formed one after the other
    // Groups of warps that take chunks in turn. 32 columns: eight warps cut a chunk as fast as 16 (Wt has 32 rows, eight warps' work), and with the other
    // eight a chunk ahead the sums wait less: 512 x 1024 x 4096 53.8 us (all 16: 58.5 us), 129 x 2304 x 768 13.8 us (14.4 us).
    static constexpr int kTurns = BN == 32 ? 2 : 1;
    static constexpr int kCutters = kWorkers / kTurns; // warps that cut a chunk
    // stFull[stages] stFree[stages] ready[parts] done[halves][parts] accFree[2], tmem slot, abort flag, flags of rows of A and Wt (1: a number without exact parts, 2: NaN),
    // whether any is set
    static constexpr int kFlagsOff = kBarrierOff + (2 * kStages + (1 + kHalves) * kParts + 2) * 8 + 16;
    static constexpr int kTotal = kFlagsOff + (kTileM + BN + 4) * 4;
    static constexpr int kDynamic = kTotal + 1024;
    static constexpr int kPitch = BN + 4; // floats: sums of a tile over the drained FP32 tiles
    static constexpr int kTmem = 512;
    static constexpr int kAccCols = kAccs * 2 * BN;
    // Columns that a worker's sums of the segments before take in tensor memory: all of them but for the 128-wide tile (half).
    static constexpr int kHeldCols = BN / 4 < (kTmem - kAccCols - kParts * 96) / 4 ? BN / 4 : (kTmem - kAccCols - kParts * 96) / 4;
    static_assert(kDynamic <= 232448, "shared memory of one CTA");
    static_assert(kTileM * kPitch * 4 + kTileM * BN / 8 + kTileM * BN / 4 + 4 <= kPlanesOff, "the sums, and what is computed again, fit the ring");
    static_assert(kAccCols + kParts * 96 + 4 * kHeldCols <= kTmem, "tensor memory");
};

// Two floats to BF16 (the first in the lower half), rounded to nearest, and what that leaves of them.
__device__ __forceinline__ uint64_t cutPair(uint64_t x, uint32_t& part)
{
    float a, b;
    unpack2(x, a, b);
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(part) : "f"(b), "f"(a));
    return fma2(pack2(__uint_as_float(part << 16), __uint_as_float(part & 0xffff0000u)), pack2(-1.f, -1.f), x);
}

// Two floats into packed BF16 parts. What is left when the last part is cut goes into the lower halves of `lost`: numbers below 2^-110 have bits
// that BF16 does not (its smallest is 2^-133); infinities, NaN and what rounds to infinity leave a NaN.
__device__ __forceinline__ void splitPair(float a, float b, uint32_t& h, uint32_t& m, uint32_t& l, uint32_t& lost)
{
    float la, lb;
    unpack2(cutPair(cutPair(pack2(a, b), h), m), la, lb);
    l = __byte_perm(__float_as_uint(la), __float_as_uint(lb), 0x7632);
    lost |= __float_as_uint(la) | __float_as_uint(lb);
}

__device__ __forceinline__ void tmemStore8(uint32_t taddr, uint32_t const (&r)[8])
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]),
                 "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}

__device__ __forceinline__ void tmemLoad8(uint32_t taddr, uint32_t (&r)[8])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ void tmemLoadWait8(uint32_t (&r)[8])
{
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7])
                 :
                 : "memory");
}

// 16 or 8 columns at two places, waited for.
__device__ __forceinline__ void tmemLoadTwo(uint32_t ta, uint32_t (&a)[16], uint32_t tb, uint32_t (&b)[16])
{
    tmemLoad16(ta, a);
    tmemLoad16(tb, b);
    tmemLoadWait16(a);
    tmemLoadWait16(b);
}
__device__ __forceinline__ void tmemLoadTwo(uint32_t ta, uint32_t (&a)[8], uint32_t tb, uint32_t (&b)[8])
{
    tmemLoad8(ta, a);
    tmemLoad8(tb, b);
    tmemLoadWait8(a);
    tmemLoadWait8(b);
}

// sums[i] += 2 * P + Q for N columns.
template <int N>
__device__ __forceinline__ void addSums(uint32_t tP, uint32_t tQ, uint64_t* sums)
{
    uint32_t x[N], y[N];
    tmemLoadTwo(tP, x, tQ, y);
    uint64_t const two = pack2(2.f, 2.f);
#pragma unroll
    for (int i = 0; i < N / 2; ++i)
        sums[i] = add2(sums[i], fma2(pack2(__uint_as_float(x[2 * i]), __uint_as_float(x[2 * i + 1])), two,
                                    pack2(__uint_as_float(y[2 * i]), __uint_as_float(y[2 * i + 1]))));
}

__device__ __forceinline__ float finishF32(FcF32TcArgs const& p, float v, float bias)
{
    v = v * p.alpha + bias;
    return p.act == BERT_B200_ACT_GELU_ERF ? geluErfF32(v) : v;
}

// Whether a sum may not be what FP32 multiply-adds give although its numbers have exact parts. The tensor core cuts off below 2^-149 with every
// addition (error on products of 2^-126 2.3e-7 instead of 1.4e-7, of 2^-132 9e-6 instead of 2.2e-6), which a sum of 2^-100 and more does
// not notice. And sums on the way may be twice as large as the result.
__device__ __forceinline__ bool sumIsInexact(float v)
{
    constexpr uint32_t kLeast = 0x0d800000u, kInf = 0x7f800000u; // 2^-100
    uint32_t const u = __float_as_uint(v) & 0x7fffffffu;
    return u != 0 && u - kLeast >= kInf - kLeast;
}

// Whether a NaN is among the k numbers (a multiple of four, 16-byte aligned), for a warp.
__device__ __forceinline__ bool hasNan(float const* row, int64_t k)
{
    bool nan = false;
#pragma unroll 4
    for (int64_t i = (threadIdx.x & 31) * 4; i < k; i += 128)
    {
        float4 const v = __ldg(reinterpret_cast<float4 const*>(row + i));
        nan |= isnan(v.x) | isnan(v.y) | isnan(v.z) | isnan(v.w);
    }
    return __any_sync(0xffffffffu, nan);
}

// The outputs of a tile whose bit in `again` (BN bits per row) is set, by FP32 multiply-adds: a warp takes 4 x 4 outputs, its lanes every 32nd four
// of K, even and odd ones apart, and their sums are added as a tree, so an output has the same bits wherever its tile lies. The chains are a
// quarter or less as long as those of fcF32Simt (error on normal values K = 768 0.9e-7 / 1.4e-7, 4096 1.6e-7 / 2.9e-7). Bound by the loads' latency for a
// few outputs, by what the L2 brings for all (4 x 4 outputs are read by 8 rows). 1024 x 2304 x 768, nothing to compute again / an infinity in A / a number
// below 2^-110 in Wt / A full of them, in the form of that time: 33.2 / 45.9 / 46.2 / 335 us (a NaN 34.9 us); a thread per output and all of K in one chain, in the kernel
// of that time, 29.6 / 140 / 169 / 10 100 us; fcF32Simt 97 us.
template <int BN>
__device__ __noinline__ void computeAgain(FcF32TcArgs const& p, uint32_t const* again, uint32_t* list, int64_t m0, int64_t n0)
{
    int const warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int kAcross = BN / 4;
    auto const maskOf = [&](int i) {
        int const r = i / kAcross * 4, c = i % kAcross * 4;
        uint32_t mask = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j)
            mask |= (again[(r + j) * (BN / 32) + c / 32] >> (c % 32) & 15u) << (4 * j);
        return mask;
    };
    for (int i = threadIdx.x; i < kTileM / 4 * kAcross; i += kThreadsF32)
        if (maskOf(i) != 0)
            list[1 + atomicAdd(list, 1u)] = i;
    __syncthreads();
    int const blocks = static_cast<int>(list[0]);
#pragma unroll 1
    for (int i = warp; i < blocks; i += kThreadsF32 / 32)
    {
        int const block = static_cast<int>(list[1 + i]);
        uint32_t const mask = maskOf(block);
        int const r = block / kAcross * 4, c = block % kAcross * 4;
        float const *a[4], *w[4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
        {
            a[j] = p.A + min(m0 + r + j, p.M - 1) * p.lda;
            w[j] = p.Wt + min(n0 + c + j, p.N - 1) * p.K;
        }
        uint64_t acc[16] = {};
#pragma unroll 1
        for (int64_t k = lane * 4; k < p.K; k += 128)
        {
            float4 av[4], wv[4];
#pragma unroll
            for (int j = 0; j < 4; ++j)
            {
                av[j] = __ldg(reinterpret_cast<float4 const*>(a[j] + k));
                wv[j] = __ldg(reinterpret_cast<float4 const*>(w[j] + k));
            }
#pragma unroll
            for (int j = 0; j < 16; ++j)
            {
                acc[j] = fma2(pack2(av[j >> 2].x, av[j >> 2].y), pack2(wv[j & 3].x, wv[j & 3].y), acc[j]);
                acc[j] = fma2(pack2(av[j >> 2].z, av[j >> 2].w), pack2(wv[j & 3].z, wv[j & 3].w), acc[j]);
            }
        }
        // lane 2 j gets the sum of output j: each step halves the outputs that a lane holds
        float v[16];
#pragma unroll
        for (int j = 0; j < 16; ++j)
        {
            float lo, hi;
            unpack2(acc[j], lo, hi);
            v[j] = lo + hi;
        }
#pragma unroll
        for (int half = 8; half >= 1; half >>= 1)
        {
            bool const upper = (lane & (2 * half)) != 0;
#pragma unroll
            for (int j = 0; j < half; ++j)
            {
                float const other = __shfl_xor_sync(0xffffffffu, upper ? v[j] : v[j + half], 2 * half);
                v[j] = (upper ? v[j + half] : v[j]) + other;
            }
        }
        v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
        int const j = lane >> 1;
        if ((lane & 1) == 0 && (mask >> j & 1u) != 0)
        {
            int64_t const n = n0 + c + (j & 3);
            p.C[(m0 + r + (j >> 2)) * p.ldc + n] = finishF32(p, v[0], p.bias ? __ldg(p.bias + n) : 0.f);
        }
    }
}

// Bound by the warps that cut operands, and by shared memory behind them: a chunk of a 128 x 128 tile takes 2900 cycles (stamps), of which the
// tensor cores are busy 1620 and shared memory serves the warps for 1130 and the products for 840 (counters, the tile's end included); of a 64-wide
// one 1870. The warps take turns with nothing any more: the columns of a 128- or 96-wide tile, whose accumulators fit tensor memory only once, are multiplied in
// two halves, so that the sums of one are read while the other's products run; all 16 warps cut every chunk beyond 32 columns (with two groups
// taking chunks in turn the sums waited for the group that was cutting); and a chunk's three barriers are asked at once (an answer takes 120 ... 150
// cycles). A chunk's place in the ring is handed back behind the stores of its parts and a proxy fence: an arrival right behind the loads does not wait
// for them, so that now and then numbers of the next tile came into the registers instead (and it saved no time). Before / after: 3400 / 2900 cycles
// per chunk; 1024 x 2304 x 768 32.7 / 28.2 us, 2000 x 3072 x 1024 117 / 101 us, 4096 x 3072 x 1024 215 / 209 us, 37 x 2304 x 768 11.3 / 10.7 us.
// Rounding costs nothing: truncation of h, other subtractions or loads further ahead leave the times as they are.
// One 128 x BN tile per CTA, or one segment of its K:
//   warp 0    : FP32 tiles of A and Wt by TMA (128-byte swizzle) into a ring.
//   warp 1    : TMEM allocation, MMA issue. The parts of A are operands in TMEM - from shared memory both operands of a
//               128 x 128 tile would take its whole bandwidth -, those of Wt in shared memory.
//   warps 2-17: the parts of every chunk (32 columns: two groups of eight, chunks in turn): 16 numbers of a row of A per thread, to TMEM, and whole
//               16-byte pieces of the parts of Wt, to shared memory. And its sums (32 rows, a quarter of the columns per warp) from TMEM into registers. Parts are
//               double-buffered, the two accumulators too where tensor memory has room (up to 64 columns).
// K is cut into segments by K alone and the segments' sums are added in order, so a row has the same bits whatever M: a CTA takes
// all segments in turn (kHold), or a cluster one per CTA, exchanging the sums through distributed shared memory.
// An output whose row of A or Wt holds numbers without exact parts (splitPair) is computed again by FP32 multiply-adds (computeAgain), unless one
// of them is NaN: then it comes out as that. So is a sum that sumIsInexact names.
template <int BN, bool kHold>
__global__ void __launch_bounds__(kThreadsF32, 1)
    fcF32TcKernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapW, const __grid_constant__ FcF32TcArgs p)
{
    using L = FcF32Smem<BN>;
    constexpr int kWidth = BN / L::kHalves; // columns of a product
    constexpr uint32_t kIdesc = makeInstrDesc(1u, 1u, 0u, 0u, 128u, static_cast<uint32_t>(kWidth));
    constexpr int kCols = BN / 4; // accumulator columns per worker thread
    constexpr uint32_t kIdescMinus = kIdesc | 1u << 13; // minus A
    constexpr uint32_t kPartsCol = L::kAccCols;

    extern __shared__ uint8_t smemRaw[];
    uint8_t* const smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smemRaw) + 1023) & ~static_cast<uintptr_t>(1023));
    uint64_t* const stFull = reinterpret_cast<uint64_t*>(smem + L::kBarrierOff);
    uint64_t* const stFree = stFull + L::kStages;
    uint64_t* const ready = stFree + L::kStages; // parts of a chunk in place
    uint64_t* const done = ready + kParts;       // [halves][parts] their products complete
    uint64_t* const accFree = done + L::kHalves * kParts; // an accumulator (or its half) has been read
    uint32_t* const tmemSlot = reinterpret_cast<uint32_t*>(accFree + 2);
    volatile uint32_t* const abortFlag = tmemSlot + 1;
    uint32_t* const flagA = reinterpret_cast<uint32_t*>(smem + L::kFlagsOff);
    uint32_t* const flagW = flagA + kTileM;
    uint32_t* const flagAny = flagW + BN;
    float* const sums = reinterpret_cast<float*>(smem);
    uint32_t* const again = reinterpret_cast<uint32_t*>(sums + kTileM * L::kPitch); // a bit per output that is computed again
    uint32_t* const list = again + kTileM * BN / 32;                               // see computeAgain

    int const warp = threadIdx.x >> 5;
    int const lane = threadIdx.x & 31;
    int const rank = p.ctas > 1 ? static_cast<int>(blockIdx.x % p.ctas) : 0;
    int64_t const tile = blockIdx.x / p.ctas;
    int64_t const m0 = tile / p.nTiles * kTileM;
    int64_t const n0 = tile % p.nTiles * BN;
    int const kChunks = static_cast<int>((p.K + kChunk - 1) / kChunk);
    auto segmentBegin = [&](int s) { return static_cast<int>(static_cast<int64_t>(kChunks) * s / p.segments); };
    int const first = p.ctas > 1 ? segmentBegin(rank) : 0;
    int const count = (p.ctas > 1 ? segmentBegin(rank + 1) : kChunks) - first;

    if (threadIdx.x == 0)
    {
        for (int i = 0; i < L::kStages; ++i)
        {
            mbarInit(&stFull[i], 1);
            mbarInit(&stFree[i], L::kCutters);
        }
        for (int i = 0; i < kParts; ++i)
            mbarInit(&ready[i], L::kCutters);
        for (int i = 0; i < L::kHalves * kParts; ++i)
            mbarInit(&done[i], 1);
        for (int i = 0; i < 2; ++i)
            mbarInit(&accFree[i], kWorkers / L::kHalves);
        *abortFlag = 0;
        fenceBarrierInit();
        prefetchTensorMap(&mapA);
        prefetchTensorMap(&mapW);
    }
    for (int i = threadIdx.x; i < kTileM + BN + 1; i += kThreadsF32)
        flagA[i] = 0;
    if (warp == 1)
        tmemAlloc(tmemSlot, L::kTmem);
    tcFenceBefore();
    __syncthreads();
    tcFenceAfter();
    uint32_t const tmemBase = *tmemSlot;
    gridDependencyLaunch();
    gridDependencyWait();

    uint64_t acc[kCols / 2] = {}; // sums over the chunks, column pairs
    if (warp == 0)
    {
        bool ok = true;
        int stage = 0;
        uint32_t phase = 1;
        for (int c = 0; c < count && ok; ++c)
        {
            uint32_t const bar = smemAddr(&stFull[stage]);
            uint32_t const a = smemAddr(smem) + stage * L::kStageBytes;
            int32_t const k = (first + c) * kChunk;
            ok = mbarWaitWarp(&stFree[stage], phase, abortFlag, kWaitStageFree);
            if (ok && electOne())
            {
                mbarArriveExpectTxAddr(bar, L::kStageBytes);
#pragma unroll
                for (int h = 0; h < 2; ++h)
                {
                    tmaLoad2dAddr(a + h * (L::kABytes / 2), &mapA, bar, k + h * 32, static_cast<int32_t>(m0));
                    tmaLoad2dAddr(a + L::kABytes + h * (L::kWBytes / 2), &mapW, bar, k + h * 32, static_cast<int32_t>(n0));
                }
            }
            __syncwarp();
            if (++stage == L::kStages)
            {
                stage = 0;
                phase ^= 1u;
            }
        }
    }
    else if (warp == 1)
    {
        uint64_t const descZero = makeSmemDesc(0, 16, 1024, kSwizzle128B);
        uint32_t const descHi = static_cast<uint32_t>(descZero >> 32);
        uint32_t const wLo = static_cast<uint32_t>(descZero) + (smemAddr(smem + L::kPlanesOff) >> 4);
        bool ok = true;
        for (int c = 0; c < count && ok; ++c)
        {
            uint32_t const s = c & 1, round = c >> 1;
            uint32_t const slot = c % L::kAccs;
            // What is there first is asked first, so that an answer is not waited for when the last one has come: two accumulators have been read before
            // a chunk's parts are ready, a single one after it (512 x 1024 x 4096, 32 columns: the other way round 55.2 us).
            bool const freeFirst = L::kAccs == 2 && c >= L::kAccs;
            ok = (!freeFirst || mbarWaitWarp(&accFree[slot], (c / L::kAccs - 1) & 1u, abortFlag, kWaitAccFree))
                && mbarWaitWarp(&ready[s], round & 1u, abortFlag, kWaitSoftmax);
#pragma unroll
            for (int h = 0; h < L::kHalves; ++h)
            {
                ok = ok && (L::kAccs == 2 || c == 0 || mbarWaitWarp(&accFree[h], (c - 1) & 1u, abortFlag, kWaitAccFree));
                tcFenceAfter();
                if (ok && electOne())
                {
                    // parts (A, Wt), the smallest products first
                    constexpr int kOrder[5][2] = {{2, 0}, {0, 2}, {1, 1}, {1, 0}, {0, 1}};
                    uint32_t const a = tmemBase + kPartsCol + s * 96;
                    uint32_t const w = wLo + s * (3 * L::kPlaneBytes >> 4) + h * (kWidth * 128 >> 4);
                    uint32_t const sumP = tmemBase + slot * 2 * BN + h * kWidth, sumQ = sumP + BN;
#pragma unroll
                    for (int i = 0; i < 5; ++i)
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            mmaF16TmemA(sumQ, a + kOrder[i][0] * 32 + k * 8, w + kOrder[i][1] * (L::kPlaneBytes >> 4) + k * 2, descHi, kIdesc,
                                i != 0 || k != 0);
#pragma unroll
                    for (int k = 0; k < 2; ++k)
                        mmaF16TmemA(sumP, a + k * 8, w + k * 2, descHi, kIdesc, k != 0);
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        mmaF16TmemA(sumQ, a + k * 8, w + k * 2, descHi, k < 2 ? kIdescMinus : kIdesc, true);
                    tcCommit(&done[h * kParts + s]);
                }
                __syncwarp();
            }
        }
    }
    else
    {
        int const quad = warp & 3;
        int const group = (warp - 2) >> 3; // takes every second 32 rows of Wt (32 columns: every second chunk)
        int const w = (warp - 2) & 7;      // which 8 of a chunk's K of Wt
        int const cols = (warp - 2) >> 2;  // which quarter of the accumulator columns, and which 16 of a chunk's K of A (32 columns: two of these)
        int const part = L::kHalves == 2 ? group : 0;
        bool const hasRows = m0 + quad * 32 < p.M; // warp-uniform; products of the other rows are never read
        uint32_t const tRow = tmemBase + (static_cast<uint32_t>(quad * 32) << 16);
        // Sums of the segments before: touched once per segment and kept out of the registers, which are all taken in the loop
        // (spilled by the compiler they cost 14 us of 1024 x 2304 x 768: beside so much shared memory the L1 holds little). What does
        // not fit tensor memory is in local memory on purpose (all of them there: 2.6 us more).
        uint32_t const tHeld = tRow + kPartsCol + kParts * 96 + cols * L::kHeldCols;
        volatile uint64_t rest[kHold && kCols > L::kHeldCols ? (kCols - L::kHeldCols) / 2 : 1];
        int segment = 0;
        int segmentEnd = segmentBegin(1);
        bool ok = true;
        // the sums of chunk c (`summed`: they are known to be complete)
        auto promote = [&](int c, bool summed) {
            if (!__all_sync(0xffffffffu, summed))
                ok = ok && mbarWaitWarp(&done[part * kParts + (c & 1)], (c >> 1) & 1u, abortFlag, kWaitAccFull);
            tcFenceAfter();
            if (hasRows)
            {
                uint32_t const t = tRow + (c % L::kAccs) * 2 * BN + cols * kCols;
#pragma unroll
                for (int g = 0; g + 16 <= kCols; g += 16)
                    addSums<16>(t + g, t + BN + g, acc + g / 2);
                if constexpr (kCols % 16 != 0)
                    addSums<8>(t + kCols - 8, t + BN + kCols - 8, acc + (kCols - 8) / 2);
            }
            tcFenceBefore();
            __syncwarp();
            if (lane == 0)
                mbarArrive(&accFree[c % L::kAccs + part]);
            if constexpr (kHold)
                if (c + 1 == segmentEnd)
                {
                    ++segment;
                    segmentEnd = segmentBegin(segment + 1);
                    constexpr int kHeldPairs = L::kHeldCols / 2, kRest = kCols / 2 - kHeldPairs;
                    if (segment > 1)
                    {
#pragma unroll
                        for (int g = 0; g < L::kHeldCols / 8; ++g)
                        {
                            uint32_t x[8];
                            tmemLoad8(tHeld + g * 8, x);
                            tmemLoadWait8(x);
#pragma unroll
                            for (int i = 0; i < 4; ++i)
                                acc[g * 4 + i] = add2(pack2(__uint_as_float(x[2 * i]), __uint_as_float(x[2 * i + 1])), acc[g * 4 + i]);
                        }
                        uint64_t x[kRest > 0 ? kRest : 1];
#pragma unroll
                        for (int i = 0; i < kRest; ++i)
                            x[i] = rest[i];
#pragma unroll
                        for (int i = 0; i < kRest; ++i)
                            acc[kHeldPairs + i] = add2(x[i], acc[kHeldPairs + i]);
                    }
                    if (segment < p.segments)
                    {
#pragma unroll
                        for (int g = 0; g < L::kHeldCols / 8; ++g)
                        {
                            uint32_t x[8];
#pragma unroll
                            for (int i = 0; i < 4; ++i)
                            {
                                float lo, hi;
                                unpack2(acc[g * 4 + i], lo, hi);
                                x[2 * i] = __float_as_uint(lo);
                                x[2 * i + 1] = __float_as_uint(hi);
                            }
                            tmemStore8(tHeld + g * 8, x);
                        }
#pragma unroll
                        for (int i = 0; i < kRest; ++i)
                            rest[i] = acc[kHeldPairs + i];
                        tmemStoreWait();
#pragma unroll
                        for (int i = 0; i < kCols / 2; ++i)
                            acc[i] = 0;
                    }
                }
        };
        int stage = 0;
        uint32_t phase = 0;
        for (int c = 0; c < count; ++c)
        {
            uint32_t const s = c & 1;
            bool const cuts = L::kTurns == 1 || static_cast<int>(s) == group;
            // A barrier answers after 120 ... 150 cycles: all are asked at once.
            bool const landed = !cuts || mbarTestAddr(smemAddr(&stFull[stage]), phase);
            if (c >= 2)
            {
                uint32_t const parity = ((c - 2) >> 1) & 1u;
                bool const summed = mbarTestAddr(smemAddr(&done[part * kParts + s]), parity);
                bool const complete = L::kHalves == 1 || part == 1 || mbarTestAddr(smemAddr(&done[kParts + s]), parity);
                promote(c - 2, summed);
                // all its products are complete: so is what they read where this chunk's parts go
                if (L::kHalves == 2 && part == 0 && !__all_sync(0xffffffffu, complete))
                {
                    ok = ok && mbarWaitWarp(&done[kParts + s], parity, abortFlag, kWaitAccFull);
                    tcFenceAfter(); // that of promote() came before this wait
                }
            }
            if (cuts)
            {
                if (!__all_sync(0xffffffffu, landed))
                    ok = ok && mbarWaitWarp(&stFull[stage], phase, abortFlag, kWaitTmaFull);
                uint8_t const* const fp = smem + stage * L::kStageBytes;
                if (hasRows)
                {
                    int const row = quad * 32 + lane;
                    uint32_t lost = 0;
#pragma unroll
                    for (int g = 0; g < L::kTurns; ++g)
                    {
                        int const at = L::kTurns == 1 ? cols : 2 * (w >> 2) + g; // which 16 of the chunk's K
                        float4 const* const src = reinterpret_cast<float4 const*>(fp + (at >> 1) * (L::kABytes / 2) + row * 128);
                        uint32_t const t = tRow + kPartsCol + s * 96 + at * 8;
                        float4 v[4];
#pragma unroll
                        for (int i = 0; i < 4; ++i)
                            v[i] = src[((at & 1) * 4 + i) ^ (row & 7)];
                        uint32_t h[8], m[8], l[8];
#pragma unroll
                        for (int i = 0; i < 4; ++i)
                        {
                            splitPair(v[i].x, v[i].y, h[2 * i], m[2 * i], l[2 * i], lost);
                            splitPair(v[i].z, v[i].w, h[2 * i + 1], m[2 * i + 1], l[2 * i + 1], lost);
                        }
                        tmemStore8(t, h);
                        tmemStore8(t + 32, m);
                        tmemStore8(t + 64, l);
                    }
                    if ((lost & 0xffffu) != 0)
                        flagA[row] = *flagAny = 1;
                }
                // eight numbers of a row of Wt: 16 bytes of each part; an odd number of 32 rows is dealt to the groups by turns
                uint8_t* const planes = smem + L::kPlanesOff + s * 3 * L::kPlaneBytes;
#pragma unroll
                for (int i = 0; i < (BN + 32) / 64; ++i)
                {
                    int const block = L::kTurns == 2 ? 0 : 2 * i + (BN % 64 == 0 ? group : (group + c) & 1);
                    if (BN % 64 != 0 && block >= BN / 32)
                        break;
                    int const row = block * 32 + lane;
                    float4 const* const src = reinterpret_cast<float4 const*>(fp + L::kABytes + (w >> 2) * (L::kWBytes / 2) + row * 128);
                    float4 const v0 = src[(2 * (w & 3)) ^ (row & 7)], v1 = src[(2 * (w & 3) + 1) ^ (row & 7)];
                    uint4 h, m, l;
                    uint32_t lost = 0;
                    splitPair(v0.x, v0.y, h.x, m.x, l.x, lost);
                    splitPair(v0.z, v0.w, h.y, m.y, l.y, lost);
                    splitPair(v1.x, v1.y, h.z, m.z, l.z, lost);
                    splitPair(v1.z, v1.w, h.w, m.w, l.w, lost);
                    uint8_t* const dst = planes + row * 128 + ((w ^ (row & 7)) << 4);
                    *reinterpret_cast<uint4*>(dst) = h;
                    *reinterpret_cast<uint4*>(dst + L::kPlaneBytes) = m;
                    *reinterpret_cast<uint4*>(dst + 2 * L::kPlaneBytes) = l;
                    if ((lost & 0xffffu) != 0)
                        flagW[row] = *flagAny = 1;
                }
                fenceProxyAsync();
                tmemStoreWait();
                tcFenceBefore();
                __syncwarp();
                if (lane == 0)
                {
                    mbarArrive(&ready[s]);
                    mbarArrive(&stFree[stage]);
                }
            }
            if (++stage == L::kStages)
            {
                stage = 0;
                phase ^= 1u;
            }
        }
        for (int c = count < 2 ? 0 : count - 2; c < count; ++c)
            promote(c, false);
    }

    __syncthreads(); // the ring is drained
    bool const aborted = *abortFlag != 0;
    if (aborted)
    {
        uint64_t const t0 = globalTimerNs();
        while (globalTimerNs() - t0 < 1000000ull)
            __nanosleep(1000);
        if (threadIdx.x == 0 && p.statusWord)
            atomicMax(p.statusWord, *abortFlag);
        __syncthreads();
    }
    if (warp == 1)
    {
        tcFenceAfter();
        tmemFree(tmemBase, L::kTmem);
    }
    if (warp >= 2)
    {
        float* const dst = sums + ((warp & 3) * 32 + lane) * L::kPitch + ((warp - 2) >> 2) * kCols;
#pragma unroll
        for (int i = 0; i < kCols / 4; ++i)
        {
            float4 v;
            unpack2(acc[2 * i], v.x, v.y);
            unpack2(acc[2 * i + 1], v.z, v.w);
            *reinterpret_cast<float4*>(dst + 4 * i) = v;
        }
    }
    for (int i = threadIdx.x; i <= kTileM * BN / 32; i += kThreadsF32)
        again[i] = 0; // and the list's length
    bool exact = true; // the same for all threads of the cluster
    if (p.ctas > 1)
    {
        clusterBarrier();
        for (int s = 0; s < p.ctas; ++s)
            exact = exact && ldSharedCluster(flagAny, s) == 0;
    }
    else
    {
        __syncthreads();
        exact = *flagAny == 0;
    }
    if (!exact)
    {
        uint32_t merged = 0; // a row's flag over all of K
        if (threadIdx.x < kTileM + BN)
            for (int s = 0; s < p.ctas; ++s)
                merged |= p.ctas > 1 ? ldSharedCluster(flagA + threadIdx.x, s) : flagA[threadIdx.x];
        if (p.ctas > 1)
            clusterBarrier();
        if (threadIdx.x < kTileM + BN)
            flagA[threadIdx.x] = merged;
        __syncthreads();
        for (int r = warp; r < kTileM + BN; r += kThreadsF32 / 32)
        {
            bool const inside = r < kTileM ? m0 + r < p.M : n0 + r - kTileM < p.N; // after an expired wait any row may be flagged
            if (inside && flagA[r] != 0 && hasNan(r < kTileM ? p.A + (m0 + r) * p.lda : p.Wt + (n0 + r - kTileM) * p.K, p.K))
                flagA[r] = 2;
        }
        __syncthreads();
    }
    // A thread keeps its four columns and goes down the rows, so what depends on the columns is formed once.
    constexpr int kPieces = BN / 4, kRows = kThreadsF32 / kPieces; // rows at a time of a CTA
    bool any = false;
    int const column = static_cast<int>(threadIdx.x % kPieces) * 4;
    int64_t const n = n0 + column;
    if (threadIdx.x < kRows * kPieces && n < p.N && !aborted)
    {
        int const inside = p.N - n < 4 ? static_cast<int>(p.N - n) : 4;
        int const rows = p.M - m0 < kTileM ? static_cast<int>(p.M - m0) : kTileM;
        bool const whole = p.wide && inside == 4;
        float bias[4] = {0.f, 0.f, 0.f, 0.f};
        if (p.bias)
        {
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (j < inside)
                    bias[j] = __ldg(p.bias + n + j);
        }
        int r = rank * kRows + static_cast<int>(threadIdx.x) / kPieces;
        float* dst = p.C + (m0 + r) * p.ldc + n;
        int64_t const step = static_cast<int64_t>(p.ctas) * kRows * p.ldc;
        for (; r < rows; r += p.ctas * kRows, dst += step)
        {
            float const* const at = sums + r * L::kPitch + column;
            float4 v;
            if (p.ctas > 1)
            {
                float4 x[kMaxSegments];
#pragma unroll
                for (int s = 0; s < kMaxSegments; ++s) // all on their way before the first is added
                    if (s < p.ctas)
                        x[s] = ldSharedCluster4(at, s);
                v = x[0];
#pragma unroll
                for (int s = 1; s < kMaxSegments; ++s)
                    if (s < p.ctas)
                        v = make_float4(v.x + x[s].x, v.y + x[s].y, v.z + x[s].z, v.w + x[s].w);
            }
            else
                v = *reinterpret_cast<float4 const*>(at);
            float o[4] = {v.x, v.y, v.z, v.w};
            uint32_t bits = 0;
#pragma unroll
            for (int j = 0; j < 4; ++j)
                bits |= sumIsInexact(o[j]) ? 1u << j : 0u;
            if (!exact)
                for (int j = 0; j < 4; ++j)
                {
                    uint32_t const flags = flagA[r] | flagW[column + j];
                    bits = (bits | (flags & 1u) << j) & ~((flags >> 1) << j);
                }
            if (inside < 4)
                bits &= (1u << inside) - 1u;
            if (bits != 0)
            {
                atomicOr(again + r * (BN / 32) + column / 32, bits << (column % 32));
                any = true;
            }
#pragma unroll
            for (int j = 0; j < 4; ++j)
                o[j] = finishF32(p, o[j], bias[j]);
            if (whole)
                *reinterpret_cast<float4*>(dst) = make_float4(o[0], o[1], o[2], o[3]);
            else
                for (int j = 0; j < inside; ++j)
                    dst[j] = o[j];
        }
    }
    if (__syncthreads_or(any))
        computeAgain<BN>(p, again, list, m0, n0);
    if (p.ctas > 1)
        clusterBarrier(); // nobody leaves while its sums are being read
}

template <int BN, bool kHold>
int32_t launchF32Tc(bert_b200_fc_params const& p, int segments, int ctas, cudaStream_t stream)
{
    CUtensorMap mapA, mapW;
    uint64_t const dimsA[2] = {static_cast<uint64_t>(p.k), static_cast<uint64_t>(p.m)}, stridesA[1] = {static_cast<uint64_t>(p.lda) * 4};
    uint64_t const dimsW[2] = {static_cast<uint64_t>(p.k), static_cast<uint64_t>(p.n)}, stridesW[1] = {static_cast<uint64_t>(p.k) * 4};
    uint32_t const boxA[2] = {32, kTileM}, boxW[2] = {32, BN};
    int32_t st = makeTensorMap(&mapA, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, p.a, dimsA, stridesA, boxA, CU_TENSOR_MAP_SWIZZLE_128B);
    if (st == BERT_B200_OK)
        st = makeTensorMap(&mapW, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, p.wt, dimsW, stridesW, boxW, CU_TENSOR_MAP_SWIZZLE_128B);
    if (st != BERT_B200_OK)
        return st;
    int64_t const mTiles = (p.m + kTileM - 1) / kTileM, nTiles = (p.n + BN - 1) / BN;
    FcF32TcArgs const args{p.m, p.n, p.k, p.lda, p.ldc, static_cast<float const*>(p.a), static_cast<float const*>(p.wt), static_cast<float*>(p.c),
        p.bias, p.activation, p.alpha, static_cast<int32_t>(nTiles), segments, ctas, p.ldc % 4 == 0 && aligned16(p.c) ? 1 : 0, p.status_word};
    static SmemOptIn optIn;
    cudaError_t const e = launchDependentCluster(&optIn, fcF32TcKernel<BN, kHold>, dim3(static_cast<unsigned>(mTiles * nTiles * ctas)),
        dim3(kThreadsF32), FcF32Smem<BN>::kDynamic, stream, ctas, mapA, mapW, args);
    if (e != cudaSuccess)
        B200_FAIL(BERT_B200_CUDA_ERROR, "fcF32TcKernel: %s", cudaGetErrorString(e));
    return checkLaunch("fcF32TcKernel");
}

} // namespace

// From K = 384 on. Error against 64 bits (2-norm) here / of the FP32 multiply-adds of fcF32Simt, in 1e-7:
//   K                        384          768          1024         3072         4096
//   normal                   0.83 / 1.34  0.89 / 1.40  0.91 / 1.58  1.03 / 2.56  1.07 / 2.93
//   rectified x normal       0.81 / 1.05  0.85 / 1.10  0.88 / 1.21  1.00 / 1.88  1.03 / 2.10
//   uniform, 0 ... 1         0.40 / 0.56  0.44 / 0.55  0.45 / 0.56  0.50 / 0.71  0.50 / 0.73
//   normal, 1 +- 0.2         0.43 / 0.55  0.48 / 0.55  0.49 / 0.55  0.54 / 0.71  0.54 / 0.72
// (mean error on the third and fourth -0.06 and +0.22; parts by truncation and 64 products in one accumulator: 1.2 and 1.0, the mean -1.1 and
// -0.9). The multiply-adds are closer where both operands have one sign and spread over orders of magnitude, since small products are cut off beside a
// large sum: softmax of 3 N(0, 1) x uniform 1.8e-7 ... 2.1e-7 / 0.8e-7 ... 1.1e-7 (before 3.0e-7 ... 3.3e-7), exp(2 N(0, 1)) on both sides 3.1e-7 ... 3.8e-7 /
// 1.0e-7 ... 1.8e-7 (before 4.1e-7 ... 5.4e-7); with normal weights they are not. A shorter K has not been measured in this form and stays with
// the multiply-adds. They also take what the TMA unit does not: rows that are no multiple of 16 bytes apart, sizes beyond its coordinates. GPU time,
// same order: 1 x 64 x 384 6.1 / 8.5 us, 1 x 768 x 768 8.2 / 8.6 us, 37 x 768 x 768 8.4 / 8.9 us, 37 x 2304 x 768 10.7 / 14.9 us, 300 x 768 x 512 9.4 /
// 18.5 us, 128 x 768 x 3072 13.5 / 44.9 us, 1024 x 2304 x 768 28.3 / 96.9 us, 4096 x 1024 x 4096 226 ... 249 / 843 us. The two tensor maps cost a call 1 us
// of the host: 10.1 instead of 9.5 us where the host is what bounds it.
int32_t fcF32(bert_b200_fc_params const& p, cudaStream_t stream)
{
    constexpr int64_t kMax = 1ll << 31;
    bool const tma = p.k % 4 == 0 && p.lda % 4 == 0 && aligned16(p.a) && aligned16(p.wt) && p.m < kMax && p.n < kMax && p.k < kMax && p.lda < (1ll << 37);
    int64_t const mTiles = (p.m + kTileM - 1) / kTileM;
    if (!tma || p.k < 384 || mTiles * ((p.n + 31) / 32) * kMaxSegments >= kMax)
        return fcF32Simt(p, stream);
    // Segments: few rows are spread over more SMs by them, and each costs a CTA that takes them in turn another pass over its sums.
    int64_t const kChunks = (p.k + kChunk - 1) / kChunk;
    int const segments = kChunks >= 24 ? 8 : kChunks >= 12 ? 4 : 2;
    // Width of the tiles, and whether a CTA takes all segments: what the measured cycles per chunk and per CTA, times the waves of CTAs,
    // make shortest: cycles of the kernel before its columns were multiplied in halves, which is now 10 % faster with 128 and 6 % with 64 columns. Over 190
    // shapes (M 1 ... 4096, N and K of encoders) the choice is still 0.3 % behind the best of the eight forms in the mean, more than 2 % behind in 13 of
    // them and 14 % at most (640 x 768 x 3072 42.5 us, 128 columns and a segment per CTA 37.4 us; 1300 x 4096 x 1024 106 us, 128 columns 99.5 us). Clusters find
    // fewer places than there are SMs. Measured with 128 / 96 / 64 / 32 columns, all segments in one CTA: 1024 x 2304 x 768 29.1 / 46.0 / 36.7 / 58.2 us, 1024 x
    // 3072 x 768 54.5 / 46.8 / 53.4 / 85.6 us, 1024 x 768 x 768 27.3 / 23.2 / 18.4 / 28.9 us; one segment per CTA, 128 / 64 columns: 1024 x 768 x 3072 72.0 /
    // 93.2 us (64 columns in one CTA 55.5 us), 128 x 768 x 3072 17.8 / 13.8 us (52.9 us).
    static constexpr int kCycles[4] = {1480, 1990, 2700, 3220}; // per chunk, of 32, 64, 96 and 128 columns
    static constexpr int kFixed[2][4] = {{12500, 13000, 16500, 26000}, {12500, 14500, 16300, 17500}}; // per CTA with all segments, with one
    int bestN = 128, bestCtas = 1;
    int64_t best = 0;
    for (int bn = 128; bn >= 32; bn -= 32)
        for (int ctas = 1; ctas <= segments; ctas += segments - 1)
        {
            int64_t const slots = smCount() * (ctas == 1 ? 148 : ctas == 2 ? 140 : ctas == 4 ? 128 : 112) / 148;
            int64_t const waves = (mTiles * ((p.n + bn - 1) / bn) * ctas + slots - 1) / slots;
            int const fixed = kFixed[ctas > 1][bn / 32 - 1] - (bn == 128 && segments == 2 && ctas == 1 ? 6000 : 0); // little to hold
            int64_t const cost = waves * ((kChunks + ctas - 1) / ctas * kCycles[bn / 32 - 1] + fixed);
            if (best == 0 || cost < best)
            {
                best = cost;
                bestN = bn;
                bestCtas = ctas;
            }
        }
    using Launch = int32_t (*)(bert_b200_fc_params const&, int, int, cudaStream_t);
    static constexpr Launch kLaunch[2][4] = {{launchF32Tc<32, false>, launchF32Tc<64, false>, launchF32Tc<96, false>, launchF32Tc<128, false>},
        {launchF32Tc<32, true>, launchF32Tc<64, true>, launchF32Tc<96, true>, launchF32Tc<128, true>}};
    return kLaunch[segments > bestCtas][bestN / 32 - 1](p, segments, bestCtas, stream);
}

} // namespace b200
