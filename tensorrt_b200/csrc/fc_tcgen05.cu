// Fully connected layer on the sm_100a tensor cores: C = epilogue(A * Wt^T).
//
// Replaces the cublasLtMatmul call of the reference FC plugin (plugin/fcPlugin/fcPlugin.cpp:551-610)
// and the separate bias / GELU / quantise layers that follow it in the reference graph.
//
// Two kernels share the epilogue arithmetic:
//   fcTcgen05PairKernel - persistent, a cluster of two CTAs per 256 x BLOCK_N tile (tcgen05.mma.cta_group::2), for problems with
//                         enough tiles to keep the SM pairs busy;
//   fcTcgen05TileKernel - one tile of 128 (64) x BLOCK_N (16 ... 128) per CTA, two CTAs per SM, for few rows: the narrow tiles spread
//                         the weights over all SMs.
// Warp roles in both: TMA producer (A and Wt tiles of 128-byte rows, 128-byte swizzle, into a shared-memory ring guarded by
// full / empty mbarriers), MMA issuer (accumulators in TMEM; tcgen05.commit releases ring stages and publishes accumulators),
// epilogue warps (tcgen05.ld, scale / bias / erf-GELU / quantise, stores).
// A row of C is the same bits whatever M and whichever kernel: every accumulator takes its K range in order.
// Every mbarrier wait is bounded (see sm100.cuh); on expiry the CTA drains, frees TMEM and exits,
// and the status word tells the host.
#include "sm100.cuh"

#include <mutex>

namespace b200
{

int32_t fcF32(bert_b200_fc_params const& p, cudaStream_t stream);

namespace
{

constexpr int kBlockM = 128;
constexpr int kRowBytes = 128; // one swizzle span = BLOCK_K * sizeof(In)
constexpr int kTmemCols = 512;
constexpr int kEpilogueWarps = 16; // pair kernel
constexpr int kFcThreads = 64 + kEpilogueWarps * 32;

struct FcArgs
{
    int64_t M, N, K;
    void* C;
    int64_t ldc;
    float const* bias;
    int32_t act;
    float alpha;
    float outScale;
    uint32_t* statusWord;
    float qLo, qHi; // clamp bounds -128 / outScale and 127 / outScale for quantised results
    // tile kernel only
    int32_t stages;       // ring stages
    int32_t aRows;        // rows of an A box: 128, or fewer when M is smaller
    int32_t weightsReady; // Wt was complete before the kernel ahead in the stream began
};

// erf-GELU through a fitted tanh form: gelu(x) = x/2 * (1 + tanh(x * (c1 + c3 x^2 + c5 x^4))), x^2 clamped at 64.
// The three coefficients are a minimax fit against 0.5 x (1 + erf(x / sqrt 2)) on [-9, 9]: |error| <= 2.6e-5
// (the classic 0.044715 cubic form is off by 4.7e-4). On top comes the error of the hardware tanh.approx
// (about 2^-11 relative), i.e. at most ~2.5e-4 |x| absolute - below FP16 resolution of the result and about
// 1 % of an INT8 step. Cost: 5 FMA-pipe operations and one MUFU operation per value.
constexpr float kGeluC1 = 7.97507884e-01f;
constexpr float kGeluC3 = 3.70056460e-02f;
constexpr float kGeluC5 = -3.51516788e-04f;

__device__ __forceinline__ float geluInner(float x)
{
    float const x2 = fminf(x * x, 64.f);
    return x * fmaf(fmaf(kGeluC5, x2, kGeluC3), x2, kGeluC1);
}

__device__ __forceinline__ float tanhApprox(float x)
{
    float y;
    asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// scale * gelu(x); `halfScale` = scale / 2
__device__ __forceinline__ float geluErf(float x, float halfScale)
{
    float const h = x * halfScale;
    return fmaf(h, tanhApprox(geluInner(x)), h);
}

// Two values at once for results that are quantised to INT8 right away: the whole tanh argument is formed in packed
// FP16 with the classic cubic x * (0.79788456 + 0.035677408 x^2) (|error| of that GELU form <= 4.7e-4, FP16 argument
// and tanh.approx.f16x2 add about 3e-4 |x|), together a few hundredths of an INT8 step at most; the product with x
// stays in FP32. 5.5 instructions per value instead of 9, and one MUFU operation per pair.
__device__ __forceinline__ void geluErfPair(float& a, float& b, float halfScale)
{
    uint32_t x, t;
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(x) : "f"(b), "f"(a));
    __half2 const xh = *reinterpret_cast<__half2 const*>(&x);
    __half2 const poly = __hfma2(__hmul2(xh, xh), __float2half2_rn(0.035677408f), __float2half2_rn(0.79788456f));
    __half2 const u = __hmul2(xh, poly);
    asm("tanh.approx.f16x2 %0, %1;" : "=r"(t) : "r"(*reinterpret_cast<uint32_t const*>(&u)));
    float2 const tf = __half22float2(*reinterpret_cast<__half2 const*>(&t));
    float const ha = a * halfScale, hb = b * halfScale;
    a = fmaf(ha, tf.x, ha);
    b = fmaf(hb, tf.y, hb);
}

// What is left to do to a value when it is quantised: multiply by s, with the clamp done before at [lo, hi].
struct QuantStep
{
    float s, lo, hi;
    bool useConvert; // round with cvt.rni.sat (conversion unit) instead of clamp + FMA
    bool unitScale;  // s == 1: the values are already scaled
};

// Without GELU the conversion unit is idle and issue slots are scarce: multiply + saturating convert. With GELU the unit is
// busy with tanh: clamp + rounding FMA on the FMA pipe instead. Same results.
__device__ __forceinline__ uint32_t quantChar4(float a, float b, float c, float d, QuantStep const& q)
{
    return q.useConvert ? (q.unitScale ? packChar4Cvt(a, b, c, d) : packChar4Cvt(a, b, c, d, q.s)) : packChar4Scaled(a, b, c, d, q.s, q.lo, q.hi);
}

// W values of one row to shared memory, in 16-byte pieces.
template <int W>
__device__ __forceinline__ void storeChunk(__half* dst, float const (&v)[W], QuantStep const&)
{
#pragma unroll
    for (int g = 0; g < W / 8; ++g)
    {
        float f[8];
#pragma unroll
        for (int j = 0; j < 8; ++j)
            f[j] = v[g * 8 + j];
        *reinterpret_cast<uint4*>(dst + g * 8) = packHalf8(f);
    }
}

template <int W>
__device__ __forceinline__ void storeChunk(int8_t* dst, float const (&v)[W], QuantStep const& q)
{
#pragma unroll
    for (int g = 0; g < W / 16; ++g)
    {
        uint32_t w[4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
            w[j] = quantChar4(v[g * 16 + 4 * j], v[g * 16 + 4 * j + 1], v[g * 16 + 4 * j + 2], v[g * 16 + 4 * j + 3], q);
        *reinterpret_cast<uint4*>(dst + g * 16) = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

// alpha / bias / activation for W accumulator columns of one row. Returns what the quantising store still has to do:
// after GELU the values are already multiplied by out_scale (it rides on the 1/2 of the GELU), otherwise the scale is
// left to the store, which folds it into its rounding FMA.
// `bias`: that of the first column (global or shared memory), null for none.
template <bool kInt8, typename Out, int W>
__device__ __forceinline__ QuantStep fcEpilogueMath(uint32_t const (&r)[W], float (&v)[W], FcArgs const& args, float const* bias, int validCols)
{
    constexpr bool kQuant = sizeof(Out) == 1;
    bool const foldScale = kQuant && bias == nullptr && args.act != BERT_B200_ACT_GELU_ERF;
    if (bias)
    {
#pragma unroll
        for (int j = 0; j < W; j += 4)
        {
            float4 b = make_float4(0.f, 0.f, 0.f, 0.f);
            if (j < validCols)
                b = *reinterpret_cast<float4 const*>(bias + j);
            float const bb[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
            for (int i = 0; i < 4; ++i)
            {
                float const a = kInt8 ? static_cast<float>(static_cast<int32_t>(r[j + i])) : __uint_as_float(r[j + i]);
                v[j + i] = fmaf(a, args.alpha, bb[i]);
            }
        }
    }
    else
    {
        // nothing between the accumulator and the quantisation: one multiply by alpha * out_scale
        float const a1 = foldScale ? args.alpha * args.outScale : args.alpha;
#pragma unroll
        for (int j = 0; j < W; ++j)
        {
            float const a = kInt8 ? static_cast<float>(static_cast<int32_t>(r[j])) : __uint_as_float(r[j]);
            v[j] = a * a1;
        }
    }
    if (args.act == BERT_B200_ACT_GELU_ERF)
    {
        if (kQuant)
        {
            float const halfScale = 0.5f * args.outScale;
#pragma unroll
            for (int j = 0; j < W; j += 2)
                geluErfPair(v[j], v[j + 1], halfScale);
        }
        else
        {
#pragma unroll
            for (int j = 0; j < W; ++j)
                v[j] = geluErf(v[j], 0.5f);
        }
        return QuantStep{1.f, -128.f, 127.f, false, true};
    }
    if (foldScale)
        return QuantStep{1.f, -128.f, 127.f, true, true};
    return QuantStep{args.outScale, args.qLo, args.qHi, true, false};
}

// ... then, in the tile kernel, storeChunk into a block of the drained ring, from which whole rows are stored;
// ... in the pair kernel into a [32 rows x 32 columns] staging tile in shared memory, laid out the way a TMA store with the 32-byte
// (INT8) or 64-byte (FP16) swizzle expects it: row `lane`, 16-byte piece c at (c ^ f(lane)) - which also spreads the
// 32 lanes' 128-bit stores over all banks.
template <typename Out>
__device__ __forceinline__ void stageChunk32(uint8_t* tile, int lane, float const (&v)[32], QuantStep const& q);

template <>
__device__ __forceinline__ void stageChunk32<__half>(uint8_t* tile, int lane, float const (&v)[32], QuantStep const&)
{
    uint8_t* const rowPtr = tile + lane * 64;
    int const x = (lane >> 1) & 3;
#pragma unroll
    for (int g = 0; g < 4; ++g)
    {
        float f[8];
#pragma unroll
        for (int j = 0; j < 8; ++j)
            f[j] = v[g * 8 + j];
        *reinterpret_cast<uint4*>(rowPtr + ((g ^ x) << 4)) = packHalf8(f);
    }
}

template <>
__device__ __forceinline__ void stageChunk32<int8_t>(uint8_t* tile, int lane, float const (&v)[32], QuantStep const& q)
{
    uint8_t* const rowPtr = tile + lane * 32;
    int const x = (lane >> 2) & 1;
#pragma unroll
    for (int g = 0; g < 2; ++g)
    {
        uint4 o;
        uint32_t* w = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
        for (int j = 0; j < 4; ++j)
        {
            w[j] = quantChar4(v[g * 16 + 4 * j], v[g * 16 + 4 * j + 1], v[g * 16 + 4 * j + 2], v[g * 16 + 4 * j + 3], q);
        }
        *reinterpret_cast<uint4*>(rowPtr + ((g ^ x) << 4)) = o;
    }
}

FcArgs makeFcArgs(bert_b200_fc_params const& p, int stages, int aRows, bool weightsReady)
{
    return FcArgs{p.m, p.n, p.k, p.c, p.ldc, p.bias, p.activation, p.alpha, p.out_scale, p.status_word,
        p.out_scale > 0.f ? -128.f / p.out_scale : 0.f, p.out_scale > 0.f ? 127.f / p.out_scale : 0.f, stages, aRows,
        weightsReady ? 1 : 0};
}

// ------------------------------------------------------------------------------------------------
// One BLOCK_M x BLOCK_N tile per CTA.
//
// With few rows a layer is bound by latency and by how fast the weights reach the SMs: one SM takes in about 100 bytes per
// clock, so the weights of a projection have to be spread over as many SMs as possible - narrow tiles. Their MMAs take 40 cycles
// each for any BLOCK_N up to 32, about as long as 128 rows of A (32 bytes each) take to come from shared memory, and a long K is
// a chain of them: up to 64 rows the tile has 64 rows. Everything around the main loop is kept short: a single tile per CTA and only
// BLOCK_N TMEM columns. Shared memory: about 100 KB where two CTAs share an SM, up to 200 KB where the tiles do not outnumber the SMs
// (37 rows: 86 KB at K = 768, 173 KB at K = 3072). Where the CTAs of the next launch fit beside the running ones, they have their
// barriers, TMEM and - where the caller says that the weights are not being written by the kernels ahead - their first
// weight tiles in place when this one ends. The other weight tiles are at least pulled into the L2 while the kernel ahead runs.
//   warp 0: TMA producer, warp 1: TMEM allocation and MMA issue, then 4 epilogue warps (8 from BLOCK_N = 64 on), one or two
//   per TMEM lane quadrant. Results go through the drained ring, so that a store instruction of a warp writes whole rows of
//   its 32 x 32 block instead of 16 bytes of each of 32 rows.
// Measured (weights from DRAM, back-to-back launches): FP16 37 x 768 x 768 in 3.0 us, 37 x 768 x 3072 in 6.3 us (3.5 us and 7.8 us
// with 128-row tiles; 18.5 us with 128 x 128 tiles and 18 warps per CTA), INT8 64 x 1024 x 4096 in 5.2 us (6.1 us), FP16 1024 x 768
// x 768 in 4.8 us (pair kernel 6.7 us).
// ------------------------------------------------------------------------------------------------
template <int BLOCK_M, int BLOCK_N>
struct FcTileSmem
{
    static constexpr int kEpiWarps = BLOCK_N >= 64 ? 8 : 4;
    static constexpr int kThreads = 64 + kEpiWarps * 32;
    // A ring stage holds kSub k-blocks: waiting for a stage, electing a lane and committing cost the issuing warp about 110
    // cycles on top of some 40 per MMA, more than four narrow MMAs take.
    static constexpr int kSub = BLOCK_N <= 32 ? 4 : BLOCK_N == 64 ? 2 : 1;
    static constexpr int kBBytes = kSub * BLOCK_N * kRowBytes;
    static constexpr int kMaxStages = 8;
    // [bias][full, empty, accFull][tmem base, abort flag][ring]
    static constexpr int kBarrierOff = BLOCK_N * 4;
    static constexpr int kRingOff = (kBarrierOff + (2 * kMaxStages + 1) * 8 + 16 + 1023) / 1024 * 1024;
    // The MMA always reads BLOCK_M rows of A: past the last A tile lie as many bytes as a full tile has more (what is read
    // there only reaches accumulator rows beyond M).
    static constexpr int bytes(int stages, int aRows)
    {
        return kRingOff + stages * (kBBytes + kSub * aRows * kRowBytes) + (BLOCK_M - aRows) * kRowBytes + 1024; // 1024: alignment
    }
    // As many stages as `budget` bytes hold or a tile has, at least 2 (which also hold the results of the epilogue warps).
    static int stagesFor(int aRows, int kSteps, int budget)
    {
        int const fit = (budget - bytes(0, aRows)) / (kBBytes + kSub * aRows * kRowBytes);
        int const most = kSteps < kMaxStages ? kSteps : kMaxStages;
        int const n = fit < most ? fit : most;
        return n < 2 ? 2 : n;
    }
};

template <typename In, int BLOCK_M, int BLOCK_N, typename Out>
__global__ void __launch_bounds__(FcTileSmem<BLOCK_M, BLOCK_N>::kThreads, 2)
    fcTcgen05TileKernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB, FcArgs const args)
{
    using L = FcTileSmem<BLOCK_M, BLOCK_N>;
    // The accumulator of a 64-row MMA takes 16 lanes of each TMEM quadrant.
    constexpr int kQuadRows = BLOCK_M / 4;
    constexpr bool kInt8 = sizeof(In) == 1;
    constexpr int kBlockK = kRowBytes / sizeof(In);
    constexpr int kUmmaKBytes = 32; // UMMA K = 16 halves or 32 bytes
    constexpr int kChunk = BLOCK_N < 32 ? BLOCK_N : 32;
    constexpr int kTmem = BLOCK_N < 32 ? 32 : BLOCK_N;
    constexpr uint32_t kIdesc
        = makeInstrDesc(kInt8 ? 2u : 1u, kInt8 ? 1u : 0u, 0u, 0u, static_cast<uint32_t>(BLOCK_M), static_cast<uint32_t>(BLOCK_N));

    extern __shared__ uint8_t smemRaw[];
    uint8_t* const smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smemRaw) + 1023) & ~static_cast<uintptr_t>(1023));
    float* const sBias = reinterpret_cast<float*>(smem);
    uint64_t* const full = reinterpret_cast<uint64_t*>(smem + L::kBarrierOff);
    uint64_t* const empty = full + L::kMaxStages;
    uint64_t* const accFull = empty + L::kMaxStages;
    uint32_t* const tmemSlot = reinterpret_cast<uint32_t*>(accFull + 1);
    volatile uint32_t* const abortFlag = tmemSlot + 1;
    uint8_t* const ring = smem + L::kRingOff; // Wt tiles of all stages, then the A tiles

    int const warp = threadIdx.x >> 5;
    int const lane = threadIdx.x & 31;
    int const stages = args.stages;
    int const tile = static_cast<int>(blockIdx.x);
    int const nBlocks = static_cast<int>((args.N + BLOCK_N - 1) / BLOCK_N);
    int32_t const m0 = tile / nBlocks * BLOCK_M;
    int32_t const n0 = tile % nBlocks * BLOCK_N;
    constexpr int kSub = L::kSub;
    constexpr int kStepK = kSub * kBlockK; // a step's k-blocks beyond K arrive as zeros
    int const count = static_cast<int>((args.K + kStepK - 1) / kStepK);
    uint32_t const fullAddr0 = smemAddr(full), emptyAddr0 = smemAddr(empty);
    uint32_t const aBytes = static_cast<uint32_t>(args.aRows * kRowBytes); // one k-block of A
    uint32_t const bAddr0 = smemAddr(ring), aAddr0 = bAddr0 + static_cast<uint32_t>(stages * L::kBBytes);
    uint32_t const stageBytes = kSub * aBytes + L::kBBytes;
    constexpr uint32_t kSubB = BLOCK_N * kRowBytes; // one k-block of Wt
    auto loadB = [&](uint32_t dst, uint32_t bar, int step) {
#pragma unroll
        for (int j = 0; j < kSub; ++j)
            tmaLoad2dAddr(dst + j * kSubB, &mapB, bar, step * kStepK + j * kBlockK, n0);
    };
    auto loadA = [&](uint32_t dst, uint32_t bar, int step) {
#pragma unroll
        for (int j = 0; j < kSub; ++j)
            tmaLoad2dAddr(dst + j * aBytes, &mapA, bar, step * kStepK + j * kBlockK, m0);
    };

    if (threadIdx.x == 0)
    {
        for (int i = 0; i < stages; ++i)
        {
            mbarInit(&full[i], 1);
            mbarInit(&empty[i], 1);
        }
        mbarInit(accFull, 1);
        *abortFlag = 0;
        fenceBarrierInit();
    }
    int const early = count < stages ? count : stages; // steps that fit the ring at once
    if (warp == 0)
    {
        __syncwarp();
        if (electOne())
        {
            prefetchTensorMap(&mapA);
            int i = 0;
            if (args.weightsReady)
                for (; i < early; ++i)
                {
                    mbarArriveExpectTxAddr(fullAddr0 + 8 * i, stageBytes);
                    loadB(bAddr0 + i * L::kBBytes, fullAddr0 + 8 * i, i);
                }
            if (m0 == 0) // the tiles of later row blocks find the weights in the L2
                for (; i < count; ++i)
#pragma unroll
                    for (int j = 0; j < kSub; ++j)
                        tmaPrefetch2d(&mapB, i * kStepK + j * kBlockK, n0);
        }
        __syncwarp();
    }
    if (warp == 1)
        tmemAlloc(tmemSlot, kTmem);
    tcFenceBefore();
    __syncthreads();
    tcFenceAfter();
    uint32_t const tmemBase = *tmemSlot;
    gridDependencyLaunch();
    // the bias, too, is usually in DRAM (a prefetch yields no value: whoever may still be writing it does not matter); 8 sequences
    // of 32 ... 384 tokens through the large INT8 encoder: 1723 -> 1703 us
    if (args.bias && m0 == 0 && threadIdx.x * 32 < BLOCK_N && n0 + static_cast<int>(threadIdx.x) * 32 < args.N)
        prefetchL2(args.bias + n0 + threadIdx.x * 32);
    gridDependencyWait();

    // Producer and MMA warp walk their loops as whole warps: every lane waits (no vote: a failed wait only stops the lane's
    // issuing, the loops end by their counts), the elected one issues. The wait stays outside the elected branch: behind a
    // polling loop the compiler no longer knows that a single lane is active.
    if (warp == 0)
    {
        bool ok = true;
        for (int i = 0; i < early; ++i)
        {
            if (electOne())
            {
                if (!args.weightsReady)
                {
                    mbarArriveExpectTxAddr(fullAddr0 + 8 * i, stageBytes);
                    loadB(bAddr0 + i * L::kBBytes, fullAddr0 + 8 * i, i);
                }
                loadA(aAddr0 + i * kSub * aBytes, fullAddr0 + 8 * i, i);
            }
            __syncwarp();
        }
        // the steps beyond, then every stage once more until its last reader is done: no commit is on its way when the CTA ends
        int stage = 0;
        uint32_t phase = 0;
        for (int i = 0; i < count; ++i)
        {
            ok = ok && mbarWaitAddr(emptyAddr0 + 8 * stage, phase, abortFlag, kWaitStageFree);
            int const step = i + stages;
            if (electOne() && ok && step < count)
            {
                mbarArriveExpectTxAddr(fullAddr0 + 8 * stage, stageBytes);
                loadB(bAddr0 + stage * L::kBBytes, fullAddr0 + 8 * stage, step);
                loadA(aAddr0 + stage * kSub * aBytes, fullAddr0 + 8 * stage, step);
            }
            __syncwarp();
            if (++stage == stages)
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
        uint32_t const aLo0 = static_cast<uint32_t>(descZero) + (aAddr0 >> 4);
        uint32_t const bLo0 = static_cast<uint32_t>(descZero) + (bAddr0 >> 4);
        constexpr uint32_t kMmas = kRowBytes / kUmmaKBytes;
        int stage = 0;
        uint32_t phase = 0;
        uint32_t off8 = 0, aLo = aLo0, bLo = bLo0;
        bool ok = true;
        for (int i = 0; i < count; ++i)
        {
            ok = ok && mbarWaitAddr(fullAddr0 + off8, phase, abortFlag, kWaitTmaFull);
            tcFenceAfter();
            if (electOne() && ok)
            {
#pragma unroll
                for (int j = 0; j < kSub; ++j)
#pragma unroll
                    for (uint32_t k = 0; k < kMmas; ++k)
                        mmaLoHi<kInt8>(tmemBase, aLo + j * (aBytes >> 4) + k * (kUmmaKBytes >> 4), descHi,
                            bLo + j * (kSubB >> 4) + k * (kUmmaKBytes >> 4), descHi, kIdesc, j != 0 || k != 0 || i != 0);
                tcCommitAddr(emptyAddr0 + off8);
            }
            __syncwarp();
            off8 += 8;
            aLo += (kSub * aBytes) >> 4;
            bLo += L::kBBytes >> 4;
            if (++stage == stages)
            {
                stage = 0;
                phase ^= 1u;
                off8 = 0;
                aLo = aLo0;
                bLo = bLo0;
            }
        }
        if (electOne() && ok)
            tcCommit(accFull);
        __syncwarp();
    }
    else
    {
        int const quad = warp & 3;
        int const part = (warp - 2) >> 2;
        int const et = static_cast<int>(threadIdx.x) - 64;
        if (args.bias && et < BLOCK_N) // read back by the other epilogue warps
            sBias[et] = n0 + et < args.N ? __ldg(args.bias + n0 + et) : 0.f;
        asm volatile("bar.sync 1, %0;" ::"n"(L::kEpiWarps * 32) : "memory");
        bool const ok = mbarWaitWarp(accFull, 0, abortFlag, kWaitAccFull);
        tcFenceAfter();
        int64_t const rowBase = static_cast<int64_t>(m0) + quad * kQuadRows;
        uint32_t const taddr = tmemBase + (static_cast<uint32_t>(quad * 32) << 16);
        Out* const C = static_cast<Out*>(args.C);
        if (ok && rowBase < args.M) // warp-uniform
        {
#pragma unroll
            for (int c = part; c < BLOCK_N / kChunk; c += L::kEpiWarps / 4)
            {
                uint32_t r[kChunk];
                if constexpr (kChunk == 16)
                {
                    tmemLoad16(taddr, r);
                    tmemLoadWait16(r);
                }
                else
                {
                    tmemLoad32(taddr + c * kChunk, r);
                    tmemLoadWait32(r);
                }
                int64_t const col = static_cast<int64_t>(n0) + c * kChunk;
                int const validCols = static_cast<int>(args.N - col < kChunk ? args.N - col : kChunk);
                if (validCols > 0) // warp-uniform
                {
                    float v[kChunk];
                    QuantStep const q = fcEpilogueMath<kInt8, Out, kChunk>(r, v, args, args.bias ? sBias + c * kChunk : nullptr, kChunk);
                    // rows of the block, padded by 16 bytes against bank conflicts; every piece is 16 bytes
                    constexpr int kRow = kChunk * static_cast<int>(sizeof(Out));
                    constexpr int kPieces = kRow / 16;
                    uint8_t* const block = ring + (warp - 2) * 32 * (kRow + 16);
                    if (kQuadRows == 32 || lane < kQuadRows)
                        storeChunk<kChunk>(reinterpret_cast<Out*>(block + lane * (kRow + 16)), v, q);
                    __syncwarp();
#pragma unroll
                    for (int i = 0; i < kPieces; ++i)
                    {
                        int const rr = i * (32 / kPieces) + lane / kPieces;
                        int const piece = lane % kPieces;
                        if ((kQuadRows == 32 || rr < kQuadRows) && rowBase + rr < args.M && piece * (16 / static_cast<int>(sizeof(Out))) < validCols)
                            *reinterpret_cast<uint4*>(reinterpret_cast<uint8_t*>(C + (rowBase + rr) * args.ldc + col) + piece * 16)
                                = *reinterpret_cast<uint4 const*>(block + rr * (kRow + 16) + piece * 16);
                    }
                    __syncwarp();
                }
            }
        }
        tcFenceBefore();
    }
    __syncthreads();
    uint32_t const aborted = *abortFlag;
    if (aborted != 0)
    {
        // Give copies / MMAs still in flight a bounded time to land before shared memory and TMEM go away.
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
        tmemFree(tmemBase, kTmem);
    }
}

template <typename In, int BLOCK_M, int BLOCK_N, typename Out>
int32_t launchFcTile(bert_b200_fc_params const& p, bool weightsReady, cudaStream_t stream)
{
    using L = FcTileSmem<BLOCK_M, BLOCK_N>;
    constexpr int kBlockK = kRowBytes / sizeof(In);
    CUtensorMapDataType const dt = sizeof(In) == 1 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
    int32_t const aRows = p.m < BLOCK_M ? static_cast<int32_t>((p.m + 7) / 8 * 8) : BLOCK_M; // no point in zero-filling the rest
    CUtensorMap mapA, mapB;
    {
        uint64_t const dims[2] = {static_cast<uint64_t>(p.k), static_cast<uint64_t>(p.m)};
        uint64_t const strides[1] = {static_cast<uint64_t>(p.lda) * sizeof(In)};
        uint32_t const box[2] = {static_cast<uint32_t>(kBlockK), static_cast<uint32_t>(aRows)};
        int32_t const st = makeTensorMap(&mapA, dt, 2, p.a, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
        if (st != BERT_B200_OK)
            return st;
    }
    {
        uint64_t const dims[2] = {static_cast<uint64_t>(p.k), static_cast<uint64_t>(p.n)};
        uint64_t const strides[1] = {static_cast<uint64_t>(p.k) * sizeof(In)};
        uint32_t const box[2] = {static_cast<uint32_t>(kBlockK), static_cast<uint32_t>(BLOCK_N)};
        int32_t const st = makeTensorMap(&mapB, dt, 2, p.wt, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
        if (st != BERT_B200_OK)
            return st;
    }
    int64_t const tiles = ((p.m + BLOCK_M - 1) / BLOCK_M) * ((p.n + BLOCK_N - 1) / BLOCK_N);
    // One CTA per SM may take a longer ring; otherwise two have to fit.
    int const kSteps = static_cast<int>((p.k + L::kSub * kBlockK - 1) / (L::kSub * kBlockK));
    int const stages = L::stagesFor(aRows, kSteps, tiles <= smCount() ? 200 * 1024 : 113 * 1024);
    auto kernel = fcTcgen05TileKernel<In, BLOCK_M, BLOCK_N, Out>;
    static SmemOptIn optIn;
    FcArgs const args = makeFcArgs(p, stages, aRows, weightsReady);
    cudaError_t const e = launchDependentCluster(
        &optIn, kernel, dim3(static_cast<unsigned>(tiles)), dim3(L::kThreads), L::bytes(stages, aRows), stream, 1, mapA, mapB, args);
    if (e != cudaSuccess)
        B200_FAIL(BERT_B200_CUDA_ERROR, "fcTcgen05TileKernel: %s", cudaGetErrorString(e));
    return checkLaunch("fcTcgen05TileKernel");
}

// ------------------------------------------------------------------------------------------------
// Two-CTA variant: a cluster of two CTAs (neighbouring SMs) computes one 256 x BLOCK_N tile with
// tcgen05.mma.cta_group::2. Each CTA loads its own 128 rows of A and its own BLOCK_N/2 rows of Wt, so a pair
// moves (256 + BLOCK_N) rows per k-block instead of 2 x (128 + BLOCK_N): the shared-memory fill bandwidth per SM,
// which bounds the one-CTA kernel, drops by a third and the ring gets deeper (6-8 stages).
//   Leader (cluster rank 0): its MMA lane issues every MMA; its "full" barriers collect the TMA bytes of both
//   CTAs; its "accEmpty" barriers collect the epilogue arrivals of both CTAs. tcgen05.commit multicasts the
//   "stage free" and "accumulator ready" arrivals to both CTAs.
// ------------------------------------------------------------------------------------------------
template <int BLOCK_N>
struct FcPairSmem
{
    static constexpr int kABytes = kBlockM * kRowBytes;            // this CTA's 128 rows of A
    static constexpr int kBBytes = (BLOCK_N / 2) * kRowBytes;      // this CTA's half of the Wt rows
    static constexpr int kStageBytes = kABytes + kBBytes;
    static constexpr int kStages = BLOCK_N == 128 ? 8 : (BLOCK_N == 160 ? 7 : 6);
    static constexpr int kOutOff = kStages * kStageBytes;          // epilogue staging: kOutWarpBytes per epilogue warp
    static constexpr int kOutWarpBytes = 2048;                     // one FP16 or two INT8 [32 x 32] chunks
    static constexpr int kBarrierOff = kOutOff + kEpilogueWarps * kOutWarpBytes;
    static constexpr int kTotal = kBarrierOff + (2 * kStages + 4) * 8 + 16;
    static constexpr int kDynamic = kTotal + 1024;
    static_assert(kDynamic <= 232448, "shared memory budget of one CTA");
};

template <typename In, int BLOCK_N, typename Out>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kFcThreads, 1)
    fcTcgen05PairKernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB,
        const __grid_constant__ CUtensorMap mapC, FcArgs const args)
{
    using L = FcPairSmem<BLOCK_N>;
    constexpr bool kInt8 = sizeof(In) == 1;
    constexpr int kBlockK = kRowBytes / sizeof(In);
    constexpr int kUmmaKBytes = 32;
    constexpr int kPairM = 2 * kBlockM;
    constexpr uint32_t kIdesc
        = makeInstrDesc(kInt8 ? 2u : 1u, kInt8 ? 1u : 0u, 0u, 0u, static_cast<uint32_t>(kPairM), static_cast<uint32_t>(BLOCK_N));

    extern __shared__ uint8_t smemRaw[];
    // the dynamic shared memory window starts at the same offset in both CTAs, so this rounding agrees too
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smemRaw) + 1023) & ~static_cast<uintptr_t>(1023));
    uint8_t* sA = smem;
    uint8_t* sB = smem + L::kStages * L::kABytes;
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + L::kBarrierOff);
    uint64_t* empty = full + L::kStages;
    uint64_t* accFull = empty + L::kStages;
    uint64_t* accEmpty = accFull + 2;
    uint32_t* tmemSlot = reinterpret_cast<uint32_t*>(accEmpty + 2);
    volatile uint32_t* abortFlag = tmemSlot + 1;

    int const warp = threadIdx.x >> 5;
    int const lane = threadIdx.x & 31;
    uint32_t const rank = clusterCtaRank();
    bool const leader = rank == 0;

    if (threadIdx.x == 0)
    {
        for (int i = 0; i < L::kStages; ++i)
        {
            mbarInit(&full[i], 1);  // the leader's producer arrives (with the byte count of both CTAs)
            mbarInit(&empty[i], 1); // one multicast commit from the leader
        }
        for (int i = 0; i < 2; ++i)
        {
            mbarInit(&accFull[i], 1);
            mbarInit(&accEmpty[i], 2 * kEpilogueWarps); // one lane per epilogue warp of both CTAs (used in the leader only)
        }
        *abortFlag = 0;
        fenceBarrierInit();
        prefetchTensorMap(&mapA);
        prefetchTensorMap(&mapB);
        prefetchTensorMap(&mapC);
    }
    if (warp == 1)
        tmemAllocPair(tmemSlot, kTmemCols);
    tcFenceBefore();
    __syncthreads();
    clusterSync(); // both CTAs' barriers are initialised before any remote arrival or TMA signal
    tcFenceAfter();
    uint32_t const tmemBase = *tmemSlot;
    // set-up done: the next kernel of the stream may start its own; the operands of this one must be complete
    gridDependencyLaunch();
    if (args.bias && blockIdx.x == 0) // see the tile kernel
        for (int64_t i = threadIdx.x * 32; i < args.N; i += kFcThreads * 32)
            prefetchL2(args.bias + i);
    gridDependencyWait();

    int64_t const mBlocks = (args.M + kPairM - 1) / kPairM;
    int64_t const nBlocks = (args.N + BLOCK_N - 1) / BLOCK_N;
    int64_t const numTiles = mBlocks * nBlocks;
    int const kBlocks = static_cast<int>((args.K + kBlockK - 1) / kBlockK);
    int64_t const firstTile = blockIdx.x / 2;
    int64_t const tileStride = gridDim.x / 2;

    if (warp == 0)
    {
        int stage = 0;
        uint32_t phase = 0;
        bool ok = true;
        // running shared-memory addresses of the stage being filled (see mmaPairLoHi for why)
        uint32_t const fullAddr0 = smemAddr(full), emptyAddr0 = smemAddr(empty);
        uint32_t const fullLeader0 = mapaShared(full, 0);
        uint32_t const aAddr0 = smemAddr(sA), bAddr0 = smemAddr(sB);
        uint32_t off8 = 0, aAddr = aAddr0, bAddr = bAddr0;
        for (int64_t tile = firstTile; tile < numTiles && ok; tile += tileStride)
        {
            int32_t const m0 = static_cast<int32_t>(tile / nBlocks) * kPairM + static_cast<int32_t>(rank) * kBlockM;
            int32_t const n0 = static_cast<int32_t>(tile % nBlocks) * BLOCK_N + static_cast<int32_t>(rank) * (BLOCK_N / 2);
            for (int kb = 0; kb < kBlocks; ++kb)
            {
                if (!mbarWaitWarp(emptyAddr0 + off8, phase ^ 1u, abortFlag, kWaitStageFree))
                {
                    ok = false;
                    break;
                }
                if (electOne())
                {
                    if (leader)
                        mbarArriveExpectTxAddr(fullAddr0 + off8, 2 * L::kStageBytes);
                    tmaLoad2dPairAddr(aAddr, &mapA, fullLeader0 + off8, kb * kBlockK, m0);
                    tmaLoad2dPairAddr(bAddr, &mapB, fullLeader0 + off8, kb * kBlockK, n0);
                }
                __syncwarp();
                off8 += 8;
                aAddr += L::kABytes;
                bAddr += L::kBBytes;
                if (++stage == L::kStages)
                {
                    stage = 0;
                    phase ^= 1u;
                    off8 = 0;
                    aAddr = aAddr0;
                    bAddr = bAddr0;
                }
            }
        }
        // Tail: every stage released, i.e. no commit arrival is still on its way to this CTA.
        for (int i = 0; i < L::kStages && ok; ++i)
        {
            ok = mbarWaitWarp(smemAddr(&empty[stage]), phase ^ 1u, abortFlag, kWaitStageFree);
            if (++stage == L::kStages)
            {
                stage = 0;
                phase ^= 1u;
            }
        }
    }
    else if (warp == 1)
    {
        if (leader)
        {
            int stage = 0;
            uint32_t phase = 0;
            int acc = 0;
            uint32_t accPhase = 0;
            bool ok = true;
            // descriptor words and barrier addresses of the stage being consumed, kept running (see mmaPairLoHi)
            uint64_t const descZero = makeSmemDesc(0, 16, 1024, kSwizzle128B);
            uint32_t const descHi = static_cast<uint32_t>(descZero >> 32);
            uint32_t const aLo0 = static_cast<uint32_t>(descZero) + (smemAddr(sA) >> 4);
            uint32_t const bLo0 = static_cast<uint32_t>(descZero) + (smemAddr(sB) >> 4);
            uint32_t const fullAddr0 = smemAddr(full), emptyAddr0 = smemAddr(empty);
            uint32_t off8 = 0, aLo = aLo0, bLo = bLo0;
            constexpr uint32_t kStep = kUmmaKBytes >> 4; // descriptor units per UMMA K step
            static_assert(kRowBytes / kUmmaKBytes == 4, "four MMAs per k-block");
            for (int64_t tile = firstTile; tile < numTiles && ok; tile += tileStride)
            {
                if (!mbarWaitWarp(smemAddr(&accEmpty[acc]), accPhase ^ 1u, abortFlag, kWaitAccFree))
                    break;
                tcFenceAfter();
                uint32_t const dTmem = tmemBase + static_cast<uint32_t>(acc * BLOCK_N);
                for (int kb = 0; kb < kBlocks; ++kb)
                {
                    if (!mbarWaitWarp(fullAddr0 + off8, phase, abortFlag, kWaitTmaFull))
                    {
                        ok = false;
                        break;
                    }
                    tcFenceAfter();
                    if (electOne())
                    {
                        if (kb == 0)
                            mmaPairLoHi<kInt8, false>(dTmem, aLo, bLo, descHi, kIdesc);
                        else
                            mmaPairLoHi<kInt8, true>(dTmem, aLo, bLo, descHi, kIdesc);
                        mmaPairLoHi<kInt8, true>(dTmem, aLo + kStep, bLo + kStep, descHi, kIdesc);
                        mmaPairLoHi<kInt8, true>(dTmem, aLo + 2 * kStep, bLo + 2 * kStep, descHi, kIdesc);
                        mmaPairLoHi<kInt8, true>(dTmem, aLo + 3 * kStep, bLo + 3 * kStep, descHi, kIdesc);
                        tcCommitPairAddr(emptyAddr0 + off8, 3);
                    }
                    __syncwarp();
                    off8 += 8;
                    aLo += L::kABytes >> 4;
                    bLo += L::kBBytes >> 4;
                    if (++stage == L::kStages)
                    {
                        stage = 0;
                        phase ^= 1u;
                        off8 = 0;
                        aLo = aLo0;
                        bLo = bLo0;
                    }
                }
                if (!ok)
                    break;
                if (electOne())
                    tcCommitPair(&accFull[acc], 3);
                __syncwarp();
                acc ^= 1;
                if (acc == 0)
                    accPhase ^= 1u;
            }
        }
    }
    else
    {
        int const quad = warp & 3;
        int const part = (warp - 2) >> 2;
        constexpr int kChunks = BLOCK_N / 32;
        constexpr int kChunksPerWarp = (kChunks + kEpilogueWarps / 4 - 1) / (kEpilogueWarps / 4); // one less in some warps
        constexpr int kChunkBytes = 32 * 32 * static_cast<int>(sizeof(Out));
        constexpr int kBufs = L::kOutWarpBytes / kChunkBytes; // staging tiles of this warp: 2 (INT8) or 1 (FP16)
        uint8_t* const stage0 = smem + L::kOutOff + (warp - 2) * L::kOutWarpBytes;
        int buf = 0;
        int acc = 0;
        uint32_t accPhase = 0;
        for (int64_t tile = firstTile; tile < numTiles; tile += tileStride)
        {
            int64_t const rowBase = (tile / nBlocks) * kPairM + static_cast<int64_t>(rank) * kBlockM + quad * 32;
            int64_t const n0 = (tile % nBlocks) * BLOCK_N;
            if (!mbarWait(&accFull[acc], accPhase, abortFlag, kWaitAccFull))
                break;
            tcFenceAfter();
            uint32_t const taddr = tmemBase + (static_cast<uint32_t>(quad * 32) << 16) + static_cast<uint32_t>(acc * BLOCK_N);
#pragma unroll
            for (int i = 0; i < kChunksPerWarp; ++i) // this warp's 32-column chunks of the tile
            {
                int const c = part + i * (kEpilogueWarps / 4);
                if (kChunks % (kEpilogueWarps / 4) != 0 && c >= kChunks)
                    break;
                uint32_t r[32];
                tmemLoad32(taddr + c * 32, r);
                tmemLoadWait32(r);
                if (c + kEpilogueWarps / 4 >= kChunks)
                {
                    // The accumulator is in registers: hand the TMEM buffer back before the arithmetic and the store.
                    tcFenceBefore();
                    __syncwarp();
                    if (lane == 0)
                        mbarArriveCluster(mapaShared(&accEmpty[acc], 0)); // the leader's barrier counts both CTAs
                }
                int64_t const col = n0 + c * 32;
                if (col < args.N && rowBase < args.M) // warp-uniform
                {
                    int const validCols = static_cast<int>(args.N - col < 32 ? args.N - col : 32);
                    float v[32];
                    QuantStep const q = fcEpilogueMath<kInt8, Out, 32>(r, v, args, args.bias ? args.bias + col : nullptr, validCols);
                    uint8_t* const tileBuf = stage0 + buf * kChunkBytes;
                    if (lane == 0)
                        bulkWaitGroupRead<kBufs - 1>(); // the store that last used this staging tile has read it
                    __syncwarp();
                    stageChunk32<Out>(tileBuf, lane, v, q);
                    fenceProxyAsync();
                    __syncwarp();
                    if (lane == 0)
                    {
                        // rows >= M and columns >= N of the box are clipped by the TMA unit
                        tmaStore2d(&mapC, tileBuf, static_cast<int32_t>(col), static_cast<int32_t>(rowBase));
                        bulkCommitGroup();
                    }
                    buf = buf + 1 == kBufs ? 0 : buf + 1;
                }
            }
            acc ^= 1;
            if (acc == 0)
                accPhase ^= 1u;
        }
        if (lane == 0)
            bulkWaitGroup<0>(); // every store of this warp has left shared memory and reached global memory
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
    tcFenceBefore();
    clusterSync(); // the peer no longer signals barriers of, or reads operands from, this CTA's shared memory
    if (warp == 1)
    {
        __syncwarp();
        tcFenceAfter();
        tmemFreePair(tmemBase, kTmemCols);
    }
}

template <typename In, int BLOCK_N, typename Out>
int32_t launchFcPair(bert_b200_fc_params const& p, cudaStream_t stream)
{
    using L = FcPairSmem<BLOCK_N>;
    constexpr int kBlockK = kRowBytes / sizeof(In);
    CUtensorMapDataType const dt = sizeof(In) == 1 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
    CUtensorMap mapA, mapB;
    {
        uint64_t const dims[2] = {static_cast<uint64_t>(p.k), static_cast<uint64_t>(p.m)};
        uint64_t const strides[1] = {static_cast<uint64_t>(p.lda) * sizeof(In)};
        uint32_t const box[2] = {static_cast<uint32_t>(kBlockK), static_cast<uint32_t>(kBlockM)};
        int32_t const st = makeTensorMap(&mapA, dt, 2, p.a, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
        if (st != BERT_B200_OK)
            return st;
    }
    {
        uint64_t const dims[2] = {static_cast<uint64_t>(p.k), static_cast<uint64_t>(p.n)};
        uint64_t const strides[1] = {static_cast<uint64_t>(p.k) * sizeof(In)};
        uint32_t const box[2] = {static_cast<uint32_t>(kBlockK), static_cast<uint32_t>(BLOCK_N / 2)};
        int32_t const st = makeTensorMap(&mapB, dt, 2, p.wt, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
        if (st != BERT_B200_OK)
            return st;
    }
    CUtensorMap mapC;
    {
        uint64_t const dims[2] = {static_cast<uint64_t>(p.n), static_cast<uint64_t>(p.m)};
        uint64_t const strides[1] = {static_cast<uint64_t>(p.ldc) * sizeof(Out)};
        uint32_t const box[2] = {32u, 32u};
        int32_t const st = makeTensorMap(&mapC, sizeof(Out) == 1 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2,
            p.c, dims, strides, box, sizeof(Out) == 1 ? CU_TENSOR_MAP_SWIZZLE_32B : CU_TENSOR_MAP_SWIZZLE_64B);
        if (st != BERT_B200_OK)
            return st;
    }
    auto kernel = fcTcgen05PairKernel<In, BLOCK_N, Out>;
    static SmemOptIn optIn;
    int64_t const tiles = ((p.m + 2 * kBlockM - 1) / (2 * kBlockM)) * ((p.n + BLOCK_N - 1) / BLOCK_N);
    int64_t const pairs = smCount() / 2;
    int const grid = static_cast<int>(2 * (tiles < pairs ? tiles : pairs));
    FcArgs const args = makeFcArgs(p, L::kStages, kBlockM, false);
    cudaError_t const le = launchDependentCluster(&optIn, kernel, dim3(grid), dim3(kFcThreads), L::kDynamic, stream, 1, mapA, mapB, mapC, args);
    if (le != cudaSuccess)
        B200_FAIL(BERT_B200_CUDA_ERROR, "fcTcgen05PairKernel: %s", cudaGetErrorString(le));
    return checkLaunch("fcTcgen05PairKernel");
}

// 256 x BLOCK_N pair tiles over the SM pairs: the width that wastes least of the last wave. A launch takes about as long as
// waves * (BLOCK_N + 110) + BLOCK_N / 2 columns of a 256-row tile: 110 for what does not grow with the width (A, hand-overs,
// epilogues of the odd widths), the last term for filling and draining the pipeline. Measured with 128 / 160 / 192 / 224 / 256
// columns: FP16 2600 x 1024 x 4096 28.8 / 33.6 / 24.2 / 26.8 / 29.5 us, 5001 x 1024 x 4096 40.5 / 36.5 / 39.7 / 43.4 / 48.0 us,
// 5001 x 4096 x 1024 40.0 / 37.6 / 35.2 / 37.3 / 35.4 us, INT8 5001 x 3072 x 1024 21.7 / 22.8 / 21.0 / 19.1 / 19.7 us,
// 24576 x 1024 x 4096 77 / 78 / 76 / 75 / 71 us.
int pickBlockNPair(int64_t m, int64_t n)
{
    int64_t const pairs = smCount() / 2;
    int best = 128;
    int64_t bestCost = 0;
    for (int bn = 128; bn <= 256 && (bn == 128 || bn - 32 < n); bn += 32)
    {
        int64_t const tiles = ((m + 2 * kBlockM - 1) / (2 * kBlockM)) * ((n + bn - 1) / bn);
        int64_t const cost = (tiles + pairs - 1) / pairs * (bn + 110) + bn / 2;
        if (bn == 128 || cost < bestCost)
        {
            best = bn;
            bestCost = cost;
        }
    }
    return best;
}

struct FcPlan
{
    bool pair;
    int blockN;
};

// Single tiles per CTA as long as they all run at once: the narrowest whose tiles do not outnumber the SMs (more SMs take part
// in loading the weights, shorter epilogue), with a short K 128-wide ones also at two CTAs per SM. Beyond, the persistent pair
// tiles are ahead: their epilogues overlap the next tile's main loop, and they load a third less per product. Measured at the
// borders, FP16: K = 768, 192 tiles 9.0 us against 10.5 us in pairs, 288 tiles 8.7 / 9.9 us, 450 tiles 15.4 / 13.8 us; 64-wide at
// two CTAs per SM (288 tiles) 6.6 us against 6.2 us with 144 128-wide ones. 4096 x 1024 (256 tiles), K = 1024 11.9 / 12.2 us, K =
// 4096 31.6 / 29.1 us; INT8 3100 x 768 (150 tiles), K = 768 7.6 / 7.6 us, K = 3072 14.5 / 12.2 us.
FcPlan planFc(bert_b200_fc_params const& p)
{
    int64_t const sms = smCount();
    int64_t const mBlocks = (p.m + kBlockM - 1) / kBlockM;
    bool const shortK = p.k * (p.type_id == BERT_B200_FP16 ? 2 : 1) < 3072;
    for (int bn = 16; bn <= 128; bn *= 2)
        if (mBlocks * ((p.n + bn - 1) / bn) <= (bn == 128 && shortK ? 2 * sms : sms))
            return {false, bn};
    if (p.m <= kBlockM) // the second CTA of a pair would have no rows
        return {false, 128};
    return {true, pickBlockNPair(p.m, p.n)};
}

} // namespace

EncodeTiledFn getEncodeTiled()
{
    static std::mutex mtx;
    static EncodeTiledFn fn = nullptr;
    std::lock_guard<std::mutex> lock(mtx);
    if (!fn)
    {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess
            && q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    }
    return fn;
}

int32_t makeTensorMap(CUtensorMap* map, CUtensorMapDataType type, int rank, void const* base, uint64_t const* dims,
    uint64_t const* stridesBytes, uint32_t const* box, CUtensorMapSwizzle swizzle)
{
    EncodeTiledFn const fn = getEncodeTiled();
    if (!fn)
        B200_FAIL(BERT_B200_NOT_INITIALIZED, "cuTensorMapEncodeTiled is not available from this driver");
    cuuint64_t d[5];
    cuuint64_t s[4];
    cuuint32_t b[5];
    cuuint32_t es[5];
    for (int i = 0; i < rank; ++i)
    {
        d[i] = dims[i];
        b[i] = box[i];
        es[i] = 1;
        if (i > 0)
            s[i - 1] = stridesBytes[i - 1];
    }
    CUresult const r = fn(map, type, static_cast<cuuint32_t>(rank), const_cast<void*>(base), d, s, b, es,
        CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS)
        B200_FAIL(BERT_B200_BAD_PARAM, "cuTensorMapEncodeTiled failed with CUresult %d", static_cast<int>(r));
    return BERT_B200_OK;
}

int32_t fcRun(bert_b200_fc_params const& p, cudaStream_t s, bool weightsReady)
{
    B200_REQUIRE(p.m >= 0 && p.n > 0 && p.k > 0, "fc: bad sizes m=%lld n=%lld k=%lld", static_cast<long long>(p.m),
        static_cast<long long>(p.n), static_cast<long long>(p.k));
    B200_REQUIRE(p.a && p.wt && p.c, "fc: null pointer");
    B200_REQUIRE(p.lda >= p.k && p.ldc >= p.n, "fc: lda/ldc smaller than the row length");
    B200_REQUIRE(p.activation == BERT_B200_ACT_NONE || p.activation == BERT_B200_ACT_GELU_ERF, "fc: unknown activation %d",
        p.activation);
    if (p.m == 0)
        return BERT_B200_OK;
    if (p.type_id == BERT_B200_FP32)
    {
        B200_REQUIRE(p.out_type_id == BERT_B200_FP32, "fc: FP32 input needs FP32 output");
        return fcF32(p, s);
    }
    B200_REQUIRE(p.type_id == BERT_B200_FP16 || p.type_id == BERT_B200_INT8, "fc: type_id %d", p.type_id);
    B200_REQUIRE(p.out_type_id != BERT_B200_INT8 || p.out_scale > 0.f, "fc: INT8 output needs out_scale > 0");
    B200_REQUIRE(p.m < (1ll << 31) && p.n < (1ll << 31) && p.k < (1ll << 31), "fc: sizes exceed the 32-bit TMA coordinates");
    int const elem = p.type_id == BERT_B200_FP16 ? 2 : 1;
    B200_REQUIRE((p.k * elem) % 16 == 0 && (p.lda * elem) % 16 == 0, "fc: row bytes of A / Wt must be a multiple of 16");
    B200_REQUIRE(aligned16(p.a) && aligned16(p.wt) && aligned16(p.c), "fc: A, Wt and C must be 16-byte aligned");
    B200_REQUIRE(p.n % 16 == 0, "fc: n=%lld must be a multiple of 16", static_cast<long long>(p.n));
    B200_REQUIRE(!p.bias || aligned16(p.bias), "fc: bias must be 16-byte aligned");
    int const outElem = p.out_type_id == BERT_B200_FP16 ? 2 : 1;
    B200_REQUIRE((p.ldc * outElem) % 16 == 0, "fc: row bytes of C must be a multiple of 16");
    FcPlan const plan = planFc(p);
    bool const shortTile = p.m <= 64; // the narrow tiles also come with 64 rows (see the kernel)
#define B200_FC_TILE(IN, OUT)                                                                                          \
    switch (plan.blockN)                                                                                               \
    {                                                                                                                  \
    case 16: return shortTile ? launchFcTile<IN, 64, 16, OUT>(p, weightsReady, s) : launchFcTile<IN, 128, 16, OUT>(p, weightsReady, s); \
    case 32: return shortTile ? launchFcTile<IN, 64, 32, OUT>(p, weightsReady, s) : launchFcTile<IN, 128, 32, OUT>(p, weightsReady, s); \
    case 64: return launchFcTile<IN, 128, 64, OUT>(p, weightsReady, s);                                                \
    default: return launchFcTile<IN, 128, 128, OUT>(p, weightsReady, s);                                               \
    }
#define B200_FC_DISPATCH(IN, OUT)                                                                                      \
    if (plan.pair)                                                                                                     \
        switch (plan.blockN)                                                                                           \
        {                                                                                                              \
        case 128: return launchFcPair<IN, 128, OUT>(p, s);                                                             \
        case 160: return launchFcPair<IN, 160, OUT>(p, s);                                                             \
        case 192: return launchFcPair<IN, 192, OUT>(p, s);                                                             \
        case 224: return launchFcPair<IN, 224, OUT>(p, s);                                                             \
        default: return launchFcPair<IN, 256, OUT>(p, s);                                                              \
        }                                                                                                              \
    B200_FC_TILE(IN, OUT)
    if (p.type_id == BERT_B200_FP16)
    {
        B200_REQUIRE(p.out_type_id == BERT_B200_FP16, "fc: FP16 input needs FP16 output");
        B200_FC_DISPATCH(__half, __half)
    }
    if (p.out_type_id == BERT_B200_INT8)
    {
        B200_FC_DISPATCH(int8_t, int8_t)
    }
    B200_REQUIRE(p.out_type_id == BERT_B200_FP16, "fc: INT8 input needs INT8 or FP16 output");
    B200_FC_DISPATCH(int8_t, __half)
#undef B200_FC_TILE
#undef B200_FC_DISPATCH
}

} // namespace b200

extern "C" int32_t bert_b200_fc(bert_b200_fc_params const* params, void* stream)
{
    B200_REQUIRE(params != nullptr, "fc: null params");
    // Nothing is known about who writes the weights: a kernel two places ahead in the stream may still be at it.
    return b200::fcRun(*params, static_cast<cudaStream_t>(stream), false);
}
