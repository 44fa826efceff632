// FP32 (type_id 0) attention, and the fully-connected layers that the tensor-core kernel of fc_f32_tcgen05.cu does not take (a short K,
// rows that are not 16-byte aligned): SIMT kernels at full FP32 precision.
// The attention kernels also serve FP16 tensors (FP32 arithmetic) for the shapes the tensor-core kernels do not
// take - heads wider than 64 or not a multiple of 16, a scale that is not positive - which the reference sends to its unfused
// runner as well.
//
// Replaces cublas{S,H}gemmStridedBatched + softmax kernels of UnfusedMHARunner::run
// (plugin/bertQKVToContextPlugin/mhaRunner.cu:533-601) and the FP32 cublasLtMatmul of the FC plugin
// (plugin/fcPlugin/fcPlugin.cpp:551-610).
#include "common.cuh"
#include "mha_f32_plan.h"

namespace b200
{

namespace
{

// ---- fully connected ------------------------------------------------------------------------------------------------
// C[m,n] = act(alpha * sum_k A[m,k] * Wt[n,k] + bias[n]).
//
// Bound by the FP32 FMA pipes (128 per clock and SM). A CTA of two warps computes a 64 x 64 tile, every thread 8 x 8
// outputs, four CTAs per SM. Both operands are K-contiguous, so they are copied to shared memory as they lie (16-byte
// cp.async, four stages) and read back as 8-byte pieces along K, those of the next two k during the FMAs of these (16-byte
// pieces left no registers for that: 3 % slower); rows are padded to 20 floats, which puts the 4 or 8 rows that a warp reads
// at once into different banks. The sums run on packed fma.rn.f32x2: one half takes the even k, the
// other the odd ones (no operand has to be duplicated), and the two are added at the end; a packed FMA takes half the
// issue slots, which leaves room for the loads. These bring 128 bytes per thread and k pair to the registers, at 128 bytes per
// clock and SM as long as the FMAs take: the loop runs at 0.6 of the FMA rate.
// K is summed in segments (1, 2, 4 or 8 of about equal length, by K alone), and the segments' sums are added in order: a row of C is the
// same bits whatever M, although the work is divided by the number of tiles. Where the tiles alone fill the SMs, a CTA takes all segments
// of its tile and keeps their sum in shared memory (16 KB, four CTAs still fit an SM); otherwise a cluster takes one per CTA, exchanges
// the sums through distributed shared memory and each CTA finishes its share of every thread's outputs.
// It takes a K below 384 and what the tensor-core kernel cannot load (see fcF32). Measured: 512 x 768 x 384 in 15.6 us; holding the sums of the
// segments costs 3 % where they are eight, exchanging them 8 %, and few rows gain (37 x 768 x 768 8.7 us, 9.7 us with a scalar exchange).
constexpr int kTile = 64;
constexpr int kTileK = 16;
constexpr int kPitch = kTileK + 4; // floats
constexpr int kStages = 4;
constexpr int kFcF32Threads = 64;
constexpr int kFcF32CtasPerSm = 4;
constexpr int kFcF32Ring = kStages * 2 * kTile * kPitch; // floats
constexpr int kFcF32Part = kTile * kTile;                // sums of a segment, as the threads hold them (see partIndex)
static_assert(kFcF32Ring >= kFcF32Part, "the last segment's sums reuse the ring");

__device__ __forceinline__ float sumPair(uint64_t v)
{
    float lo, hi;
    unpack2(v, lo, hi);
    return lo + hi;
}

// kBytes (16 or 4) from global to shared memory, zeros when `valid` is false.
template <int kBytes>
__device__ __forceinline__ void cpAsync(uint32_t dst, void const* src, bool valid)
{
    int const n = valid ? kBytes : 0;
    if constexpr (kBytes == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}

__device__ __forceinline__ void cpAsyncCommit()
{
    asm volatile("cp.async.commit_group;" ::: "memory");
}

template <int N>
__device__ __forceinline__ void cpAsyncWait()
{
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

struct FcF32Args
{
    int64_t M, N, K;
    float const* A;
    int64_t lda;
    float const* Wt;
    float* C;
    int64_t ldc;
    float const* bias;
    int32_t act;
    float alpha;
    int32_t nTiles;   // tiles along N
    int32_t segments; // of K
};

__device__ __forceinline__ float fcF32Epilogue(FcF32Args const& p, float v, int64_t n)
{
    v = v * p.alpha + (p.bias ? p.bias[n] : 0.f);
    return p.act == BERT_B200_ACT_GELU_ERF ? geluErfF32(v) : v;
}

// Columns n, n + 8, n + 16 and n + 24 of row m.
__device__ __forceinline__ void storeF32(FcF32Args const& p, float4 v, int64_t m, int64_t n)
{
    float const vv[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int c = 0; c < 4; ++c)
        if (m < p.M && n + 8 * c < p.N)
            p.C[m * p.ldc + n + 8 * c] = fcF32Epilogue(p, vv[c], n + 8 * c);
}

// Where the segment's sums of outputs (i, j ... j + 3) of a thread lie: group i * 2 + j / 4, consecutive lanes at consecutive 16
// bytes (no bank conflicts).
__device__ __forceinline__ int partIndex(int i, int j, int tid)
{
    return ((i * 2 + (j >> 2)) * kFcF32Threads + tid) * 4 + (j & 3);
}

// kVec: floats per copy (4, or 1 where K, lda or an address is not a multiple of 16 bytes). kAlone: a CTA takes all segments of its
// tile, otherwise a cluster takes one per CTA.
template <int kVec, bool kAlone>
__global__ void __launch_bounds__(kFcF32Threads, kFcF32CtasPerSm) fcF32Kernel(FcF32Args const p)
{
    extern __shared__ __align__(16) float smRaw[]; // the ring, then (kAlone) the sum of the segments so far
    float(*const sm)[2][kTile][kPitch] = reinterpret_cast<float(*)[2][kTile][kPitch]>(smRaw);
    float* const held = smRaw + kFcF32Ring;
    int const tid = threadIdx.x;
    int const lane = tid & 31;
    int const ty = lane >> 3;
    int const tx = lane & 7;
    int const row0 = (tid >> 5) * 32 + ty; // rows row0 + 4 i, columns tx + 8 j
    int const rank = kAlone ? 0 : static_cast<int>(blockIdx.x % p.segments);
    int64_t const tile = kAlone ? blockIdx.x : blockIdx.x / p.segments;
    int64_t const m0 = tile / p.nTiles * kTile;
    int64_t const n0 = tile % p.nTiles * kTile;
    int64_t const kBlocks = (p.K + kTileK - 1) / kTileK;
    auto segmentBegin = [&](int s) { return static_cast<int>(kBlocks * s / p.segments); };
    int const kbFirst = segmentBegin(rank);
    int const kbEnd = kAlone ? static_cast<int>(kBlocks) : segmentBegin(rank + 1);

    gridDependencyLaunch();
    gridDependencyWait();

    uint32_t const smBase = static_cast<uint32_t>(__cvta_generic_to_shared(smRaw));
    auto load = [&](int kb, int stage) {
        constexpr int kPieces = kTileK / kVec; // per row
        constexpr int kRowStep = kFcF32Threads / kPieces;
        int const piece = tid % kPieces;
        int64_t const k = static_cast<int64_t>(kb) * kTileK + piece * kVec;
        bool const kOk = k < p.K;
#pragma unroll
        for (int r = tid / kPieces; r < 2 * kTile; r += kRowStep)
        {
            bool const isA = r < kTile;
            int64_t const g = isA ? m0 + r : n0 + r - kTile;
            bool const ok = kOk && g < (isA ? p.M : p.N);
            float const* const src = isA ? p.A + g * p.lda + k : p.Wt + g * p.K + k;
            cpAsync<4 * kVec>(smBase + 4u * (static_cast<uint32_t>(stage * 2 * kTile + r) * kPitch + piece * kVec), ok ? src : p.A, ok);
        }
    };

    uint64_t acc[8][8] = {};
    for (int s = 0; s < kStages - 1; ++s)
    {
        if (kbFirst + s < kbEnd)
            load(kbFirst + s, s);
        cpAsyncCommit();
    }
    int stage = 0;
    int segment = 0;
    int segmentEnd = kAlone ? segmentBegin(1) : kbEnd;
#pragma unroll 1
    for (int kb = kbFirst; kb < kbEnd; ++kb)
    {
        if (kAlone && kb == segmentEnd)
        {
            // the segment's sums to those before it (a thread reads what it has written itself)
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 8; j += 4)
                {
                    float4* const h = reinterpret_cast<float4*>(held + partIndex(i, j, tid));
                    float4 v = make_float4(sumPair(acc[i][j]), sumPair(acc[i][j + 1]), sumPair(acc[i][j + 2]), sumPair(acc[i][j + 3]));
                    if (segment > 0)
                    {
                        float4 const before = *h;
                        v = make_float4(before.x + v.x, before.y + v.y, before.z + v.z, before.w + v.w);
                    }
                    *h = v;
                    acc[i][j] = acc[i][j + 1] = acc[i][j + 2] = acc[i][j + 3] = 0;
                }
            ++segment;
            segmentEnd = segmentBegin(segment + 1);
        }
        cpAsyncWait<kStages - 2>();
        __syncthreads(); // this stage has landed; everybody is done with the one that is filled next
        int const ahead = stage == 0 ? kStages - 1 : stage - 1;
        if (kb + kStages - 1 < kbEnd)
            load(kb + kStages - 1, ahead);
        cpAsyncCommit();
        float const(*const a)[kPitch] = sm[stage][0];
        float const(*const b)[kPitch] = sm[stage][1];
        // two k at a time; the next two are on their way from shared memory during the FMAs of these
        uint64_t av[2][8], bv[2][8];
        auto fetch = [&](int buf, int k) {
#pragma unroll
            for (int i = 0; i < 8; ++i)
                av[buf][i] = *reinterpret_cast<uint64_t const*>(&a[row0 + 4 * i][k]);
#pragma unroll
            for (int j = 0; j < 8; ++j)
                bv[buf][j] = *reinterpret_cast<uint64_t const*>(&b[tx + 8 * j][k]);
        };
        fetch(0, 0);
#pragma unroll
        for (int k = 0; k < kTileK; k += 2)
        {
            int const cur = (k >> 1) & 1;
            if (k + 2 < kTileK)
                fetch(cur ^ 1, k + 2);
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    acc[i][j] = fma2(av[cur][i], bv[cur][j], acc[i][j]);
        }
        stage = stage + 1 == kStages ? 0 : stage + 1;
    }
    if constexpr (kAlone)
    {
#pragma unroll
        for (int i = 0; i < 8; ++i)
        {
            int64_t const m = m0 + row0 + 4 * i;
#pragma unroll
            for (int j = 0; j < 8; j += 4)
            {
                float4 v = make_float4(sumPair(acc[i][j]), sumPair(acc[i][j + 1]), sumPair(acc[i][j + 2]), sumPair(acc[i][j + 3]));
                if (p.segments > 1)
                {
                    float4 const before = *reinterpret_cast<float4 const*>(held + partIndex(i, j, tid));
                    v = make_float4(before.x + v.x, before.y + v.y, before.z + v.z, before.w + v.w);
                }
                storeF32(p, v, m, n0 + tx + 8 * j);
            }
        }
        return;
    }
    cpAsyncWait<0>();
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; j += 4)
            *reinterpret_cast<float4*>(smRaw + partIndex(i, j, tid))
                = make_float4(sumPair(acc[i][j]), sumPair(acc[i][j + 1]), sumPair(acc[i][j + 2]), sumPair(acc[i][j + 3]));
    clusterBarrier();
    for (int g = rank; g < 16; g += p.segments)
    {
        int const i = g >> 1, j = (g & 1) * 4;
        int const at = partIndex(i, j, tid);
        float4 x[8];
#pragma unroll
        for (int s = 0; s < 8; ++s) // all on their way before the first is added
            if (s < p.segments)
                x[s] = ldSharedCluster4(smRaw + at, s);
        float4 v = x[0];
#pragma unroll
        for (int s = 1; s < 8; ++s)
            if (s < p.segments)
                v = make_float4(v.x + x[s].x, v.y + x[s].y, v.z + x[s].z, v.w + x[s].w);
        int64_t const m = m0 + row0 + 4 * i;
        storeF32(p, v, m, n0 + tx + 8 * j);
    }
    clusterBarrier(); // nobody leaves while its partial sums are being read
}

__device__ __forceinline__ float toFloat(float v)
{
    return v;
}
__device__ __forceinline__ float toFloat(__half v)
{
    return __half2float(v);
}
__device__ __forceinline__ void fromFloat(float& dst, float v)
{
    dst = v;
}
__device__ __forceinline__ void fromFloat(__half& dst, float v)
{
    dst = __float2half_rn(v);
}

// ---- attention ------------------------------------------------------------------------------------------------------
// Where the rows of one (sequence, head) lie.
struct SeqRows
{
    int rows, len;  // query rows, valid keys
    int64_t row0, rowStride;
};

__device__ __forceinline__ SeqRows seqRows(int b, int B, int S, int32_t const* cu, int32_t const* maskIdx)
{
    if (cu)
        return {cu[b + 1] - cu[b], cu[b + 1] - cu[b], cu[b], 1};
    return {S, maskIdx ? min(max(maskIdx[b], 0), S) : S, b, B};
}

// Four consecutive elements of a row, as FP32.
__device__ __forceinline__ float4 load4(float const* p)
{
    return __ldg(reinterpret_cast<float4 const*>(p));
}
__device__ __forceinline__ float4 load4(__half const* p)
{
    uint2 const v = __ldg(reinterpret_cast<uint2 const*>(p));
    float2 const lo = __half22float2(*reinterpret_cast<__half2 const*>(&v.x));
    float2 const hi = __half22float2(*reinterpret_cast<__half2 const*>(&v.y));
    return make_float4(lo.x, lo.y, hi.x, hi.y);
}
__device__ __forceinline__ void store4(float* p, float4 v)
{
    *reinterpret_cast<float4*>(p) = v;
}
__device__ __forceinline__ void store4(__half* p, float4 v)
{
    __half2 const lo = __floats2half2_rn(v.x, v.y), hi = __floats2half2_rn(v.z, v.w);
    *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<uint32_t const*>(&lo), *reinterpret_cast<uint32_t const*>(&hi));
}

// 16 bytes into shared memory, or zeros.
__device__ __forceinline__ void copy16(void* to, void const* from, bool ok)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(to))), "l"(from), "r"(ok ? 16u : 0u)
                 : "memory");
}
__device__ __forceinline__ void copyGroup()
{
    asm volatile("cp.async.commit_group;" ::: "memory");
}
template <int N> // groups that may still be on their way
__device__ __forceinline__ void copyWait()
{
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// 64 or 32 queries of one (sequence, head) per CTA against blocks of 64 keys, running maximum and sum per row.
//
// Bound by the FP32 pipes and the shared-memory loads that feed them. Every warp owns 16 query rows, so its scores,
// probabilities and row sums are its own business; a thread computes 4 rows x
// 8 keys of the scores with 16-byte loads along d (packed FMAs, even and odd channels apart, as in the FC above), and 4
// rows x D / 8 columns of the context. Rows are padded by 4 floats against bank conflicts. Which form, and how many CTAs share an SM: see planAtt.
// Measured, heads of 64 channels: 8 sequences of 128 tokens, 12 heads 19.6 us (a warp per query row, keys and values from global memory: 509 us).
constexpr int kAttKeys = 64;

template <int D, int WARPS> // head size rounded up to 32, 64, 96 or 128; channels beyond d are zero
struct AttSmem
{
    static constexpr int kAttRows = 16 * WARPS;
    float q[kAttRows][D + 4];
    float k[kAttKeys][D + 4];
    float v[kAttKeys][D];
    float p[kAttRows][kAttKeys + 4];
};

// Context of rows row0 + 4 i: keys c ... c + 3 of the block.
template <typename Smem, int COLS>
__device__ __forceinline__ void addFourKeys(Smem const& sm, int const row0, int const tx, int const c, float4 (&o)[4][COLS])
{
    float4 pr[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
        pr[i] = *reinterpret_cast<float4 const*>(&sm.p[row0 + 4 * i][c]);
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int j = 0; j < COLS; ++j)
        {
            float4 const v = *reinterpret_cast<float4 const*>(&sm.v[c + k][tx * 4 + 32 * j]);
#pragma unroll
            for (int i = 0; i < 4; ++i)
            {
                float const w = k == 0 ? pr[i].x : k == 1 ? pr[i].y : k == 2 ? pr[i].z : pr[i].w;
                o[i][j].x = fmaf(w, v.x, o[i][j].x);
                o[i][j].y = fmaf(w, v.y, o[i][j].y);
                o[i][j].z = fmaf(w, v.z, o[i][j].z);
                o[i][j].w = fmaf(w, v.w, o[i][j].w);
            }
        }
}

// ASYNC: FP32 keys and values come by asynchronous copies, the next keys during the softmax and the second product, the next values during the scores (with one
// barrier less each, values during scores and softmax, keys during the second product: 16 x 128, 12 heads 31.7 us instead of 27.5 us). That takes four
// barriers per block of keys instead of two.
// SKIP: keys beyond the sequence, which have no weight, are left out of the second product, four or eight at a time (the scores' product takes all 64).
template <typename T, int D, int WARPS, bool ASYNC, bool SKIP>
__global__ void __launch_bounds__(32 * WARPS) mhaTiledKernel(int32_t const B, int32_t const S, int32_t const N, int32_t const d,
    T const* __restrict__ qkv, T* __restrict__ out, int32_t const* __restrict__ cu, int32_t const* __restrict__ maskIdx, float const scale)
{
    static_assert(!ASYNC || (sizeof(T) == 4 && SKIP), "FP16 is converted on the way");
    extern __shared__ float smRaw[];
    using Smem = AttSmem<D, WARPS>;
    Smem& sm = *reinterpret_cast<Smem*>(smRaw);
    constexpr int kAttRows = Smem::kAttRows, kAttThreads = 32 * WARPS;
    constexpr int kVecs = D / 4;
    constexpr int kCols = D / 32; // float4 columns of the context per thread
    int const lane = threadIdx.x & 31;
    int const ty = lane >> 3;
    int const tx = lane & 7;
    int const row0 = (threadIdx.x >> 5) * 16 + ty; // rows row0 + 4 i

    gridDependencyLaunch();
    gridDependencyWait();

    SeqRows const seq = seqRows(blockIdx.y, B, S, cu, maskIdx);
    int const q0 = blockIdx.z * kAttRows;
    if (q0 >= seq.rows)
        return;
    int64_t const tokStride = static_cast<int64_t>(3) * N * d;
    T const* const base = qkv + seq.row0 * tokStride + static_cast<int64_t>(blockIdx.x) * 3 * d;
    int64_t const rowStep = seq.rowStride * tokStride;
    float4 const zero = make_float4(0.f, 0.f, 0.f, 0.f);

    for (int i = threadIdx.x; i < kAttRows * kVecs; i += kAttThreads)
    {
        int const r = i / kVecs, c = i % kVecs * 4;
        bool const ok = q0 + r < seq.rows && c < d;
        if constexpr (ASYNC)
            copy16(&sm.q[r][c], ok ? base + (q0 + r) * rowStep + c : base, ok);
        else
            *reinterpret_cast<float4*>(&sm.q[r][c]) = ok ? load4(base + (q0 + r) * rowStep + c) : zero;
    }
    // Scores of keys beyond the sequence are never looked at, so such rows are left as they are; a value row with them has to be a number.
    [[maybe_unused]] auto fetchKeys = [&](int k0) {
        if constexpr (sizeof(T) != 4)
            return;
        int const rows = min(kAttKeys, seq.len - k0);
#pragma unroll 2
        for (int i = threadIdx.x; i < rows * kVecs; i += kAttThreads)
        {
            int const r = i / kVecs, c = i % kVecs * 4;
            copy16(&sm.k[r][c], c < d ? base + (k0 + r) * rowStep + c + d : base, c < d);
        }
        copyGroup();
    };
    [[maybe_unused]] auto fetchValues = [&](int k0) {
        if constexpr (sizeof(T) != 4)
            return;
        int const rows = min(kAttKeys, (seq.len - k0 + 3) & ~3);
#pragma unroll 2
        for (int i = threadIdx.x; i < rows * kVecs; i += kAttThreads)
        {
            int const r = i / kVecs, c = i % kVecs * 4;
            bool const ok = k0 + r < seq.len && c < d;
            copy16(&sm.v[r][c], ok ? base + (k0 + r) * rowStep + c + 2 * d : base, ok);
        }
        copyGroup();
    };
    if constexpr (ASYNC)
    {
        fetchKeys(0); // and the queries
        fetchValues(0);
    }
    float4 o[4][kCols];
    float mx[4], sum[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
    {
        mx[i] = -INFINITY;
        sum[i] = 0.f;
#pragma unroll
        for (int j = 0; j < kCols; ++j)
            o[i][j] = zero;
    }
    for (int k0 = 0; k0 < seq.len; k0 += kAttKeys)
    {
        if constexpr (ASYNC)
            copyWait<1>(); // keys
        else
        {
            __syncthreads(); // the previous block of keys is done with
#pragma unroll 4
            for (int i = threadIdx.x; i < kAttKeys * kVecs; i += kAttThreads)
            {
                int const r = i / kVecs, c = i % kVecs * 4;
                bool const ok = k0 + r < seq.len && c < d;
                T const* const src = base + (k0 + r) * rowStep + c;
                *reinterpret_cast<float4*>(&sm.k[r][c]) = ok ? load4(src + d) : zero;
                *reinterpret_cast<float4*>(&sm.v[r][c]) = ok ? load4(src + 2 * d) : zero;
            }
        }
        __syncthreads();
        uint64_t acc[4][8] = {};
#pragma unroll 4
        for (int c = 0; c < D; c += 4)
        {
            ulonglong2 a[4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
                a[i] = *reinterpret_cast<ulonglong2 const*>(&sm.q[row0 + 4 * i][c]);
#pragma unroll
            for (int j = 0; j < 8; ++j)
            {
                ulonglong2 const b = *reinterpret_cast<ulonglong2 const*>(&sm.k[tx + 8 * j][c]);
#pragma unroll
                for (int i = 0; i < 4; ++i)
                {
                    acc[i][j] = fma2(a[i].x, b.x, acc[i][j]);
                    acc[i][j] = fma2(a[i].y, b.y, acc[i][j]);
                }
            }
        }
        if constexpr (ASYNC)
        {
            __syncthreads();
            fetchKeys(k0 + kAttKeys);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
        {
            float s[8];
            float m = -INFINITY;
#pragma unroll
            for (int j = 0; j < 8; ++j)
            {
                s[j] = k0 + tx + 8 * j < seq.len ? sumPair(acc[i][j]) * scale : -INFINITY;
                m = fmaxf(m, s[j]);
            }
#pragma unroll
            for (int x = 1; x < 8; x <<= 1)
                m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, x));
            float const next = fmaxf(mx[i], m);
            float const ref = next == -INFINITY ? 0.f : next; // every score so far has overflowed to -inf: no weight
            float const rescale = expf(mx[i] - ref);
            mx[i] = next;
            sum[i] *= rescale;
#pragma unroll
            for (int j = 0; j < kCols; ++j)
            {
                o[i][j].x *= rescale;
                o[i][j].y *= rescale;
                o[i][j].z *= rescale;
                o[i][j].w *= rescale;
            }
#pragma unroll
            for (int j = 0; j < 8; ++j)
            {
                float const e = expf(s[j] - ref);
                sum[i] += e;
                sm.p[row0 + 4 * i][tx + 8 * j] = e;
            }
        }
        if constexpr (ASYNC)
        {
            copyWait<1>(); // values
            __syncthreads();
        }
        else
            __syncwarp();
        if constexpr (ASYNC)
        {
            auto product = [&](int const keys) {
#pragma unroll 2
                for (int c = 0; c < keys; c += 4)
                    addFourKeys(sm, row0, tx, c, o);
            };
            if (seq.len - k0 >= kAttKeys) // a loop of its own: with a variable end it is 2.5 % slower
                product(kAttKeys);
            else
                product(seq.len - k0);
        }
        else if constexpr (SKIP)
        {
            int const keys = min(kAttKeys, seq.len - k0);
#pragma unroll 1
            for (int c = 0; c < keys; c += 8)
            {
                addFourKeys(sm, row0, tx, c, o);
                addFourKeys(sm, row0, tx, c + 4, o);
            }
        }
        else // addFourKeys written out: called, heads of 128 channels are 2.5 % slower
        {
#pragma unroll 2
            for (int c = 0; c < kAttKeys; c += 4)
            {
                float4 pr[4];
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    pr[i] = *reinterpret_cast<float4 const*>(&sm.p[row0 + 4 * i][c]);
#pragma unroll
                for (int k = 0; k < 4; ++k)
#pragma unroll
                    for (int j = 0; j < kCols; ++j)
                    {
                        float4 const v = *reinterpret_cast<float4 const*>(&sm.v[c + k][tx * 4 + 32 * j]);
#pragma unroll
                        for (int i = 0; i < 4; ++i)
                        {
                            float const w = k == 0 ? pr[i].x : k == 1 ? pr[i].y : k == 2 ? pr[i].z : pr[i].w;
                            o[i][j].x = fmaf(w, v.x, o[i][j].x);
                            o[i][j].y = fmaf(w, v.y, o[i][j].y);
                            o[i][j].z = fmaf(w, v.z, o[i][j].z);
                            o[i][j].w = fmaf(w, v.w, o[i][j].w);
                        }
                    }
            }
        }
        if constexpr (ASYNC)
        {
            __syncthreads();
            fetchValues(k0 + kAttKeys);
        }
    }
    if constexpr (ASYNC)
        copyWait<0>();
#pragma unroll
    for (int i = 0; i < 4; ++i)
    {
        float t = sum[i];
#pragma unroll
        for (int x = 1; x < 8; x <<= 1)
            t += __shfl_xor_sync(0xffffffffu, t, x);
        int const r = q0 + row0 + 4 * i;
        if (r >= seq.rows)
            continue;
        float const inv = seq.len > 0 ? 1.f / t : 0.f;
        T* const dst = out + (seq.row0 + r * seq.rowStride) * (static_cast<int64_t>(N) * d) + static_cast<int64_t>(blockIdx.x) * d;
#pragma unroll
        for (int j = 0; j < kCols; ++j)
            if (tx * 4 + 32 * j < d)
                store4(dst + tx * 4 + 32 * j, make_float4(o[i][j].x * inv, o[i][j].y * inv, o[i][j].z * inv, o[i][j].w * inv));
    }
}

// Heads wider than 128, of a size that is no multiple of 4, or tensors that are not aligned to four elements.
// One warp per query row. Scores of the row live in shared memory ([warps][S]); all arithmetic in FP32.
template <typename T>
__global__ void __launch_bounds__(128) mhaSimtKernel(int32_t const B, int32_t const S, int32_t const N, int32_t const d,
    T const* __restrict__ qkv, T* __restrict__ out, int32_t const* __restrict__ cu,
    int32_t const* __restrict__ maskIdx, float const scale)
{
    extern __shared__ float sm[];
    int const lane = threadIdx.x & 31;
    int const warp = threadIdx.x >> 5;
    int const b = blockIdx.y;
    int const n = blockIdx.x;
    float* scores = sm + warp * (S + d);
    float* qs = scores + S;

    SeqRows const seq = seqRows(b, B, S, cu, maskIdx);
    int const rows = seq.rows, len = seq.len;
    int64_t const row0 = seq.row0, rowStride = seq.rowStride;
    int64_t const tokStride = static_cast<int64_t>(3) * N * d;
    int64_t const headOff = static_cast<int64_t>(n) * 3 * d;
    for (int s = blockIdx.z * 4 + warp; s < rows; s += gridDim.z * 4)
    {
        T const* q = qkv + (row0 + s * rowStride) * tokStride + headOff;
        for (int i = lane; i < d; i += 32)
            qs[i] = toFloat(q[i]);
        __syncwarp();
        float mx = -INFINITY;
        for (int j = lane; j < len; j += 32)
        {
            T const* k = qkv + (row0 + j * rowStride) * tokStride + headOff + d;
            float acc = 0.f;
            for (int i = 0; i < d; ++i)
                acc = fmaf(qs[i], toFloat(k[i]), acc);
            acc *= scale;
            scores[j] = acc;
            mx = fmaxf(mx, acc);
        }
        mx = warpMax(mx);
        float sum = 0.f;
        for (int j = lane; j < len; j += 32)
        {
            float const p = expf(scores[j] - mx);
            scores[j] = p;
            sum += p;
        }
        sum = warpSum(sum);
        float const inv = len > 0 ? 1.f / sum : 0.f;
        __syncwarp();
        T* o = out + (row0 + s * rowStride) * (static_cast<int64_t>(N) * d) + static_cast<int64_t>(n) * d;
        for (int i = lane; i < d; i += 32)
        {
            float acc = 0.f;
            for (int j = 0; j < len; ++j)
                acc = fmaf(scores[j], toFloat(qkv[(row0 + j * rowStride) * tokStride + headOff + 2 * d + i]), acc);
            fromFloat(o[i], acc * inv);
        }
        __syncwarp();
    }
}

} // namespace

// Segments of K: eight from K = 768 on, else 192 products or more each. More of them are more CTAs for few rows and more sums to hold
// or exchange for many: with 4 / 8, 37 x 3072 x 768 22.5 / 15.2 us, 37 x 768 x 3072 47 / 26 us, 300 x 768 x 768 25.8 / 15.8 us, and 8192 x
// 768 x 768 255 / 262 us.
static int segmentsF32(int64_t kBlocks)
{
    return kBlocks >= 48 ? 8 : kBlocks >= 24 ? 4 : kBlocks >= 12 ? 2 : 1;
}

// Whether a CTA takes all segments of its tile: where the tiles alone are nearly all the CTAs that fit at once; with a long K (2048 and
// more), where a CTA of the last wave runs for long, only when that wave is nearly full. Measured with one CTA per tile / one per
// segment (waves of 592): 37 x 768 x 768 (12 tiles) 51 / 8.9 us, 300 x 3072 x 768 (240) 90 / 51 us, 2048 x 1024 x 1024 (512) 123 / 124 us,
// 4096 x 1024 x 1024 (1024) 233 / 237 us, 8192 x 768 x 768 (1536) 262 / 280 us, 3000 x 768 x 3072 (564) 350 / 366 us, 4096 x 1024 x 4096 (1024)
// 878 / 843 us.
static bool aloneF32(int64_t tiles, int64_t kBlocks)
{
    if (kBlocks < 2048 / kTileK)
        return tiles >= 17 * smCount() / 5;
    int64_t const wave = static_cast<int64_t>(kFcF32CtasPerSm) * smCount();
    return 10 * tiles >= 9 * ((tiles + wave - 1) / wave * wave);
}

int32_t fcF32Simt(bert_b200_fc_params const& p, cudaStream_t stream)
{
    int64_t const mTiles = (p.m + kTile - 1) / kTile;
    int64_t const nTiles = (p.n + kTile - 1) / kTile;
    int64_t const kBlocks = (p.k + kTileK - 1) / kTileK;
    bool const vec = p.k % 4 == 0 && p.lda % 4 == 0 && aligned16(p.a) && aligned16(p.wt);
    int const segments = segmentsF32(kBlocks);
    bool const alone = segments == 1 || aloneF32(mTiles * nTiles, kBlocks);
    int const ctas = alone ? 1 : segments; // per tile
    B200_REQUIRE(mTiles * nTiles * ctas < (1ll << 31), "fc (FP32): m=%lld, n=%lld too large", static_cast<long long>(p.m), static_cast<long long>(p.n));
    FcF32Args const args{p.m, p.n, p.k, static_cast<float const*>(p.a), p.lda, static_cast<float const*>(p.wt), static_cast<float*>(p.c), p.ldc,
        p.bias, p.activation, p.alpha, static_cast<int32_t>(nTiles), segments};
    size_t const smem = sizeof(float) * (kFcF32Ring + (alone && segments > 1 ? kFcF32Part : 0));
    auto const kernel = alone ? (vec ? fcF32Kernel<4, true> : fcF32Kernel<1, true>) : (vec ? fcF32Kernel<4, false> : fcF32Kernel<1, false>);
    static SmemOptIn optIn[2];
    cudaError_t const e = launchDependentCluster(alone ? &optIn[vec] : nullptr, kernel, dim3(static_cast<unsigned>(mTiles * nTiles * ctas)),
        dim3(kFcF32Threads), smem, stream, ctas, args);
    if (e != cudaSuccess)
        B200_FAIL(BERT_B200_CUDA_ERROR, "fcF32Kernel: %s", cudaGetErrorString(e));
    return checkLaunch("fcF32Kernel");
}

namespace
{

// perSm: how many CTAs may share an SM (0: as many as fit), by the shared memory that is asked for.
template <typename T, int D, int WARPS, bool ASYNC, bool SKIP>
int32_t launchMhaTiled(bert_b200_mha_params const& p, int perSm, cudaStream_t stream)
{
    int32_t const rowBlocks = (p.S - 1) / (16 * WARPS) + 1;
    B200_REQUIRE(rowBlocks <= 65535, "mha (SIMT): S=%d too large", p.S); // the grid's third dimension
    constexpr size_t kSmem = sizeof(AttSmem<D, WARPS>), kSm = 227 * 1024;
    size_t const share = perSm > 0 ? kSm / perSm - 2048 : 0;
    static SmemOptIn optIn;
    cudaError_t const e = launchDependentCluster(&optIn, mhaTiledKernel<T, D, WARPS, ASYNC, SKIP>, dim3(p.num_heads, p.B, rowBlocks),
        dim3(32 * WARPS), share > kSmem ? share : kSmem, stream, 1, p.B, p.S, p.num_heads, p.head_size, static_cast<T const*>(p.qkv),
        static_cast<T*>(p.out), p.cu_seqlens, p.mask_idx, p.scale_bmm1);
    if (e != cudaSuccess)
        B200_FAIL(BERT_B200_CUDA_ERROR, "mhaTiledKernel: %s", cudaGetErrorString(e));
    return checkLaunch("mhaTiledKernel");
}

template <typename T, int D>
int32_t launchMhaTiled(bert_b200_mha_params const& p, cudaStream_t stream)
{
    if constexpr (sizeof(T) == 4 && D <= 64)
    {
        bool const full = p.cu_seqlens != nullptr ? p.total == static_cast<int64_t>(p.B) * p.S : p.mask_idx == nullptr;
        AttPlan const plan = planAtt(p.B, p.num_heads, p.S, D, full, smCount());
        if (plan.rows == 32)
            return launchMhaTiled<T, D, 2, true, true>(p, plan.perSm, stream);
        if constexpr (D == 64)
        {
            if (plan.async)
                return launchMhaTiled<T, D, 4, true, true>(p, plan.perSm, stream);
            if (!plan.skip)
                return launchMhaTiled<T, D, 4, false, false>(p, plan.perSm, stream);
        }
        return launchMhaTiled<T, D, 4, false, true>(p, plan.perSm, stream);
    }
    else
        return launchMhaTiled<T, D, 4, false, false>(p, 0, stream);
}

template <typename T>
int32_t launchMhaSimt(bert_b200_mha_params const& p, cudaStream_t stream)
{
    uintptr_t const bits = reinterpret_cast<uintptr_t>(p.qkv) | reinterpret_cast<uintptr_t>(p.out);
    if (p.head_size % 4 == 0 && p.head_size <= 128 && bits % (4 * sizeof(T)) == 0)
        return p.head_size <= 32 ? launchMhaTiled<T, 32>(p, stream)
            : p.head_size <= 64  ? launchMhaTiled<T, 64>(p, stream)
            : p.head_size <= 96  ? launchMhaTiled<T, 96>(p, stream)
                                 : launchMhaTiled<T, 128>(p, stream);
    size_t const smem = 4 * static_cast<size_t>(p.S + p.head_size) * sizeof(float);
    B200_REQUIRE(smem <= 200 * 1024, "mha (SIMT): S=%d with head size %d does not fit shared memory", p.S, p.head_size);
    auto kernel = mhaSimtKernel<T>;
    if (smem > 48 * 1024)
    {
        static SmemOptIn optIn;
        cudaError_t const e = optIn.set(kernel, smem, true);
        if (e != cudaSuccess)
            B200_FAIL(BERT_B200_CUDA_ERROR, "mha (SIMT): cudaFuncSetAttribute: %s", cudaGetErrorString(e));
    }
    int const z = (p.S + 3) / 4 < 32 ? (p.S + 3) / 4 : 32;
    dim3 const grid(p.num_heads, p.B, z > 0 ? z : 1);
    kernel<<<grid, 128, smem, stream>>>(p.B, p.S, p.num_heads, p.head_size, static_cast<T const*>(p.qkv),
        static_cast<T*>(p.out), p.cu_seqlens, p.mask_idx, p.scale_bmm1);
    return checkLaunch("mhaSimtKernel");
}

} // namespace

// FP32 always; FP16 for the shapes outside the tensor-core kernel.
int32_t mhaSimt(bert_b200_mha_params const& p, cudaStream_t stream)
{
    B200_REQUIRE(!p.interleaved, "mha (SIMT): the interleaved layout is INT8 only");
    return p.type_id == BERT_B200_FP16 ? launchMhaSimt<__half>(p, stream) : launchMhaSimt<float>(p, stream);
}

} // namespace b200
