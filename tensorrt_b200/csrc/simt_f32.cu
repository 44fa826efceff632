// FP32 (type_id 0) fully-connected and attention kernels. FP32 has no tensor-core path that keeps
// full precision (TF32 would break the 1e-5 tolerance the reference configuration states for FP32,
// plugin/bertQKVToContextPlugin/CustomQKVToContextPluginDynamic_PluginConfig.yaml:72-76), so these
// are SIMT kernels; the FP16 / INT8 paths live in fc_tcgen05.cu and mha_tcgen05.cu.
// The attention kernel also serves FP16 tensors (FP32 arithmetic) for the shapes the tensor-core kernel does not
// take - heads wider than 64 or not a multiple of 16, sequences longer than 512 - the shapes the reference sends
// to its unfused runner as well.
//
// Replaces cublas{S,H}gemmStridedBatched + softmax kernels of UnfusedMHARunner::run
// (plugin/bertQKVToContextPlugin/mhaRunner.cu:533-601) and the FP32 cublasLtMatmul of the FC plugin
// (plugin/fcPlugin/fcPlugin.cpp:551-610).
#include "common.cuh"

namespace b200
{

namespace
{

__device__ __forceinline__ float geluErf(float x)
{
    return 0.5f * x * (1.f + erff(x * 0.70710678118654752440f));
}

// ---- fully connected ------------------------------------------------------------------------------------------------
// C[m,n] = act(alpha * sum_k A[m,k] * Wt[n,k] + bias[n]).
//
// Bound by the FP32 FMA pipes (128 per clock and SM). A CTA of two warps computes a 64 x 64 tile, every thread 8 x 8
// outputs, four CTAs per SM. Both operands are K-contiguous, so they are copied to shared memory as they lie (16-byte
// cp.async, four stages) and read back as 8-byte pieces along K, those of the next two k during the FMAs of these (16-byte
// pieces left no registers for that: 3 % slower); rows are padded to 20 floats, which puts the 4 or 8 rows that a warp reads
// at once into different banks. The sums run on packed fma.rn.f32x2: one half takes the even k, the
// other the odd ones (no operand has to be duplicated), and the two are added at the end; a packed FMA takes half the
// issue slots, which leaves room for the loads. These bring 64 bytes per thread and k pair to the registers, at 128 bytes per
// clock and SM as long as the FMAs take: the loop runs at 0.6 of the FMA rate.
// A cluster of `split` CTAs divides the K range of a tile where the tiles alone leave SMs idle or fill the last wave badly;
// its CTAs exchange partial sums through distributed shared memory, each finishing every split-th row.
// Measured: 1024 x 2304 x 768 in 96 us (38 TFLOP/s; a 4 x 4-per-thread kernel with scalar copies took 195 us), 1024 x 768 x
// 3072 in 141 us (700 us).
constexpr int kTile = 64;
constexpr int kTileK = 16;
constexpr int kPitch = kTileK + 4; // floats
constexpr int kStages = 4;
constexpr int kFcF32Threads = 64;
constexpr int kFcF32CtasPerSm = 4;

__device__ __forceinline__ void fma2(uint64_t& c, uint64_t a, uint64_t b)
{
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
}

__device__ __forceinline__ float sumPair(uint64_t v)
{
    return __uint_as_float(static_cast<uint32_t>(v)) + __uint_as_float(static_cast<uint32_t>(v >> 32));
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
    int32_t nTiles; // tiles along N
    int32_t split;  // CTAs per tile = cluster size
};

__device__ __forceinline__ float fcF32Epilogue(FcF32Args const& p, float v, int64_t n)
{
    v = v * p.alpha + (p.bias ? p.bias[n] : 0.f);
    return p.act == BERT_B200_ACT_GELU_ERF ? geluErf(v) : v;
}

// kVec: floats per copy (4, or 1 where K, lda or an address is not a multiple of 16 bytes)
template <int kVec>
__global__ void __launch_bounds__(kFcF32Threads, kFcF32CtasPerSm) fcF32Kernel(FcF32Args const p)
{
    __shared__ __align__(16) float sm[kStages][2][kTile][kPitch];
    static_assert(sizeof(sm) >= kTile * kTile * sizeof(float), "partial sums reuse the ring");
    int const tid = threadIdx.x;
    int const lane = tid & 31;
    int const ty = lane >> 3;
    int const tx = lane & 7;
    int const row0 = (tid >> 5) * 32 + ty; // rows row0 + 4 i, columns tx + 8 j
    int const rank = static_cast<int>(blockIdx.x % p.split);
    int64_t const tile = blockIdx.x / p.split;
    int64_t const m0 = tile / p.nTiles * kTile;
    int64_t const n0 = tile % p.nTiles * kTile;
    int64_t const kBlocks = (p.K + kTileK - 1) / kTileK;
    int const kbFirst = static_cast<int>(kBlocks * rank / p.split);
    int const kbEnd = static_cast<int>(kBlocks * (rank + 1) / p.split);

    gridDependencyLaunch();
    gridDependencyWait();

    uint32_t const smBase = static_cast<uint32_t>(__cvta_generic_to_shared(&sm[0][0][0][0]));
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
    for (int kb = kbFirst; kb < kbEnd; ++kb)
    {
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
                    fma2(acc[i][j], av[cur][i], bv[cur][j]);
        }
        stage = stage + 1 == kStages ? 0 : stage + 1;
    }
    if (p.split == 1)
    {
#pragma unroll
        for (int i = 0; i < 8; ++i)
        {
            int64_t const m = m0 + row0 + 4 * i;
#pragma unroll
            for (int j = 0; j < 8; ++j)
            {
                int64_t const n = n0 + tx + 8 * j;
                if (m < p.M && n < p.N)
                    p.C[m * p.ldc + n] = fcF32Epilogue(p, sumPair(acc[i][j]), n);
            }
        }
        return;
    }
    cpAsyncWait<0>();
    __syncthreads();
    float* const part = &sm[0][0][0][0];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j)
            part[(row0 + 4 * i) * kTile + tx + 8 * j] = sumPair(acc[i][j]);
    clusterBarrier();
    int const rows = static_cast<int>(p.M - m0 < kTile ? p.M - m0 : kTile);
    int64_t const n = n0 + tid; // one column per thread, every split-th row
    for (int r = rank; r < rows; r += p.split)
    {
        float v = 0.f;
        for (int q = 0; q < p.split; ++q)
            v += ldSharedCluster(part + r * kTile + tid, q);
        if (n < p.N)
            p.C[(m0 + r) * p.ldc + n] = fcF32Epilogue(p, v, n);
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

// 64 queries of one (sequence, head) per CTA against blocks of 64 keys, running maximum and sum per row.
//
// Bound by the FP32 pipes and the shared-memory loads that feed them. Every warp owns 16 query rows, so its scores,
// probabilities and row sums are its own business (a warp-level sync between the two products); a thread computes 4 rows x
// 8 keys of the scores with 16-byte loads along d (packed FMAs, even and odd channels apart, as in the FC above), and 4
// rows x D / 8 columns of the context. Rows are padded by 4 floats against bank conflicts. Measured: 8 sequences of 128
// tokens, 12 heads of 64 channels in 26 us (a warp per query row, keys and values from global memory: 509 us).
constexpr int kAttRows = 64;
constexpr int kAttKeys = 64;
constexpr int kAttThreads = 128;

template <int D> // head size rounded up to 32, 64, 96 or 128; channels beyond d are zero
struct AttSmem
{
    float q[kAttRows][D + 4];
    float k[kAttKeys][D + 4];
    float v[kAttKeys][D];
    float p[kAttRows][kAttKeys + 4];
};

template <typename T, int D>
__global__ void __launch_bounds__(kAttThreads) mhaTiledKernel(int32_t const B, int32_t const S, int32_t const N, int32_t const d,
    T const* __restrict__ qkv, T* __restrict__ out, int32_t const* __restrict__ cu, int32_t const* __restrict__ maskIdx, float const scale)
{
    extern __shared__ float smRaw[];
    AttSmem<D>& sm = *reinterpret_cast<AttSmem<D>*>(smRaw);
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
        *reinterpret_cast<float4*>(&sm.q[r][c]) = ok ? load4(base + (q0 + r) * rowStep + c) : zero;
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
                    fma2(acc[i][j], a[i].x, b.x);
                    fma2(acc[i][j], a[i].y, b.y);
                }
            }
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
        __syncwarp();
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

// CTAs per tile: the smallest of 1, 2, 4, 8 that gives the SMs nearly all the CTAs that fit at once; with a long K (2048 and more
// per CTA) twice as many, so that the last ones do not run alone for long. Other cluster sizes leave SMs idle (clusters of three:
// some SMs none, others four); fewer CTAs leave FMA pipes idle, more exchange partial sums for nothing. Measured with 1 / 2 / 4 / 8
// per tile: 1024 x 768 x 3072 (192 tiles) 273 / 183 / 141 / 147 us (three: 184), 1024 x 3072 x 768 (768 tiles) 139 / 149 / 151 us,
// 128 x 768 x 3072 (24 tiles) 182 / 100 / 52 / 44 us, 4096 x 1024 x 4096 (1024 tiles) 890 / 780 us.
static int pickSplitF32(int64_t tiles, int64_t kBlocks)
{
    int split = 1;
    while (split < 8 && 2 * split <= kBlocks)
    {
        int64_t const enough = kBlocks / split >= 2048 / kTileK ? 8 * smCount() : 17 * smCount() / 5;
        if (tiles * split >= enough)
            break;
        split *= 2;
    }
    return split;
}

int32_t fcF32(bert_b200_fc_params const& p, cudaStream_t stream)
{
    int64_t const mTiles = (p.m + kTile - 1) / kTile;
    int64_t const nTiles = (p.n + kTile - 1) / kTile;
    bool const vec = p.k % 4 == 0 && p.lda % 4 == 0 && aligned16(p.a) && aligned16(p.wt);
    int const split = pickSplitF32(mTiles * nTiles, (p.k + kTileK - 1) / kTileK);
    B200_REQUIRE(mTiles * nTiles * split < (1ll << 31), "fc (FP32): m=%lld, n=%lld too large", static_cast<long long>(p.m), static_cast<long long>(p.n));
    FcF32Args const args{p.m, p.n, p.k, static_cast<float const*>(p.a), p.lda, static_cast<float const*>(p.wt), static_cast<float*>(p.c), p.ldc,
        p.bias, p.activation, p.alpha, static_cast<int32_t>(nTiles), split};
    cudaError_t const e = launchDependentCluster(nullptr, vec ? fcF32Kernel<4> : fcF32Kernel<1>, dim3(static_cast<unsigned>(mTiles * nTiles * split)),
        dim3(kFcF32Threads), 0, stream, split, args);
    if (e != cudaSuccess)
        B200_FAIL(BERT_B200_CUDA_ERROR, "fcF32Kernel: %s", cudaGetErrorString(e));
    return checkLaunch("fcF32Kernel");
}

namespace
{

template <typename T, int D>
int32_t launchMhaTiled(bert_b200_mha_params const& p, cudaStream_t stream)
{
    static SmemOptIn optIn;
    cudaError_t const e = launchDependentCluster(&optIn, mhaTiledKernel<T, D>, dim3(p.num_heads, p.B, (p.S + kAttRows - 1) / kAttRows),
        dim3(kAttThreads), sizeof(AttSmem<D>), stream, 1, p.B, p.S, p.num_heads, p.head_size, static_cast<T const*>(p.qkv),
        static_cast<T*>(p.out), p.cu_seqlens, p.mask_idx, p.scale_bmm1);
    if (e != cudaSuccess)
        B200_FAIL(BERT_B200_CUDA_ERROR, "mhaTiledKernel: %s", cudaGetErrorString(e));
    return checkLaunch("mhaTiledKernel");
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
