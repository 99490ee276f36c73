// Learned surrogate of the absorption factor: an ensemble of small MLPs that
// map (omega, incident and diffracted unit vectors in the crystal frame) to
// log A_h, trained on the GPU on absorption factors the plain tracer computes.
//
// Network (per ensemble member): 7 inputs -> 64 Fourier features
// [sin 2pi(Bx), cos 2pi(Bx)] with a fixed seeded B (32 x 7; its omega column
// is integer so the features are periodic in omega) -> 4 hidden layers of 256
// with GELU -> 1 output, the standardised log A_h.  Weights are FP32 masters
// with BF16 copies in [out][in] and [in][out] order; every matrix product is a
// tcgen05 BF16 GEMM with FP32 accumulation in tensor memory (umma_gemm.cuh),
// all members in one launch.  Training is Adam on the mean squared error with
// hand-written forward, backward and optimiser kernels; one training step is
// captured in a CUDA graph and replayed.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <new>
#include <random>
#include <vector>

#include "anacor_gb300.h"
#include "anacor_internal.h"
#include "gelu.cuh"
#include "umma_gemm.cuh"

namespace anacor {
int report_status(int st, const char *msg);
}

using namespace anacor;
using bf16 = __nv_bfloat16;

namespace {

constexpr int kIn = 7;        // omega + two unit vectors
constexpr int kFeat = 64;     // Fourier features
constexpr int kWidth = 256;
constexpr int kDepth = 4;     // hidden layers

// parameter offsets of one member (FP32 masters)
__host__ __device__ constexpr long long off_w(int l) { return l == 0 ? 0 : 16640 + (long long)(l - 1) * 65792; }
__host__ __device__ constexpr long long off_b(int l) { return off_w(l) + (long long)kWidth * (l == 0 ? kFeat : kWidth); }
constexpr long long kOffW5 = 214016;
constexpr long long kOffB5 = 214272;
constexpr long long kParams = 214280;   // per member, padded to a multiple of 8
__host__ __device__ constexpr int in_dim(int l) { return l == 0 ? kFeat : kWidth; }
static_assert(off_b(3) + kWidth == kOffW5, "parameter layout");

constexpr int kSplitK = 16;             // K splits of the weight-gradient GEMMs
constexpr int kMaxMembers = 16;
constexpr int kPredictChunk = 1 << 18;  // rows per inference pass

enum Epi { kEpiStoreF32 = 0, kEpiBiasGelu = 1 };

struct GemmArgs {
    const bf16 *A;
    long long lda, sA;
    const bf16 *B;
    long long ldb, sB;
    int M, N, K;
    int ksplit;            // z = member * ksplit + split; 0 or 1 = no split
    int mode;
    const float *bias;
    long long sBias;
    float *of;             // fp32 [M][N]  (with ksplit > 1: one slice per z)
    long long ldf, sF;
    bf16 *ob;              // bf16 [M][N]
    long long ldob, sOb;
    int *err;
};

// Stage one K-chunk of 64 of A (128 rows) and B (BN rows) into the canonical
// no-swizzle K-major tile layout with 16-byte cp.async copies.
template <int BN>
__device__ __forceinline__ void load_chunk(uint8_t *As, uint8_t *Bs, const bf16 *A, long long lda, const bf16 *B,
                                           long long ldb, int k0)
{
    for (int c = threadIdx.x; c < umma::kBM * 8; c += umma::kThreads) {
        const int r = c >> 3, kc = c & 7;
        umma::cp_async16(As + umma::tile_off(r, kc * 8), A + (long long)r * lda + k0 + kc * 8);
    }
    for (int c = threadIdx.x; c < BN * 8; c += umma::kThreads) {
        const int r = c >> 3, kc = c & 7;
        umma::cp_async16(Bs + umma::tile_off(r, kc * 8), B + (long long)r * ldb + k0 + kc * 8);
    }
    umma::cp_async_commit();
}

// One 128 x BN tile per CTA, two shared-memory stages: the copy of chunk k+1
// overlaps the tensor-core work on chunk k.  A stage is refilled only after
// the MMAs that read it have signalled their mbarrier.
template <int BN>
__global__ void __launch_bounds__(umma::kThreads, 1) gemm_kernel(GemmArgs g)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    constexpr int kStageA = umma::kBM * umma::kBK * 2, kStageB = BN * umma::kBK * 2;
    __shared__ uint64_t bar[2];
    __shared__ uint32_t tslot;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int ks = g.ksplit > 1 ? g.ksplit : 1;
    const int z = blockIdx.z, e = z / ks, sp = z - e * ks;
    const int Kc = g.K / ks;
    const int m0 = blockIdx.y * umma::kBM, n0 = blockIdx.x * BN;
    const bf16 *A = g.A + e * g.sA + (long long)m0 * g.lda + (long long)sp * Kc;
    const bf16 *B = g.B + e * g.sB + (long long)n0 * g.ldb + (long long)sp * Kc;
    constexpr int kStage = kStageA + kStageB;   // stage s: A at s * kStage, B after it

    if (tid == 0) {
        umma::mbar_init(&bar[0], 1);
        umma::mbar_init(&bar[1], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0)
        umma::tmem_alloc(&tslot, BN);
    umma::tc_fence_before();
    __syncthreads();
    umma::tc_fence_after();
    const uint32_t tmem = tslot;
    constexpr uint32_t idesc = umma::idesc_bf16_f32(BN);

    const int nk = Kc / umma::kBK;
    uint32_t phase[2] = {0u, 0u};
    bool ok = true;
    load_chunk<BN>(smem, smem + kStageA, A, g.lda, B, g.ldb, 0);
    for (int k = 0; k < nk; k++) {
        const int s = k & 1;
        umma::cp_async_wait_all();
        umma::fence_async_smem();
        __syncthreads();
        if (tid == 0) {
            umma::tc_fence_after();
            const uint32_t a0 = umma::smem_u32(smem + s * kStage), b0 = a0 + kStageA;
#pragma unroll
            for (int kk = 0; kk < umma::kBK / 16; kk++) {
                const uint64_t ad = umma::smem_desc(a0 + kk * 256, 128, 1024);
                const uint64_t bd = umma::smem_desc(b0 + kk * 256, 128, 1024);
                umma::mma_bf16(tmem, ad, bd, idesc, (k > 0 || kk > 0) ? 1u : 0u);
            }
            umma::mma_commit(&bar[s]);
        }
        if (k + 1 < nk) {
            const int t = s ^ 1;
            if (k >= 1) {   // stage t was read by the MMAs of chunk k-1
                ok = umma::mbar_wait(&bar[t], phase[t]) && ok;
                phase[t] ^= 1u;
            }
            load_chunk<BN>(smem + t * kStage, smem + t * kStage + kStageA, A, g.lda, B, g.ldb, (k + 1) * umma::kBK);
        }
    }
    // the last commit covers every MMA issued before it
    ok = umma::mbar_wait(&bar[(nk - 1) & 1], phase[(nk - 1) & 1]) && ok;
    umma::tc_fence_after();
    ok = __all_sync(0xffffffffu, ok);
    if (!ok) {
        if (lane == 0)
            atomicOr(g.err, 1);
    } else {
        const int row = m0 + warp * 32 + lane;
        const long long zo = ks > 1 ? z : e;
        for (int c0 = 0; c0 < BN; c0 += 16) {
            float v[16];
            uint32_t t[8];   // 16 BF16
            umma::tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c0, v);
            const int n = n0 + c0;
            if (g.mode == kEpiStoreF32) {
                float *o = g.of + zo * g.sF + (long long)row * g.ldf + n;
#pragma unroll
                for (int i = 0; i < 16; i += 4)
                    *reinterpret_cast<float4 *>(o + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
                continue;
            }
            gelu::values_bf16<8>(v, g.bias + e * g.sBias + n, t);
            bf16 *o = g.ob + e * g.sOb + (long long)row * g.ldob + n;
            *reinterpret_cast<uint4 *>(o) = make_uint4(t[0], t[1], t[2], t[3]);
            *reinterpret_cast<uint4 *>(o + 8) = make_uint4(t[4], t[5], t[6], t[7]);
        }
    }
    umma::tc_fence_before();
    __syncthreads();
    if (warp == 0)
        umma::tmem_dealloc(tmem, BN);
}

constexpr int gemm_smem(int bn) { return 2 * (umma::kBM + bn) * umma::kBK * 2; }

std::once_flag g_gemm_once[64];
cudaError_t g_gemm_init_err[64];

// opt every tile width into its shared-memory size once per device (outside
// any stream capture)
cudaError_t gemm_init()
{
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e)
        return e;
    if (dev < 0 || dev >= 64)
        return cudaErrorInvalidDevice;
    std::call_once(g_gemm_once[dev], [dev] {
        cudaError_t r = cudaFuncSetAttribute(gemm_kernel<256>, cudaFuncAttributeMaxDynamicSharedMemorySize, gemm_smem(256));
        if (!r)
            r = cudaFuncSetAttribute(gemm_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, gemm_smem(128));
        if (!r)
            r = cudaFuncSetAttribute(gemm_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, gemm_smem(64));
        g_gemm_init_err[dev] = r;
    });
    return g_gemm_init_err[dev];
}

// tile width: the widest that still gives at least one CTA per SM
int pick_bn(int M, int N, int zcount)
{
    const int tiles_m = M / umma::kBM;
    for (int bn : {256, 128})
        if (N % bn == 0 && (long long)(N / bn) * tiles_m * zcount >= 148)
            return bn;
    if (N % 128 == 0)
        return 128;
    return N % 64 == 0 ? 64 : 0;
}

cudaError_t gemm(const GemmArgs &g, int members, cudaStream_t st)
{
    const int ks = g.ksplit > 1 ? g.ksplit : 1;
    if (g.M % umma::kBM || g.K % (umma::kBK * ks))
        return cudaErrorInvalidValue;
    const int bn = pick_bn(g.M, g.N, members * ks);
    if (!bn)
        return cudaErrorInvalidValue;
    dim3 grid(g.N / bn, g.M / umma::kBM, members * ks);
    if (bn == 256)
        gemm_kernel<256><<<grid, umma::kThreads, gemm_smem(256), st>>>(g);
    else if (bn == 128)
        gemm_kernel<128><<<grid, umma::kThreads, gemm_smem(128), st>>>(g);
    else
        gemm_kernel<64><<<grid, umma::kThreads, gemm_smem(64), st>>>(g);
    return cudaGetLastError();
}

// ------------------------------------------------------------ small kernels

struct Geometry {
    double xray[3], axis[3], F[9];
};

// x7 = (omega / 2pi wrapped to [0, 1), incident and diffracted unit vectors
// in the crystal frame).  The rotation is T = (R(axis, omega) F)^T as the
// reference builds it (AnACor/src/ray_tracing.c:397-407, matrices.h:49-68).
__global__ void inputs_kernel(const double *__restrict__ omega, const double *__restrict__ s1, long long n,
                              Geometry geo, float *__restrict__ x7)
{
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    const double w = omega[i];
    double c, s;
    sincos(w, &s, &c);
    const double x = geo.axis[0], y = geo.axis[1], z = geo.axis[2], k = 1.0 - c;
    const double R[9] = {c + x * x * k,      x * y * k - z * s, y * s + x * z * k,
                         z * s + x * y * k,  c + y * y * k,     -x * s + y * z * k,
                         -y * s + x * z * k, x * s + y * z * k, c + z * z * k};
    double M[9];
#pragma unroll
    for (int r = 0; r < 3; r++)
#pragma unroll
        for (int q = 0; q < 3; q++)
            M[r * 3 + q] = R[r * 3 + 0] * geo.F[q] + R[r * 3 + 1] * geo.F[3 + q] + R[r * 3 + 2] * geo.F[6 + q];
    double a[3], b[3];
    const double *sv = s1 + 3 * i;
#pragma unroll
    for (int r = 0; r < 3; r++) {   // T = M^T
        a[r] = M[r] * geo.xray[0] + M[3 + r] * geo.xray[1] + M[6 + r] * geo.xray[2];
        b[r] = M[r] * sv[0] + M[3 + r] * sv[1] + M[6 + r] * sv[2];
    }
    const double na = rsqrt(a[0] * a[0] + a[1] * a[1] + a[2] * a[2]);
    const double nb = rsqrt(b[0] * b[0] + b[1] * b[1] + b[2] * b[2]);
    float *o = x7 + 7 * i;
    const double turns = w * 0.15915494309189535;
    o[0] = (float)(turns - floor(turns));
#pragma unroll
    for (int r = 0; r < 3; r++) {
        o[1 + r] = (float)(a[r] * na);
        o[4 + r] = (float)(b[r] * nb);
    }
}

// Fourier features of rows 0..n-1 (rows n..rows_pad-1 are written as zeros)
__global__ void features_kernel(const float *__restrict__ x7, const float *__restrict__ Bf, long long n,
                                long long rows_pad, bf16 *__restrict__ out)
{
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const long long i = t / (kFeat / 2);
    const int j = (int)(t % (kFeat / 2));
    if (i >= rows_pad)
        return;
    float sv = 0.0f, cv = 0.0f;
    if (i < n) {
        const float *x = x7 + 7 * i;
        float p = 0.0f;
#pragma unroll
        for (int q = 0; q < kIn; q++)
            p += Bf[j * kIn + q] * x[q];
        sincospif(2.0f * p, &sv, &cv);
    }
    out[i * kFeat + j] = __float2bfloat16_rn(sv);
    out[i * kFeat + kFeat / 2 + j] = __float2bfloat16_rn(cv);
}

__device__ __forceinline__ uint32_t mix32(uint32_t x)
{
    x ^= x >> 16;
    x *= 0x7feb352dU;
    x ^= x >> 15;
    x *= 0x846ca68bU;
    x ^= x >> 16;
    return x;
}

// output layer, one warp per row: y = A4 . w5 + b5
__global__ void head_kernel(const bf16 *__restrict__ A4, const float *__restrict__ params, int rows,
                            float *__restrict__ y)
{
    const int e = blockIdx.y;
    const int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (r >= rows)
        return;
    const float *P = params + e * kParams;
    const long long base = (long long)e * rows + r;
    const uint4 av = reinterpret_cast<const uint4 *>(A4 + base * kWidth)[lane];
    const bf16 *a = reinterpret_cast<const bf16 *>(&av);
    float acc = 0.0f;
#pragma unroll
    for (int q = 0; q < 8; q++)
        acc += __bfloat162float(a[q]) * P[kOffW5 + lane * 8 + q];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0)
        y[base] = acc + P[kOffB5];
}

// ensemble mean of A_h = exp(mu + sd * y) and its relative spread (standard
// deviation over members / mean)
__global__ void ensemble_kernel(const float *__restrict__ y, int E, long long rows, long long ld, float mu, float sd,
                                float *__restrict__ mean, float *__restrict__ spread, float *__restrict__ members,
                                long long ldm)
{
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= rows)
        return;
    // two passes (mean, then squared deviations): the members agree to
    // ~1e-3, so a one-pass E[a^2] - E[a]^2 would cancel away the spread
    float a[kMaxMembers];
    float s = 0.0f;
#pragma unroll
    for (int e = 0; e < kMaxMembers; e++) {
        if (e < E) {
            const float la = mu + sd * y[e * ld + i];
            if (members)
                members[e * ldm + i] = la;
            a[e] = expf(la);
            s += a[e];
        }
    }
    const float m = s / E;
    float v = 0.0f;
#pragma unroll
    for (int e = 0; e < kMaxMembers; e++)
        if (e < E)
            v += (a[e] - m) * (a[e] - m);
    mean[i] = m;
    spread[i] = sqrtf(v / E) / m;
}

// audit flags: bit 0 = in the seeded random audit sample, bit 1 = ensemble
// spread above the threshold (or not finite)
__global__ void audit_kernel(const float *__restrict__ spread, long long n, uint32_t seed, uint32_t cut,
                             float threshold, uint8_t *__restrict__ flags)
{
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    const uint32_t h = mix32(seed ^ mix32((uint32_t)i ^ mix32((uint32_t)(i >> 32) + 0x632BE5ABu)));
    const float sp = spread[i];
    flags[i] = (uint8_t)((h < cut ? 1u : 0u) | (!(sp <= threshold) ? 2u : 0u));
}

// ------------------------------------------------- fused inference kernel
//
// The four hidden layers and the head of every member for a 128-row tile in
// one persistent kernel: the tile's Fourier features and each layer's
// activations stay in shared memory, the accumulators in tensor memory, and
// only the weights stream in (from L2: 1.7 MB for four members), as 16 KiB
// K-chunks copied by the bulk-copy engine (cp.async.bulk) into a 4-stage ring.
//
// Two members are in flight at a time, on two "streams" with their own
// 256-column TMEM accumulator and 128 x 256 activation tile: while the sixteen
// epilogue warps apply bias and GELU to one member's layer, the MMA warp issues
// the other member's MMAs (it never waits for one) and a copy warp keeps the
// weight ring full.  The streams hand over through mbarriers: acc_full[s] (the
// layer's MMAs are done), act_ready[s] (its epilogue has read the accumulator
// and written the next operand), x0_ready (a tile's features, which are
// computed while the tile before it is still in its last layers).  An epilogue
// warp owns 32 rows x 64 columns of every layer and loads the next 16 columns
// from tensor memory while it works on the last; warps meet only around the
// head's sums, in groups of four.  (Eight warps for each stream instead: 10 %
// slower, a stream's MMAs leave the other's eight too little to fill the SM.)
//
// What bounds it is the epilogue: alone it takes 2.9 of the 3.2 ms for a
// million rows x 4 members (18 instructions a value, issue slots at 61 %, FMA
// pipe at 52 %); the MMAs alone with their hand-overs take 1.7 ms, the weight
// copies alone 1.3 ms (13.3 GB from L2).  Before the packed GELU, the copy
// warp of its own and the features ahead of time it took 5.95 ms.
//
// The arithmetic is the layered path's: the same MMAs in the same K order,
// the same epilogue values and the head's and ensemble's summation orders, so
// the outputs are the same numbers without the per-layer round trips through
// HBM.
//
// A call whose tiles leave more than half of the SMs idle runs each tile on a
// cluster of two, four or eight CTAs that share its members; their outputs
// meet in the first CTA's shared memory.

constexpr int kWChunkK = 32;                                          // K per weight chunk
constexpr int kChunkBytes = kWidth * kWChunkK * 2;                    // 256 rows x 32 BF16 = 16 KiB
constexpr int kChunksPerMember = (kFeat + (kDepth - 1) * kWidth) / kWChunkK;   // 2 + 3 * 8 = 26
constexpr int kInferStages = 4;
constexpr int kEpiWarps = 16;                                         // four per TMEM lane quarter
constexpr int kEpiThreads = 32 * kEpiWarps;
constexpr int kInferThreads = kEpiThreads + 64;                       // + the MMA and the copy warp
constexpr int kTileRows = umma::kBM;                                  // 128
constexpr int kActChunk = kTileRows * umma::kBK * 2;                 // 128 rows x 64 BF16 = 16 KiB
constexpr int kActBytes = (kWidth / umma::kBK) * kActChunk;          // 64 KiB
constexpr int kInferMaxMembers = 8;
constexpr int kOffInferAct = kInferStages * kChunkBytes;             // two activation tiles
constexpr int kOffInferX0 = kOffInferAct + 2 * kActBytes;
constexpr int kOffInferY = kOffInferX0 + kActChunk;
constexpr int kInferSmem = kOffInferY + kInferMaxMembers * kTileRows * 4;
// The head's partial sums (32 per row) live in the stream's activation tile,
// which the last layer's MMAs have finished reading when the head writes them:
// each TMEM lane quarter's in the bytes of its own 32 rows of the first
// K-chunk, so that the only warps that write there next are the quarter's.
constexpr int kQuarterBytes = 32 * 32 * 4;
static_assert(kQuarterBytes == 4 * 1024, "a quarter's rows of a K-chunk");
static_assert(kInferSmem + 512 <= 227 * 1024, "fused inference shared memory");
static_assert(kEpiWarps / 4 * 64 == kWidth, "an epilogue warp owns 64 columns");

// byte offset of element (r, k) of a rows x 32 K-major weight chunk in the
// canonical no-swizzle layout (8-row groups 512 bytes apart)
__host__ __device__ constexpr uint32_t wchunk_off(int r, int k)
{
    return (uint32_t)(((r >> 3) * (kWChunkK / 8) + (k >> 3)) * 128 + (r & 7) * 16 + (k & 7) * 2);
}

// The work of one tile on E members as jobs (stream s, member e, layer l), in
// the order that the copy, MMA and epilogue warps take them: members
// in pairs (2p on stream 0, 2p + 1 on stream 1), layer by layer, alternating
// streams; an odd last member alone on stream 0.
__host__ __device__ inline void job_of(int j, int E, int &s, int &e, int &l)
{
    const int pairs = E / 2;
    if (j < pairs * 2 * kDepth) {
        const int p = j / (2 * kDepth), r = j % (2 * kDepth);
        l = r / 2;
        s = r % 2;
        e = 2 * p + s;
        return;
    }
    s = 0;
    e = E - 1;
    l = j - pairs * 2 * kDepth;
}

// the last job that reads the tile's features
__host__ __device__ inline int last_feature_job(int E)
{
    return E % 2 ? E / 2 * 2 * kDepth : (E / 2 - 1) * 2 * kDepth + 1;
}

__host__ __device__ constexpr int job_chunks(int l) { return in_dim(l) / kWChunkK; }

// index of K-chunk kq of layer l of member e in the weight image
__host__ __device__ constexpr int chunk_index(int e, int l, int kq)
{
    return e * kChunksPerMember + (l == 0 ? 0 : job_chunks(0) + (l - 1) * job_chunks(1)) + kq;
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(umma::smem_u32(bar)), "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t *bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(umma::smem_u32(bar)) : "memory");
}

// bulk copy of `bytes` (a multiple of 16, both addresses 16-byte aligned)
// from global to this CTA's shared memory, completing on `bar`
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, uint32_t bytes, uint64_t *bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     umma::smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(umma::smem_u32(bar))
                 : "memory");
}

// bounded wait that also gives up once another thread has aborted the CTA;
// a thread whose own wait runs out raises the abort flag
__device__ __forceinline__ bool wait_or_abort(uint64_t *bar, uint32_t parity, volatile int *abort)
{
    const uint32_t addr = umma::smem_u32(bar);
    for (unsigned it = 0; it < umma::kWaitLimit; it++) {
        uint32_t done;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(done)
            : "r"(addr), "r"(parity)
            : "memory");
        if (done)
            return true;
        if ((it & 255u) == 255u && *abort)
            return false;
    }
    *abort = 1;
    return false;
}

// barrier over the four epilogue warps of a TMEM lane quarter
__device__ __forceinline__ void quarter_sync(int quarter)
{
    asm volatile("bar.sync %0, 128;" ::"r"(1 + quarter) : "memory");
}

struct InferArgs {
    const float *x7;
    long long n;
    const float *Bf;
    const uint8_t *wimg;
    const float *params;
    int E;
    int share;   // CTAs of a cluster that share a tile's members (1: no cluster)
    float mu, sd;
    float *mean, *spread, *members;
    long long ldm;
    int *err;
};

// Fourier features of a tile (features_kernel's expressions), BF16 into the
// layer-0 operand tile; rows past n are zeros.  Thread t: row t / 4, eight
// frequencies.
__device__ __forceinline__ void tile_features(const InferArgs &a, long long row0, int t, uint8_t *X0s)
{
    const int r = t >> 2, h = t & 3;
    const long long i = row0 + r;
    float sv[8], cv[8];
#pragma unroll
    for (int jj = 0; jj < 8; jj++) {
        sv[jj] = 0.0f;
        cv[jj] = 0.0f;
    }
    if (i < a.n) {
        const float *x = a.x7 + 7 * i;
#pragma unroll
        for (int jj = 0; jj < 8; jj++) {
            const int j = 8 * h + jj;
            float p = 0.0f;
#pragma unroll
            for (int q = 0; q < kIn; q++)
                p += __ldg(a.Bf + j * kIn + q) * __ldg(x + q);
            sincospif(2.0f * p, &sv[jj], &cv[jj]);
        }
    }
    uint32_t u[4], w[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
        u[q] = gelu::bf16x2(sv[2 * q], sv[2 * q + 1]);
        w[q] = gelu::bf16x2(cv[2 * q], cv[2 * q + 1]);
    }
    *reinterpret_cast<uint4 *>(X0s + umma::tile_off(r, 8 * h)) = make_uint4(u[0], u[1], u[2], u[3]);
    *reinterpret_cast<uint4 *>(X0s + umma::tile_off(r, kFeat / 2 + 8 * h)) = make_uint4(w[0], w[1], w[2], w[3]);
    umma::fence_async_smem();
}

__global__ void __launch_bounds__(kInferThreads, 1) infer_kernel(InferArgs a)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ uint64_t full[kInferStages], empty[kInferStages], acc_full[2], act_ready[2], x0_ready;
    __shared__ uint32_t tslot;
    __shared__ int s_abort;
    uint8_t *Ws = smem;
    uint8_t *X0s = smem + kOffInferX0;
    float *ys = reinterpret_cast<float *>(smem + kOffInferY);
    volatile int *abort = &s_abort;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rank = a.share > 1 ? (int)(blockIdx.x % a.share) : 0;
    const long long first = blockIdx.x / a.share, step = gridDim.x / a.share;   // tiles of this CTA (cluster)
    const long long tiles = (a.n + kTileRows - 1) / kTileRows;
    const long long my_tiles = tiles > first ? (tiles - 1 - first) / step + 1 : 0;
    const int e0 = rank * a.E / a.share, E = (rank + 1) * a.E / a.share - e0;    // this CTA's members
    const int jobs = kDepth * E;

    if (tid == 0) {
        for (int s = 0; s < kInferStages; s++) {
            umma::mbar_init(&full[s], 1);
            umma::mbar_init(&empty[s], 1);
        }
        for (int s = 0; s < 2; s++) {
            umma::mbar_init(&acc_full[s], 1);
            umma::mbar_init(&act_ready[s], kEpiWarps);
        }
        umma::mbar_init(&x0_ready, kEpiWarps);
        s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0)
        umma::tmem_alloc(&tslot, 2 * kWidth);   // one accumulator per stream
    umma::tc_fence_before();
    __syncthreads();
    umma::tc_fence_after();
    const uint32_t tmem = tslot;
    if (a.share > 1) {   // the first CTA has started before its shared memory is written to
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }

    if (warp == kEpiWarps + 1) {
        // ---- copy warp: lane 0 streams the weight chunks in the order the
        // MMAs take them, each into its stage once the MMAs that read the
        // stage's previous chunk are done
        if (lane == 0) {
            const long long total = my_tiles * E * kChunksPerMember;
            int j = 0, kq = 0;
            long long q = 0;
            for (; q < total; q++) {
                const int st = (int)(q % kInferStages);
                if (q >= kInferStages && !wait_or_abort(&empty[st], (uint32_t)((q / kInferStages - 1) & 1), abort))
                    break;
                int s, e, l;
                job_of(j, E, s, e, l);
                mbar_expect_tx(&full[st], kChunkBytes);
                bulk_g2s(Ws + st * kChunkBytes, a.wimg + (long long)chunk_index(e0 + e, l, kq) * kChunkBytes,
                         kChunkBytes, &full[st]);
                if (++kq == job_chunks(l)) {
                    kq = 0;
                    j = j + 1 == jobs ? 0 : j + 1;
                }
            }
            // copies still in flight complete before the CTA's shared memory
            // goes away (bounded: a failed copy does not hold the exit)
            for (long long p = q > kInferStages ? q - kInferStages : 0; p < q; p++)
                wait_or_abort(&full[p % kInferStages], (uint32_t)((p / kInferStages) & 1), abort);
        }
        __syncwarp();
    } else if (warp == kEpiWarps) {
        // ---- MMA warp: lane 0 issues the MMAs and never waits for one
        if (lane == 0) {
            constexpr uint32_t idesc = umma::idesc_bf16_f32(kWidth);
            long long q = 0;
            uint32_t kjob[2] = {0u, 0u};
            bool ok = true;
            for (long long ti = 0; ti < my_tiles && ok; ti++) {
                for (int j = 0; j < jobs && ok; j++) {
                    int s, e, l;
                    job_of(j, E, s, e, l);
                    // the operand: the tile's features (layer 0) or the stream's
                    // previous epilogue, which also freed its accumulator
                    if (j == 0)
                        ok = wait_or_abort(&x0_ready, (uint32_t)(ti & 1), abort);
                    if (ok && kjob[s] > 0)
                        ok = wait_or_abort(&act_ready[s], (kjob[s] - 1u) & 1u, abort);
                    if (!ok)
                        break;
                    umma::tc_fence_after();
                    const uint8_t *A = l == 0 ? X0s : smem + kOffInferAct + s * kActBytes;
                    const int nk = job_chunks(l);
                    for (int kc = 0; kc < nk; kc++, q++) {
                        const int st = (int)(q % kInferStages);
                        if (!wait_or_abort(&full[st], (uint32_t)((q / kInferStages) & 1), abort)) {
                            ok = false;
                            break;
                        }
#pragma unroll
                        for (int kk = 0; kk < kWChunkK / 16; kk++) {
                            const int k0 = kc * kWChunkK + kk * 16;
                            const uint32_t a0 = umma::smem_u32(A + (k0 / umma::kBK) * kActChunk) +
                                                (uint32_t)((k0 % umma::kBK) / 16) * 256;
                            const uint32_t b0 = umma::smem_u32(Ws + st * kChunkBytes) + (uint32_t)kk * 256;
                            umma::mma_bf16(tmem + (uint32_t)(s * kWidth), umma::smem_desc(a0, 128, 1024),
                                           umma::smem_desc(b0, 128, 512), idesc, (kc > 0 || kk > 0) ? 1u : 0u);
                        }
                        umma::mma_commit(&empty[st]);
                    }
                    umma::mma_commit(&acc_full[s]);
                    kjob[s]++;
                }
            }
            if (!ok)
                *abort = 1;
        }
        __syncwarp();
    } else {
        // ---- epilogue warps: features, bias + GELU per layer, head, ensemble.
        // A warp whose wait runs out goes on through the loops without waiting
        // or writing, so that the others still meet it at the barriers.
        const int quarter = warp & 3;                   // TMEM lanes 32 * quarter ..
        const int rl = 32 * quarter + lane;             // this thread's row of the tile
        const int cb = 64 * (warp >> 2);                // its accumulator columns cb .. cb + 63
        const uint32_t lane_base = (uint32_t)(32 * quarter) << 16;
        const int jx0 = last_feature_job(E);
        uint32_t ejob[2] = {0u, 0u};
        bool ok = true;
        if (my_tiles > 0) {
            tile_features(a, first * kTileRows, tid, X0s);
            __syncwarp();
            if (lane == 0)
                mbar_arrive(&x0_ready);
        }
        for (long long ti = 0; ti < my_tiles; ti++) {
            const long long row0 = (first + ti * step) * kTileRows;
            for (int j = 0; j < jobs; j++) {
                int s, e, l;
                job_of(j, E, s, e, l);
                uint8_t *Act = smem + kOffInferAct + s * kActBytes;
                float *gs = reinterpret_cast<float *>(Act + quarter * kQuarterBytes) + 32 * lane;
                const float *P = a.params + (long long)(e0 + e) * kParams;
                const float *bias = P + off_b(l) + cb;
                const uint32_t acc = tmem + (uint32_t)(s * kWidth + cb) + lane_base;
                ok = ok && wait_or_abort(&acc_full[s], ejob[s] & 1u, abort);
                ejob[s]++;
                ok = __all_sync(0xffffffffu, ok);
                if (l == 0)
                    quarter_sync(quarter);   // the stream's previous head sums have been read
                if (ok) {
                    umma::tc_fence_after();
                    float v[2][16];
                    umma::tmem_ld16_start(acc, v[0]);
#pragma unroll
                    for (int g = 0; g < 4; g++) {
                        float *x = v[g & 1];
                        float bs[16];
#pragma unroll
                        for (int q = 0; q < 4; q++)
                            *reinterpret_cast<float4 *>(bs + 4 * q) =
                                __ldg(reinterpret_cast<const float4 *>(bias + 16 * g) + q);
                        umma::tmem_ld16_wait(x);
                        if (g < 3)
                            umma::tmem_ld16_start(acc + 16 * (g + 1), v[(g + 1) & 1]);
                        uint32_t t[8];
                        gelu::values_bf16<8>(x, bs, t);
                        const int c0 = cb + 16 * g;
                        if (l < kDepth - 1) {
                            uint8_t *dst = Act + (c0 / umma::kBK) * kActChunk;
                            const int k = c0 % umma::kBK;
                            *reinterpret_cast<uint4 *>(dst + umma::tile_off(rl, k)) =
                                make_uint4(t[0], t[1], t[2], t[3]);
                            *reinterpret_cast<uint4 *>(dst + umma::tile_off(rl, k + 8)) =
                                make_uint4(t[4], t[5], t[6], t[7]);
                        } else {
                            // the head's per-8-column partial sums, as head_kernel's lanes form them
                            const float4 *w5 = reinterpret_cast<const float4 *>(P + kOffW5 + c0);
#pragma unroll
                            for (int h = 0; h < 2; h++) {
                                const float4 wa = __ldg(w5 + 2 * h), wb = __ldg(w5 + 2 * h + 1);
                                const float ws[8] = {wa.x, wa.y, wa.z, wa.w, wb.x, wb.y, wb.z, wb.w};
                                float sum = 0.0f;
#pragma unroll
                                for (int q = 0; q < 8; q++) {
                                    const uint32_t w = t[4 * h + (q >> 1)];
                                    sum += __uint_as_float(q & 1 ? w & 0xffff0000u : w << 16) * ws[q];
                                }
                                gs[(c0 / 8 + h) ^ lane] = sum;
                            }
                        }
                    }
                    umma::tc_fence_before();
                    umma::fence_async_smem();
                }
                __syncwarp();
                if (lane == 0)
                    mbar_arrive(&act_ready[s]);
                if (l == kDepth - 1) {
                    quarter_sync(quarter);
                    if (ok && warp < 4) {
                        // head_kernel's shuffle tree over the 32 partial sums (lane 0's order)
                        float g[32];
#pragma unroll
                        for (int jj = 0; jj < 32; jj++)
                            g[jj] = gs[jj ^ lane];
#pragma unroll
                        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                            for (int jj = 0; jj < o; jj++)
                                g[jj] = g[jj] + g[jj + o];
                        const float y = g[0] + __ldg(P + kOffB5);
                        if (rank == 0) {
                            ys[(e0 + e) * kTileRows + rl] = y;
                        } else {   // into the first CTA's shared memory
                            uint32_t dst;
                            asm volatile("mapa.shared::cluster.u32 %0, %1, 0;"
                                         : "=r"(dst)
                                         : "r"(umma::smem_u32(ys + (e0 + e) * kTileRows + rl)));
                            asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(dst), "f"(y) : "memory");
                        }
                    }
                }
                if (j == jx0 && ti + 1 < my_tiles) {
                    // the tile's features have been read: the next tile's
                    if (ok)
                        tile_features(a, row0 + step * kTileRows, tid, X0s);
                    __syncwarp();
                    if (lane == 0)
                        mbar_arrive(&x0_ready);
                }
            }
            __syncwarp();
            if (a.share > 1) {   // one tile per cluster: the other CTAs' outputs arrive
                asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
                asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
            }
            if (ok && rank == 0 && warp < 4 && row0 + rl < a.n) {
                // ensemble_kernel's statistics (this thread's own row of ys)
                const long long i = row0 + rl;
                float av[kInferMaxMembers];
                float sum = 0.0f;
#pragma unroll
                for (int e = 0; e < kInferMaxMembers; e++) {
                    if (e < a.E) {
                        const float la = a.mu + a.sd * ys[e * kTileRows + rl];
                        if (a.members)
                            a.members[e * a.ldm + i] = la;
                        av[e] = expf(la);
                        sum += av[e];
                    }
                }
                const float m = sum / a.E;
                float var = 0.0f;
#pragma unroll
                for (int e = 0; e < kInferMaxMembers; e++)
                    if (e < a.E)
                        var += (av[e] - m) * (av[e] - m);
                a.mean[i] = m;
                a.spread[i] = sqrtf(var / a.E) / m;
            }
        }
    }
    if (a.share > 1 && warp >= kEpiWarps) {   // the MMA and copy warps' part of the cluster barrier
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
    umma::tc_fence_before();
    __syncthreads();
    if (tid == 0 && s_abort)
        atomicOr(a.err, 1);
    if (warp == 0)
        umma::tmem_dealloc(tmem, 2 * kWidth);
}

// The error path of the tensor-core kernels' bounded waits, on its own: a CTA
// allocates tensor memory as they do, waits for an mbarrier phase that
// nothing completes (an arrival count of 2 with one arrival) with an
// iteration limit, then records the error, releases the tensor memory and
// returns.
__global__ void wait_guard_kernel(unsigned limit, int *err)
{
    __shared__ uint64_t bar;
    __shared__ uint32_t tslot;
    if (threadIdx.x == 0) {
        umma::mbar_init(&bar, 2);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (threadIdx.x < 32)
        umma::tmem_alloc(&tslot, 32);
    umma::tc_fence_before();
    __syncthreads();
    umma::tc_fence_after();
    if (threadIdx.x == 0)
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(umma::smem_u32(&bar)) : "memory");
    const bool ok = umma::mbar_wait(&bar, 0u, limit);
    if (!__syncthreads_and(ok) && threadIdx.x == 0)
        atomicOr(err, 1);
    umma::tc_fence_before();
    __syncthreads();
    if (threadIdx.x < 32)
        umma::tmem_dealloc(tslot, 32);
}

// every float through the layers' BF16 GELU and the bounds of its derivative:
// counts[0] the values whose bits differ from the reference evaluation's or
// whose derivative is out of bounds, counts[1] those the approximation
// left to it
__global__ void gelu_check_kernel(unsigned long long *counts)
{
    unsigned long long wrong = 0, open = 0;
    for (unsigned long long t = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; t < (1ull << 31);
         t += (unsigned long long)gridDim.x * blockDim.x) {
        float v[2] = {__uint_as_float((uint32_t)(2 * t)), __uint_as_float((uint32_t)(2 * t + 1))};
        const uint32_t want = gelu::bf16x2(gelu::value(v[0]), gelu::value(v[1]));
        uint32_t r, o;
        const uint32_t p = gelu::value_bf16x2(gelu::f2(v[0], v[1]), o);
        o ^= p;
        gelu::values_bf16<1>(v, nullptr, &r);
        const uint32_t d = r ^ want;
        wrong += ((d & 0xffffu) != 0) + ((d >> 16) != 0);
        // the derivative lies between its bounds (finite values of it)
        gelu::F2 lo, hi;
        gelu::grad_bounds(gelu::f2(v[0], v[1]), lo, hi);
        float l0, l1, h0, h1;
        gelu::split(lo, l0, l1);
        gelu::split(hi, h0, h1);
        const float g0 = gelu::grad(v[0]), g1 = gelu::grad(v[1]);
        wrong += (isfinite(g0) && !(l0 <= g0 && g0 <= h0)) + (isfinite(g1) && !(l1 <= g1 && g1 <= h1));
        open += ((o & 0xffffu) != 0) + ((o >> 16) != 0);
    }
    atomicAdd(&counts[0], wrong);
    atomicAdd(&counts[1], open);
}

std::once_flag g_infer_once[64];
cudaError_t g_infer_init_err[64];

// opt the fused kernel into its shared-memory size once per device
cudaError_t infer_init(int dev)
{
    if (dev < 0 || dev >= 64)
        return cudaErrorInvalidDevice;
    std::call_once(g_infer_once[dev], [dev] {
        g_infer_init_err[dev] =
            cudaFuncSetAttribute(infer_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kInferSmem);
    });
    return g_infer_init_err[dev];
}

#include "surrogate_train.cuh"

std::once_flag g_train_once[64];
cudaError_t g_train_init_err[64];

// opt the training kernels into their shared-memory sizes once per device
// (outside any stream capture)
cudaError_t train_init(int dev)
{
    if (dev < 0 || dev >= 64)
        return cudaErrorInvalidDevice;
    std::call_once(g_train_once[dev], [dev] {
        cudaError_t e = cudaFuncSetAttribute(chain_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kChainSmem);
        if (!e)
            e = cudaFuncSetAttribute(update_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kGradSmem);
        g_train_init_err[dev] = e;
    });
    return g_train_init_err[dev];
}

}  // namespace

// ------------------------------------------------------------------ state

struct anacor_surrogate {
    int E = 4;
    uint32_t seed = 0;
    cudaStream_t st = nullptr;
    float *params = nullptr, *m = nullptr, *v = nullptr, *grad = nullptr;
    bf16 *W[kDepth] = {};                   // BF16 weights [E][256][K] (the layer-by-layer path)
    uint8_t *wimg = nullptr, *wtimg = nullptr;   // and as the chunks of W and W^T that the fused kernels read
    float *Bf = nullptr;                    // Fourier matrix [32][7]
    double t_mean = 0.0, t_std = 1.0;       // log A_h = t_mean + t_std * y
    // training data
    long long n_data = 0;
    float *target = nullptr;
    bf16 *feat = nullptr;
    // inference workspace of the layer-by-layer path for `rows` rows per member
    int rows = 0;
    bf16 *X0 = nullptr, *A[2] = {};
    float *y = nullptr;
    // training workspace for `train_rows` rows per member (see surrogate_train.cuh)
    int train_rows = 0;
    uint4 *X0i = nullptr, *Ai[kDepth] = {}, *dHi[kDepth] = {};
    float4 *Hi[2] = {};
    float *ty = nullptr, *dy = nullptr;
    float *loss_acc = nullptr;              // zero between steps
    unsigned *step = nullptr, *ticket = nullptr;   // steps taken; blocks of a step that have read it
    float *loss_hist = nullptr;
    int hist_len = 0;
    int *err = nullptr;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    int graph_rows = 0;
    AdamArgs adam{1e-3f, 1e-5f, 0.9f, 0.999f, 1e-8f, 0u};
    int fused = 1;                  // inference by the fused kernel (1) or layer by layer (0)
};

namespace {

template <class T>
cudaError_t dalloc(T **p, size_t n)
{
    *p = nullptr;
    return cudaMalloc(reinterpret_cast<void **>(p), sizeof(T) * std::max<size_t>(n, 1));
}

template <class T>
void dfree(T *&p)
{
    if (p)
        cudaFree(p);
    p = nullptr;
}

void drop_graph(anacor_surrogate *s)
{
    if (s->exec)
        cudaGraphExecDestroy(s->exec);
    if (s->graph)
        cudaGraphDestroy(s->graph);
    s->exec = nullptr;
    s->graph = nullptr;
    s->graph_rows = 0;
}

void free_work(anacor_surrogate *s)
{
    dfree(s->X0); dfree(s->A[0]); dfree(s->A[1]); dfree(s->y);
    s->rows = 0;
}

void free_train(anacor_surrogate *s)
{
    drop_graph(s);
    dfree(s->X0i);
    for (int l = 0; l < kDepth; l++) {
        dfree(s->Ai[l]); dfree(s->dHi[l]);
    }
    dfree(s->Hi[0]); dfree(s->Hi[1]); dfree(s->ty); dfree(s->dy);
    s->train_rows = 0;
}

// layer-by-layer inference for exactly `rows` rows per member
int ensure_work(anacor_surrogate *s, int rows)
{
    if (rows <= 0 || rows % umma::kBM)
        return report_status(kErrArgs, "surrogate: rows must be a positive multiple of 128");
    if (s->rows == rows)
        return kOk;
    free_work(s);
    const size_t E = s->E, R = rows;
    if (dalloc(&s->X0, E * R * kFeat) || dalloc(&s->y, E * R) || dalloc(&s->A[0], E * R * kWidth) ||
        dalloc(&s->A[1], E * R * kWidth)) {
        free_work(s);
        return report_status(kErrCuda, "surrogate: device allocation failed");
    }
    s->rows = rows;
    return kOk;
}

// training on batches of exactly `rows` rows per member
int ensure_train(anacor_surrogate *s, int rows)
{
    if (rows <= 0 || rows % (umma::kBK * kSplitK))
        return report_status(kErrArgs, "surrogate: the training batch must be a multiple of 1024");
    int dev = 0;
    cudaError_t e;
    if ((e = cudaGetDevice(&dev)) || (e = train_init(dev)))
        return report_status(kErrCuda, cudaGetErrorString(e));
    if (s->train_rows == rows)
        return kOk;
    free_train(s);
    const size_t E = s->E, R = rows;
    bool ok = !dalloc(&s->X0i, E * R * kFeat / 8) && !dalloc(&s->ty, E * R) && !dalloc(&s->dy, E * R) &&
              !dalloc(&s->Hi[0], E * R * kWidth / 4) &&
              !dalloc(&s->Hi[1], E * R * kWidth / 4);
    for (int l = 0; l < kDepth && ok; l++)
        ok = !dalloc(&s->Ai[l], E * R * kWidth / 8) && !dalloc(&s->dHi[l], E * R * kWidth / 8);
    if (!ok) {
        free_train(s);
        return report_status(kErrCuda, "surrogate: device allocation failed");
    }
    s->train_rows = rows;
    return kOk;
}

int cuda_fail(cudaError_t e) { return report_status(kErrCuda, cudaGetErrorString(e)); }

int check_err(anacor_surrogate *s, cudaStream_t st)
{
    int h = 0;
    cudaError_t e;
    if ((e = cudaMemcpyAsync(&h, s->err, sizeof(int), cudaMemcpyDeviceToHost, st)) || (e = cudaStreamSynchronize(st)))
        return cuda_fail(e);
    if (h)
        return report_status(kErrCuda, "surrogate: a tensor-core wait timed out");
    return report_status(kOk, "");
}

WeightCopies weight_copies(const anacor_surrogate *s)
{
    WeightCopies c;
    for (int l = 0; l < kDepth; l++)
        c.w[l] = s->W[l];
    c.wimg = s->wimg;
    c.wtimg = s->wtimg;
    return c;
}

// the BF16 copies of the weights, after the masters have changed
cudaError_t convert_all(anacor_surrogate *s, cudaStream_t st)
{
    copies_kernel<<<512, 256, 0, st>>>(s->params, s->E, weight_copies(s));
    return cudaGetLastError();
}

// Forward of every member over `rows` rows of the shared X0 [rows][64]; the
// buffer that holds the last hidden activation.
bf16 *forward(anacor_surrogate *s, int rows, cudaStream_t st, cudaError_t &err)
{
    const long long R = rows;
    const bf16 *in = s->X0;
    bf16 *out = nullptr;
    for (int l = 0; l < kDepth; l++) {
        GemmArgs g{};
        const int K = in_dim(l);
        out = s->A[l & 1];
        g.A = in;
        g.lda = K;
        g.sA = l == 0 ? 0 : R * K;
        g.B = s->W[l];
        g.ldb = K;
        g.sB = (long long)kWidth * K;
        g.M = rows; g.N = kWidth; g.K = K;
        g.mode = kEpiBiasGelu;
        g.bias = s->params + off_b(l);
        g.sBias = kParams;
        g.ob = out;
        g.ldob = kWidth; g.sOb = R * kWidth;
        g.err = s->err;
        if ((err = gemm(g, s->E, st)))
            return nullptr;
        in = out;
    }
    err = cudaSuccess;
    return out;
}

// One step on batches of s->train_rows rows: drawn from the training set, or
// (ordered) the first rows of `feat` and `target` for every member.  With
// `update` the Adam step, the weight copies and the step count, else the
// gradients into s->grad.
cudaError_t train_step(anacor_surrogate *s, const bf16 *feat, const float *target, long long n, bool ordered,
                       bool update, int sms, cudaStream_t st)
{
    ChainArgs c{};
    c.feat = feat;
    c.target = target;
    c.n_data = n;
    c.batch = s->train_rows;
    c.ordered = ordered;
    c.seed = s->seed;
    c.step = s->step;
    c.params = s->params;
    c.wimg = s->wimg;
    c.wtimg = s->wtimg;
    c.E = s->E;
    c.X0 = s->X0i;
    for (int l = 0; l < kDepth; l++) {
        c.A[l] = s->Ai[l];
        c.dH[l] = s->dHi[l];
    }
    c.H[0] = s->Hi[0];
    c.H[1] = s->Hi[1];
    c.y = s->ty;
    c.dy = s->dy;
    c.loss_acc = s->loss_acc;
    c.err = s->err;
    const int units = s->train_rows / kTileRows * s->E;
    chain_kernel<<<std::min(units, sms), kChainThreads, kChainSmem, st>>>(c);
    UpdateArgs u{};
    u.X0 = s->X0i;
    for (int l = 0; l < kDepth; l++) {
        u.A[l] = s->Ai[l];
        u.dH[l] = s->dHi[l];
    }
    u.dy = s->dy;
    u.batch = s->train_rows;
    u.E = s->E;
    u.params = s->params;
    u.m = s->m;
    u.v = s->v;
    u.grad = s->grad;
    u.adam = s->adam;
    u.update = update;
    u.copies = weight_copies(s);
    u.step = s->step;
    u.ticket = s->ticket;
    u.loss_acc = s->loss_acc;
    u.loss_hist = s->loss_hist;
    u.hist_len = s->hist_len;
    u.err = s->err;
    // the column sums take the SMs that the tiles' last wave leaves, or a wave
    // of their own where these are few (one block too many is a wave more: 6 us)
    const int grad_tiles = s->E * kGradTiles, left = sms - grad_tiles % sms;
    const int sums = std::min(s->E * kVectors, left < sms / 4 ? left + sms : left);
    update_kernel<<<grad_tiles + sums, kGradThreads, kGradSmem, st>>>(u);
    return cudaGetLastError();
}

// He-style initialisation of every member (host RNG, seeded)
void init_params(std::vector<float> &p, int E, uint32_t seed)
{
    std::mt19937 rng(seed);
    for (int e = 0; e < E; e++) {
        float *P = p.data() + e * kParams;
        for (int l = 0; l < kDepth; l++) {
            std::normal_distribution<float> nd(0.0f, std::sqrt(2.0f / (float)in_dim(l)));
            for (long long i = 0; i < (long long)kWidth * in_dim(l); i++)
                P[off_w(l) + i] = nd(rng);
            for (int i = 0; i < kWidth; i++)
                P[off_b(l) + i] = 0.0f;
        }
        std::normal_distribution<float> nd(0.0f, std::sqrt(1.0f / (float)kWidth));
        for (int i = 0; i < kWidth; i++)
            P[kOffW5 + i] = nd(rng);
        P[kOffB5] = 0.0f;
    }
}

// features of n rows of device x7 into X0 (padded to rows_pad), forward, head
// and ensemble statistics; all on `st`, no synchronisation
cudaError_t predict_pass(anacor_surrogate *s, const float *d_x7, long long n, int rows_pad, float *d_mean,
                         float *d_spread, float *d_members, long long ldm, cudaStream_t st)
{
    cudaError_t e;
    features_kernel<<<(unsigned)(((long long)rows_pad * (kFeat / 2) + 255) / 256), 256, 0, st>>>(d_x7, s->Bf, n,
                                                                                                 rows_pad, s->X0);
    bf16 *a4 = forward(s, rows_pad, st, e);
    if (e)
        return e;
    head_kernel<<<dim3((rows_pad * 32 + 255) / 256, s->E), 256, 0, st>>>(a4, s->params, rows_pad, s->y);
    ensemble_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(s->y, s->E, n, rows_pad, (float)s->t_mean,
                                                                 (float)s->t_std, d_mean, d_spread, d_members, ldm);
    return cudaGetLastError();
}

Geometry make_geometry(const double *xray, const double *axis, const double *F)
{
    Geometry g;
    std::memcpy(g.xray, xray, sizeof(g.xray));
    std::memcpy(g.axis, axis, sizeof(g.axis));
    std::memcpy(g.F, F, sizeof(g.F));
    return g;
}

}  // namespace

extern "C" {

anacor_surrogate *anacor_surrogate_create(int n_members, uint32_t seed, float fourier_scale)
{
    if (n_members < 1 || n_members > kMaxMembers || !(fourier_scale > 0.0f)) {
        report_status(kErrArgs, "surrogate: 1..16 members and a positive Fourier scale");
        return nullptr;
    }
    if (cudaError_t e = gemm_init()) {
        cuda_fail(e);
        return nullptr;
    }
    anacor_surrogate *s = new (std::nothrow) anacor_surrogate();
    if (!s) {
        report_status(kErrNoMem, "out of host memory");
        return nullptr;
    }
    s->E = n_members;
    s->seed = seed;
    const size_t np = (size_t)kParams * n_members;
    bool ok = !cudaStreamCreateWithFlags(&s->st, cudaStreamNonBlocking) && !dalloc(&s->params, np) &&
              !dalloc(&s->m, np) && !dalloc(&s->v, np) && !dalloc(&s->grad, np) && !dalloc(&s->Bf, 32 * kIn) &&
              !dalloc(&s->loss_acc, 16) && !dalloc(&s->step, 1) && !dalloc(&s->ticket, 1) && !dalloc(&s->err, 1) &&
              !dalloc(&s->wimg, (size_t)n_members * kChunksPerMember * kChunkBytes) &&
              !dalloc(&s->wtimg, (size_t)n_members * kChunksBack * kChunkBytes);
    for (int l = 0; l < kDepth && ok; l++) {
        const size_t n = (size_t)kWidth * in_dim(l) * n_members;
        ok = !dalloc(&s->W[l], n);
    }
    std::vector<float> p(np, 0.0f);
    init_params(p, n_members, seed);
    std::vector<float> B(32 * kIn);
    std::mt19937 rng(seed ^ 0x5bd1e995u);
    std::normal_distribution<float> nd(0.0f, fourier_scale);
    for (int j = 0; j < 32; j++)
        for (int q = 0; q < kIn; q++)   // integer omega frequencies: features periodic in omega
            B[j * kIn + q] = q == 0 ? std::nearbyint(nd(rng)) : nd(rng);
    cudaError_t e = cudaSuccess;
    if (ok && ((e = cudaMemcpy(s->params, p.data(), np * sizeof(float), cudaMemcpyHostToDevice)) ||
               (e = cudaMemset(s->m, 0, np * sizeof(float))) || (e = cudaMemset(s->v, 0, np * sizeof(float))) ||
               (e = cudaMemset(s->grad, 0, np * sizeof(float))) || (e = cudaMemset(s->step, 0, sizeof(unsigned))) ||
               (e = cudaMemset(s->ticket, 0, sizeof(unsigned))) ||
               (e = cudaMemset(s->err, 0, sizeof(int))) || (e = cudaMemset(s->loss_acc, 0, 16 * sizeof(float))) ||
               (e = cudaMemcpy(s->Bf, B.data(), B.size() * sizeof(float), cudaMemcpyHostToDevice)) ||
               (e = convert_all(s, s->st)) || (e = cudaStreamSynchronize(s->st))))
        ok = false;
    if (!ok) {
        if (e)
            cuda_fail(e);
        else
            report_status(kErrCuda, "surrogate: device allocation failed");
        anacor_surrogate_destroy(s);
        return nullptr;
    }
    report_status(kOk, "");
    return s;
}

void anacor_surrogate_destroy(anacor_surrogate *s)
{
    if (!s)
        return;
    if (s->st)
        cudaStreamSynchronize(s->st);
    free_work(s);
    free_train(s);
    dfree(s->params); dfree(s->m); dfree(s->v); dfree(s->grad); dfree(s->Bf);
    dfree(s->loss_acc); dfree(s->step); dfree(s->ticket); dfree(s->err); dfree(s->loss_hist); dfree(s->wimg); dfree(s->wtimg);
    dfree(s->target); dfree(s->feat);
    for (int l = 0; l < kDepth; l++) {
        dfree(s->W[l]);
    }
    if (s->st)
        cudaStreamDestroy(s->st);
    delete s;
}

int64_t anacor_surrogate_param_count(void) { return kParams; }

int anacor_surrogate_members(const anacor_surrogate *s) { return s ? s->E : 0; }

int anacor_surrogate_params(anacor_surrogate *s, float *host, int to_device)
{
    if (!s || !host)
        return report_status(kErrArgs, "bad arguments");
    const size_t n = (size_t)kParams * s->E * sizeof(float);
    cudaError_t e = cudaStreamSynchronize(s->st);
    if (!e)
        e = to_device ? cudaMemcpy(s->params, host, n, cudaMemcpyHostToDevice)
                      : cudaMemcpy(host, s->params, n, cudaMemcpyDeviceToHost);
    if (!e && to_device)
        e = convert_all(s, s->st);
    if (!e)
        e = cudaStreamSynchronize(s->st);
    return e ? cuda_fail(e) : report_status(kOk, "");
}

int anacor_surrogate_fourier(anacor_surrogate *s, float *host32x7, int to_device)
{
    if (!s || !host32x7)
        return report_status(kErrArgs, "bad arguments");
    cudaError_t e = to_device ? cudaMemcpy(s->Bf, host32x7, 32 * kIn * sizeof(float), cudaMemcpyHostToDevice)
                              : cudaMemcpy(host32x7, s->Bf, 32 * kIn * sizeof(float), cudaMemcpyDeviceToHost);
    return e ? cuda_fail(e) : report_status(kOk, "");
}

int anacor_surrogate_scale(anacor_surrogate *s, double *mean, double *std_dev, int set)
{
    if (!s || !mean || !std_dev || (set && !(*std_dev > 0.0)))
        return report_status(kErrArgs, "bad arguments");
    if (set) {
        s->t_mean = *mean;
        s->t_std = *std_dev;
    } else {
        *mean = s->t_mean;
        *std_dev = s->t_std;
    }
    return report_status(kOk, "");
}

int anacor_surrogate_inputs_device(const double *d_omega, const double *d_s1, int64_t n, const double *xray,
                                   const double *omega_axis, const double *F, float *d_x7, void *stream)
{
    if (n < 0 || (n > 0 && (!d_omega || !d_s1 || !xray || !omega_axis || !F || !d_x7)))
        return report_status(kErrArgs, "bad arguments");
    if (n == 0)
        return report_status(kOk, "");
    inputs_kernel<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(
        d_omega, d_s1, n, make_geometry(xray, omega_axis, F), d_x7);
    cudaError_t e = cudaGetLastError();
    return e ? cuda_fail(e) : report_status(kOk, "");
}

int anacor_surrogate_inputs(const double *omega, const double *s1, int64_t n, const double *xray,
                            const double *omega_axis, const double *F, float *x7_out)
{
    if (n < 0 || (n > 0 && (!omega || !s1 || !xray || !omega_axis || !F || !x7_out)))
        return report_status(kErrArgs, "bad arguments");
    if (n == 0)
        return report_status(kOk, "");
    double *d_om = nullptr, *d_s1 = nullptr;
    float *d_x = nullptr;
    cudaError_t e;
    if (!(e = dalloc(&d_om, n)) && !(e = dalloc(&d_s1, 3 * n)) && !(e = dalloc(&d_x, 7 * n)) &&
        !(e = cudaMemcpy(d_om, omega, n * sizeof(double), cudaMemcpyHostToDevice)) &&
        !(e = cudaMemcpy(d_s1, s1, 3 * n * sizeof(double), cudaMemcpyHostToDevice))) {
        inputs_kernel<<<(unsigned)((n + 255) / 256), 256>>>(d_om, d_s1, n, make_geometry(xray, omega_axis, F), d_x);
        if (!(e = cudaGetLastError()))
            e = cudaMemcpy(x7_out, d_x, 7 * n * sizeof(float), cudaMemcpyDeviceToHost);
    }
    dfree(d_om); dfree(d_s1); dfree(d_x);
    return e ? cuda_fail(e) : report_status(kOk, "");
}

// training set: x7 rows and log A_h targets; the targets are standardised
// with their mean and standard deviation, which become the output scale
int anacor_surrogate_set_data(anacor_surrogate *s, const float *x7, const double *log_ah, int64_t n)
{
    if (!s || n < 2 || !x7 || !log_ah)
        return report_status(kErrArgs, "bad arguments");
    double mu = 0.0, m2 = 0.0;
    for (int64_t i = 0; i < n; i++) {
        if (!std::isfinite(log_ah[i]))
            return report_status(kErrArgs, "surrogate: non-finite training target");
        const double d = log_ah[i] - mu;
        mu += d / (double)(i + 1);
        m2 += d * (log_ah[i] - mu);
    }
    double sd = std::sqrt(m2 / (double)(n - 1));
    if (!(sd > 1e-12))
        sd = 1.0;
    std::vector<float> t(n);
    for (int64_t i = 0; i < n; i++)
        t[i] = (float)((log_ah[i] - mu) / sd);
    cudaStreamSynchronize(s->st);
    drop_graph(s);
    dfree(s->target);
    dfree(s->feat);
    float *d_x = nullptr;
    cudaError_t e;
    if (!(e = dalloc(&d_x, 7 * n)) && !(e = dalloc(&s->target, n)) && !(e = dalloc(&s->feat, n * kFeat)) &&
        !(e = cudaMemcpy(d_x, x7, 7 * n * sizeof(float), cudaMemcpyHostToDevice)) &&
        !(e = cudaMemcpy(s->target, t.data(), n * sizeof(float), cudaMemcpyHostToDevice))) {
        features_kernel<<<(unsigned)((n * (kFeat / 2) + 255) / 256), 256, 0, s->st>>>(d_x, s->Bf, n, n, s->feat);
        if (!(e = cudaGetLastError()))
            e = cudaStreamSynchronize(s->st);
    }
    dfree(d_x);
    if (e) {
        dfree(s->target);
        dfree(s->feat);
        s->n_data = 0;
        return cuda_fail(e);
    }
    s->n_data = n;
    s->t_mean = mu;
    s->t_std = sd;
    return report_status(kOk, "");
}

int anacor_surrogate_train(anacor_surrogate *s, int steps, int batch, float lr_max, float lr_min, int total_steps,
                           float *loss_out)
{
    if (!s || steps < 0 || batch <= 0 || !s->n_data || !(lr_max > 0.0f) || lr_min < 0.0f || total_steps < 0)
        return report_status(kErrArgs, "surrogate: bad training arguments");
    if (int st = ensure_train(s, batch))
        return st;
    int dev = 0, sms = 0;
    unsigned start = 0;
    cudaError_t e;
    if ((e = cudaGetDevice(&dev)) || (e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) ||
        (e = cudaStreamSynchronize(s->st)) ||
        (e = cudaMemcpy(&start, s->step, sizeof(unsigned), cudaMemcpyDeviceToHost)))
        return cuda_fail(e);
    const AdamArgs a{lr_max, lr_min, 0.9f, 0.999f, 1e-8f, (unsigned)total_steps};
    if (std::memcmp(&a, &s->adam, sizeof(a)) != 0) {
        s->adam = a;
        drop_graph(s);   // the graph holds the Adam arguments by value
    }
    const int need = (int)start + steps;
    if (need > s->hist_len) {
        float *h = nullptr;
        if (dalloc(&h, (size_t)need + 1024))
            return report_status(kErrCuda, "surrogate: device allocation failed");
        if (s->loss_hist)
            cudaMemcpy(h, s->loss_hist, s->hist_len * sizeof(float), cudaMemcpyDeviceToDevice);
        dfree(s->loss_hist);
        s->loss_hist = h;
        s->hist_len = need + 1024;
        drop_graph(s);   // ... and the history pointer
    }
    if (!s->exec || s->graph_rows != batch) {
        drop_graph(s);
        if ((e = cudaStreamBeginCapture(s->st, cudaStreamCaptureModeThreadLocal)))
            return cuda_fail(e);
        const cudaError_t le = train_step(s, s->feat, s->target, s->n_data, false, true, sms, s->st);
        e = cudaStreamEndCapture(s->st, &s->graph);
        if (le || e) {
            drop_graph(s);
            return cuda_fail(le ? le : e);
        }
        if ((e = cudaGraphInstantiate(&s->exec, s->graph, 0))) {
            drop_graph(s);
            return cuda_fail(e);
        }
        s->graph_rows = batch;
    }
    for (int i = 0; i < steps; i++)
        if ((e = cudaGraphLaunch(s->exec, s->st)))
            return cuda_fail(e);
    if (int st = check_err(s, s->st))
        return st;
    if (loss_out && steps > 0 &&
        (e = cudaMemcpy(loss_out, s->loss_hist + start, steps * sizeof(float), cudaMemcpyDeviceToHost)))
        return cuda_fail(e);
    return report_status(kOk, "");
}

int anacor_surrogate_gradients(anacor_surrogate *s, const float *x7, const float *target, int rows,
                               float *grads_out, float *y_out)
{
    if (!s || rows <= 0 || !x7 || !target)
        return report_status(kErrArgs, "bad arguments");
    if (int st = ensure_train(s, rows))
        return st;
    const size_t R = rows;
    float *d_x = nullptr, *d_t = nullptr;
    bf16 *d_f = nullptr;
    int dev = 0, sms = 0;
    cudaError_t e;
    if (!(e = cudaGetDevice(&dev)) && !(e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) &&
        !(e = cudaStreamSynchronize(s->st)) && !(e = dalloc(&d_x, 7 * R)) && !(e = dalloc(&d_t, R)) &&
        !(e = dalloc(&d_f, R * kFeat)) && !(e = cudaMemcpy(d_x, x7, 7 * R * sizeof(float), cudaMemcpyHostToDevice)) &&
        !(e = cudaMemcpy(d_t, target, R * sizeof(float), cudaMemcpyHostToDevice))) {
        features_kernel<<<(unsigned)((R * (kFeat / 2) + 255) / 256), 256, 0, s->st>>>(d_x, s->Bf, rows, rows, d_f);
        // the same batch, rows in order, for every member
        if (!(e = cudaGetLastError()) && !(e = train_step(s, d_f, d_t, rows, true, false, sms, s->st)))
            e = cudaStreamSynchronize(s->st);
    }
    if (!e && grads_out)
        e = cudaMemcpy(grads_out, s->grad, (size_t)kParams * s->E * sizeof(float), cudaMemcpyDeviceToHost);
    if (!e && y_out)
        e = cudaMemcpy(y_out, s->ty, R * s->E * sizeof(float), cudaMemcpyDeviceToHost);
    dfree(d_x); dfree(d_t); dfree(d_f);
    if (e)
        return cuda_fail(e);
    return check_err(s, s->st);
}

int anacor_surrogate_predict_device(anacor_surrogate *s, const float *d_x7, int64_t n, float *d_mean,
                                    float *d_spread, float *d_members, void *stream)
{
    if (!s || n < 0 || (n > 0 && (!d_x7 || !d_mean || !d_spread)))
        return report_status(kErrArgs, "bad arguments");
    if (n == 0)
        return report_status(kOk, "");
    cudaStream_t st = stream ? (cudaStream_t)stream : s->st;
    if (s->fused && s->E <= kInferMaxMembers) {
        // one launch over all n rows: no activation workspace
        int dev = 0, sms = 0;
        cudaError_t e;
        if ((e = cudaGetDevice(&dev)) || (e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) ||
            (e = infer_init(dev)))
            return cuda_fail(e);
        InferArgs ia;
        ia.x7 = d_x7;
        ia.n = n;
        ia.Bf = s->Bf;
        ia.wimg = s->wimg;
        ia.params = s->params;
        ia.E = s->E;
        ia.mu = (float)s->t_mean;
        ia.sd = (float)s->t_std;
        ia.mean = d_mean;
        ia.spread = d_spread;
        ia.members = d_members;
        ia.ldm = n;
        ia.err = s->err;
        const long long tiles = (n + kTileRows - 1) / kTileRows;
        // few tiles: share each one's members between the CTAs of a cluster
        // while every cluster still has SMs of its own
        ia.share = 1;
        while (ia.share * 2 <= s->E && tiles * ia.share * 2 <= sms)
            ia.share *= 2;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)(ia.share > 1 ? tiles * ia.share : std::min<long long>(tiles, sms)));
        cfg.blockDim = dim3(kInferThreads);
        cfg.dynamicSmemBytes = kInferSmem;
        cfg.stream = st;
        cudaLaunchAttribute attr;
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = (unsigned)ia.share;
        attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
        cfg.attrs = &attr;
        cfg.numAttrs = ia.share > 1 ? 1 : 0;
        if ((e = cudaLaunchKernelEx(&cfg, infer_kernel, ia)))
            return cuda_fail(e);
        if ((e = cudaGetLastError()))
            return cuda_fail(e);
        return report_status(kOk, "");
    }
    const int chunk = (int)std::min<int64_t>(kPredictChunk, (n + umma::kBM - 1) / umma::kBM * umma::kBM);
    if (s->rows != chunk) {
        // the workspace is about to be replaced: nothing may still use it
        cudaError_t e;
        if ((e = cudaStreamSynchronize(s->st)) || (stream && (e = cudaStreamSynchronize(st))))
            return cuda_fail(e);
        if (int r = ensure_work(s, chunk))
            return r;
    }
    for (int64_t i0 = 0; i0 < n; i0 += chunk) {
        const long long m = std::min<int64_t>(chunk, n - i0);
        const int rows = (int)((m + umma::kBM - 1) / umma::kBM * umma::kBM);
        if (cudaError_t e = predict_pass(s, d_x7 + 7 * i0, m, rows, d_mean + i0, d_spread + i0,
                                         d_members ? d_members + i0 : nullptr, n, st))
            return cuda_fail(e);
    }
    return report_status(kOk, "");
}

int anacor_surrogate_set_inference(anacor_surrogate *s, int fused)
{
    if (!s || (fused != 0 && fused != 1))
        return report_status(kErrArgs, "bad arguments");
    if (s->st)
        cudaStreamSynchronize(s->st);
    s->fused = fused;
    return report_status(kOk, "");
}

int anacor_surrogate_predict(anacor_surrogate *s, const float *x7, int64_t n, float *mean_out, float *spread_out,
                             float *members_out)
{
    if (!s || n < 0 || (n > 0 && (!x7 || !mean_out || !spread_out)))
        return report_status(kErrArgs, "bad arguments");
    if (n == 0)
        return report_status(kOk, "");
    float *d_x = nullptr, *d_mean = nullptr, *d_spread = nullptr, *d_mem = nullptr;
    cudaError_t e;
    int st = kOk;
    if (!(e = dalloc(&d_x, 7 * (size_t)n)) && !(e = dalloc(&d_mean, n)) && !(e = dalloc(&d_spread, n)) &&
        !(members_out && (e = dalloc(&d_mem, (size_t)n * s->E))) &&
        !(e = cudaMemcpyAsync(d_x, x7, 7 * (size_t)n * sizeof(float), cudaMemcpyHostToDevice, s->st))) {
        st = anacor_surrogate_predict_device(s, d_x, n, d_mean, d_spread, d_mem, s->st);
        if (!st && !(e = cudaMemcpyAsync(mean_out, d_mean, n * sizeof(float), cudaMemcpyDeviceToHost, s->st)) &&
            !(e = cudaMemcpyAsync(spread_out, d_spread, n * sizeof(float), cudaMemcpyDeviceToHost, s->st)) &&
            !(members_out && (e = cudaMemcpyAsync(members_out, d_mem, (size_t)n * s->E * sizeof(float),
                                                  cudaMemcpyDeviceToHost, s->st))))
            e = cudaStreamSynchronize(s->st);
    }
    dfree(d_x); dfree(d_mean); dfree(d_spread); dfree(d_mem);
    if (st)
        return st;
    if (e)
        return cuda_fail(e);
    return check_err(s, s->st);
}

int anacor_surrogate_audit_flags(const float *d_spread, int64_t n, uint32_t seed, double audit_fraction,
                                 float spread_threshold, uint8_t *d_flags, void *stream)
{
    if (n < 0 || (n > 0 && (!d_spread || !d_flags)) || !(audit_fraction >= 0.0 && audit_fraction <= 1.0))
        return report_status(kErrArgs, "bad arguments");
    if (n == 0)
        return report_status(kOk, "");
    const double c = std::ldexp(audit_fraction, 32);
    const uint32_t cut = c >= 4294967295.0 ? 0xFFFFFFFFu : (uint32_t)c;
    audit_kernel<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(d_spread, n, seed, cut,
                                                                                spread_threshold, d_flags);
    cudaError_t e = cudaGetLastError();
    return e ? cuda_fail(e) : report_status(kOk, "");
}

int anacor_surrogate_save(anacor_surrogate *s, const char *path)
{
    if (!s || !path)
        return report_status(kErrArgs, "bad arguments");
    std::vector<float> p((size_t)kParams * s->E), B(32 * kIn);
    cudaError_t e;
    if ((e = cudaStreamSynchronize(s->st)) ||
        (e = cudaMemcpy(p.data(), s->params, p.size() * sizeof(float), cudaMemcpyDeviceToHost)) ||
        (e = cudaMemcpy(B.data(), s->Bf, B.size() * sizeof(float), cudaMemcpyDeviceToHost)))
        return cuda_fail(e);
    FILE *f = std::fopen(path, "wb");
    if (!f)
        return report_status(kErrArgs, "surrogate: cannot open the checkpoint for writing");
    const uint32_t hdr[4] = {0x41484750u, 1u, (uint32_t)s->E, (uint32_t)kParams};
    const double scale[2] = {s->t_mean, s->t_std};
    bool ok = std::fwrite(hdr, sizeof(hdr), 1, f) == 1 && std::fwrite(scale, sizeof(scale), 1, f) == 1 &&
              std::fwrite(B.data(), sizeof(float), B.size(), f) == B.size() &&
              std::fwrite(p.data(), sizeof(float), p.size(), f) == p.size();
    ok = (std::fclose(f) == 0) && ok;
    return report_status(ok ? kOk : kErrArgs, ok ? "" : "surrogate: checkpoint write failed");
}

int anacor_surrogate_load(anacor_surrogate *s, const char *path)
{
    if (!s || !path)
        return report_status(kErrArgs, "bad arguments");
    FILE *f = std::fopen(path, "rb");
    if (!f)
        return report_status(kErrArgs, "surrogate: cannot open the checkpoint");
    uint32_t hdr[4];
    double scale[2];
    std::vector<float> p((size_t)kParams * s->E), B(32 * kIn);
    bool ok = std::fread(hdr, sizeof(hdr), 1, f) == 1 && hdr[0] == 0x41484750u && hdr[1] == 1u &&
              hdr[2] == (uint32_t)s->E && hdr[3] == (uint32_t)kParams && std::fread(scale, sizeof(scale), 1, f) == 1 &&
              std::fread(B.data(), sizeof(float), B.size(), f) == B.size() &&
              std::fread(p.data(), sizeof(float), p.size(), f) == p.size() && scale[1] > 0.0;
    std::fclose(f);
    if (!ok)
        return report_status(kErrArgs, "surrogate: the checkpoint does not match this network");
    cudaError_t e;
    if ((e = cudaStreamSynchronize(s->st)) ||
        (e = cudaMemcpy(s->params, p.data(), p.size() * sizeof(float), cudaMemcpyHostToDevice)) ||
        (e = cudaMemcpy(s->Bf, B.data(), B.size() * sizeof(float), cudaMemcpyHostToDevice)) ||
        (e = convert_all(s, s->st)) || (e = cudaStreamSynchronize(s->st)))
        return cuda_fail(e);
    s->t_mean = scale[0];
    s->t_std = scale[1];
    if (s->n_data) {   // the cached training features used the old Fourier matrix
        dfree(s->target);
        dfree(s->feat);
        s->n_data = 0;
        drop_graph(s);
    }
    return report_status(kOk, "");
}

int anacor_wait_guard_check(unsigned iterations, int32_t *status)
{
    if (!status || iterations == 0 || iterations > (1u << 20))
        return report_status(kErrArgs, "iterations must lie in [1, 2^20]");
    int *d_err = nullptr;
    cudaError_t e;
    if ((e = dalloc(&d_err, 1)))
        return cuda_fail(e);
    int h = 0;
    if (!(e = cudaMemset(d_err, 0, sizeof(int)))) {
        wait_guard_kernel<<<1, 128>>>(iterations, d_err);
        if (!(e = cudaGetLastError()) && !(e = cudaDeviceSynchronize()))
            e = cudaMemcpy(&h, d_err, sizeof(int), cudaMemcpyDeviceToHost);
    }
    dfree(d_err);
    if (e)
        return cuda_fail(e);
    *status = h;
    return report_status(kOk, "");
}

int anacor_gelu_check(uint64_t *wrong, uint64_t *open)
{
    if (!wrong || !open)
        return report_status(kErrArgs, "bad arguments");
    unsigned long long *d = nullptr, h[2] = {0, 0};
    cudaError_t e;
    if (!(e = dalloc(&d, 2)) && !(e = cudaMemset(d, 0, sizeof(h)))) {
        gelu_check_kernel<<<1024, 256>>>(d);
        if (!(e = cudaGetLastError()) && !(e = cudaDeviceSynchronize()))
            e = cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost);
    }
    dfree(d);
    if (e)
        return cuda_fail(e);
    *wrong = h[0];
    *open = h[1];
    return report_status(kOk, "");
}

int anacor_tc_gemm_check(const float *A, const float *B, int M, int N, int K, int batch, int ksplit, float *C)
{
    if (!A || !B || !C || M <= 0 || N <= 0 || K <= 0 || batch <= 0 || ksplit < 1)
        return report_status(kErrArgs, "bad arguments");
    if (M % umma::kBM || N % 64 || K % (umma::kBK * ksplit))
        return report_status(kErrArgs, "tc_gemm: M % 128, N % 64 and K % (64 * ksplit) must be 0");
    if (cudaError_t e = gemm_init())
        return cuda_fail(e);
    std::vector<bf16> ha((size_t)batch * M * K), hb((size_t)batch * N * K);
    for (size_t i = 0; i < ha.size(); i++)
        ha[i] = __float2bfloat16_rn(A[i]);
    for (size_t i = 0; i < hb.size(); i++)
        hb[i] = __float2bfloat16_rn(B[i]);
    bf16 *da = nullptr, *db = nullptr;
    float *dc = nullptr;
    int *derr = nullptr;
    const size_t nc = (size_t)batch * ksplit * M * N;
    cudaError_t e;
    int herr = 0;
    std::vector<float> part(nc);
    if (!(e = dalloc(&da, ha.size())) && !(e = dalloc(&db, hb.size())) && !(e = dalloc(&dc, nc)) &&
        !(e = dalloc(&derr, 1)) && !(e = cudaMemcpy(da, ha.data(), ha.size() * sizeof(bf16), cudaMemcpyHostToDevice)) &&
        !(e = cudaMemcpy(db, hb.data(), hb.size() * sizeof(bf16), cudaMemcpyHostToDevice)) &&
        !(e = cudaMemset(derr, 0, sizeof(int)))) {
        GemmArgs g{};
        g.A = da; g.lda = K; g.sA = (long long)M * K;
        g.B = db; g.ldb = K; g.sB = (long long)N * K;
        g.M = M; g.N = N; g.K = K;
        g.ksplit = ksplit;
        g.mode = kEpiStoreF32;
        g.of = dc; g.ldf = N; g.sF = (long long)M * N;
        g.err = derr;
        if (!(e = gemm(g, batch, 0)) && !(e = cudaDeviceSynchronize()) &&
            !(e = cudaMemcpy(part.data(), dc, nc * sizeof(float), cudaMemcpyDeviceToHost)))
            e = cudaMemcpy(&herr, derr, sizeof(int), cudaMemcpyDeviceToHost);
    }
    dfree(da); dfree(db); dfree(dc); dfree(derr);
    if (e)
        return cuda_fail(e);
    if (herr)
        return report_status(kErrCuda, "tc_gemm: a tensor-core wait timed out");
    const size_t mn = (size_t)M * N;
    for (int z = 0; z < batch; z++)
        for (size_t i = 0; i < mn; i++) {
            float acc = 0.0f;
            for (int sp = 0; sp < ksplit; sp++)
                acc += part[((size_t)z * ksplit + sp) * mn + i];
            C[(size_t)z * mn + i] = acc;
        }
    return report_status(kOk, "");
}

}  // extern "C"
