// One training step of the surrogate as three kernels.  Included by
// surrogate.cu after the fused inference kernel, whose helpers it uses.
//
//   chain_kernel   a 128-row tile of one member's batch: gather, the four
//                  forward layers, head and loss, and the three backward
//                  products dH_{l-1} = (dH_l W_l) gelu'(H_{l-1}), all of which
//                  need the tile's own rows only;
//   dw_kernel      the weight gradients dH_l^T A_{l-1}, K-split over the rows;
//   update_kernel  sums of the splits and of the biases, Adam, and the BF16
//                  weights in the layouts the products read.
//
// Step by step (a GEMM per layer and direction, transposed copies, sums,
// Adam, conversions: 40 launches) it took 411 us for four members at a batch
// of 4,096.  The numbers are the same: every product accumulates over the same
// K order, the splits and column sums are added in the same order and the
// BF16 roundings are the same.
//
// Activations and gradients leave the chain only as "row images" for the dW
// products, which contract over the rows: blocks of 64 rows, in each the
// columns in groups of eight, [group][64 rows][8], so that a block is one bulk
// copy and its bytes are the canonical no-swizzle MN-major operand (8 x 8 core
// matrices of 128 bytes, the next eight rows 128 bytes on, the next eight
// columns 1,024), and 32 lanes holding 32 rows write 512 contiguous bytes.

// 16-byte element (row, 8 columns from 8 * group) of a row image of C columns
__host__ __device__ constexpr long long row_image(long long row, int group, int C)
{
    return ((row >> 6) * (C / 8) + group) * 64 + (row & 63);
}

// pre-activations of a tile kept for its own backward pass: [4-column group][128 rows][4] floats
__host__ __device__ constexpr long long pre_image(long long tile, int group4, int row)
{
    return (tile * (kWidth / 4) + group4) * kTileRows + row;
}

constexpr int kChunksBack = (kDepth - 1) * (kWidth / kWChunkK);   // chunks of W_l^T, l = 1 .. 3, per member

struct ChainArgs {
    const bf16 *feat;         // [n][64]
    const float *target;      // [n], standardised
    long long n_data;
    int batch;
    int ordered;              // rows 0 .. batch - 1 for every member instead of a drawn batch
    uint32_t seed;
    const unsigned *step;
    const float *params;
    const uint8_t *wimg;      // W_l chunks (weight_image's layout)
    const uint8_t *wtimg;     // W_l^T chunks, l = 1 .. 3
    int E;
    uint4 *X0;                // row images: [E][batch][64], then [E][batch][256] per layer
    uint4 *A[kDepth], *dH[kDepth];
    float4 *H[2];             // pre-activations of layers 0 and 1
    float *y, *dy, *loss_acc;
    int *err;
};

constexpr int kOffChainAct = 8 * kChunkBytes;                     // eight weight stages: a whole layer
constexpr int kOffChainX0 = kOffChainAct + kActBytes;
constexpr int kOffChainDy = kOffChainX0 + kActChunk;
constexpr int kChainSmem = kOffChainDy + kTileRows * 4;
constexpr int kChainStages = 8;
static_assert(kChainSmem + 512 <= 227 * 1024, "chain kernel shared memory");
constexpr int kChainJobs = 2 * kDepth - 1;                        // four forward, three backward products

// Row drawn for (member, batch row): the hash of (seed, step, member, row)
__device__ __forceinline__ long long drawn_row(const ChainArgs &a, unsigned step, int e, int b)
{
    if (a.ordered)
        return b;
    const uint32_t h = mix32(a.seed ^ mix32(step * 0x9E3779B9u ^ mix32((uint32_t)e * 0x85EBCA6Bu ^ (uint32_t)b)));
    return (long long)(((uint64_t)h * (uint64_t)a.n_data) >> 32);
}

__global__ void __launch_bounds__(kInferThreads, 1) chain_kernel(ChainArgs a)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ uint64_t full[kChainStages], empty[kChainStages], acc_full, act_ready, x0_ready;
    __shared__ uint32_t tslot;
    __shared__ int s_abort;
    uint8_t *Ws = smem, *Act = smem + kOffChainAct, *X0s = smem + kOffChainX0;
    float *dys = reinterpret_cast<float *>(smem + kOffChainDy);
    volatile int *abort = &s_abort;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int tiles = a.batch / kTileRows;
    const int units = tiles * a.E;   // unit u: member u / tiles, tile u % tiles

    if (tid == 0) {
        for (int s = 0; s < kChainStages; s++) {
            umma::mbar_init(&full[s], 1);
            umma::mbar_init(&empty[s], 1);
        }
        umma::mbar_init(&acc_full, 1);
        umma::mbar_init(&act_ready, kEpiWarps);
        umma::mbar_init(&x0_ready, kEpiWarps);
        s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0)
        umma::tmem_alloc(&tslot, 2 * kWidth);
    umma::tc_fence_before();
    __syncthreads();
    umma::tc_fence_after();
    const uint32_t tmem = tslot;

    // product j of a unit: 0 .. 3 forward layers, 4 .. 6 dH_3, dH_2, dH_1 times
    // W_3, W_2, W_1; its accumulator (layer 2's pre-activations stay in the
    // first one until the first backward product is done)
    auto job_nk = [](int j) { return (j == 0 ? kFeat : kWidth) / kWChunkK; };
    auto job_acc = [](int j) { return j < 4 ? j & 1 : (j == 4 ? 1 : j & 1); };

    if (warp == kEpiWarps + 1) {
        if (lane == 0) {
            long long q = 0;
            bool ok = true;
            for (int u = blockIdx.x; u < units && ok; u += gridDim.x) {
                const int e = u / tiles;
                for (int j = 0; j < kChainJobs && ok; j++)
                    for (int kq = 0; kq < job_nk(j); kq++, q++) {
                        const int st = (int)(q % kChainStages);
                        if (q >= kChainStages &&
                            !wait_or_abort(&empty[st], (uint32_t)((q / kChainStages - 1) & 1), abort)) {
                            ok = false;
                            break;
                        }
                        const uint8_t *src =
                            j < kDepth ? a.wimg + (long long)chunk_index(e, j, kq) * kChunkBytes
                                       : a.wtimg + ((long long)e * kChunksBack + (kChainJobs - 1 - j) * 8 + kq) * kChunkBytes;
                        mbar_expect_tx(&full[st], kChunkBytes);
                        bulk_g2s(Ws + st * kChunkBytes, src, kChunkBytes, &full[st]);
                    }
            }
            // copies in flight land before the shared memory goes away
            for (long long p = q > kChainStages ? q - kChainStages : 0; p < q; p++)
                wait_or_abort(&full[p % kChainStages], (uint32_t)((p / kChainStages) & 1), abort);
        }
        __syncwarp();
    } else if (warp == kEpiWarps) {
        if (lane == 0) {
            constexpr uint32_t idesc = umma::idesc_bf16_f32(kWidth);
            long long q = 0;
            uint32_t jobs = 0, unit = 0;
            bool ok = true;
            for (int u = blockIdx.x; u < units && ok; u += gridDim.x, unit++) {
                for (int j = 0; j < kChainJobs && ok; j++, jobs++) {
                    if (j == 0)
                        ok = wait_or_abort(&x0_ready, unit & 1u, abort);
                    if (ok && jobs > 0)
                        ok = wait_or_abort(&act_ready, (jobs - 1u) & 1u, abort);
                    if (!ok)
                        break;
                    umma::tc_fence_after();
                    const uint8_t *A = j == 0 ? X0s : Act;
                    const uint32_t d = tmem + (uint32_t)(job_acc(j) * kWidth);
                    for (int kc = 0; kc < job_nk(j); kc++, q++) {
                        const int st = (int)(q % kChainStages);
                        if (!wait_or_abort(&full[st], (uint32_t)((q / kChainStages) & 1), abort)) {
                            ok = false;
                            break;
                        }
#pragma unroll
                        for (int kk = 0; kk < kWChunkK / 16; kk++) {
                            const int k0 = kc * kWChunkK + kk * 16;
                            const uint32_t a0 = umma::smem_u32(A + (k0 / umma::kBK) * kActChunk) +
                                                (uint32_t)((k0 % umma::kBK) / 16) * 256;
                            const uint32_t b0 = umma::smem_u32(Ws + st * kChunkBytes) + (uint32_t)kk * 256;
                            umma::mma_bf16(d, umma::smem_desc(a0, 128, 1024), umma::smem_desc(b0, 128, 512), idesc,
                                           (kc > 0 || kk > 0) ? 1u : 0u);
                        }
                        umma::mma_commit(&empty[st]);
                    }
                    umma::mma_commit(&acc_full);
                }
            }
            if (!ok)
                *abort = 1;
        }
        __syncwarp();
    } else {
        // ---- epilogue warps (a warp whose wait runs out goes on through the
        // loops without waiting or writing, see infer_kernel)
        const int quarter = warp & 3, rl = 32 * quarter + lane, cb = 64 * (warp >> 2);
        const uint32_t lane_base = (uint32_t)(32 * quarter) << 16;
        float *gs = reinterpret_cast<float *>(Act + quarter * kQuarterBytes) + 32 * lane;
        const unsigned step = *a.step;
        uint32_t jobs = 0;
        bool ok = true;
        // a unit's features: into the layer-0 operand and its row image
        auto gather = [&](int u) {
            const int e = u / tiles, t = u - e * tiles;
            const int r = tid >> 2, part = tid & 3;
            const int b = t * kTileRows + r;
            const uint4 *src = reinterpret_cast<const uint4 *>(a.feat + drawn_row(a, step, e, b) * kFeat) + 2 * part;
            const uint4 v0 = __ldg(src), v1 = __ldg(src + 1);
            *reinterpret_cast<uint4 *>(X0s + umma::tile_off(r, 16 * part)) = v0;
            *reinterpret_cast<uint4 *>(X0s + umma::tile_off(r, 16 * part + 8)) = v1;
            uint4 *img = a.X0 + (long long)e * a.batch * (kFeat / 8);
            img[row_image(b, 2 * part, kFeat)] = v0;
            img[row_image(b, 2 * part + 1, kFeat)] = v1;
            umma::fence_async_smem();
        };
        auto wait_job = [&]() {
            ok = ok && wait_or_abort(&acc_full, jobs & 1u, abort);
            jobs++;
            ok = __all_sync(0xffffffffu, ok);
            if (ok)
                umma::tc_fence_after();
        };
        auto done_job = [&]() {
            umma::tc_fence_before();
            umma::fence_async_smem();
            __syncwarp();
            if (lane == 0)
                mbar_arrive(&act_ready);
        };
        if ((int)blockIdx.x < units) {
            gather(blockIdx.x);
            __syncwarp();
            if (lane == 0)
                mbar_arrive(&x0_ready);
        }
        for (int u = blockIdx.x; u < units; u += gridDim.x) {
            const int e = u / tiles, t = u - e * tiles;
            const long long row = (long long)t * kTileRows + rl;     // of the member's batch
            const long long tile = (long long)e * tiles + t;
            const long long img = (long long)e * a.batch * (kWidth / 8);
            const float *P = a.params + (long long)e * kParams;
            const float *w5 = P + kOffW5 + cb;
            // ---- forward
            for (int l = 0; l < kDepth; l++) {
                const uint32_t acc = tmem + (uint32_t)(job_acc(l) * kWidth + cb) + lane_base;
                const float *bias = P + off_b(l) + cb;
                wait_job();
                if (ok) {
#pragma unroll 1
                    for (int g = 0; g < 4; g++) {
                        const int c0 = cb + 16 * g;
                        float v[16], bs[16];
                        umma::tmem_ld16_start(acc + 16 * g, v);
#pragma unroll
                        for (int q = 0; q < 4; q++)
                            *reinterpret_cast<float4 *>(bs + 4 * q) =
                                __ldg(reinterpret_cast<const float4 *>(bias + 16 * g) + q);
                        umma::tmem_ld16_wait(v);
                        uint32_t w[8];
                        gelu::values_bf16<8>(v, bs, w);
                        if (l < 2) {
                            float4 *h = a.H[l];
#pragma unroll
                            for (int q = 0; q < 4; q++)
                                h[pre_image(tile, c0 / 4 + q, rl)] =
                                    make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
                        }
                        const uint4 lo = make_uint4(w[0], w[1], w[2], w[3]), hi = make_uint4(w[4], w[5], w[6], w[7]);
                        uint4 *im = a.A[l] + img;
                        im[row_image(row, c0 / 8, kWidth)] = lo;
                        im[row_image(row, c0 / 8 + 1, kWidth)] = hi;
                        if (l < kDepth - 1) {
                            uint8_t *dst = Act + (c0 / umma::kBK) * kActChunk;
                            const int k = c0 % umma::kBK;
                            *reinterpret_cast<uint4 *>(dst + umma::tile_off(rl, k)) = lo;
                            *reinterpret_cast<uint4 *>(dst + umma::tile_off(rl, k + 8)) = hi;
                        } else {
                            // the head's per-8-column partial sums, as head_kernel's lanes form them
#pragma unroll
                            for (int h = 0; h < 2; h++) {
                                float sum = 0.0f;
#pragma unroll
                                for (int q = 0; q < 8; q++) {
                                    const uint32_t b = w[4 * h + (q >> 1)];
                                    sum += __uint_as_float(q & 1 ? b & 0xffff0000u : b << 16) *
                                           __ldg(w5 + 16 * g + 8 * h + q);
                                }
                                gs[(c0 / 8 + h) ^ lane] = sum;
                            }
                        }
                    }
                }
                if (l < kDepth - 1) {
                    done_job();
                    if (l == 0 && u + (int)gridDim.x < units) {   // the features have been read: the next unit's
                        if (ok)
                            gather(u + gridDim.x);
                        __syncwarp();
                        if (lane == 0)
                            mbar_arrive(&x0_ready);
                    }
                }
            }
            // ---- head, loss
            quarter_sync(quarter);
            if (ok && warp < 4) {
                float g[32];
#pragma unroll
                for (int jj = 0; jj < 32; jj++)
                    g[jj] = gs[jj ^ lane];
#pragma unroll
                for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                    for (int jj = 0; jj < o; jj++)
                        g[jj] = g[jj] + g[jj + o];
                const float out = g[0] + __ldg(P + kOffB5);
                const float diff = out - __ldg(a.target + drawn_row(a, step, e, (int)row));
                const float d = 2.0f * diff / (float)a.batch;
                a.y[(long long)e * a.batch + row] = out;
                a.dy[(long long)e * a.batch + row] = d;
                dys[rl] = d;
                float loss = diff * diff / (float)a.batch;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1)
                    loss += __shfl_xor_sync(0xffffffffu, loss, o);
                if (lane == 0)
                    atomicAdd(a.loss_acc + e, loss);
            }
            quarter_sync(quarter);
            // ---- dH_3 (the last hidden layer's), from its accumulator again
            if (ok) {
                const float gd = dys[rl];
                const float *bias = P + off_b(kDepth - 1) + cb;
                const uint32_t acc = tmem + (uint32_t)(job_acc(kDepth - 1) * kWidth + cb) + lane_base;
#pragma unroll 1
                for (int g = 0; g < 4; g++) {
                    const int c0 = cb + 16 * g;
                    float h[16], v[16];
                    umma::tmem_ld16_start(acc + 16 * g, h);
#pragma unroll
                    for (int q = 0; q < 16; q++)
                        v[q] = gd * __ldg(w5 + 16 * g + q);
                    umma::tmem_ld16_wait(h);
#pragma unroll
                    for (int q = 0; q < 16; q++)
                        h[q] += __ldg(bias + 16 * g + q);
                    uint32_t w[8];
                    gelu::grads_bf16<8>(v, h, w);
                    const uint4 lo = make_uint4(w[0], w[1], w[2], w[3]), hi = make_uint4(w[4], w[5], w[6], w[7]);
                    uint4 *im = a.dH[kDepth - 1] + img;
                    im[row_image(row, c0 / 8, kWidth)] = lo;
                    im[row_image(row, c0 / 8 + 1, kWidth)] = hi;
                    uint8_t *dst = Act + (c0 / umma::kBK) * kActChunk;
                    const int k = c0 % umma::kBK;
                    *reinterpret_cast<uint4 *>(dst + umma::tile_off(rl, k)) = lo;
                    *reinterpret_cast<uint4 *>(dst + umma::tile_off(rl, k + 8)) = hi;
                }
            }
            done_job();
            // ---- backward
            for (int l = kDepth - 2; l >= 0; l--) {
                const int j = 2 * kDepth - 2 - l;   // product 4 gives layer 2's gradient, 6 layer 0's
                const uint32_t acc = tmem + (uint32_t)(job_acc(j) * kWidth + cb) + lane_base;
                const uint32_t hacc = tmem + (uint32_t)(job_acc(2) * kWidth + cb) + lane_base;
                const float *bias = P + off_b(l) + cb;
                const float4 *hs = l < 2 ? a.H[l] : nullptr;
                wait_job();
                if (ok) {
#pragma unroll 1
                    for (int g = 0; g < 4; g++) {
                        const int c0 = cb + 16 * g;
                        float h[16], v[16];
                        if (l == 2) {
                            umma::tmem_ld16_start(hacc + 16 * g, h);
                            umma::tmem_ld16_start(acc + 16 * g, v);
                            umma::tmem_ld16_wait(h);
                            umma::tmem_ld16_wait(v);
#pragma unroll
                            for (int q = 0; q < 16; q++)
                                h[q] += __ldg(bias + 16 * g + q);
                        } else {
                            umma::tmem_ld16_start(acc + 16 * g, v);
#pragma unroll
                            for (int q = 0; q < 4; q++)
                                *reinterpret_cast<float4 *>(h + 4 * q) = hs[pre_image(tile, c0 / 4 + q, rl)];
                            umma::tmem_ld16_wait(v);
                        }
                        uint32_t w[8];
                        gelu::grads_bf16<8>(v, h, w);
                        const uint4 lo = make_uint4(w[0], w[1], w[2], w[3]), hi = make_uint4(w[4], w[5], w[6], w[7]);
                        uint4 *im = a.dH[l] + img;
                        im[row_image(row, c0 / 8, kWidth)] = lo;
                        im[row_image(row, c0 / 8 + 1, kWidth)] = hi;
                        if (l > 0) {
                            uint8_t *dst = Act + (c0 / umma::kBK) * kActChunk;
                            const int k = c0 % umma::kBK;
                            *reinterpret_cast<uint4 *>(dst + umma::tile_off(rl, k)) = lo;
                            *reinterpret_cast<uint4 *>(dst + umma::tile_off(rl, k + 8)) = hi;
                        }
                    }
                }
                done_job();
            }
        }
    }
    umma::tc_fence_before();
    __syncthreads();
    if (tid == 0 && s_abort)
        atomicOr(a.err, 1);
    if (warp == 0)
        umma::tmem_dealloc(tmem, 2 * kWidth);
}

// ---------------------------------------------------------------- gradients
//
// dW_l = dH_l^T A_{l-1} for one (member, layer, K split, half of the 256
// rows of dW_l): M = 128, N = 256 or 64, K = batch / 16 rows in blocks of 64,
// both operands MN-major straight from the row images.  Partial sums go out
// as [4-column group][128 rows][4], 512 contiguous bytes a warp and store.

constexpr int kDwStages = 2;
constexpr int kDwA = 16 * 1024;                     // 128 columns of a dH block
constexpr int kDwStage = kDwA + 32 * 1024;          // and 256 of an activation block
constexpr int kDwSmem = kDwStages * kDwStage;       // two CTAs an SM
constexpr int kDwThreads = 192;                     // four epilogue warps, copy, MMA

// floats of the partial sums before layer l of a member
__host__ __device__ constexpr long long part_off(int l)
{
    return l == 0 ? 0 : (long long)kSplitK * kWidth * (kFeat + (l - 1) * kWidth);
}
constexpr long long kPartFloats = (long long)kSplitK * kWidth * (kFeat + (kDepth - 1) * kWidth);

struct DwArgs {
    const uint4 *X0, *A[kDepth], *dH[kDepth];
    int batch;
    float4 *part;             // [E][kPartFloats]
    // the first block also closes the step's loss: its mean over the members
    // into the history and the step count (when there is one to close)
    unsigned *step;
    float *loss_acc, *loss_hist;
    int E, hist_len, count_step;
    int *err;
};

__global__ void __launch_bounds__(kDwThreads, 2) dw_kernel(DwArgs a)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ uint64_t full[kDwStages], empty[kDwStages], acc_full;
    __shared__ uint32_t tslot;
    __shared__ int s_abort;
    volatile int *abort = &s_abort;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int mh = blockIdx.x & 1, sp = (blockIdx.x >> 1) % kSplitK, l = (blockIdx.x >> 1) / kSplitK;
    const int e = blockIdx.y;
    const int K = l == 0 ? kFeat : kWidth;
    const int rows = a.batch / kSplitK, blocks = rows / 64;
    const long long block0 = (long long)sp * blocks;

    if (tid == 0) {
        for (int s = 0; s < kDwStages; s++) {
            umma::mbar_init(&full[s], 1);
            umma::mbar_init(&empty[s], 1);
        }
        umma::mbar_init(&acc_full, 1);
        s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0)
        umma::tmem_alloc(&tslot, kWidth);
    if (blockIdx.x == 0 && blockIdx.y == 0 && tid == 64) {
        float acc = 0.0f;
        for (int m = 0; m < a.E; m++) {
            acc += a.loss_acc[m];
            a.loss_acc[m] = 0.0f;
        }
        if (a.count_step) {
            const unsigned s = *a.step;
            if ((int)s < a.hist_len)
                a.loss_hist[s] = acc / (float)a.E;
            *a.step = s + 1u;
        }
    }
    umma::tc_fence_before();
    __syncthreads();
    umma::tc_fence_after();
    const uint32_t tmem = tslot;
    const uint32_t b_bytes = (uint32_t)K * 128u;    // 64 rows x K columns

    if (warp == 4) {
        if (lane == 0) {
            const uint8_t *A = reinterpret_cast<const uint8_t *>(a.dH[l] + (long long)e * a.batch * (kWidth / 8));
            const uint8_t *B =
                reinterpret_cast<const uint8_t *>((l == 0 ? a.X0 : a.A[l - 1]) + (long long)e * a.batch * (K / 8));
            int c = 0;
            for (; c < blocks; c++) {
                const int st = c % kDwStages;
                if (c >= kDwStages && !wait_or_abort(&empty[st], (uint32_t)((c / kDwStages - 1) & 1), abort))
                    break;
                uint8_t *dst = smem + st * kDwStage;
                mbar_expect_tx(&full[st], kDwA + b_bytes);
                bulk_g2s(dst, A + (block0 + c) * (kWidth * 128) + mh * kDwA, kDwA, &full[st]);
                bulk_g2s(dst + kDwA, B + (block0 + c) * b_bytes, b_bytes, &full[st]);
            }
            for (int p = c > kDwStages ? c - kDwStages : 0; p < c; p++)   // none in flight at the end
                wait_or_abort(&full[p % kDwStages], (uint32_t)((p / kDwStages) & 1), abort);
        }
        __syncwarp();
    } else if (warp == 5) {
        if (lane == 0) {
            // both operands MN-major (transpose bits of the instruction descriptor)
            const uint32_t idesc = umma::idesc_bf16_f32(K) | (1u << 15) | (1u << 16);
            bool ok = true;
            for (int c = 0; c < blocks; c++) {
                const int st = c % kDwStages;
                if (!wait_or_abort(&full[st], (uint32_t)((c / kDwStages) & 1), abort)) {
                    ok = false;
                    break;
                }
                const uint32_t a0 = umma::smem_u32(smem + st * kDwStage), b0 = a0 + kDwA;
#pragma unroll
                for (int kk = 0; kk < 4; kk++)   // 16 rows each
                    umma::mma_bf16(tmem, umma::smem_desc(a0 + kk * 256, 128, 1024),
                                   umma::smem_desc(b0 + kk * 256, 128, 1024), idesc, (c > 0 || kk > 0) ? 1u : 0u);
                umma::mma_commit(&empty[st]);
            }
            umma::mma_commit(&acc_full);
            if (!ok)
                *abort = 1;
        }
        __syncwarp();
    } else {
        bool ok = wait_or_abort(&acc_full, 0u, abort);
        ok = __all_sync(0xffffffffu, ok);
        if (ok) {
            umma::tc_fence_after();
            float4 *out = a.part + ((long long)e * kPartFloats + part_off(l) +
                                    (long long)(sp * 2 + mh) * (128 * K)) / 4;
            const uint32_t acc = tmem + ((uint32_t)(32 * warp) << 16);
            for (int c0 = 0; c0 < K; c0 += 16) {
                float v[16];
                umma::tmem_ld16(acc + c0, v);
#pragma unroll
                for (int q = 0; q < 4; q++)
                    out[(c0 / 4 + q) * 128 + 32 * warp + lane] =
                        make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
            }
        }
    }
    umma::tc_fence_before();
    __syncthreads();
    if (tid == 0 && s_abort)
        atomicOr(a.err, 1);
    if (warp == 0)
        umma::tmem_dealloc(tmem, kWidth);
}

// ------------------------------------------------------------------- update

struct AdamArgs {
    float lr_max, lr_min, b1, b2, eps;
    unsigned total;   // cosine decay from lr_max to lr_min over `total` steps
};

struct AdamStep {
    float lr, c1, c2;   // learning rate; 1 - b1^t, 1 - b2^t
};

// step s (counting from 0): t = s + 1
__device__ __forceinline__ AdamStep adam_step(const AdamArgs &a, unsigned s)
{
    const float t = (float)(s + 1u);
    const float frac = a.total ? fminf((float)s / (float)a.total, 1.0f) : 0.0f;
    AdamStep r;
    r.lr = a.lr_min + (a.lr_max - a.lr_min) * 0.5f * (1.0f + cospif(frac));
    r.c1 = 1.0f - powf(a.b1, t);
    r.c2 = 1.0f - powf(a.b2, t);
    return r;
}

__device__ __forceinline__ float adam(const AdamArgs &a, const AdamStep &s, float g, float &m, float &v, float p)
{
    // the fused products are spelled out: training amplifies a last bit
    const float mi = __fmaf_rn(1.0f - a.b1, g, __fmul_rn(a.b1, m));
    const float vi = __fmaf_rn(__fmul_rn(1.0f - a.b2, g), g, __fmul_rn(a.b2, v));
    m = mi;
    v = vi;
    const float mh = mi / s.c1;
    const float vh = vi / s.c2;
    return p - s.lr * mh / (sqrtf(vh) + a.eps);
}

// BF16 copies of a weight matrix: W[e][n][k] for the layer-by-layer path,
// the chunks of W for the forward products and of W^T for the backward ones
struct WeightCopies {
    bf16 *w[kDepth];
    uint8_t *wimg, *wtimg;
};

// byte offset of W_l[n][k] in the chunks of W_l of member e
__host__ __device__ constexpr long long image_off(int e, int l, int n, int k)
{
    return (long long)chunk_index(e, l, k / kWChunkK) * kChunkBytes + wchunk_off(n, k % kWChunkK);
}

// and of W_l^T (l >= 1): rows k, contraction over n
__host__ __device__ constexpr long long back_image_off(int e, int l, int n, int k)
{
    return ((long long)e * kChunksBack + (l - 1) * 8 + n / kWChunkK) * kChunkBytes + wchunk_off(k, n % kWChunkK);
}

struct UpdateArgs {
    const float4 *part;
    const uint4 *A3, *dH[kDepth];   // last activation, layer gradients (row images)
    const float *dy;
    int batch, E;
    float *params, *m, *v, *grad;
    const unsigned *step;           // already counted
    AdamArgs adam;
    int update;                     // Adam and the copies, or (0) the gradients into `grad`
    WeightCopies copies;
};

constexpr int kPatch = 32;          // weights in patches of 32 x 32
constexpr int kPatches0 = (kWidth / kPatch) * (kFeat / kPatch), kPatchesL = (kWidth / kPatch) * (kWidth / kPatch);
constexpr int kPatches = kPatches0 + (kDepth - 1) * kPatchesL;
constexpr int kVectors = (kDepth + 1) * (kWidth / 8) + 1;   // column sums: four biases, w5 (8 columns each); b5

// Blocks 0 .. kPatches - 1 of a member: a 32 x 32 patch of a weight matrix.
// The rest: column sums over the batch (bias gradients, the output weights'
// and bias's), each thread's rows and the order of the sums as in a block of
// 256 threads striding over the batch.
__global__ void __launch_bounds__(256) update_kernel(UpdateArgs a)
{
    const int e = blockIdx.y, tid = threadIdx.x;
    const AdamStep st = a.update ? adam_step(a.adam, *a.step - 1u) : AdamStep{0.0f, 1.0f, 1.0f};
    float *P = a.params + (long long)e * kParams;
    const long long pe = (long long)e * kParams;
    __shared__ float g[kPatch][kPatch + 1];
    if (blockIdx.x < kPatches) {
        int b = blockIdx.x, l = 0;
        if (b >= kPatches0) {
            b -= kPatches0;
            l = 1 + b / kPatchesL;
            b %= kPatchesL;
        }
        const int K = in_dim(l), per_row = K / kPatch;
        const int n0 = b / per_row * kPatch, k0 = b % per_row * kPatch;
        {
            // thread: row n0 + lane, columns k0 + 4 * warp ..; the splits in order
            const int lane = tid & 31, c4 = k0 / 4 + (tid >> 5);
            const float4 *p = a.part + (pe / kParams * kPartFloats + part_off(l)) / 4 +
                              ((long long)(n0 / 128) * (K / 4) + c4) * 128 + n0 % 128 + lane;
            const long long stride = (long long)2 * 32 * K;   // float4s of a split: 256 K / 4
            float4 v[kSplitK];
#pragma unroll
            for (int s = 0; s < kSplitK; s++)
                v[s] = __ldg(p + s * stride);
            float4 t = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
            for (int s = 0; s < kSplitK; s++) {
                t.x += v[s].x;
                t.y += v[s].y;
                t.z += v[s].z;
                t.w += v[s].w;
            }
            float *row = &g[lane][4 * (tid >> 5)];
            row[0] = t.x;
            row[1] = t.y;
            row[2] = t.z;
            row[3] = t.w;
        }
        __syncthreads();
        const int r = tid >> 3, c = 4 * (tid & 7);   // four weights along k
        const long long o = pe + off_w(l) + (long long)(n0 + r) * K + k0 + c;
        if (!a.update) {
            *reinterpret_cast<float4 *>(a.grad + o) = make_float4(g[r][c], g[r][c + 1], g[r][c + 2], g[r][c + 3]);
            return;
        }
        float4 p4 = *reinterpret_cast<float4 *>(a.params + o), m4 = *reinterpret_cast<float4 *>(a.m + o),
               v4 = *reinterpret_cast<float4 *>(a.v + o);
        float *pp = &p4.x, *mm = &m4.x, *vv = &v4.x;
#pragma unroll
        for (int q = 0; q < 4; q++)
            pp[q] = adam(a.adam, st, g[r][c + q], mm[q], vv[q], pp[q]);
        *reinterpret_cast<float4 *>(a.params + o) = p4;
        *reinterpret_cast<float4 *>(a.m + o) = m4;
        *reinterpret_cast<float4 *>(a.v + o) = v4;
        const uint2 w = make_uint2(gelu::bf16x2(pp[0], pp[1]), gelu::bf16x2(pp[2], pp[3]));
        *reinterpret_cast<uint2 *>(a.copies.w[l] + (long long)e * kWidth * K + (long long)(n0 + r) * K + k0 + c) = w;
        *reinterpret_cast<uint2 *>(a.copies.wimg + image_off(e, l, n0 + r, k0 + c)) = w;
        if (l > 0) {
            __syncthreads();
#pragma unroll
            for (int q = 0; q < 4; q++)
                g[r][c + q] = pp[q];
            __syncthreads();
            // four weights along n of column k0 + r
            const uint2 wt = make_uint2(gelu::bf16x2(g[c][r], g[c + 1][r]), gelu::bf16x2(g[c + 2][r], g[c + 3][r]));
            *reinterpret_cast<uint2 *>(a.copies.wtimg + back_image_off(e, l, n0 + c, k0 + r)) = wt;
        }
        return;
    }
    // ---- column sums
    const int b = blockIdx.x - kPatches;
    const int lane = tid & 31, warp = tid >> 5;
    __shared__ float red[8][8];
    const bool last = b == kVectors - 1;             // b5
    const int l = b / (kWidth / 8), group = b % (kWidth / 8);
    float acc[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    const float *dy = a.dy + (long long)e * a.batch;
    if (last) {
        for (int r = tid; r < a.batch; r += 256)
            acc[0] += dy[r];
    } else {
        const uint4 *im = (l < kDepth ? a.dH[l] : a.A3) + (long long)e * a.batch * (kWidth / 8);
#pragma unroll 4
        for (int r = tid; r < a.batch; r += 256) {
            const uint4 x = __ldg(im + row_image(r, group, kWidth));
            const float w = l < kDepth ? 1.0f : dy[r];
            const uint32_t u[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
            for (int q = 0; q < 8; q++)
                acc[q] += __uint_as_float(q & 1 ? u[q >> 1] & 0xffff0000u : u[q >> 1] << 16) * w;
        }
    }
#pragma unroll
    for (int q = 0; q < 8; q++) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            acc[q] += __shfl_xor_sync(0xffffffffu, acc[q], o);
        if (lane == 0)
            red[q][warp] = acc[q];
    }
    __syncthreads();
    if (tid < (last ? 1 : 8)) {
        float s[8];
#pragma unroll
        for (int w = 0; w < 8; w++)
            s[w] = red[tid][w];
#pragma unroll
        for (int o = 4; o > 0; o >>= 1)
#pragma unroll
            for (int w = 0; w < o; w++)
                s[w] += s[w + o];
        const long long o = last ? kOffB5 : (l < kDepth ? off_b(l) + 8 * group + tid : kOffW5 + 8 * group + tid);
        if (!a.update) {
            a.grad[pe + o] = s[0];
        } else {
            P[o] = adam(a.adam, st, s[0], a.m[pe + o], a.v[pe + o], P[o]);
        }
    }
}

// BF16 copies of all weights from the FP32 masters
__global__ void copies_kernel(const float *__restrict__ params, int E, WeightCopies c)
{
    constexpr int kPer = kWidth * (kFeat + (kDepth - 1) * kWidth);
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < (long long)E * kPer;
         t += (long long)gridDim.x * blockDim.x) {
        const int e = (int)(t / kPer);
        int i = (int)(t - (long long)e * kPer), l = 0;
        if (i >= kWidth * kFeat) {
            i -= kWidth * kFeat;
            l = 1 + i / (kWidth * kWidth);
            i %= kWidth * kWidth;
        }
        const int K = in_dim(l), n = i / K, k = i % K;
        const bf16 w = __float2bfloat16_rn(params[e * kParams + off_w(l) + i]);
        c.w[l][(long long)e * kWidth * K + i] = w;
        *reinterpret_cast<bf16 *>(c.wimg + image_off(e, l, n, k)) = w;
        if (l > 0)
            *reinterpret_cast<bf16 *>(c.wtimg + back_image_off(e, l, n, k)) = w;
    }
}
