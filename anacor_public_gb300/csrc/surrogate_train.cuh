// One training step of the surrogate as two kernels.  Included by
// surrogate.cu after the fused inference kernel, whose helpers it uses.
//
//   chain_kernel   a 128-row tile of one member's batch: gather, the four
//                  forward layers, head and loss, and the three backward
//                  products dH_{l-1} = (dH_l W_l) gelu'(H_{l-1}), all of which
//                  need the tile's own rows only;
//   update_kernel  the weight gradients dH_l^T A_{l-1} and the sums for the
//                  biases, Adam, and the BF16 weights in the layouts the
//                  products read.
//
// Step by step (a GEMM per layer and direction, transposed copies, sums,
// Adam, conversions: 40 launches) it took 411 us for four members at a batch
// of 4,096.  The numbers are the same: every product accumulates over the same
// K order, the K splits and column sums are added in the same order and the
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
constexpr int kOffChainVec = kOffChainDy + kTileRows * 4;          // a unit's biases and output weights, two units
constexpr int kVecFloats = (kDepth + 1) * kWidth;
constexpr int kChainSmem = kOffChainVec + 2 * kVecFloats * 4;
constexpr int kChainStages = 8;
constexpr int kActChunks = kWidth / umma::kBK;                    // 64-column chunks of an operand
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

// Bound by the epilogues, one after the other: a layer's 32,768 values a tile
// take 8 to 12 thousand cycles (issue 55 % busy meanwhile, the pre-activations'
// 128 KB a layer to L2 and back, values that the rounding test leaves open in
// one warp or other), its product 2 to 4.5 thousand, of which the first
// three quarters run beside the epilogue before it where the accumulator is
// free.  Four members, a batch of 4,096 (128 tiles): 64.6 us with a product
// waiting for its whole operand, biases from L2 for every 16 columns and the
// pre-activations fetched where they are used; 58 us so.  (Two accumulator
// pieces in flight a warp spill: 96 registers are all that 18 warps leave.)
constexpr int kChainThreads = 32 * (kEpiWarps + 2);                // the epilogue's, MMA, copy

__global__ void __launch_bounds__(kChainThreads, 1) chain_kernel(ChainArgs a)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ uint64_t full[kChainStages], empty[kChainStages], acc_full, act_ready[kActChunks], x0_ready;
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
        for (int s = 0; s < kActChunks; s++)
            umma::mbar_init(&act_ready[s], kEpiWarps);
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
    // whether product j may start on the first columns of its operand while the
    // epilogue writes the others: its accumulator is not being read by it
    auto job_early = [](int j) { return (j >= 1 && j <= 3) || j == 6; };

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
                    int ready = 0;   // column chunks of the operand known to be written
                    const int at_least = job_early(j) ? 1 : kActChunks;
                    for (; ok && jobs > 0 && ready < at_least; ready++)
                        ok = wait_or_abort(&act_ready[ready], (jobs - 1u) & 1u, abort);
                    if (!ok)
                        break;
                    umma::tc_fence_after();
                    const uint8_t *A = j == 0 ? X0s : Act;
                    const uint32_t d = tmem + (uint32_t)(job_acc(j) * kWidth);
                    for (int kc = 0; kc < job_nk(j); kc++, q++) {
                        const int st = (int)(q % kChainStages);
                        for (; ok && jobs > 0 && ready <= kc * kWChunkK / umma::kBK; ready++)
                            ok = wait_or_abort(&act_ready[ready], (jobs - 1u) & 1u, abort);
                        if (!ok || !wait_or_abort(&full[st], (uint32_t)((q / kChainStages) & 1), abort)) {
                            ok = false;
                            break;
                        }
                        umma::tc_fence_after();
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
        // piece g of a warp: columns 64 g + cb .. + 15, so that all warps finish
        // a 64-column chunk of the next operand together
        const int quarter = warp & 3, rl = 32 * quarter + lane, cb = 16 * (warp >> 2);
        const uint32_t lane_base = (uint32_t)(32 * quarter) << 16;
        float *gs = reinterpret_cast<float *>(Act + quarter * kQuarterBytes) + 32 * lane;
        const unsigned step = *a.step;
        uint32_t jobs = 0;
        bool ok = true;
        // a unit's features: into the layer-0 operand and its row image
        // the unit after `unit` units of this CTA: also its biases and output
        // weights, which from global memory cost each piece an L2 access
        auto gather = [&](int u, uint32_t unit) {
            const int e = u / tiles, t = u - e * tiles;
            float *vec = reinterpret_cast<float *>(smem + kOffChainVec) + (unit & 1u) * kVecFloats;
            const float *P = a.params + (long long)e * kParams;
            for (int i = tid; i < kVecFloats; i += 32 * kEpiWarps)
                vec[i] = i < kDepth * kWidth ? __ldg(P + off_b(i / kWidth) + i % kWidth)
                                             : __ldg(P + kOffW5 + i - kDepth * kWidth);
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
        auto done_chunk = [&](int g) {
            umma::tc_fence_before();
            umma::fence_async_smem();
            __syncwarp();
            if (lane == 0)
                mbar_arrive(&act_ready[g]);
        };
        // 16 values of a row to its image and into the next operand
        auto keep = [&](uint4 *im, long long row, int c0, const uint32_t *w, bool operand) {
            const uint4 lo = make_uint4(w[0], w[1], w[2], w[3]), hi = make_uint4(w[4], w[5], w[6], w[7]);
            if (operand) {
                uint8_t *dst = Act + (c0 / umma::kBK) * kActChunk;
                const int k = c0 % umma::kBK;
                *reinterpret_cast<uint4 *>(dst + umma::tile_off(rl, k)) = lo;
                *reinterpret_cast<uint4 *>(dst + umma::tile_off(rl, k + 8)) = hi;
            }
            im[row_image(row, c0 / 8, kWidth)] = lo;
            im[row_image(row, c0 / 8 + 1, kWidth)] = hi;
        };
        if ((int)blockIdx.x < units) {
            gather(blockIdx.x, 0u);
            __syncwarp();
            if (lane == 0)
                mbar_arrive(&x0_ready);
        }
        uint32_t unit = 0;
        for (int u = blockIdx.x; u < units; u += gridDim.x, unit++) {
            const int e = u / tiles, t = u - e * tiles;
            const long long row = (long long)t * kTileRows + rl;     // of the member's batch
            const long long tile = (long long)e * tiles + t;
            const long long img = (long long)e * a.batch * (kWidth / 8);
            const float *P = a.params + (long long)e * kParams;
            const float *vec = reinterpret_cast<const float *>(smem + kOffChainVec) + (unit & 1u) * kVecFloats + cb;
            const float *w5 = vec + kDepth * kWidth;
            asm volatile("bar.sync 5, 512;" ::: "memory");   // `vec` is written by all epilogue warps
            // ---- forward
            for (int l = 0; l < kDepth; l++) {
                const uint32_t acc = tmem + (uint32_t)(job_acc(l) * kWidth + cb) + lane_base;
                const float *bias = vec + l * kWidth;
                wait_job();
                auto piece = [&](int g, float *v) {
                    const int c0 = 64 * g + cb;
                    uint32_t w[8];
                    gelu::values_bf16<8>(v, bias + 64 * g, w);
                    keep(a.A[l] + img, row, c0, w, l < kDepth - 1);
                    if (l < 2) {
                        float4 *h = a.H[l];
#pragma unroll
                        for (int q = 0; q < 4; q++)
                            h[pre_image(tile, c0 / 4 + q, rl)] =
                                make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
                    }
                    if (l == kDepth - 1) {
                        // the head's per-8-column partial sums, as head_kernel's lanes form them
#pragma unroll
                        for (int h = 0; h < 2; h++) {
                            float sum = 0.0f;
#pragma unroll
                            for (int q = 0; q < 8; q++) {
                                const uint32_t b = w[4 * h + (q >> 1)];
                                sum += __uint_as_float(q & 1 ? b & 0xffff0000u : b << 16) * w5[64 * g + 8 * h + q];
                            }
                            gs[(c0 / 8 + h) ^ lane] = sum;
                        }
                    }
                };
#pragma unroll 1
                for (int g = 0; g < 4; g++) {
                    if (ok) {
                        float v[16];
                        umma::tmem_ld16(acc + 64 * g, v);
                        piece(g, v);
                    }
                    if (l < kDepth - 1)
                        done_chunk(g);
                }
                if (l == 0 && u + (int)gridDim.x < units) {   // the features have been read: the next unit's
                    if (ok)
                        gather(u + gridDim.x, unit + 1u);
                    __syncwarp();
                    if (lane == 0)
                        mbar_arrive(&x0_ready);
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
            {
                const float gd = ok ? dys[rl] : 0.0f;
                const float *bias = vec + (kDepth - 1) * kWidth;
                const uint32_t acc = tmem + (uint32_t)(job_acc(kDepth - 1) * kWidth + cb) + lane_base;
#pragma unroll 1
                for (int g = 0; g < 4; g++) {
                    if (ok) {
                        float h[16], v[16];
                        umma::tmem_ld16_start(acc + 64 * g, h);
#pragma unroll
                        for (int q = 0; q < 16; q++)
                            v[q] = gd * w5[64 * g + q];
                        umma::tmem_ld16_wait(h);
#pragma unroll
                        for (int q = 0; q < 16; q++)
                            h[q] += bias[64 * g + q];
                        uint32_t w[8];
                        gelu::grads_bf16<8>(v, h, w);
                        keep(a.dH[kDepth - 1] + img, row, 64 * g + cb, w, true);
                    }
                    done_chunk(g);
                }
            }
            // ---- backward
            for (int l = kDepth - 2; l >= 0; l--) {
                const int j = 2 * kDepth - 2 - l;   // product 4 gives layer 2's gradient, 6 layer 0's
                const uint32_t acc = tmem + (uint32_t)(job_acc(j) * kWidth + cb) + lane_base;
                const uint32_t hacc = tmem + (uint32_t)(job_acc(2) * kWidth + cb) + lane_base;
                const float *bias = vec + l * kWidth;
                const float4 *hs = l < 2 ? a.H[l] : nullptr;
                // layers 0 and 1: the pre-activations come from L2, a piece ahead
                auto fetch = [&](int g, float *h) {
#pragma unroll
                    for (int q = 0; q < 4; q++)
                        *reinterpret_cast<float4 *>(h + 4 * q) = hs[pre_image(tile, (64 * g + cb) / 4 + q, rl)];
                };
                auto piece = [&](int g, float *h, float *v) {
                    if (l == 2) {
                        umma::tmem_ld16_start(hacc + 64 * g, h);
                        umma::tmem_ld16_start(acc + 64 * g, v);
                        umma::tmem_ld16_wait(h);
                        umma::tmem_ld16_wait(v);
#pragma unroll
                        for (int q = 0; q < 16; q++)
                            h[q] += bias[64 * g + q];
                    } else {
                        umma::tmem_ld16(acc + 64 * g, v);
                    }
                    uint32_t w[8];
                    gelu::grads_bf16<8>(v, h, w);
                    keep(a.dH[l] + img, row, 64 * g + cb, w, l > 0);
                };
                float h[16];
                if (ok && l < 2)
                    fetch(0, h);
                wait_job();
#pragma unroll 1
                for (int g = 0; g < 4; g++) {
                    if (ok) {
                        float v[16];
                        piece(g, h, v);
                        if (l < 2 && g + 1 < 4)
                            fetch(g + 1, h);
                    }
                    done_chunk(g);
                }
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

// --------------------------------------------------------- gradients, update

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

// One launch for the weight gradients dW_l = dH_l^T A_{l-1}, the column sums
// over the batch (bias gradients, the output weights' and bias's), Adam and
// the weights' BF16 copies.
//
// Blocks 0 .. E * kGradTiles - 1: a tile of 128 x 64 weights of one matrix, the
// whole batch.  Both operands come MN-major straight from the row images, 64
// rows a stage; each K split (batch / kSplitK rows) has an accumulator of its
// own, four of them in a ring, and the epilogue adds the splits in order while
// the next are computed, so no partial sums are stored: a kernel with a CTA a
// split and one that added them moved 110 MB between them.  Bound by the
// operands' way from L2, 1.5 MB a tile (64 columns a tile are 104 tiles for
// four members at a batch of 4,096, one an SM; 32 columns would be 2.5 MB an
// SM), with eight stages of 24 KB in flight, and by Adam's quotients at the
// end.  23 + 22 us as two kernels, 40 so.
// The rest: column sums, a task (eight columns of an image) after the other,
// on the SMs that the tiles leave; each thread's rows and the order of the
// sums as in a block of 256 threads striding over the batch.

struct UpdateArgs {
    const uint4 *X0, *A[kDepth], *dH[kDepth];   // row images
    const float *dy;
    int batch, E;
    float *params, *m, *v, *grad;
    AdamArgs adam;
    int update;                     // Adam, the copies and the step count, or (0) the gradients into `grad`
    WeightCopies copies;
    // The last block to have read the step count closes the step: the loss, its
    // mean over the members into the history, and the count.
    unsigned *step, *ticket;
    float *loss_acc, *loss_hist;
    int hist_len;
    int *err;
};

constexpr int kGradCols = 64;
constexpr int kGradTiles = 2 + (kDepth - 1) * 2 * (kWidth / kGradCols);   // per member
constexpr int kGradStages = 8;
constexpr int kGradA = 16 * 1024;                              // 128 columns of a dH block
constexpr int kGradStage = kGradA + kGradCols * 128;           // and 64 of an activation block
constexpr int kGradSmem = kGradStages * kGradStage;            // 192 KB: one CTA an SM
constexpr int kGradAccs = 4;
constexpr int kGradThreads = 320;                              // eight epilogue warps, copy, MMA
constexpr int kGradPitch = kGradCols + 1;                      // floats a row of the gradient tile
static_assert(128 * kGradPitch * 4 <= kGradSmem, "the gradient tile reuses the stages");
constexpr int kVectors = (kDepth + 1) * (kWidth / 8) + 1;      // column sums: four biases, w5 (8 columns each); b5

__device__ __forceinline__ void sync_256() { asm volatile("bar.sync 1, 256;" ::: "memory"); }

// column sums of task b of member e (256 threads)
__device__ __forceinline__ void column_sums(const UpdateArgs &a, const AdamStep &st, int e, int b, float (*red)[8])
{
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const long long pe = (long long)e * kParams;
    const bool last = b == kVectors - 1;             // b5
    const int l = b / (kWidth / 8), group = b % (kWidth / 8);
    float acc[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    const float *dy = a.dy + (long long)e * a.batch;
    if (last) {
        for (int r = tid; r < a.batch; r += 256)
            acc[0] += dy[r];
    } else {
        const uint4 *im = (l < kDepth ? a.dH[l] : a.A[kDepth - 1]) + (long long)e * a.batch * (kWidth / 8);
#pragma unroll 16
        for (int r = tid; r < a.batch; r += 256) {
            const uint4 x = __ldg(im + row_image(r, group, kWidth));
            const float w = l < kDepth ? 1.0f : dy[r];
            const uint32_t u[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
            for (int q = 0; q < 8; q++)
                acc[q] += __uint_as_float(q & 1 ? u[q >> 1] & 0xffff0000u : u[q >> 1] << 16) * w;
        }
    }
    sync_256();   // the last task's sums have been read
#pragma unroll
    for (int q = 0; q < 8; q++) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            acc[q] += __shfl_xor_sync(0xffffffffu, acc[q], o);
        if (lane == 0)
            red[q][warp] = acc[q];
    }
    sync_256();
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
        const long long o = pe + (last ? kOffB5 : (l < kDepth ? off_b(l) : kOffW5) + 8 * group + tid);
        if (!a.update)
            a.grad[o] = s[0];
        else
            a.params[o] = adam(a.adam, st, s[0], a.m[o], a.v[o], a.params[o]);
    }
}

// Adam and the copies of the tile g of gradients (256 threads): rows n0 ..,
// columns k0 .. of W_l of member e
__device__ __forceinline__ void update_tile(const UpdateArgs &a, const AdamStep &st, int e, int l, int n0, int k0,
                                            float (*g)[kGradPitch])
{
    const int tid = threadIdx.x, K = in_dim(l);
    const long long base = (long long)e * kParams + off_w(l);
    // four weights along k a thread and pass; the loads of four passes together
    constexpr int kPasses = 128 * (kGradCols / 4) / 256, kAhead = 4;
    const int c = 4 * (tid % (kGradCols / 4)), r0 = tid / (kGradCols / 4);
    constexpr int kRowStep = 256 / (kGradCols / 4);
    for (int i0 = 0; i0 < kPasses; i0 += kAhead) {
        float4 p4[kAhead], m4[kAhead], v4[kAhead];
#pragma unroll
        for (int i = 0; i < kAhead; i++) {
            const int r = r0 + (i0 + i) * kRowStep;
            const long long o = base + (long long)(n0 + r) * K + k0 + c;
            if (!a.update) {
                *reinterpret_cast<float4 *>(a.grad + o) = make_float4(g[r][c], g[r][c + 1], g[r][c + 2], g[r][c + 3]);
                continue;
            }
            p4[i] = *reinterpret_cast<const float4 *>(a.params + o);
            m4[i] = *reinterpret_cast<const float4 *>(a.m + o);
            v4[i] = *reinterpret_cast<const float4 *>(a.v + o);
        }
        if (!a.update)
            continue;
#pragma unroll
        for (int i = 0; i < kAhead; i++) {
            const int r = r0 + (i0 + i) * kRowStep;
            const long long o = base + (long long)(n0 + r) * K + k0 + c;
            float *pp = &p4[i].x, *mm = &m4[i].x, *vv = &v4[i].x;
#pragma unroll
            for (int q = 0; q < 4; q++) {
                pp[q] = adam(a.adam, st, g[r][c + q], mm[q], vv[q], pp[q]);
                g[r][c + q] = pp[q];
            }
            *reinterpret_cast<float4 *>(a.params + o) = p4[i];
            *reinterpret_cast<float4 *>(a.m + o) = m4[i];
            *reinterpret_cast<float4 *>(a.v + o) = v4[i];
            const uint2 w = make_uint2(gelu::bf16x2(pp[0], pp[1]), gelu::bf16x2(pp[2], pp[3]));
            *reinterpret_cast<uint2 *>(a.copies.w[l] + (long long)e * kWidth * K + (long long)(n0 + r) * K + k0 + c) =
                w;
            *reinterpret_cast<uint2 *>(a.copies.wimg + image_off(e, l, n0 + r, k0 + c)) = w;
        }
    }
    if (!a.update || l == 0)
        return;
    sync_256();
#pragma unroll 2
    for (int i = tid; i < kGradCols * 32; i += 256) {
        const int r = i / 32, n = 4 * (i % 32);   // four weights along n of column k0 + r
        const uint2 w = make_uint2(gelu::bf16x2(g[n][r], g[n + 1][r]), gelu::bf16x2(g[n + 2][r], g[n + 3][r]));
        *reinterpret_cast<uint2 *>(a.copies.wtimg + back_image_off(e, l, n0 + n, k0 + r)) = w;
    }
}

__global__ void __launch_bounds__(kGradThreads, 1) update_kernel(UpdateArgs a)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ uint64_t full[kGradStages], empty[kGradStages], acc_full[kGradAccs], acc_empty[kGradAccs];
    __shared__ uint32_t tslot;
    __shared__ int s_abort, s_bad;   // s_bad: of the epilogue warps, decided at a barrier
    __shared__ float red[8][8];
    volatile int *abort = &s_abort;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int tiles = a.E * kGradTiles;
    const bool is_tile = (int)blockIdx.x < tiles;
    const AdamStep st = a.update ? adam_step(a.adam, *(volatile unsigned *)a.step) : AdamStep{0.0f, 1.0f, 1.0f};

    if (tid == 0) {
        for (int s = 0; s < kGradStages; s++) {
            umma::mbar_init(&full[s], 1);
            umma::mbar_init(&empty[s], 1);
        }
        for (int s = 0; s < kGradAccs; s++) {
            umma::mbar_init(&acc_full[s], 1);
            umma::mbar_init(&acc_empty[s], 8);
        }
        s_abort = s_bad = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0 && is_tile)
        umma::tmem_alloc(&tslot, kGradAccs * kGradCols);
    umma::tc_fence_before();
    __syncthreads();
    umma::tc_fence_after();
    if (tid == 0) {   // this block has read the step count
        __threadfence();
        if (atomicAdd(a.ticket, 1u) == gridDim.x - 1) {
            *a.ticket = 0u;
            float acc = 0.0f;
            for (int m = 0; m < a.E; m++) {
                acc += a.loss_acc[m];
                a.loss_acc[m] = 0.0f;
            }
            if (a.update) {
                const unsigned s = *(volatile unsigned *)a.step;
                if ((int)s < a.hist_len)
                    a.loss_hist[s] = acc / (float)a.E;
                *a.step = s + 1u;
            }
        }
    }
    if (!is_tile) {
        if (warp < 8)
            for (int q = (int)blockIdx.x - tiles; q < a.E * kVectors; q += (int)gridDim.x - tiles)
                column_sums(a, st, q / kVectors, q % kVectors, red);
        return;
    }

    const uint32_t tmem = tslot;
    const int e = blockIdx.x / kGradTiles, t = blockIdx.x % kGradTiles;
    const int l = t < 2 ? 0 : 1 + (t - 2) / (2 * (kWidth / kGradCols));
    const int mh = t & 1, nt = t < 2 ? 0 : (t - 2) / 2 % (kWidth / kGradCols);
    const int per = a.batch / kSplitK / 64, blocks = kSplitK * per;   // 64-row blocks of a split, of the batch
    if (warp == 8) {
        if (lane == 0) {
            const int K = in_dim(l);
            const uint8_t *A =
                reinterpret_cast<const uint8_t *>(a.dH[l] + (long long)e * a.batch * (kWidth / 8)) + mh * kGradA;
            const uint8_t *B =
                reinterpret_cast<const uint8_t *>((l == 0 ? a.X0 : a.A[l - 1]) + (long long)e * a.batch * (K / 8)) +
                nt * (kGradCols * 128);
            int c = 0;
            for (; c < blocks; c++) {
                const int s = c % kGradStages;
                if (c >= kGradStages && !wait_or_abort(&empty[s], (uint32_t)((c / kGradStages - 1) & 1), abort))
                    break;
                uint8_t *dst = smem + s * kGradStage;
                mbar_expect_tx(&full[s], kGradStage);
                bulk_g2s(dst, A + (long long)c * (kWidth * 128), kGradA, &full[s]);
                bulk_g2s(dst + kGradA, B + (long long)c * (K * 128), kGradCols * 128, &full[s]);
            }
            for (int p = c > kGradStages ? c - kGradStages : 0; p < c; p++)   // none in flight at the end
                wait_or_abort(&full[p % kGradStages], (uint32_t)((p / kGradStages) & 1), abort);
        }
        __syncwarp();
    } else if (warp == 9) {
        if (lane == 0) {
            // both operands MN-major (transpose bits of the instruction descriptor)
            constexpr uint32_t idesc = umma::idesc_bf16_f32(kGradCols) | (1u << 15) | (1u << 16);
            bool ok = true;
            for (int sp = 0, c = 0; sp < kSplitK && ok; sp++) {
                const int q = sp % kGradAccs;
                if (sp >= kGradAccs)
                    ok = wait_or_abort(&acc_empty[q], (uint32_t)((sp / kGradAccs - 1) & 1), abort);
                umma::tc_fence_after();
                for (int i = 0; i < per && ok; i++, c++) {
                    const int s = c % kGradStages;
                    ok = wait_or_abort(&full[s], (uint32_t)((c / kGradStages) & 1), abort);
                    if (!ok)
                        break;
                    const uint32_t a0 = umma::smem_u32(smem + s * kGradStage), b0 = a0 + kGradA;
#pragma unroll
                    for (int kk = 0; kk < 4; kk++)   // 16 rows each
                        umma::mma_bf16(tmem + (uint32_t)(q * kGradCols), umma::smem_desc(a0 + kk * 256, 128, 1024),
                                       umma::smem_desc(b0 + kk * 256, 128, 1024), idesc, (i > 0 || kk > 0) ? 1u : 0u);
                    umma::mma_commit(&empty[s]);
                }
                if (ok)
                    umma::mma_commit(&acc_full[q]);
            }
            if (!ok)
                *abort = 1;
        }
        __syncwarp();
    } else {
        const int quarter = warp & 3, c0 = 32 * (warp >> 2);
        const uint32_t acc = tmem + ((uint32_t)(32 * quarter) << 16) + (uint32_t)c0;
        float sum[32];
#pragma unroll
        for (int j = 0; j < 32; j++)
            sum[j] = 0.0f;
        bool ok = true;
        for (int sp = 0; sp < kSplitK; sp++) {
            const int q = sp % kGradAccs;
            ok = ok && wait_or_abort(&acc_full[q], (uint32_t)((sp / kGradAccs) & 1), abort);
            ok = __all_sync(0xffffffffu, ok);
            if (ok) {
                float v[16], w[16];
                umma::tc_fence_after();
                umma::tmem_ld16_start(acc + q * kGradCols, v);
                umma::tmem_ld16_start(acc + q * kGradCols + 16, w);
                umma::tmem_ld16_wait(v);
                umma::tmem_ld16_wait(w);
#pragma unroll
                for (int j = 0; j < 16; j++) {
                    sum[j] += v[j];
                    sum[16 + j] += w[j];
                }
                umma::tc_fence_before();
            }
            __syncwarp();
            if (lane == 0)
                mbar_arrive(&acc_empty[q]);
        }
        // all products are done: the stages hold the gradient tile now
        float(*g)[kGradPitch] = reinterpret_cast<float(*)[kGradPitch]>(smem);
        if (!ok)
            s_bad = s_abort = 1;
        sync_256();
        if (!s_bad) {
#pragma unroll
            for (int j = 0; j < 32; j++)
                g[32 * quarter + lane][c0 + j] = sum[j];
            sync_256();
            update_tile(a, st, e, l, 128 * mh, kGradCols * nt, g);
        }
    }
    umma::tc_fence_before();
    __syncthreads();
    if (tid == 0 && s_abort)
        atomicOr(a.err, 1);
    if (warp == 0)
        umma::tmem_dealloc(tmem, kGradAccs * kGradCols);
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
