// Interpolation kernels of the gridding (absorption-map) mode.
//
// The reference's interpolation (AnACor/src/gridding_interpolation.c:100-163)
// takes, per reflection, the two legs' polar angles, reads each voxel's map
// value at both (nearest neighbour, :16-45, or GSL bilinear, :48-76) and
// averages exp(-(z_incident + z_diffracted)) over the voxels.  The host
// computes the grid rows and weights of every reflection exactly as the
// reference does (FP64, same expressions); one CTA per reflection then streams
// the voxels: with the map stored direction-major ([direction][voxel]) the
// two (or eight) rows a reflection reads are contiguous, so the kernel is a
// coalesced read of 2 x 4 bytes per voxel (HBM-bound), four voxels per 16-byte
// load.  For nearest lookups exp runs in FP32 on the FP32 sum of the two map
// values (within 1e-7 relative of the reference's FP64 sum and exp); bilinear
// lookups carry the FP64 weights and the range reduction on pairs of floats.  The mean is a
// compensated FP32 sum.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "device_math.cuh"
#include "trace_launch.h"

namespace anacor {
namespace {

constexpr int kInterpBlock = 256;

template <class T>
__device__ __forceinline__ double leg_value(const T *mk, const long long *o, const double *w, bool linear)
{
    if (!linear)
        return (double)mk[o[0]];
    // (((w0 z0 + w1 z1) + w2 z2) + w3 z3): the bilinear sum's left-to-right order
    double z = __dmul_rn(w[0], (double)mk[o[0]]);
    z = __dadd_rn(z, __dmul_rn(w[1], (double)mk[o[1]]));
    z = __dadd_rn(z, __dmul_rn(w[2], (double)mk[o[2]]));
    return __dadd_rn(z, __dmul_rn(w[3], (double)mk[o[3]]));
}

template <class T, bool kVec4>
__global__ void __launch_bounds__(kInterpBlock) gridding_interp_kernel(const T *__restrict__ map, long long sK,
                                                                       long long sR, int n_vox,
                                                                       const InterpRow *__restrict__ rows,
                                                                       long long n_refl, int linear,
                                                                       double *__restrict__ out)
{
    __shared__ float red_s[kInterpBlock / 32], red_c[kInterpBlock / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (long long r = blockIdx.x; r < n_refl; r += gridDim.x) {
        long long o0[4], o1[4];
        double w0[4], w1[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            o0[j] = __ldg(&rows[r].row[0][j]) * sR;
            o1[j] = __ldg(&rows[r].row[1][j]) * sR;
            w0[j] = __ldg(&rows[r].w[0][j]);
            w1[j] = __ldg(&rows[r].w[1][j]);
        }
        float s = 0.0f, c = 0.0f;
        int k0 = 0;
        if (kVec4 && !linear) {
            // direction-major float map, nearest lookups: both rows are
            // contiguous, 16-byte aligned (row stride a multiple of 4 floats):
            // four voxels per load, exp in FP32 of the FP32 sum z_0 + z_1
            const float4 *r0 = reinterpret_cast<const float4 *>(map + o0[0]);
            const float4 *r1 = reinterpret_cast<const float4 *>(map + o1[0]);
            const int n4 = n_vox >> 2;
#pragma unroll 2
            for (int q = tid; q < n4; q += kInterpBlock) {
                const float4 a = __ldg(r0 + q), b = __ldg(r1 + q);
                const float t[4] = {expf(-(a.x + b.x)), expf(-(a.y + b.y)), expf(-(a.z + b.z)), expf(-(a.w + b.w))};
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    float ns, e;
                    two_sum(s, t[j], ns, e);
                    s = ns;
                    c += e;
                }
            }
            k0 = n4 << 2;
        }
        for (int k = k0 + tid; k < n_vox; k += kInterpBlock) {
            const T *mk = map + (long long)k * sK;
            const double a = __dadd_rn(leg_value(mk, o0, w0, linear), leg_value(mk, o1, w1, linear));
            float ns, e;
            two_sum(s, exp_neg(a), ns, e);
            s = ns;
            c += e;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float so = __shfl_down_sync(0xffffffffu, s, o);
            const float co = __shfl_down_sync(0xffffffffu, c, o);
            float ns, e;
            two_sum(s, so, ns, e);
            s = ns;
            c = c + co + e;
        }
        if (lane == 0) {
            red_s[warp] = s;
            red_c[warp] = c;
        }
        __syncthreads();
        if (tid == 0) {
            float bs = red_s[0], bc = red_c[0];
            for (int w = 1; w < kInterpBlock / 32; w++) {
                float ns, e;
                two_sum(bs, red_s[w], ns, e);
                bs = ns;
                bc = bc + red_c[w] + e;
            }
            out[r] = ((double)bs + (double)bc) / (double)n_vox;
        }
        __syncthreads();
    }
}

// Bilinear lookups on the direction-major float map.  A reflection's eight
// rows are streamed four voxels a load by kGroup warps; the weights, the
// eight-term sum and the reduction to exp's range run on pairs of floats
// (about 46 bits, so the FP32 argument of expf is the FP64 evaluation's but
// for near ties): in FP64 the 16 multiply-adds per voxel bound the kernel, at
// 1.04 ms for 20,000 reflections of 960 voxels; now 614 MB of map rows take
// 0.14 ms in one launch.  One warp per reflection when there are enough of
// them to fill the device (no block barrier), else a whole block.
template <int kGroup>
__global__ void __launch_bounds__(kInterpBlock) gridding_bilinear_kernel(const float *__restrict__ map, long long sR,
                                                                         int n_vox,
                                                                         const InterpRow *__restrict__ rows,
                                                                         long long n_refl, double *__restrict__ out)
{
    constexpr int kWarpsPerBlock = kInterpBlock / 32, kGroups = kWarpsPerBlock / kGroup;
    __shared__ float red_s[kWarpsPerBlock], red_c[kWarpsPerBlock];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int t = tid % (32 * kGroup);
    for (long long r = (long long)blockIdx.x * kGroups + warp / kGroup; r < n_refl;
         r += (long long)gridDim.x * kGroups) {
        const float4 *row[8];
        FloatPair w[8];
        // a weight each for eight lanes, then to all: the conversion is the only
        // FP64 left, and eight a thread had that pipe 79 % busy in whole blocks
        // (2,048 reflections: 40 -> 23 us)
        const FloatPair mine = pair_of(__ldg(&rows[r].w[(lane >> 2) & 1][lane & 3]));
#pragma unroll
        for (int j = 0; j < 8; j++) {
            row[j] = reinterpret_cast<const float4 *>(map + __ldg(&rows[r].row[j >> 2][j & 3]) * sR);
            w[j].h = __shfl_sync(0xffffffffu, mine.h, j);
            w[j].l = __shfl_sync(0xffffffffu, mine.l, j);
        }
        float s = 0.0f, c = 0.0f;
        auto add = [&](const float *z) {
            float h = __fmul_rn(w[0].h, z[0]);
            float l = __fmaf_rn(w[0].l, z[0], __fmaf_rn(w[0].h, z[0], -h));
#pragma unroll
            for (int j = 1; j < 8; j++) {
                const float p = __fmul_rn(w[j].h, z[j]);
                const float e = __fmaf_rn(w[j].l, z[j], __fmaf_rn(w[j].h, z[j], -p));
                float ns, d;
                two_sum(h, p, ns, d);
                h = ns;
                l = __fadd_rn(l, __fadd_rn(d, e));
            }
            float ns, e;
            two_sum(s, exp_neg(pair_norm(h, l)), ns, e);
            s = ns;
            c += e;
        };
        const int n4 = n_vox >> 2;
        for (int q = t; q < n4; q += 32 * kGroup) {
            float4 v[8];
#pragma unroll
            for (int j = 0; j < 8; j++)
                v[j] = __ldg(row[j] + q);
            float z[8];
#pragma unroll
            for (int j = 0; j < 8; j++)
                z[j] = v[j].x;
            add(z);
#pragma unroll
            for (int j = 0; j < 8; j++)
                z[j] = v[j].y;
            add(z);
#pragma unroll
            for (int j = 0; j < 8; j++)
                z[j] = v[j].z;
            add(z);
#pragma unroll
            for (int j = 0; j < 8; j++)
                z[j] = v[j].w;
            add(z);
        }
        if (const int k = (n4 << 2) + t; k < n_vox) {   // the last one to three voxels
            float z[8];
#pragma unroll
            for (int j = 0; j < 8; j++)
                z[j] = __ldg(reinterpret_cast<const float *>(row[j]) + k);
            add(z);
        }
        __syncwarp();
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float so = __shfl_down_sync(0xffffffffu, s, o);
            const float co = __shfl_down_sync(0xffffffffu, c, o);
            float ns, e;
            two_sum(s, so, ns, e);
            s = ns;
            c = c + co + e;
        }
        if (kGroup == 1) {
            if (lane == 0)
                out[r] = ((double)s + (double)c) / (double)n_vox;
            continue;
        }
        if (lane == 0) {
            red_s[warp] = s;
            red_c[warp] = c;
        }
        __syncthreads();
        if (tid == 0) {
            float bs = red_s[0], bc = red_c[0];
            for (int i = 1; i < kWarpsPerBlock; i++) {
                float ns, e;
                two_sum(bs, red_s[i], ns, e);
                bs = ns;
                bc = bc + red_c[i] + e;
            }
            out[r] = ((double)bs + (double)bc) / (double)n_vox;
        }
        __syncthreads();
    }
}

template <class T>
cudaError_t launch_interp(const T *map, long long sK, long long sR, int n_vox, const InterpRow *rows, long long n_refl,
                          int linear, double *out, cudaStream_t st)
{
    if (n_refl <= 0)
        return cudaSuccess;
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess)
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const long long grid = std::min<long long>(n_refl, (long long)sms * 8);
    if constexpr (sizeof(T) == 4) {
        if (linear && sK == 1 && sR % 4 == 0 && ((uintptr_t)map & 15) == 0) {
            // Warps of a device at eight blocks an SM: one reflection each once
            // there are that many (9,728 of 960 voxels: 76 us, a block each 100;
            // of 1,658: 113 and 144).  Prepared and asynchronous lookups launch
            // all their rows at once; a synchronous call launches 2,048 at a time,
            // blocks, which its host lookups hide.
            if (n_refl >= (long long)sms * 64)
                gridding_bilinear_kernel<1><<<(unsigned)std::min<long long>((n_refl + 7) / 8, (long long)sms * 8),
                                              kInterpBlock, 0, st>>>(map, sR, n_vox, rows, n_refl, out);
            else
                gridding_bilinear_kernel<8><<<(unsigned)grid, kInterpBlock, 0, st>>>(map, sR, n_vox, rows, n_refl, out);
            return cudaGetLastError();
        }
    }
    // the vectorised path: float rows (sK == 1) with a stride of whole float4s
    if (sizeof(T) == 4 && sK == 1 && sR % 4 == 0 && ((uintptr_t)map & 15) == 0)
        gridding_interp_kernel<T, true><<<(unsigned)grid, kInterpBlock, 0, st>>>(map, sK, sR, n_vox, rows, n_refl,
                                                                                 linear, out);
    else
        gridding_interp_kernel<T, false><<<(unsigned)grid, kInterpBlock, 0, st>>>(map, sK, sR, n_vox, rows, n_refl,
                                                                                  linear, out);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_gridding_interp_f32(const float *map, long long sK, long long sR, int n_vox, const InterpRow *rows,
                                       long long n_refl, int linear, double *out, cudaStream_t st)
{
    return launch_interp(map, sK, sR, n_vox, rows, n_refl, linear, out, st);
}

cudaError_t launch_gridding_interp_f64(const double *map, long long sK, long long sR, int n_vox,
                                       const InterpRow *rows, long long n_refl, int linear, double *out,
                                       cudaStream_t st)
{
    return launch_interp(map, sK, sR, n_vox, rows, n_refl, linear, out, st);
}

}  // namespace anacor
