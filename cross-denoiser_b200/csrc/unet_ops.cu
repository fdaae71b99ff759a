// The U-Net's non-convolution layers, their backward passes, the gradient
// reductions and the optimizer (scripts/main.py:74-118, 300-303):
//   input packing      Concatenate of the five 3-channel inputs (:101-102)
//   Conv2DTranspose    kernel 1, stride 2, 'same' (:92, :96): out[2i,2j] =
//                      K x[i,j] + b, every other position b; Keras kernel
//                      layout [1][1][cout][cin]
//   head               Conv2D(6, 1) in fp32, band = 1 / (p^2 + 1e-4),
//                      alpha = sigmoid (:106-111)
//   max-pool backward  the gradient goes to the first maximum of each 2x2
//                      window (row-major), added to the skip connection's
//                      gradient, times the ReLU derivative
//   Adam               Keras semantics: m += (g - m)(1 - b1),
//                      v += (g^2 - v)(1 - b2),
//                      w -= lr sqrt(1 - b2^t) / (1 - b1^t) m / (sqrt(v) + eps)
// Per-block partial sums of the parameter gradients are reduced in a fixed
// order by reduce_kernel, so the gradients are deterministic.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include "cd_common.cuh"
#include "launch.cuh"
#include "unet.cuh"
#include "unet_ops.cuh"

namespace cd {
namespace unet {
namespace {

CD_DEV void ld8(const __nv_bfloat16 *p, float *v)
{
    const uint4 raw = *reinterpret_cast<const uint4 *>(p);
    const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(&raw);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const float2 f = __bfloat1622float2(h[e]);
        v[2 * e] = f.x;
        v[2 * e + 1] = f.y;
    }
}
CD_DEV uint4 pack8(const float *v)
{
    uint4 o;
    __nv_bfloat162 *h = reinterpret_cast<__nv_bfloat162 *>(&o);
#pragma unroll
    for (int e = 0; e < 4; ++e) h[e] = __floats2bfloat162_rn(v[2 * e], v[2 * e + 1]);
    return o;
}
CD_DEV void st8(__nv_bfloat16 *p, const float *v) { *reinterpret_cast<uint4 *>(p) = pack8(v); }

// [ols1, ols2, prev_out, albedo, normal] (fp32, 3 channels each) -> bf16, 16
// channels (15 + zero) in two row-chunk planes; n = B * H * W pixels, W wide
__global__ void __launch_bounds__(256) pack_input_kernel(const float *a, const float *b,
                                                         const float *c, const float *d,
                                                         const float *e, __nv_bfloat16 *__restrict__ x,
                                                         size_t n, int W)
{
    chain_wait();
    chain_next();
    const size_t p = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    const int row = (int)(p / W), px = (int)(p - (size_t)row * W);
    float v[16];
    const float *src[5] = {a, b, c, d, e};
#pragma unroll
    for (int k = 0; k < 5; ++k) {
        v[3 * k] = src[k][3 * p];
        v[3 * k + 1] = src[k][3 * p + 1];
        v[3 * k + 2] = src[k][3 * p + 2];
    }
    v[15] = 0.f;
    st8(x + act_idx(0, row, 0, px, 0, W, 2) * 8, v);
    st8(x + act_idx(0, row, 1, px, 0, W, 2) * 8, v + 8);
}

// Conv2DTranspose(kernel 1, stride 2) forward: output (2i, 2j) = K x + b
// (each channel summed over ci in order, K rows read as float4), outputs
// (2i, 2j + 1), (2i + 1, 2j), (2i + 1, 2j + 1) = b.  A weight read from
// shared memory costs its 128 bytes per warp whatever the lanes share, and
// with one pixel per thread those reads bound the kernel, so a thread takes
// kPix input pixels (a block apart) per weight, and lanes trade pixels so that
// every store is 512 consecutive bytes: 32 channels at 480x270 22 -> 16 us, 16
// at 960x540 27 -> 18.
template <int CI, int CO, int kPix>
__global__ void __launch_bounds__(256) tconv_fwd_kernel(const __nv_bfloat16 *in,
                                                        const float *K, const float *bias,
                                                        __nv_bfloat16 *__restrict__ out, int Hi, int Wi, int B)
{
    chain_wait();
    chain_next();
    __shared__ __align__(16) float sK[CO * CI + CO];
    for (int i = threadIdx.x; i < CO * CI + CO; i += blockDim.x) sK[i] = i < CO * CI ? K[i] : bias[i - CO * CI];
    __syncthreads();
    const int Ho = 2 * Hi, Wo = 2 * Wi;
    const size_t n = (size_t)B * Hi * Wi, p0 = (size_t)blockIdx.x * blockDim.x * kPix + threadIdx.x;
    float x[kPix][CI];
    unsigned at[kPix];   // output (2i, 2j), chunk 0, in 8-channel units; kNone past the last pixel
    constexpr unsigned kNone = 0xFFFFFFFFu;
#pragma unroll
    for (int k = 0; k < kPix; ++k) {
        const size_t p = p0 + (size_t)k * blockDim.x, q = p < n ? p : 0;
        const int xi = (int)(q % Wi), yi = (int)((q / Wi) % Hi), b = (int)(q / ((size_t)Wi * Hi));
        at[k] = p < n ? (unsigned)act_idx(b, 2 * yi, 0, 2 * xi, Ho, Wo, CO / 8) : kNone;
#pragma unroll
        for (int c = 0; c < CI; c += 8) ld8(in + act_idx(b, yi, c / 8, xi, Hi, Wi, CI / 8) * 8, x[k] + c);
    }
    const int lane = threadIdx.x & 31;
    uint4 *out4 = reinterpret_cast<uint4 *>(out);
#pragma unroll 1
    for (int c = 0; c < CO; c += 8) {
        float o[kPix][8], ob[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            ob[e] = sK[CO * CI + c + e];
#pragma unroll
            for (int k = 0; k < kPix; ++k) o[k][e] = ob[e];
            const float4 *kr = reinterpret_cast<const float4 *>(sK + (c + e) * CI);
#pragma unroll
            for (int c4 = 0; c4 < CI / 4; ++c4) {
                const float4 k4 = kr[c4];
#pragma unroll
                for (int k = 0; k < kPix; ++k) {
                    float t = fmaf(k4.x, x[k][4 * c4], o[k][e]);
                    t = fmaf(k4.y, x[k][4 * c4 + 1], t);
                    t = fmaf(k4.z, x[k][4 * c4 + 2], t);
                    o[k][e] = fmaf(k4.w, x[k][4 * c4 + 3], t);
                }
            }
        }
        const uint4 vb = pack8(ob);
#pragma unroll
        for (int k = 0; k < kPix; ++k) {
            // the warp's 64 output pixels of each row, 32 consecutive ones per
            // store: lane l takes pixel 32 j + l, input pixel (32 j + l) / 2's
            const uint4 v = pack8(o[k]);
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int src = 16 * j + (lane >> 1);
                const unsigned base = __shfl_sync(0xffffffffu, at[k], src);
                uint4 t;
                t.x = __shfl_sync(0xffffffffu, v.x, src);
                t.y = __shfl_sync(0xffffffffu, v.y, src);
                t.z = __shfl_sync(0xffffffffu, v.z, src);
                t.w = __shfl_sync(0xffffffffu, v.w, src);
                if (base == kNone) continue;
                const size_t i = (size_t)base + (size_t)(c / 8) * Wo + (lane & 1);
                out4[i] = lane & 1 ? vb : t;
                out4[i + (size_t)(CO / 8) * Wo] = vb;
            }
        }
    }
}

// Conv2DTranspose backward: for every chunk of kN input pixels, d_in =
// K^T d_out[2i,2j] (times the ReLU derivative of `in`) and the chunk's
// contribution to dK[co][ci] and db[co] (db over all four output positions
// of each input pixel).  Blocks walk chunks blockIdx.x, + gridDim.x, ...
// and keep their dK / db sums in registers: one partial row per block.
template <int CI, int CO, int kN>
__global__ void __launch_bounds__(kN) tconv_bwd_kernel(const __nv_bfloat16 *in,
                                                        const __nv_bfloat16 *dout,
                                                        const float *K,
                                                        __nv_bfloat16 *__restrict__ dz_in, float *__restrict__ partial,
                                                        int Hi, int Wi, int B)
{
    chain_wait();
    chain_next();
    // dK in 4 x 4 register tiles: kTiles tiles cover CO x CI, and the
    // threads split into kGroups pixel groups, each summing its share of a
    // chunk's pixels (in order) into every tile; the groups' sums are added
    // in group order at the end.  Then db.
    constexpr int TM = 4, TN = 4, kTiles = (CO / TM) * (CI / TN), kGroups = kN / kTiles;
    static_assert(kGroups >= 1 && kGroups * kTiles == kN && kN % kGroups == 0, "tiles x groups cover the block");
    __shared__ __align__(16) float sK[CO * CI];
    __shared__ float sx[kN][CI + 1], sd[kN][CO + 1], sb[kN][CO + 1];
    for (int i = threadIdx.x; i < CO * CI; i += blockDim.x) sK[i] = K[i];
    const size_t n = (size_t)B * Hi * Wi, nchunk = (n + kN - 1) / kN;
    const int t = threadIdx.x;
    const int tile = t % kTiles, grp = t / kTiles;
    const int tci = tile % (CI / TN), tco = tile / (CI / TN);
    const int ci0 = TN * tci, co0 = TM * tco;
    constexpr int kPer = kN / kGroups;   // pixels of a chunk per group
    float acc[TM][TN];
#pragma unroll
    for (int a = 0; a < TM; ++a)
#pragma unroll
        for (int c = 0; c < TN; ++c) acc[a][c] = 0.f;
    float bacc = 0.f;
    for (size_t chunk = blockIdx.x; chunk < nchunk; chunk += gridDim.x) {
        const size_t p = chunk * kN + t;
        float x[CI], d[CO];
#pragma unroll
        for (int c = 0; c < CI; ++c) x[c] = 0.f;
#pragma unroll
        for (int c = 0; c < CO; ++c) d[c] = 0.f;
        float bsum[CO];
#pragma unroll
        for (int c = 0; c < CO; ++c) bsum[c] = 0.f;
        const int xi = (int)(p % Wi), yi = (int)((p / Wi) % Hi), b = (int)(p / ((size_t)Wi * Hi));
        if (p < n) {
#pragma unroll
            for (int c = 0; c < CI; c += 8) ld8(in + act_idx(b, yi, c / 8, xi, Hi, Wi, CI / 8) * 8, x + c);
            const int Wo = 2 * Wi, Ho = 2 * Hi;
            for (int a = 0; a < 4; ++a) {
                const int yo = 2 * yi + (a >> 1), xo = 2 * xi + (a & 1);
                float g[CO];
#pragma unroll
                for (int c = 0; c < CO; c += 8) ld8(dout + act_idx(b, yo, c / 8, xo, Ho, Wo, CO / 8) * 8, g + c);
#pragma unroll
                for (int c = 0; c < CO; ++c) {
                    bsum[c] += g[c];
                    if (a == 0) d[c] = g[c];
                }
            }
        }
#pragma unroll
        for (int c = 0; c < CI; ++c) sx[t][c] = x[c];
#pragma unroll
        for (int c = 0; c < CO; ++c) {
            sd[t][c] = d[c];
            sb[t][c] = bsum[c];
        }
        __syncthreads();
        if (p < n) {
            // co outer, ci inner: each g[ci] still sums over co in order, and a
            // row of K is read as float4s
            float g[CI];
#pragma unroll
            for (int ci = 0; ci < CI; ++ci) g[ci] = 0.f;
#pragma unroll
            for (int co = 0; co < CO; ++co) {
                const float4 *kr = reinterpret_cast<const float4 *>(sK + co * CI);
#pragma unroll
                for (int c4 = 0; c4 < CI / 4; ++c4) {
                    const float4 k4 = kr[c4];
                    g[4 * c4] = fmaf(k4.x, d[co], g[4 * c4]);
                    g[4 * c4 + 1] = fmaf(k4.y, d[co], g[4 * c4 + 1]);
                    g[4 * c4 + 2] = fmaf(k4.z, d[co], g[4 * c4 + 2]);
                    g[4 * c4 + 3] = fmaf(k4.w, d[co], g[4 * c4 + 3]);
                }
            }
#pragma unroll
            for (int ci = 0; ci < CI; ++ci) g[ci] = x[ci] > 0.f ? g[ci] : 0.f;
#pragma unroll
            for (int c = 0; c < CI; c += 8) st8(dz_in + act_idx(b, yi, c / 8, xi, Hi, Wi, CI / 8) * 8, g + c);
        }
        for (int k = grp * kPer; k < (grp + 1) * kPer; ++k) {
            float dv[TM], xv[TN];
#pragma unroll
            for (int a = 0; a < TM; ++a) dv[a] = sd[k][co0 + a];
#pragma unroll
            for (int c = 0; c < TN; ++c) xv[c] = sx[k][ci0 + c];
#pragma unroll
            for (int a = 0; a < TM; ++a)
#pragma unroll
                for (int c = 0; c < TN; ++c) acc[a][c] = fmaf(dv[a], xv[c], acc[a][c]);
        }
        if (t < CO)
            for (int k = 0; k < kN; ++k) bacc += sb[k][t];
        __syncthreads();   // the chunk's tiles are read before the next one is written
    }
    float *out = partial + (size_t)blockIdx.x * (CO * CI + CO);
    if (kGroups == 1) {
#pragma unroll
        for (int a = 0; a < TM; ++a)
#pragma unroll
            for (int c = 0; c < TN; ++c) out[(co0 + a) * CI + ci0 + c] = acc[a][c];
    } else {
        // the groups' tiles through shared memory (sx is free now: kN x (CI + 1)
        // floats hold the kGroups x CO x CI sums)
        float *red = &sx[0][0];
        static_assert(kGroups * CO * CI <= kN * (CI + 1), "the group sums fit sx");
#pragma unroll
        for (int a = 0; a < TM; ++a)
#pragma unroll
            for (int c = 0; c < TN; ++c) red[(grp * CO + co0 + a) * CI + ci0 + c] = acc[a][c];
        __syncthreads();
        for (int j = t; j < CO * CI; j += kN) {
            float v = 0.f;
            for (int g = 0; g < kGroups; ++g) v += red[g * CO * CI + j];
            out[j] = v;
        }
    }
    if (t < CO) out[CO * CI + t] = bacc;
}

// Head: param = Kh^T c5_1 + bh (Kh[ci][co], 8 x 6), band = 1 / (p^2 + 1e-4), alpha = sigmoid(p5).
// A thread takes two pixels per weight read (as tconv_fwd_kernel), 256
// apart; a block's band values (five per pixel) go out through shared
// memory as float4 stores.  2560x1440: 41 -> 32 us.
constexpr int kHeadThreads = 256;

// param co of a pixel's v, weights sT[co][ci] (co = 0..5), summed over ci in order
CD_DEV void head_params(const float4 *sT, const float *bias, const float (&v)[2][8], float (&q)[2][6])
{
#pragma unroll
    for (int co = 0; co < 6; ++co) {
        const float4 k0 = sT[2 * co], k1 = sT[2 * co + 1];
        const float kk[8] = {k0.x, k0.y, k0.z, k0.w, k1.x, k1.y, k1.z, k1.w}, bc = bias[co];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            float t = bc;
#pragma unroll
            for (int ci = 0; ci < 8; ++ci) t = fmaf(kk[ci], v[i][ci], t);
            q[i][co] = t;
        }
    }
}

__global__ void __launch_bounds__(kHeadThreads) head_fwd_kernel(const __nv_bfloat16 *x,
                                                                const float *K,
                                                                const float *bias,
                                                                float *__restrict__ band, float *__restrict__ alpha,
                                                                size_t n)
{
    chain_wait();
    chain_next();
    __shared__ __align__(16) float sT[48];
    __shared__ float sB[6];
    __shared__ __align__(16) float sb[2 * kHeadThreads * 5];   // the block's band values, written out as float4
    const int tid = threadIdx.x;
    const size_t p0 = (size_t)blockIdx.x * (2 * kHeadThreads);
    float v[2][8];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const size_t p = p0 + i * kHeadThreads + tid;
        ld8(x + 8 * (p < n ? p : 0), v[i]);
    }
    if (tid < 48) sT[(tid % 6) * 8 + tid / 6] = K[tid];
    if (tid < 6) sB[tid] = bias[tid];
    __syncthreads();
    float q[2][6];
    head_params(reinterpret_cast<const float4 *>(sT), sB, v, q);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int t = i * kHeadThreads + tid;
#pragma unroll
        for (int k = 0; k < 5; ++k) sb[5 * t + k] = 1.f / (q[i][k] * q[i][k] + 1e-4f);
        if (p0 + t < n) alpha[p0 + t] = 1.f / (1.f + expf(-q[i][5]));
    }
    __syncthreads();
    const int cnt = 5 * (int)(n - p0 < 2 * kHeadThreads ? n - p0 : 2 * kHeadThreads);
    float *dst = band + 5 * p0;
    int i = tid;
    if (!(reinterpret_cast<uintptr_t>(dst) & 15)) {
        for (; i < cnt / 4; i += kHeadThreads)
            reinterpret_cast<float4 *>(dst)[i] = reinterpret_cast<const float4 *>(sb)[i];
        i = (cnt / 4) * 4 + tid;
    }
    for (; i < cnt; i += kHeadThreads) dst[i] = sb[i];
}

// Head backward: dZ of c5_1 (times its ReLU derivative) and the block's
// partial sums of dKh[ci][co] and dbh[co].  Each thread walks pixels
// p = thread, thread + grid size, ... accumulating its 54 parameter-gradient
// terms in registers (in that order); the block then reduces them (lanes,
// then warps, in a fixed order) to one partial row.
//
// 128 registers leave two blocks an SM, too few loads in flight to cover
// DRAM from registers: every warp copies its pixels' inputs (32 activations,
// band and alpha gradients) kHeadAhead iterations ahead into slots of its
// own (cp.async, no block barrier).  Two iterations at a time share the weight
// reads.  2560x1440: 98 -> 60 us.
constexpr int kHeadMaxBlocks = 592;
constexpr int kHeadAhead = 4, kHeadSlots = kHeadAhead + 2;
struct __align__(16) HeadSlot {
    uint4 x[32];
    float gband[160], galpha[32];
};
constexpr int kHeadBwdSmem = kHeadSlots * (kHeadThreads / 32) * (int)sizeof(HeadSlot);

CD_DEV void head_cp(void *dst, const void *src, int bytes)   // bytes: 4 or 16
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    if (bytes == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src) : "memory");
}

__global__ void __launch_bounds__(kHeadThreads, 2) head_bwd_kernel(const __nv_bfloat16 *x,
                                                                   const float *K,
                                                                   const float *bias,
                                                                   const float *gband,
                                                                   const float *galpha,
                                                                   __nv_bfloat16 *__restrict__ dz,
                                                                   float *__restrict__ partial, size_t n)
{
    chain_wait();
    chain_next();
    extern __shared__ __align__(16) uint8_t head_smem[];
    __shared__ __align__(16) float sK[48], sT[48];   // Kh[ci][co], and transposed
    __shared__ float sB[6];
    __shared__ float red[kHeadThreads / 32][54];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    HeadSlot *slots = reinterpret_cast<HeadSlot *>(head_smem) + warp * kHeadSlots;
    const bool aligned = ((reinterpret_cast<uintptr_t>(gband) | reinterpret_cast<uintptr_t>(galpha)) & 15) == 0;
    const size_t w0 = (size_t)blockIdx.x * kHeadThreads + warp * 32, step = (size_t)gridDim.x * kHeadThreads;
    auto fetch = [&](int k) {   // iteration k's inputs, one group
        const size_t p = w0 + k * step;
        HeadSlot &s = slots[k % kHeadSlots];
        if (p + 32 <= n && aligned) {
            head_cp(&s.x[lane], x + 8 * (p + lane), 16);
            head_cp(&s.gband[4 * lane], gband + 5 * p + 4 * lane, 16);
            if (lane < 8) {
                head_cp(&s.gband[128 + 4 * lane], gband + 5 * p + 128 + 4 * lane, 16);
                head_cp(&s.galpha[4 * lane], galpha + p + 4 * lane, 16);
            }
        } else if (p + lane < n) {
            head_cp(&s.x[lane], x + 8 * (p + lane), 16);
#pragma unroll
            for (int e = 0; e < 5; ++e) head_cp(&s.gband[5 * lane + e], gband + 5 * (p + lane) + e, 4);
            head_cp(&s.galpha[lane], galpha + p + lane, 4);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int k = 0; k < kHeadAhead; ++k) fetch(k);
    if (tid < 48) {
        const float w = K[tid];
        sK[tid] = w;
        sT[(tid % 6) * 8 + tid / 6] = w;
    }
    if (tid < 6) sB[tid] = bias[tid];
    __syncthreads();
    float acc[54];
#pragma unroll
    for (int j = 0; j < 54; ++j) acc[j] = 0.f;
    for (int k = 0; w0 + k * step < n; k += 2) {
        fetch(k + kHeadAhead);
        fetch(k + kHeadAhead + 1);
        asm volatile("cp.async.wait_group %0;" ::"n"(kHeadAhead) : "memory");
        __syncwarp();
        float v[2][8], g[2][6], d[2][8];
        bool in[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const HeadSlot &s = slots[(k + i) % kHeadSlots];
            in[i] = w0 + (k + i) * step + lane < n;
            ld8(reinterpret_cast<const __nv_bfloat16 *>(&s.x[lane]), v[i]);
#pragma unroll
            for (int e = 0; e < 5; ++e) g[i][e] = s.gband[5 * lane + e];
            g[i][5] = s.galpha[lane];
        }
        float q[2][6];
        head_params(reinterpret_cast<const float4 *>(sT), sB, v, q);
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int co = 0; co < 6; ++co) {
                const float t = q[i][co];
                if (co < 5) {
                    // d band / d t = -2 t / (t^2 + 1e-4)^2, with one fast
                    // reciprocal (a gradient: FP32 tolerance, not the forward's
                    // rounding)
                    const float r = __fdividef(1.f, t * t + 1e-4f);
                    g[i][co] = g[i][co] * (-2.f * t * r * r);
                } else {
                    const float a = 1.f / (1.f + expf(-t));
                    g[i][co] = g[i][co] * a * (1.f - a);
                }
            }
#pragma unroll
        for (int ci = 0; ci < 8; ci += 2) {   // two rows of Kh: twelve weights
            const float4 *kr = reinterpret_cast<const float4 *>(sK + 6 * ci);
            const float4 k0 = kr[0], k1 = kr[1], k2 = kr[2];
            const float kk[12] = {k0.x, k0.y, k0.z, k0.w, k1.x, k1.y, k1.z, k1.w, k2.x, k2.y, k2.z, k2.w};
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    float t = 0.f;
#pragma unroll
                    for (int co = 0; co < 6; ++co) t = fmaf(kk[6 * c + co], g[i][co], t);
                    d[i][ci + c] = v[i][ci + c] > 0.f ? t : 0.f;
                }
        }
#pragma unroll
        for (int i = 0; i < 2; ++i)
            if (in[i]) {
                st8(dz + 8 * (w0 + (k + i) * step + lane), d[i]);
#pragma unroll
                for (int ci = 0; ci < 8; ++ci)
#pragma unroll
                    for (int co = 0; co < 6; ++co) acc[ci * 6 + co] = fmaf(v[i][ci], g[i][co], acc[ci * 6 + co]);
#pragma unroll
                for (int co = 0; co < 6; ++co) acc[48 + co] += g[i][co];
            }
        __syncwarp();   // both slots are read before a later fetch writes them
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
    for (int j = 0; j < 54; ++j) {
        float s = acc[j];
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) red[warp][j] = s;
    }
    __syncthreads();
    if (tid < 54) {
        float s = 0.f;
        for (int w = 0; w < kHeadThreads / 32; ++w) s += red[w][tid];
        partial[(size_t)blockIdx.x * 54 + tid] = s;
    }
}

// dZ = (maxpool backward of dpool + dskip) * [act > 0], C channels (multiple
// of 8).  One thread per pooled pixel (H and W even): it reads the four
// pixels of its 2x2 window once per 8-channel chunk; the pooled gradient
// goes to the first maximum of the window (row-major), as in the forward.
template <int C>
__global__ void __launch_bounds__(256) pool_bwd_kernel(const __nv_bfloat16 *act,
                                                       const __nv_bfloat16 *pooled,
                                                       const __nv_bfloat16 *dpool,
                                                       const __nv_bfloat16 *dskip,
                                                       __nv_bfloat16 *__restrict__ dz, int H, int W, int B)
{
    chain_wait();
    chain_next();
    constexpr int NC = C / 8;
    const int PH = H / 2, PW = W / 2;
    const size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= (size_t)B * PH * PW) return;
    const int px = (int)(q % PW), py = (int)((q / PW) % PH), b = (int)(q / ((size_t)PW * PH));
#pragma unroll
    for (int c = 0; c < NC; ++c) {
        float m[8], dp[8], a[4][8], g[4][8];
        ld8(pooled + act_idx(b, py, c, px, PH, PW, NC) * 8, m);
        ld8(dpool + act_idx(b, py, c, px, PH, PW, NC) * 8, dp);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const size_t r = act_idx(b, 2 * py + (k >> 1), c, 2 * px + (k & 1), H, W, NC) * 8;
            ld8(act + r, a[k]);
            ld8(dskip + r, g[k]);
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            bool taken = false;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (!taken && a[k][e] == m[e]) {
                    g[k][e] += dp[e];
                    taken = true;
                }
            }
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
#pragma unroll
            for (int e = 0; e < 8; ++e)
                if (!(a[k][e] > 0.f)) g[k][e] = 0.f;
            st8(dz + act_idx(b, 2 * py + (k >> 1), c, 2 * px + (k & 1), H, W, NC) * 8, g[k]);
        }
    }
}

// Fixed-order reduction of partial sums, one launch for every parameter
// tensor: a block owns 32 output columns of one job (lane = column) and its
// 32 warps take the rows t = warp, warp + 32, ... in order; the warps' sums
// are then added in warp order.  The same partials always give the same
// result.  One launch per tensor, each waiting for the one before it, took
// 61 us of a 1920x1080 backward (12 launches), one launch at the end 15 us.
constexpr int kReduceWarps = 32;

__global__ void __launch_bounds__(32 * kReduceWarps) reduce_kernel(const __grid_constant__ ReduceJobs J)
{
    chain_wait();
    chain_next();
    __shared__ float red[kReduceWarps][33];
    int k = 0, blk = blockIdx.x;
    while (k + 1 < J.n && blk >= (J.job[k].n + 31) / 32) blk -= (J.job[k++].n + 31) / 32;
    const float *partial = J.job[k].partial;
    const int n = J.job[k].n, rows = J.job[k].rows;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int j = blk * 32 + lane;
    float s = 0.f;
    if (j < n) {
#pragma unroll 4
        for (int t = warp; t < rows; t += kReduceWarps) s += partial[(size_t)t * n + j];
    }
    red[warp][lane] = s;
    __syncthreads();
    if (warp == 0 && j < n) {
        float v = 0.f;
        for (int w = 0; w < kReduceWarps; ++w) v += red[w][lane];
        J.job[k].out[j] = v;
    }
}

// The update count lives in device memory (so a captured graph replays
// correct steps): t = *step + 1, lr_t = lr sqrt(1 - b2^t) / (1 - b1^t) in
// float as Keras computes it; step_kernel then advances the counter.
__global__ void __launch_bounds__(256) adam_kernel(float *w, const float *g, float *m, float *v, int n,
                                                   const int *step, float lr, float b1, float b2,
                                                   float eps)
{
    chain_wait();
    chain_next();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float t = (float)(*step + 1);
    const float lr_t = lr * sqrtf(1.f - powf(b2, t)) / (1.f - powf(b1, t));
    const float gi = g[i];
    const float mi = m[i] + (gi - m[i]) * (1.f - b1);
    const float vi = v[i] + (gi * gi - v[i]) * (1.f - b2);
    m[i] = mi;
    v[i] = vi;
    w[i] -= (mi * lr_t) / (sqrtf(vi) + eps);
}

__global__ void step_kernel(int *step)
{
    chain_wait();
    *step += 1;
}

}  // namespace

cudaError_t launch_pack_input(const float *a, const float *b, const float *c, const float *d, const float *e,
                              __nv_bfloat16 *x, size_t n, int W, cudaStream_t st)
{
    return launch_chained(pack_input_kernel, (unsigned)((n + 255) / 256), 256, 0, st, a, b, c, d, e, x, n, W);
}

cudaError_t launch_tconv_fwd(int ci, int co, const __nv_bfloat16 *in, const float *K, const float *bias,
                             __nv_bfloat16 *out, int Hi, int Wi, int B, cudaStream_t st)
{
    const size_t n = (size_t)B * Hi * Wi;
    auto go = [&](auto kern, int threads, int pix) {
        return launch_chained(kern, (unsigned)((n + threads * pix - 1) / (threads * pix)), threads, 0, st, in, K, bias,
                              out, Hi, Wi, B);
    };
    if (ci == 32 && co == 32) return go(tconv_fwd_kernel<32, 32, 2>, 64, 2);
    if (ci == 16 && co == 16) return go(tconv_fwd_kernel<16, 16, 2>, 128, 2);
    return cudaErrorInvalidValue;
}

// pixels per block of the transposed-conv backward (static shared memory < 48 KB)
static int tconv_bwd_px(int ci) { return ci == 32 ? 64 : 128; }

// Blocks of the transposed-conv backward (and partial rows it writes): one
// per chunk of input pixels up to 8 per SM of a 148-SM part.
constexpr size_t kTconvMaxBlocks = 1184;
size_t tconv_blocks(int ci, int Hi, int Wi, int B)
{
    const int k = tconv_bwd_px(ci);
    const size_t chunks = ((size_t)B * Hi * Wi + k - 1) / k;
    return chunks < kTconvMaxBlocks ? chunks : kTconvMaxBlocks;
}

cudaError_t launch_tconv_bwd(int ci, int co, const __nv_bfloat16 *in, const __nv_bfloat16 *dout, const float *K,
                             __nv_bfloat16 *dz_in, float *partial, int Hi, int Wi, int B, cudaStream_t st)
{
    const unsigned g = (unsigned)tconv_blocks(ci, Hi, Wi, B);
    if (ci == 32 && co == 32) return launch_chained(tconv_bwd_kernel<32, 32, 64>, g, 64, 0, st, in, dout, K, dz_in,
                                                    partial, Hi, Wi, B);
    if (ci == 16 && co == 16)
        return launch_chained(tconv_bwd_kernel<16, 16, 128>, g, 128, 0, st, in, dout, K, dz_in, partial, Hi, Wi, B);
    return cudaErrorInvalidValue;
}

cudaError_t launch_head_fwd(const __nv_bfloat16 *x, const float *K, const float *bias, float *band, float *alpha,
                            size_t n, cudaStream_t st)
{
    return launch_chained(head_fwd_kernel, (unsigned)((n + 2 * kHeadThreads - 1) / (2 * kHeadThreads)), kHeadThreads, 0,
                          st, x, K, bias, band, alpha, n);
}

size_t head_blocks(size_t n)
{
    const size_t g = (n + kHeadThreads - 1) / kHeadThreads;
    return g < (size_t)kHeadMaxBlocks ? g : (size_t)kHeadMaxBlocks;
}

cudaError_t launch_head_bwd(const __nv_bfloat16 *x, const float *K, const float *bias, const float *gband,
                            const float *galpha, __nv_bfloat16 *dz, float *partial, size_t n, cudaStream_t st)
{
    cudaError_t e = cudaFuncSetAttribute(head_bwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kHeadBwdSmem);
    if (e != cudaSuccess) return e;
    return launch_chained(head_bwd_kernel, (unsigned)head_blocks(n), kHeadThreads, kHeadBwdSmem, st, x, K, bias, gband,
                          galpha, dz, partial, n);
}

cudaError_t launch_pool_bwd(int C, const __nv_bfloat16 *act, const __nv_bfloat16 *pooled,
                            const __nv_bfloat16 *dpool, const __nv_bfloat16 *dskip, __nv_bfloat16 *dz, int H, int W,
                            int B, cudaStream_t st)
{
    if ((H | W) & 1) return cudaErrorInvalidValue;   // the network's levels are even-sized
    const size_t n = (size_t)B * (H / 2) * (W / 2);
    const unsigned g = (unsigned)((n + 255) / 256);
    if (C == 8) return launch_chained(pool_bwd_kernel<8>, g, 256, 0, st, act, pooled, dpool, dskip, dz, H, W, B);
    if (C == 16) return launch_chained(pool_bwd_kernel<16>, g, 256, 0, st, act, pooled, dpool, dskip, dz, H, W, B);
    return cudaErrorInvalidValue;
}

cudaError_t launch_reduce(const ReduceJobs &J, cudaStream_t st)
{
    if (J.n < 1 || J.n > kMaxReduceJobs) return cudaErrorInvalidValue;
    int blocks = 0;
    for (int k = 0; k < J.n; ++k) blocks += (J.job[k].n + 31) / 32;
    return launch_chained(reduce_kernel, blocks, 32 * kReduceWarps, 0, st, J);
}

cudaError_t launch_adam(float *w, const float *g, float *m, float *v, int n, int *step, float lr, float b1, float b2,
                        float eps, cudaStream_t st)
{
    const cudaError_t e = launch_chained(adam_kernel, (n + 255) / 256, 256, 0, st, w, g, m, v, n, step, lr, b1, b2, eps);
    return e != cudaSuccess ? e : launch_chained(step_kernel, 1, 1, 0, st, step);
}

}  // namespace unet
}  // namespace cd
