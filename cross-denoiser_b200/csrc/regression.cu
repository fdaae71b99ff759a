// Cross-regression on sm_100a: variance estimate, per-centre weighted least
// squares and block reconstruction.
//
// Reference semantics: ops/regression.cu.cc:206-500 (EstInputVarianceKernel,
// RegressionKernel with cholesky_color / forward_backward_solver, BlockRecon,
// CrossRegressionFunc).  Buffer A regresses imgb (target) on imga's features
// and buffer B the converse; both are computed by the same threads so the
// albedo / normal differences and the shared tile are read once.
//
// Coefficient layout in the workspace: beta[buf][b][j][i][r][ch] with
// r = 0..5 the regression coefficient (constant, colour, albedo, normal.xyz)
// and ch = 0..2 the colour channel; 18 floats per centre and buffer.
#include <type_traits>
#include <cuda_runtime.h>
#include "cd_common.cuh"
#include "launch.cuh"
#include "f32x2.cuh"
#include "window_rows.cuh"

namespace cd {
namespace {

constexpr int kP = 6;            // coefficients per channel (ops/regression.cu.cc:30)
constexpr int kBeta = kP * 3;    // floats per centre and buffer

// ---------------------------------------------------------------------------
// Variance: var = |mean of the in-bounds 3x3 neighbours minus the centre -
// centre|^2 summed over channels (ops/regression.cu.cc:244-276).  Also
// writes sqrt(var) to a workspace plane: the regression and reconstruction
// read the standard deviation of every tap.
//
// variance_kernel: one thread per pixel computes both buffers from the
// block's footprint in shared memory (rows of 40 pixels from x0 - 4, as
// stored: 3 floats per pixel), each row copied by one warp with one float4
// per lane.  Needs W % 4 == 0 and 16-byte aligned images, so that every
// float4 lies wholly inside or wholly outside an image row.
// variance_px_kernel (any W): one thread per pixel and buffer, global loads.
// blockIdx.z = 2 * batch + buffer there.
// ---------------------------------------------------------------------------
constexpr int kVX = 32, kVY = 8;
constexpr int kVRow = 3 * (kVX + 8), kVTH = kVY + 2;   // footprint row: 40 pixels x 3 floats

__global__ void __launch_bounds__(kVX * kVY) variance_kernel(const float *imga,
                                                             const float *imgb,
                                                             float *__restrict__ vara,
                                                             float *__restrict__ varb,
                                                             float *__restrict__ sda,
                                                             float *__restrict__ sdb, int H, int W)
{
    chain_wait();
    chain_next();
    __shared__ __align__(16) float tile[2][kVTH][kVRow];
    const int x0 = blockIdx.x * kVX, y0 = blockIdx.y * kVY, xa = x0 - 4;
    const size_t base = (size_t)blockIdx.z * H * W;
    const int lane = threadIdx.x, warp = threadIdx.y;
    constexpr int kRows = 2 * kVTH, kIt = (kRows + kVY - 1) / kVY;
    float4 v[kIt];
    // every load issued before the first store
#pragma unroll
    for (int k = 0; k < kIt; ++k) {
        const int rr = warp + k * kVY, buf = rr >= kVTH, ty = rr - buf * kVTH, gy = y0 - 1 + ty;
        const int f = 3 * xa + 4 * lane;   // float offset in the image row
        v[k] = make_float4(0.f, 0.f, 0.f, 0.f);   // outside the image: never read
        if (rr < kRows && 4 * lane < kVRow && gy >= 0 && gy < H && f >= 0 && f + 4 <= 3 * W)
            v[k] = *reinterpret_cast<const float4 *>((buf ? imgb : imga) + 3 * (base + (size_t)gy * W) + f);
    }
#pragma unroll
    for (int k = 0; k < kIt; ++k) {
        const int rr = warp + k * kVY, buf = rr >= kVTH, ty = rr - buf * kVTH;
        if (rr < kRows && 4 * lane < kVRow) *reinterpret_cast<float4 *>(&tile[buf][ty][4 * lane]) = v[k];
    }
    __syncthreads();
    const int cx = x0 + lane, cy = y0 + warp;
    if (cx >= W || cy >= H) return;
    const size_t p = base + (size_t)cy * W + cx;
#pragma unroll
    for (int buf = 0; buf < 2; ++buf) {
        float ax = 0.f, ay = 0.f, az = 0.f;
        int n = 0;
#pragma unroll
        for (int dy = -1; dy <= 1; ++dy)
#pragma unroll
            for (int dx = -1; dx <= 1; ++dx) {
                if (dy == 0 && dx == 0) continue;
                const int ix = cx + dx, iy = cy + dy;
                if (ix < 0 || ix >= W || iy < 0 || iy >= H) continue;
                const float *t = &tile[buf][warp + 1 + dy][3 * (lane + 4 + dx)];
                ax += t[0];
                ay += t[1];
                az += t[2];
                ++n;
            }
        const float *t = &tile[buf][warp + 1][3 * (lane + 4)];
        float mx, my, mz;
        if (n == 8) {
            // interior pixels: a quotient by 8 is the product by 1/8, exactly
            // (__fmul_rn: rounded on its own, never fused into the subtraction)
            mx = __fmul_rn(ax, 0.125f);
            my = __fmul_rn(ay, 0.125f);
            mz = __fmul_rn(az, 0.125f);
        } else {
            const float fn = (float)n;
            mx = ax / fn;
            my = ay / fn;
            mz = az / fn;
        }
        const float var = norm2(mx - t[0], my - t[1], mz - t[2]);
        (buf ? varb : vara)[p] = var;
        (buf ? sdb : sda)[p] = sqrtf(var);
    }
}

__global__ void __launch_bounds__(256) variance_px_kernel(const float *imga,
                                                       const float *imgb,
                                                       float *__restrict__ vara,
                                                       float *__restrict__ varb,
                                                       float *__restrict__ sda,
                                                       float *__restrict__ sdb, int H, int W)
{
    chain_wait();
    chain_next();
    const int cx = blockIdx.x * blockDim.x + threadIdx.x;
    const int cy = blockIdx.y * blockDim.y + threadIdx.y;
    if (cx >= W || cy >= H) return;
    const int buf = blockIdx.z & 1;
    const size_t base = (size_t)(blockIdx.z >> 1) * H * W;
    const float *img = (buf ? imgb : imga) + 3 * base;
    float *var = (buf ? varb : vara) + base;
    float *sd = (buf ? sdb : sda) + base;
    const int sx = max(0, cx - 1), ex = min(W - 1, cx + 1);
    const int sy = max(0, cy - 1), ey = min(H - 1, cy + 1);
    float ax = 0.f, ay = 0.f, az = 0.f;
    int n = 0;
    for (int iy = sy; iy <= ey; ++iy)
        for (int ix = sx; ix <= ex; ++ix) {
            if (iy == cy && ix == cx) continue;
            const float3 v = ld3(img, (size_t)iy * W + ix);
            ax += v.x;
            ay += v.y;
            az += v.z;
            ++n;
        }
    const float3 c = ld3(img, (size_t)cy * W + cx);
    float mx, my, mz;
    if (n == 8) {
        // interior pixels: a quotient by 8 is the product by 1/8, exactly
        // (__fmul_rn: rounded on its own, never fused into the subtraction)
        mx = __fmul_rn(ax, 0.125f);
        my = __fmul_rn(ay, 0.125f);
        mz = __fmul_rn(az, 0.125f);
    } else {
        const float fn = (float)n;
        mx = ax / fn;
        my = ay / fn;
        mz = az / fn;
    }
    const float v = norm2(mx - c.x, my - c.y, mz - c.z);
    var[(size_t)cy * W + cx] = v;
    sd[(size_t)cy * W + cx] = sqrtf(v);
}

// ---------------------------------------------------------------------------
// Normal-equation accumulators of one buffer.  The 6x6 per-channel systems
// share every entry that involves only the constant and the normal
// differences, so 61 scalars describe all three channels:
//   shared (10): A00 A03 A04 A05 A33 A34 A35 A44 A45 A55
//   per channel (11 x 3): A01 A02 A11 A12 A13 A14 A15 A22 A23 A24 A25
//   right-hand side (6 x 3): X0..X5
// 58 of them are kept as packed FP32x2 pairs updated by one fma.rn.f32x2
// each, every lane rounded as the scalar update and in the same order:
// channels 0 and 1 side by side (p, px; low lane channel 0), and the shared
// terms with channel 2's (q, x) so that the two lanes share one factor (w,
// w dn_i, w d1 or w da) and the other is a pair at hand, (dn0, dn1), (dn2, y)
// or (d1, da).  a05x0 = (A05, channel 2's X0), and so on.
// ---------------------------------------------------------------------------
struct Normal {
    float a00, a44, q22;
    x2::f2 a03a04, a05x0, a33a34, a35x3, a45x4, a55x5, q01q02, q11q12, q13q14, q15x1, q23q24, q25x2;
    x2::f2 p01, p02, p11, p12, p13, p14, p15, p22, p23, p24, p25;   // channels 0, 1
    x2::f2 px0, px1, px2, px3, px4, px5;
};

CD_DEV void normal_zero(Normal &n)
{
    n.a00 = n.a44 = n.q22 = 0.f;
    const x2::f2 z = 0ull;   // +0.0f in both lanes
    n.a03a04 = n.a05x0 = n.a33a34 = n.a35x3 = n.a45x4 = n.a55x5 = z;
    n.q01q02 = n.q11q12 = n.q13q14 = n.q15x1 = n.q23q24 = n.q25x2 = z;
    n.p01 = n.p02 = n.p11 = n.p12 = n.p13 = n.p14 = n.p15 = n.p22 = n.p23 = n.p24 = n.p25 = z;
    n.px0 = n.px1 = n.px2 = n.px3 = n.px4 = n.px5 = z;
}

// channel k (0, 1: a lane of the pair; 2: q) of a per-channel term
CD_DEV float chan(x2::f2 p, float q, int k) { return k == 0 ? x2::lo(p) : k == 1 ? x2::hi(p) : q; }

// |v|^2 as the reference's compiled norm2 rounds it: fma(z, z, fma(x, x, y*y))
// (the contraction the reference kernels were observed to use for
// x*x + y*y + z*z, see reproject.cu).
CD_DEV float sqnorm(float x, float y, float z) { return fmaf(z, z, fmaf(x, x, y * y)); }

// exp(x) = 2^(x log2 e) on the ex2.approx.ftz instruction (subnormal results
// flushed to zero).
CD_DEV float exp_ftz(float x)
{
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x * 1.44269504088896341f));
    return y;
}

// Quotients by a shared divisor (P. Markstein, "Computation of elementary
// functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34,
// 1990): with y the reciprocal of b rounded to nearest, q = RN(a y) and the
// exact residual r = a - q b, RN(q + r y) is the IEEE quotient a / b.  y is
// the hardware approximation after one Newton step: the rounded reciprocal
// of every significand (run on sm_100a over all 2^23 of them at nine
// exponents; 7e10 quotients there equal the division's).
// Holds for b in [2^-14, 2^100) and a = 0 or |a| in [2^-102, 2^100) with a
// normal quotient.  Below, the residual (a multiple of 2^-47 of a) underflows
// and the result may be an ulp off.  That is not seen: with the taps' divisors
// of 1e-2 and more it is a difference quotient below 2^-95, whose square
// vanishes beside the ridge of 1e-3 on the diagonal, and whose coefficient
// multiplies a quotient as small in the reconstruction; a distance below
// 2^-88 leaves its weight at 1.
CD_DEV float reciprocal(float b)
{
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(b));
    return fmaf(y, fmaf(-b, y, 1.f), y);
}
CD_DEV float quotient(float a, float b, float y)
{
    const float q = __fmul_rn(a, y);
    return fmaf(fmaf(-q, b, a), y, q);
}
constexpr float kQuotientMax = 0x1p100f;
// The same for any a and any b not below 1e-4 (or NaN), for the repeated
// windows.  An operand that is not finite leaves no rounding to get right:
// inf / b is that infinity, a / inf a zero, the rest NaN.  The division
// instruction sequence takes its slow path there, which made such a window
// cost twice a finite one.
CD_DEV float quotient_any(float a, float b, float y)
{
    if (fabsf(a) < kQuotientMax && b < kQuotientMax) return quotient(a, b, y);
    const bool b_finite = b < INFINITY;
    if (fabsf(a) < INFINITY && b_finite) return a / b;
    return b_finite ? a : a * __fdividef(1.f, b);
}

// The centre's own values: features, albedo and normal (channels 0, 1 as a
// pair), variance and standard deviation.
struct Centre {
    x2::f2 f01, a01, n01;
    float f2, a2, n2, v, sd;
};

// One window tap of one buffer: f4 = (features, variance), y4 = (target, .),
// a4 = (albedo, .), n4 = (normal, .), sdt the features' standard deviation.
// Follows ops/regression.cu.cc:418-445: delta = [1, (f_t-f_c)/(sd_c+sd_t+1e-2),
// alb_t-alb_c, n_t-n_c], w = exp(-|f_t-f_c|^2/(v_c+v_t+1e-4)) + 1e-7.
//
// The tap's four quotients are the IEEE quotients (but for the smallest, see
// quotient()): the normal equations amplify their last bits.  kFast takes them
// with quotient() from two reciprocals instead of four divisions (about 20
// instructions each, with a branch): 1080p, window 17, the kernel 505 -> 433
// us (and 407 us with the pairs, the fixed row layout and the launch bound
// below).  That needs the divisors (at least 1e-4) and the squared distance
// below kQuotientMax, which bounds the other operands from above too (sd =
// sqrt(v)); `sane` turns false where a tap is not, and the caller starts its
// window again with kFast off at the end of that row.  256x256, window 15, one
// NaN pixel: 125 us (151 with four divisions throughout, 197 when the window
// was swept to its end and repeated with them); 1080p, window 17, 3000 of
// them: 952 (1110, 1406).  The vote per row costs a finite frame 0.5 %.
template <bool kFast>
CD_DEV void normal_tap(Normal &n, float4 f4, float4 y4, float4 a4, float4 n4, float sdt, const Centre &c, bool &sane)
{
    using namespace x2;
    const f2 df01 = sub2(pack(f4.x, f4.y), c.f01), da01 = sub2(pack(a4.x, a4.y), c.a01);
    const f2 dn01 = sub2(pack(n4.x, n4.y), c.n01);
    const float df2 = f4.z - c.f2, da2 = a4.z - c.a2, dn2 = n4.z - c.n2;
    const float den = (c.sd + sdt) + 1e-2f;
    const float denw = (c.v + f4.w) + 1e-4f, sq = sqnorm(lo(df01), hi(df01), df2);
    float dist, d1[3];
    if (kFast) {
        sane = sane && denw < kQuotientMax && sq < kQuotientMax;
        const float rden = reciprocal(den), rw = reciprocal(denw);
        dist = quotient(sq, denw, rw);
        d1[0] = quotient(lo(df01), den, rden);
        d1[1] = quotient(hi(df01), den, rden);
        d1[2] = quotient(df2, den, rden);
    } else {
        const float rden = reciprocal(den), rw = reciprocal(denw);
        dist = quotient_any(sq, denw, rw);
        d1[0] = quotient_any(lo(df01), den, rden);
        d1[1] = quotient_any(hi(df01), den, rden);
        d1[2] = quotient_any(df2, den, rden);
    }
    // a weight below 2^-126 and its flush to zero both give 1e-7 after the addition
    const float w = exp_ftz(-dist) + 1e-7f;
    const f2 wP = pack(w, w), d1P = pack(d1[0], d1[1]), yP = pack(y4.x, y4.y);
    const f2 dda = pack(d1[2], da2), dny = pack(dn2, y4.z);   // channel 2's (d1, da) and (dn2, y)
    const f2 wd1P = mul2(wP, d1P), wd2P = mul2(wP, da01), wdda = mul2(wP, dda), wn01 = mul2(wP, dn01);
    const f2 dn0P = pack(lo(dn01), lo(dn01)), dn1P = pack(hi(dn01), hi(dn01)), dn2P = pack(dn2, dn2);
    const f2 wn0P = pack(lo(wn01), lo(wn01)), wn1P = pack(hi(wn01), hi(wn01));
    const float wn2 = w * dn2;
    const f2 wn2P = pack(wn2, wn2);
    n.p01 = fma2(wP, d1P, n.p01);
    n.p02 = fma2(wP, da01, n.p02);
    n.p11 = fma2(wd1P, d1P, n.p11);
    n.p12 = fma2(wd1P, da01, n.p12);
    n.p13 = fma2(wd1P, dn0P, n.p13);
    n.p14 = fma2(wd1P, dn1P, n.p14);
    n.p15 = fma2(wd1P, dn2P, n.p15);
    n.p22 = fma2(wd2P, da01, n.p22);
    n.p23 = fma2(wd2P, dn0P, n.p23);
    n.p24 = fma2(wd2P, dn1P, n.p24);
    n.p25 = fma2(wd2P, dn2P, n.p25);
    n.px0 = fma2(wP, yP, n.px0);
    n.px1 = fma2(wd1P, yP, n.px1);
    n.px2 = fma2(wd2P, yP, n.px2);
    n.px3 = fma2(wn0P, yP, n.px3);
    n.px4 = fma2(wn1P, yP, n.px4);
    n.px5 = fma2(wn2P, yP, n.px5);
    // shared terms and channel 2
    const float wd1 = lo(wdda), wd2 = hi(wdda);
    const f2 wd1D = pack(wd1, wd1), wd2D = pack(wd2, wd2);
    n.a00 += w;
    n.a44 = fmaf(hi(wn01), hi(dn01), n.a44);
    n.q22 = fmaf(wd2, da2, n.q22);
    n.a03a04 = fma2(wP, dn01, n.a03a04);
    n.a05x0 = fma2(wP, dny, n.a05x0);
    n.a33a34 = fma2(wn0P, dn01, n.a33a34);
    n.a35x3 = fma2(wn0P, dny, n.a35x3);
    n.a45x4 = fma2(wn1P, dny, n.a45x4);
    n.a55x5 = fma2(wn2P, dny, n.a55x5);
    n.q01q02 = fma2(wP, dda, n.q01q02);
    n.q11q12 = fma2(wd1D, dda, n.q11q12);
    n.q13q14 = fma2(wd1D, dn01, n.q13q14);
    n.q15x1 = fma2(wd1D, dny, n.q15x1);
    n.q23q24 = fma2(wd2D, dn01, n.q23q24);
    n.q25x2 = fma2(wd2D, dny, n.q25x2);
}

// Cholesky factorisation + forward / backward substitution of one channel's
// ridge-regularised 6x6 system, in the reference's operation order
// (ops/regression.cu.cc:206-242, 449-467): diagonal pivots
// sqrt(max(1e-5, a_ii - s)), off-diagonals (1/L_jj) * (a_ji - s).
// Lo (nullable) receives the factor, row-major packed lower triangle
// (21 floats per channel), for the backward pass.
//
// FP64 fallback (cond_limit > 0, off by default): when the factor's pivots
// give a condition estimate (max L_ii / min L_ii)^2 above cond_limit, the
// same FP32 normal equations are factored and solved again in double and
// *fallbacks is incremented.  The reference has no such path; with the
// fallback off the result is the reference's.
CD_DEV void solve_fp64(const float (*A)[kP], const float *X, int k, float *beta)
{
    double L[kP][kP];
#pragma unroll
    for (int i = 0; i < kP; ++i) {
#pragma unroll
        for (int j = 0; j <= i; ++j) {
            double s = 0.0;
#pragma unroll
            for (int q = 0; q < j; ++q) s = fma(L[i][q], L[j][q], s);
            if (i == j)
                L[i][i] = sqrt(fmax(1e-12, (double)A[i][i] - s));
            else
                L[i][j] = ((double)A[j][i] - s) / L[j][j];
        }
    }
    double Y[kP], bt[kP];
#pragma unroll
    for (int i = 0; i < kP; ++i) {
        double s = X[i];
#pragma unroll
        for (int q = 0; q < i; ++q) s -= L[i][q] * Y[q];
        Y[i] = s / L[i][i];
    }
#pragma unroll
    for (int i = kP - 1; i >= 0; --i) {
        double s = Y[i];
#pragma unroll
        for (int q = i + 1; q < kP; ++q) s -= L[q][i] * bt[q];
        bt[i] = s / L[i][i];
    }
#pragma unroll
    for (int r = 0; r < kP; ++r) beta[r * 3 + k] = (float)bt[r];
}

CD_DEV void solve_channel(const Normal &n, int k, float *beta, float *Lo, float cond_limit = 0.f,
                          unsigned *fallbacks = nullptr)
{
    float A[kP][kP];
    using x2::lo;
    using x2::hi;
    A[0][0] = n.a00; A[0][1] = chan(n.p01, lo(n.q01q02), k); A[0][2] = chan(n.p02, hi(n.q01q02), k);
    A[0][3] = lo(n.a03a04); A[0][4] = hi(n.a03a04); A[0][5] = lo(n.a05x0);
    A[1][1] = chan(n.p11, lo(n.q11q12), k); A[1][2] = chan(n.p12, hi(n.q11q12), k);
    A[1][3] = chan(n.p13, lo(n.q13q14), k); A[1][4] = chan(n.p14, hi(n.q13q14), k);
    A[1][5] = chan(n.p15, lo(n.q15x1), k);
    A[2][2] = chan(n.p22, n.q22, k); A[2][3] = chan(n.p23, lo(n.q23q24), k);
    A[2][4] = chan(n.p24, hi(n.q23q24), k); A[2][5] = chan(n.p25, lo(n.q25x2), k);
    A[3][3] = lo(n.a33a34); A[3][4] = hi(n.a33a34); A[3][5] = lo(n.a35x3);
    A[4][4] = n.a44; A[4][5] = lo(n.a45x4);
    A[5][5] = lo(n.a55x5);
#pragma unroll
    for (int r = 0; r < kP; ++r) A[r][r] += 1e-3f;
    const float X[kP] = {chan(n.px0, hi(n.a05x0), k), chan(n.px1, hi(n.q15x1), k), chan(n.px2, hi(n.q25x2), k),
                         chan(n.px3, hi(n.a35x3), k), chan(n.px4, hi(n.a45x4), k), chan(n.px5, hi(n.a55x5), k)};
    float L[kP][kP];
#pragma unroll
    for (int i = 0; i < kP; ++i) {
#pragma unroll
        for (int j = 0; j <= i; ++j) {
            float s = 0.f;
#pragma unroll
            for (int q = 0; q < j; ++q) s = fmaf(L[i][q], L[j][q], s);
            if (i == j)
                L[i][i] = sqrtf(fmaxf(1e-5f, A[i][i] - s));
            else
                L[i][j] = (1.f / L[j][j]) * (A[j][i] - s);
        }
    }
    if (Lo) {
#pragma unroll
        for (int i = 0; i < kP; ++i)
#pragma unroll
            for (int j = 0; j <= i; ++j) Lo[21 * k + i * (i + 1) / 2 + j] = L[i][j];
    }
    if (cond_limit > 0.f) {
        float dmin = L[0][0], dmax = L[0][0];
#pragma unroll
        for (int i = 1; i < kP; ++i) {
            dmin = fminf(dmin, L[i][i]);
            dmax = fmaxf(dmax, L[i][i]);
        }
        if (dmax * dmax > cond_limit * (dmin * dmin)) {
            solve_fp64(A, X, k, beta);
            if (fallbacks) atomicAdd(fallbacks, 1u);
            return;
        }
    }
    float Y[kP];
    Y[0] = X[0] / L[0][0];
#pragma unroll
    for (int i = 1; i < kP; ++i) {
        float s = 0.f;
#pragma unroll
        for (int q = 0; q < i; ++q) s = fmaf(L[i][q], Y[q], s);
        Y[i] = (X[i] - s) / L[i][i];
    }
    float bt[kP];
    bt[kP - 1] = Y[kP - 1] / L[kP - 1][kP - 1];
#pragma unroll
    for (int i = kP - 2; i >= 0; --i) {
        float s = 0.f;
#pragma unroll
        for (int q = kP - 1; q > i; --q) s = fmaf(L[q][i], bt[q], s);
        bt[i] = (Y[i] - s) / L[i][i];
    }
#pragma unroll
    for (int r = 0; r < kP; ++r) beta[r * 3 + k] = bt[r];
}

// ---------------------------------------------------------------------------
// Regression kernel.
// A CTA owns 32 consecutive centres of one centre row; warp 0 solves buffer A
// and warp 1 buffer B, one thread per (centre, buffer), so every centre sums
// its window taps in the reference's order (rows, then columns) with the
// reference's per-tap arithmetic.  The window rows stream through two
// shared-memory row slots (cp.async, double buffered; layout in
// window_rows.cuh): row r + 1 is copied while row r is consumed, and a tap
// is four conflict-free LDS.128.
// ---------------------------------------------------------------------------
constexpr int kCX = kRowCentres;   // centres per CTA
constexpr int kThreads = 64;

// two row slots of 4 float4 groups, then the per-position tables
//
// SP > 0: the sparsity as a template parameter, and a fixed row layout
// (row_q(SP) positions per de-interleaved run, enough for windows to 19), so
// that a tap's four loads and the SP taps of a run are constant offsets from
// one pointer.  SP = 4, the reference's, and 2; others take SP = 0.  The
// positions are no more than the windows need: a longer run measured slower
// (40 instead of 36 at SP = 4: 713 against 706 us per 1080p
// cross-regression, window 17), shared memory being taken from the L1 that
// the neighbouring CTAs' rows hit.
__host__ __device__ constexpr int row_q(int sp) { return kCX - 1 + (19 + sp - 1) / sp; }

template <int SP>
__host__ __device__ inline RowGeom regression_geom(int hw, int sp)
{
    RowGeom g = row_geom(hw, sp);
    if (SP > 0) {
        g.q = row_q(SP);
        g.npos = SP * g.q;
    }
    return g;
}

inline bool fixed_rows(int hw, int sp) { return (sp == 2 || sp == 4) && row_geom(hw, sp).q <= row_q(sp); }

__host__ __device__ inline size_t regression_smem(const RowGeom &g)
{
    return (size_t)2 * 4 * g.npos * sizeof(float4) + (size_t)2 * g.rw * sizeof(int);
}

// Launch bound 8 CTAs per SM (128 registers): 706 us per 1080p
// cross-regression, window 17, against 733 under a bound of 7, 776 under 6
// (154 registers, 12 warps per SM) and 757 under 9 (112, spills in the sums).
// Not launched chained (launch.cuh): the waits before its loads cost it
// registers (256x256 cross-regression 77 against 64 us).
template <int SP>
__global__ void __launch_bounds__(kThreads, 8) regression_kernel(
    const float *__restrict__ imga, const float *__restrict__ imgb,
    const float *__restrict__ albedo, const float *__restrict__ normal,
    const float *__restrict__ vara, const float *__restrict__ varb,
    const float *__restrict__ sda, const float *__restrict__ sdb, float *__restrict__ beta,
    float *__restrict__ chol, float cond_limit, unsigned *__restrict__ fallbacks, int H, int W, int hw, int sp_rt)
{
    extern __shared__ float4 sm4[];
    const int sp = SP > 0 ? SP : sp_rt;
    const RowGeom g = regression_geom<SP>(hw, sp);
    const int slot = 4 * g.npos;                                   // float4s per slot
    int *pos_gx = reinterpret_cast<int *>(sm4 + 2 * slot);
    int *pos_dst = pos_gx + g.rw;
    const int Ws = W / sp, Hs = H / sp;
    const int b = blockIdx.z;
    const size_t px = (size_t)H * W;
    imga += 3 * px * b;
    imgb += 3 * px * b;
    albedo += 3 * px * b;
    normal += 3 * px * b;
    vara += px * b;
    varb += px * b;
    sda += px * b;
    sdb += px * b;

    const int i0 = blockIdx.x * kCX;
    const int cy = blockIdx.y * sp;
    const int x0 = i0 * sp - hw;
    const int buf = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int R = 2 * hw + 1;

    row_positions(pos_gx, pos_dst, g, x0, W, sp, threadIdx.x, kThreads);
    __syncthreads();

    auto stage = [&](int r, int s) {
        stage_window_row(reinterpret_cast<float *>(sm4 + s * slot), g, pos_gx, pos_dst,
                         clampi(mirror(cy - hw + r, H), 0, H - 1), W, imga, imgb, albedo, normal, vara, varb, sda,
                         sdb, threadIdx.x, kThreads);
    };

    // centre values, read directly (clamped for lanes past the last centre)
    const int ci = min(i0 + lane, Ws - 1);
    const size_t c = (size_t)cy * W + (size_t)ci * sp;
    const float3 fc = ldg3(buf ? imgb : imga, c);
    const float3 alc = ldg3(albedo, c), nrc = ldg3(normal, c);
    const float vc = __ldg((buf ? varb : vara) + c), sdc = __ldg((buf ? sdb : sda) + c);
    const Centre cen = {x2::pack(fc.x, fc.y), x2::pack(alc.x, alc.y), x2::pack(nrc.x, nrc.y), fc.z, alc.z, nrc.z,
                        vc, sdc};
    // groups read by this buffer: own features + variance, target, albedo, normal
    const int gf = buf ? 1 : 0, gy_ = buf ? 0 : 1;

    Normal nm;
    // the sum over the window's taps; false once a quotient was out of range
    auto sweep = [&](auto fast) {
        bool sane = true;
        normal_zero(nm);
        stage(0, 0);
        cp_async_commit();
        for (int r = 0; r < R; ++r) {
            if (r + 1 < R) {
                stage(r + 1, (r + 1) & 1);
                cp_async_commit();
                cp_async_wait<1>();
            } else {
                cp_async_wait<0>();
            }
            __syncthreads();
            const float4 *P = sm4 + (r & 1) * slot;
            const float4 *Gf = P + gf * g.npos + lane, *Gy = P + gy_ * g.npos + lane;
            const float4 *Gn = P + 3 * g.npos + lane;   // albedo: g.npos before it
            auto tap = [&](int o) {
                const float4 f4 = Gf[o], y4 = Gy[o], a4 = Gn[o - g.npos], n4 = Gn[o];
                // own standard deviation: sdA rides in g2.w, sdB in g3.w
                normal_tap<decltype(fast)::value>(nm, f4, y4, a4, n4, buf ? n4.w : a4.w, cen, sane);
            };
            if (SP > 0) {
                for (int t = 0; t < R; t += sp, ++Gf, ++Gy, ++Gn) {
#pragma unroll
                    for (int tm = 0; tm < SP; ++tm)
                        if (t + tm < R) tap(tm * g.q);
                }
            } else {
                int tm = 0, td = 0;
                for (int t = 0; t < R; ++t) {
                    tap(tm * g.q + td);
                    if (++tm == sp) {
                        tm = 0;
                        ++td;
                    }
                }
            }
            if (!__syncthreads_and(sane)) return false;
        }
        return true;
    };
    if (!sweep(std::true_type())) sweep(std::false_type());

    if (i0 + lane >= Ws) return;
    const size_t nb_img = (size_t)Hs * Ws;
    const size_t cidx = (size_t)b * nb_img + (size_t)blockIdx.y * Ws + (i0 + lane);
    float *bo = beta + (size_t)buf * gridDim.z * nb_img * kBeta + cidx * kBeta;
    float *lo = chol ? chol + ((size_t)buf * gridDim.z * nb_img + cidx) * 63 : nullptr;
    solve_channel(nm, 0, bo, lo, cond_limit, fallbacks);
    solve_channel(nm, 1, bo, lo, cond_limit, fallbacks);
    solve_channel(nm, 2, bo, lo, cond_limit, fallbacks);
}

// ---------------------------------------------------------------------------
// Block reconstruction (ops/regression.cu.cc:289-365).  A CTA owns 32x4
// output pixels.  The centres their windows reach are staged in shared
// memory as 13 float4 records each.  Each thread sums, over the centres of
// its own window (the reference's clamped iDivUp range, in its order),
// w * (beta_c . delta(p, c)) with delta taken as (p - c).  The quotients use
// a reciprocal and a multiply: unlike the regression's normal equations,
// nothing downstream amplifies their last-bit differences.
//
// Buffers A and B share every centre and pixel pair, so their arithmetic
// runs as packed FP32x2 pairs (low lane A, high lane B; same operation
// order and per-lane rounding as the scalar formulation, ops/regression.cu.cc
// :465-500).  Record of a centre (pairs (A, B) unless noted):
//   0..8   coefficients j = r * 3 + ch, two per record: (A_j, B_j, A_j+1, B_j+1)
//   9      (feature.x, feature.y)      10  (feature.z, variance)
//   11     (sd, albedo.x albedo.y)     12  albedo.z normal.xyz (scalars)
// ---------------------------------------------------------------------------
constexpr int kRX = 32, kRThreadRows = 4;
constexpr int kRec = 13;   // float4 per staged centre

// The three forms of the kernel and where each runs (us per cross-regression,
// all with the same results):
//   two pixels per thread (128 registers, four CTAs' worth) where a pixel
//     reaches more than two centres a row, the grid still has two CTAs per SM
//     of a 148-SM part, and three CTAs' centres fit an SM's shared memory.
//     1080p, window 17, sparsity 4: 615 against 697 lean; 256x384 (384 CTAs),
//     window 17: 72 against 75; below the lines: 192x192 (144 CTAs), window
//     17: 65 against 64 lean, 64x96 64 against 62, 720p, window 5, sparsity 4:
//     101 against 95, window 1, sparsity 2: 145 against 129;
//   one, lean (72 registers, seven CTAs, the column loop not unrolled), while
//     the centres of six CTAs fit: 720p, window 7, sparsity 4: 111 us, in the
//     unrolled form of 111 registers 133;
//   one, unrolled, for more centres than that, which leave few CTAs to an SM:
//     720p, window 5, sparsity 1: 619 against 646 lean.
constexpr size_t kReconPairSmem = 74 * 1024, kReconLeanSmem = 36 * 1024;
constexpr long kReconPairCtas = 2 * 148;

__host__ __device__ inline int floordiv(int a, int b) { return a >= 0 ? a / b : -((-a + b - 1) / b); }

__host__ __device__ inline size_t recon_smem(int hw, int sp, int rs, int rows)
{
    const int cxmax = ((kRX - 1) * rs + 2 * hw) / sp + 2;
    const int cymax = ((rows - 1) * rs + 2 * hw) / sp + 2;
    return (size_t)kRec * cxmax * cymax * sizeof(float4);
}

// One output pixel's own values ((A, B) pairs, shared scalars) and its sums.
struct ReconPixel {
    x2::f2 f0, f1, f2, var, sd;
    float3 al, nr;
    x2::f2 o0, o1, o2, sw;
};

// NP: output pixels per thread, in consecutive rows.  A record is 208 bytes
// per lane, and shared memory returns 128 bytes per cycle and SM whatever
// the lanes share, so with one pixel per thread the kernel runs at that rate
// (92 % of it, 52 cycles per warp and centre against 19 of packed
// arithmetic); two pixels per thread read each record once for both.  The
// rows of a warp's pixels are the same, so the centre rows that only one of
// them reaches are a uniform branch.
template <int NP, bool kLean>
__global__ void __launch_bounds__(kRX * kRThreadRows, NP == 2 ? 4 : kLean ? 7 : 1) recon_kernel(
    const float *imga, const float *imgb,
    const float *albedo, const float *normal,
    const float *vara, const float *varb,
    const float *sda, const float *sdb,
    const float *beta, float *__restrict__ outa, float *__restrict__ outb,
    float *__restrict__ state, int H, int W, int hw, int sp, int rs)
{
    chain_wait();
    chain_next();
    using namespace x2;
    extern __shared__ float4 rec[];
    constexpr int kRows = NP * kRThreadRows, kBlock = kRX * kRThreadRows;
    const int Wr = W / rs, Hr = H / rs;
    const int Ws = W / sp, Hs = H / sp;
    const int b = blockIdx.z;
    const size_t px = (size_t)H * W;
    imga += 3 * px * b;
    imgb += 3 * px * b;
    albedo += 3 * px * b;
    normal += 3 * px * b;
    vara += px * b;
    varb += px * b;
    sda += px * b;
    sdb += px * b;
    const size_t nb_img = (size_t)Hs * Ws;
    const float *betaA = beta + (size_t)b * nb_img * kBeta;
    const float *betaB = beta + (size_t)gridDim.z * nb_img * kBeta + (size_t)b * nb_img * kBeta;

    // centres any pixel of this tile can reach (a superset of every
    // per-pixel range below)
    const int ox0 = blockIdx.x * kRX, oy0 = blockIdx.y * kRows;
    const int ox1 = min(ox0 + kRX - 1, Wr - 1), oy1 = min(oy0 + kRows - 1, Hr - 1);
    const int cx_lo = max(0, floordiv(ox0 * rs - hw, sp));
    const int cx_hi = min(Ws - 1, (ox1 * rs + hw) / sp);
    const int cy_lo = max(0, floordiv(oy0 * rs - hw, sp));
    const int cy_hi = min(Hs - 1, (oy1 * rs + hw) / sp);
    const int ncx = cx_hi - cx_lo + 1, ncy = cy_hi - cy_lo + 1;
    const int nc = ncx * ncy;

    const int tid = threadIdx.y * kRX + threadIdx.x;
    for (int e = tid; e < nc * 9; e += kBlock) {
        const int n = e / 9, f = e - 9 * n;
        const int iy = cy_lo + n / ncx, ix = cx_lo + n % ncx;
        const size_t cb = ((size_t)iy * Ws + ix) * kBeta + 2 * f;
        rec[n * kRec + f] = make_float4(betaA[cb], betaB[cb], betaA[cb + 1], betaB[cb + 1]);
    }
    for (int n = tid; n < nc; n += kBlock) {
        const int iy = cy_lo + n / ncx, ix = cx_lo + n % ncx;
        const size_t t = (size_t)(iy * sp) * W + ix * sp;
        const float3 fa = ld3(imga, t), fb = ld3(imgb, t), al = ld3(albedo, t), nr = ld3(normal, t);
        rec[n * kRec + 9] = make_float4(fa.x, fb.x, fa.y, fb.y);
        rec[n * kRec + 10] = make_float4(fa.z, fb.z, vara[t], varb[t]);
        rec[n * kRec + 11] = make_float4(sda[t], sdb[t], al.x, al.y);
        rec[n * kRec + 12] = make_float4(al.z, nr.x, nr.y, nr.z);
    }
    __syncthreads();

    const int cx = ox0 + threadIdx.x, cy = oy0 + NP * threadIdx.y;
    if (cx >= Wr || cy >= Hr) return;
    const int pxo = cx * rs;
    const int sx = max(0, idivup(pxo - hw, sp));
    const int ex = min((W - 1) / sp, (pxo + hw) / sp);
    int sy[NP], ey[NP];
    ReconPixel px_[NP];
#pragma unroll
    for (int i = 0; i < NP; ++i) {
        const bool in = cy + i < Hr;
        const int pyo = (in ? cy + i : cy) * rs;
        const size_t p = (size_t)pyo * W + pxo;
        sy[i] = max(0, idivup(pyo - hw, sp));
        ey[i] = in ? min((H - 1) / sp, (pyo + hw) / sp) : -1;   // no centre row for a pixel past the image
        const float3 fa = ld3(imga, p), fb = ld3(imgb, p);
        ReconPixel &q = px_[i];
        q.al = ld3(albedo, p);
        q.nr = ld3(normal, p);
        q.f0 = pack(fa.x, fb.x);
        q.f1 = pack(fa.y, fb.y);
        q.f2 = pack(fa.z, fb.z);
        q.var = pack(vara[p], varb[p]);
        q.sd = pack(sda[p], sdb[p]);
        q.o0 = q.o1 = q.o2 = q.sw = 0ull;   // +0.0f in both lanes
    }
    const f2 k1e2 = pack(1e-2f, 1e-2f), k1e4 = pack(1e-4f, 1e-4f), k1e7 = pack(1e-7f, 1e-7f);
    // the centres of row iy, for the pixels [i0, i0 + n)
    auto centre_row = [&](int iy, auto first, auto count) {
        constexpr int i0 = decltype(first)::value, n = decltype(count)::value;
        const float4 *R4 = rec + ((iy - cy_lo) * ncx - cx_lo + sx) * kRec;
        auto centre = [&]() {
            const ulonglong2 *R = reinterpret_cast<const ulonglong2 *>(R4);
            const ulonglong2 F9 = R[9], F10 = R[10], F11 = R[11];
            const float4 L12 = R4[12];
            f2 e0[n], e1[n], e2[n], w[n];
#pragma unroll
            for (int i = 0; i < n; ++i) {
                const ReconPixel &q = px_[i0 + i];
                const f2 d0 = sub2(q.f0, F9.x), d1 = sub2(q.f1, F9.y), d2 = sub2(q.f2, F10.x);
                const f2 den_r = add2(add2(q.sd, F11.x), k1e2);
                const f2 rden = pack(__fdividef(1.f, lo(den_r)), __fdividef(1.f, hi(den_r)));
                const f2 den_w = add2(add2(q.var, F10.y), k1e4);
                const f2 dist =
                    mul2(sqnorm2(d0, d1, d2), pack(__fdividef(1.f, lo(den_w)), __fdividef(1.f, hi(den_w))));
                // exp(-dist) + 1e-7 with exp as 2^(-dist log2 e) on ex2.approx.ftz:
                // the same weight as __expf wherever it is a normal float, and
                // where it is not, both round to 1e-7 after the addition
                w[i] = add2(pack(exp_ftz(-lo(dist)), exp_ftz(-hi(dist))), k1e7);
                e0[i] = mul2(d0, rden);
                e1[i] = mul2(d1, rden);
                e2[i] = mul2(d2, rden);
            }
            const ulonglong2 c0 = R[0], c1 = R[1], c2 = R[2], c3 = R[3], c4 = R[4], c5 = R[5], c6 = R[6], c7 = R[7],
                             c8 = R[8];
#pragma unroll
            for (int i = 0; i < n; ++i) {
                ReconPixel &q = px_[i0 + i];
                const float da0 = q.al.x - lo(F11.y), da1 = q.al.y - hi(F11.y), da2 = q.al.z - L12.x;
                const float dn0 = q.nr.x - L12.y, dn1 = q.nr.y - L12.z, dn2 = q.nr.z - L12.w;
                // coefficient j = r * 3 + ch sits in record j / 2, half j % 2:
                // r 0: c0.x c0.y c1.x | r 1: c1.y c2.x c2.y | r 2: c3.x c3.y c4.x
                // r 3: c4.y c5.x c5.y | r 4: c6.x c6.y c7.x | r 5: c7.y c8.x c8.y
                f2 p0 = fma2(c1.y, e0[i], c0.x);
                f2 p1 = fma2(c2.x, e1[i], c0.y);
                f2 p2 = fma2(c2.y, e2[i], c1.x);
                p0 = fma2(c3.x, pack(da0, da0), p0);
                p1 = fma2(c3.y, pack(da1, da1), p1);
                p2 = fma2(c4.x, pack(da2, da2), p2);
                const f2 n0 = pack(dn0, dn0), n1 = pack(dn1, dn1), n2 = pack(dn2, dn2);
                p0 = fma2(c4.y, n0, p0);
                p1 = fma2(c5.x, n0, p1);
                p2 = fma2(c5.y, n0, p2);
                p0 = fma2(c6.x, n1, p0);
                p1 = fma2(c6.y, n1, p1);
                p2 = fma2(c7.x, n1, p2);
                p0 = fma2(c7.y, n2, p0);
                p1 = fma2(c8.x, n2, p1);
                p2 = fma2(c8.y, n2, p2);
                q.o0 = fma2(w[i], p0, q.o0);
                q.o1 = fma2(w[i], p1, q.o1);
                q.o2 = fma2(w[i], p2, q.o2);
                q.sw = add2(q.sw, w[i]);
            }
        };
        if (kLean) {
#pragma unroll 1
            for (int ix = sx; ix <= ex; ++ix, R4 += kRec) centre();
        } else {
            for (int ix = sx; ix <= ex; ++ix, R4 += kRec) centre();
        }
    };
    using std::integral_constant;
    const int iy1 = NP == 2 ? max(ey[0], ey[NP - 1]) : ey[0];
    for (int iy = NP == 2 ? min(sy[0], sy[NP - 1]) : sy[0]; iy <= iy1; ++iy) {
        const bool in0 = iy >= sy[0] && iy <= ey[0], in1 = iy >= sy[NP - 1] && iy <= ey[NP - 1];
        if (NP == 1 || !in1) {
            if (in0) centre_row(iy, integral_constant<int, 0>(), integral_constant<int, 1>());
        } else if (in0) {
            centre_row(iy, integral_constant<int, 0>(), integral_constant<int, NP>());
        } else {
            centre_row(iy, integral_constant<int, NP - 1>(), integral_constant<int, 1>());
        }
    }
#pragma unroll
    for (int i = 0; i < NP; ++i) {
        if (cy + i >= Hr) break;
        const ReconPixel &q = px_[i];
        const float dA = fmaxf(lo(q.sw), 1e-7f), dB = fmaxf(hi(q.sw), 1e-7f);
        const size_t o = (size_t)b * Hr * Wr + (size_t)(cy + i) * Wr + cx;
        const float3 qa = make_float3(fmaxf(0.f, lo(q.o0) / dA), fmaxf(0.f, lo(q.o1) / dA), fmaxf(0.f, lo(q.o2) / dA));
        const float3 qb = make_float3(fmaxf(0.f, hi(q.o0) / dB), fmaxf(0.f, hi(q.o1) / dB), fmaxf(0.f, hi(q.o2) / dB));
        if (outa) {
            st3(outa, o, qa);
            st3(outb, o, qb);
        }
        if (state) {   // for the backward: the outputs and the weight sums D, [buffer][pixel]
            float4 *S = reinterpret_cast<float4 *>(state);
            S[o] = make_float4(qa.x, qa.y, qa.z, lo(q.sw));
            S[(size_t)gridDim.z * Hr * Wr + o] = make_float4(qb.x, qb.y, qb.z, hi(q.sw));
        }
    }
}

}  // namespace

cudaError_t launch_variance(const float *imga, const float *imgb, float *vara, float *varb, float *sda,
                            float *sdb, int B, int H, int W, cudaStream_t st)
{
    dim3 block(kVX, kVY);
    const bool vec = W % 4 == 0 && ((reinterpret_cast<uintptr_t>(imga) | reinterpret_cast<uintptr_t>(imgb)) & 15) == 0;
    if (vec) {
        dim3 grid((W + kVX - 1) / kVX, (H + kVY - 1) / kVY, B);
        return launch_chained(variance_kernel, grid, block, 0, st, imga, imgb, vara, varb, sda, sdb, H, W);
    }
    dim3 grid((W + kVX - 1) / kVX, (H + kVY - 1) / kVY, 2 * B);
    return launch_chained(variance_px_kernel, grid, block, 0, st, imga, imgb, vara, varb, sda, sdb, H, W);
}

size_t regression_smem_bytes(int win, int sp) { return regression_smem(row_geom(win / 2, sp)); }
size_t recon_smem_bytes(int win, int sp, int rs) { return recon_smem(win / 2, sp, rs, kRThreadRows); }

cudaError_t launch_regression(const float *imga, const float *imgb, const float *albedo,
                              const float *normal, const float *vara, const float *varb,
                              const float *sda, const float *sdb, float *beta, int B, int H, int W,
                              int win, int sp, cudaStream_t st, float *chol, float cond_limit,
                              unsigned *fallbacks)
{
    const int hw = win / 2;
    const int Ws = W / sp, Hs = H / sp;
    dim3 grid((Ws + kCX - 1) / kCX, Hs, B);
    auto go = [&](auto kern, const RowGeom &g) {
        const size_t smem = regression_smem(g);
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        kern<<<grid, kThreads, smem, st>>>(imga, imgb, albedo, normal, vara, varb, sda, sdb, beta, chol, cond_limit,
                                           fallbacks, H, W, hw, sp);
        return cudaGetLastError();
    };
    if (!fixed_rows(hw, sp)) return go(regression_kernel<0>, regression_geom<0>(hw, sp));
    return sp == 4 ? go(regression_kernel<4>, regression_geom<4>(hw, sp))
                   : go(regression_kernel<2>, regression_geom<2>(hw, sp));
}

cudaError_t launch_recon(const float *imga, const float *imgb, const float *albedo,
                         const float *normal, const float *vara, const float *varb, const float *sda,
                         const float *sdb, const float *beta, float *outa, float *outb, int B, int H,
                         int W, int win, int sp, int rs, cudaStream_t st, float *state)
{
    const int hw = win / 2;
    const int Wr = W / rs, Hr = H / rs;
    auto go = [&](auto kern, int np) {
        const int rows = np * kRThreadRows;
        const size_t smem = recon_smem(hw, sp, rs, rows);
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        dim3 block(kRX, kRThreadRows), grid((Wr + kRX - 1) / kRX, (Hr + rows - 1) / rows, B);
        return launch_chained(kern, grid, block, smem, st, imga, imgb, albedo, normal, vara, varb, sda, sdb, beta,
                              outa, outb, state, H, W, hw, sp, rs);
    };
    constexpr int pair_rows = 2 * kRThreadRows;
    const long pair_ctas = (long)B * ((Wr + kRX - 1) / kRX) * ((Hr + pair_rows - 1) / pair_rows);
    if (win > 2 * sp && pair_ctas >= kReconPairCtas && recon_smem(hw, sp, rs, pair_rows) <= kReconPairSmem)
        return go(recon_kernel<2, false>, 2);
    return recon_smem(hw, sp, rs, kRThreadRows) <= kReconLeanSmem ? go(recon_kernel<1, true>, 1)
                                                                  : go(recon_kernel<1, false>, 1);
}

}  // namespace cd
