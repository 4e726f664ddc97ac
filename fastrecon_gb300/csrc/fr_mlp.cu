// fr_mlp.cu -- the learned-DCF network: 5 -> 64 -> 64 -> 1, tanh, predicting
// log-DCF from sample-density features.  No counterpart in the reference.
//
// Parameters are kept as an FP32 master copy (optimiser state) and a BF16
// copy that the forward and backward kernels read; all arithmetic is FP32.
// Layout (FR_MLP_PARAMS values): W1[64][5] | b1[64] | W2[64][64] | b2[64] |
// W3[64] | b3.
//
//  * mlp_forward_mma_kernel (inference): the hidden layer on the tensor
//    cores (mma.sync, BF16 operands in three terms, FP32 accumulation).
//  * mlp_forward_kernel (FR_MLP_SIMT=1): one thread per sample, the BF16
//    parameters widened into shared memory once per CTA; first-layer units
//    are produced one at a time and scattered into the 64 second-layer
//    accumulators held in registers.
//  * backward: mlp_step_kernel does the forward and reverse pass of tiles of
//    64 samples in shared memory and keeps the gradient of its tiles in
//    registers, one partial gradient per CTA; mlp_reduce_kernel sums the
//    partials in a fixed order (the gradient is deterministic).
//  * mlp_adam_kernel: Adam on the master copy, then the BF16 copy.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>

#include "fr_internal.h"

namespace fr {
namespace {

constexpr int NI = FR_MLP_IN;
constexpr int NH = FR_MLP_HIDDEN;
constexpr int OFF_W1 = 0;
constexpr int OFF_B1 = OFF_W1 + NH * NI;
constexpr int OFF_W2 = OFF_B1 + NH;
constexpr int OFF_B2 = OFF_W2 + NH * NH;
constexpr int OFF_W3 = OFF_B2 + NH;
constexpr int OFF_B3 = OFF_W3 + NH;
constexpr int NP = OFF_B3 + 1;
static_assert(NP == FR_MLP_PARAMS, "parameter layout");

constexpr int kFwdThreads = 128;

// Widen the BF16 parameters into shared memory, W2 transposed (row i of the
// shared copy holds W2[.][i]) so that both passes read it along rows.
__device__ __forceinline__ void load_params(const __nv_bfloat16 *__restrict__ pb, float *ps)
{
    for (int p = threadIdx.x; p < NP; p += blockDim.x) {
        int q = p;
        if (p >= OFF_W2 && p < OFF_B2) {
            const int j = (p - OFF_W2) / NH, i = (p - OFF_W2) % NH;
            q = OFF_W2 + i * NH + j;
        }
        ps[q] = __bfloat162float(pb[p]);
    }
    __syncthreads();
}

// Hidden unit i of the first layer.
__device__ __forceinline__ float unit1(const float *ps, const float *x, int i)
{
    float a = ps[OFF_B1 + i];
#pragma unroll
    for (int k = 0; k < NI; ++k) a = fmaf(ps[OFF_W1 + i * NI + k], x[k], a);
    return tanhf(a);
}

// acc[j] += W2[j][i] * v for all j (row i of the transposed copy).
__device__ __forceinline__ void axpy_row(const float *ps, int i, float v, float *acc)
{
    const float4 *w = reinterpret_cast<const float4 *>(ps + OFF_W2 + i * NH);
#pragma unroll
    for (int q = 0; q < NH / 4; ++q) {
        const float4 c = w[q];
        acc[4 * q] = fmaf(c.x, v, acc[4 * q]);
        acc[4 * q + 1] = fmaf(c.y, v, acc[4 * q + 1]);
        acc[4 * q + 2] = fmaf(c.z, v, acc[4 * q + 2]);
        acc[4 * q + 3] = fmaf(c.w, v, acc[4 * q + 3]);
    }
}

// Second-layer activations h2 (in place of the pre-activations) and the output.
__device__ __forceinline__ float forward_sample(const float *ps, const float *xs, float *h2)
{
#pragma unroll
    for (int j = 0; j < NH; ++j) h2[j] = ps[OFF_B2 + j];
#pragma unroll 1
    for (int i = 0; i < NH; ++i) axpy_row(ps, i, unit1(ps, xs, i), h2);
    float out = ps[OFF_B3];
#pragma unroll
    for (int j = 0; j < NH; ++j) {
        h2[j] = tanhf(h2[j]);
        out = fmaf(ps[OFF_W3 + j], h2[j], out);
    }
    return out;
}

__global__ void __launch_bounds__(kFwdThreads) mlp_forward_kernel(const __nv_bfloat16 *__restrict__ pb,
                                                                  const float *__restrict__ x, long long n, int exp_out,
                                                                  int residual, float scale, float *__restrict__ y)
{
    __shared__ __align__(16) float ps[NP + 3];
    load_params(pb, ps);
    for (long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x; s < n; s += (long long)gridDim.x * blockDim.x) {
        float xs[NI], h2[NH];
#pragma unroll
        for (int k = 0; k < NI; ++k) xs[k] = x[s * NI + k];
        float out = forward_sample(ps, xs, h2);
        if (residual) out = __fsub_rn(out, xs[1]);  // the network predicts log-DCF + log density (radius 2)
        y[s] = exp_out ? __fmul_rn(scale, expf(out)) : out;
    }
}

// Two floats in one 64-bit register and their packed arithmetic (one issue
// slot for both).
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float a, float b)
{
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 unpack2(f32x2 v)
{
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c)
{
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b)
{
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b)
{
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ float ex2_approx(float a)
{
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
    return r;
}
__device__ __forceinline__ float rcp_approx(float a)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
    return r;
}
// tanh of two values, branch-free.  Below 0.65: x + x t Q(t), t = x^2, Q the polynomial
// of degree 4 through (tanh(sqrt t) / sqrt t - 1) / t at the 5 Chebyshev points of
// [0, 0.65^2] (relative error of the result 2.6e-8, in floats within 1.1 ulp).  Above: the
// identity 1 - 2 / (e^2|x| + 1) with x's sign, whose errors are those of the approximate
// exponential and reciprocal times the subtracted term over the result, 0.75 at 0.65
// and falling (+-1 and NaN come out by themselves).  Within 1.7 ulp of FP64 at 1.0 M
// points, where tanhf promises 2.  A split further out costs the polynomial a degree
// for each 0.1 to 0.2: 5.1 M samples 602 us (588 since the tables are staged faster), at 0.75
// with degree 5 625 us and 1.5 ulp, at 1 with degree 6 641 us and 1.2 ulp; without the absolute
// value and sign 590 us, but 1 - 2 / (e^2x + 1) of a negative x cancels: 3.8 ulp.
__device__ __forceinline__ f32x2 tanh2(f32x2 x)
{
    const f32x2 one = pack2(1.f, 1.f);
    const f32x2 t = mul2(x, x);
    f32x2 q = fma2(t, pack2(-0.0059237261f, -0.0059237261f), pack2(0.020873461f, 0.020873461f));
    q = fma2(q, t, pack2(-0.053823758f, -0.053823758f));
    q = fma2(q, t, pack2(0.13332583f, 0.13332583f));
    q = fma2(q, t, pack2(-0.33333328f, -0.33333328f));
    const float2 p = unpack2(fma2(mul2(q, t), x, x)), v = unpack2(x);
    constexpr float k = 2.885390081777927f;  // 2 / ln 2
    const float2 e = unpack2(add2(pack2(ex2_approx(fabsf(v.x) * k), ex2_approx(fabsf(v.y) * k)), one));
    const float2 h = unpack2(fma2(pack2(rcp_approx(e.x), rcp_approx(e.y)), pack2(-2.f, -2.f), one));
    return pack2(fabsf(v.x) < 0.65f ? p.x : copysignf(h.x, v.x), fabsf(v.y) < 0.65f ? p.y : copysignf(h.y, v.y));
}

// The forward pass with the hidden layer (64 x 64) on the tensor cores:
// mma.sync m16n8k16, BF16 operands, FP32 accumulation.  One warp holds a
// tile of 16 samples: each lane evaluates, in FP32, exactly the first-layer
// activations its A fragments hold (2 samples x 16 units, units in pairs),
// splits each into three BF16 terms hi + mid + lo (the residual of a BF16
// rounding, twice: together within ~2^-24 of the FP32 value), and the warp
// accumulates W2 h1 = W2 hi + W2 mid + W2 lo into FP32 fragments that start
// from b2; the weights are BF16 already, so every product is exact and the
// sums carry FP32 rounding only.  The output layer reduces each lane's 16
// units and the 4 lanes of a row with shuffles.
// Bound: the pipes of tanh (special functions 45 %, FMA 39 % of the time), the
// tensor pipe (34 %) and issue (51 %).  5.1 M samples: 775 us with W2 rows of
// 128 bytes (8-way bank conflicts, the shared pipe 83 % busy), tanhf, and
// first-layer weights read as single BF16; 600 us so.
__device__ __forceinline__ unsigned pack_bf16(float lo_half, float hi_half)
{
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo_half, hi_half);
    return *reinterpret_cast<const unsigned *>(&v);
}

__device__ __forceinline__ void mma_bf16_16816(float *d, const unsigned *a, unsigned b0, unsigned b1)
{
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
        "{%0, %1, %2, %3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

constexpr int kMmaThreads = 128;  // 4 warps, 16 samples each per step
constexpr int kW2Row = NH + 8;    // BF16 per shared row of W2: rows 4 banks apart

__global__ void __launch_bounds__(kMmaThreads, 4) mlp_forward_mma_kernel(const __nv_bfloat16 *__restrict__ pb,
                                                                         const float *__restrict__ x, long long n,
                                                                         int exp_out, int residual, float scale,
                                                                         float *__restrict__ y)
{
    __shared__ __align__(16) float w1[NH / 2][NI + 1][2];  // unit pairs: weights per input, then biases
    __shared__ __align__(16) __nv_bfloat16 w2s[NH * kW2Row];
    __shared__ __align__(16) float b2s[NH], w3s[NH];
    __shared__ float b3s;
    // the tables, which a small batch waits for: every thread's loads at once, W2 in
    // 16-byte pieces where the parameters are aligned (as one loop over all parameters with
    // a branch for each: 3 k samples 12.6 us, so 8.0)
    if ((reinterpret_cast<uintptr_t>(pb + OFF_W2) & 15) == 0) {
        uint4 q[NH * NH / 8 / kMmaThreads];
#pragma unroll
        for (int k = 0; k < NH * NH / 8 / kMmaThreads; ++k)
            q[k] = reinterpret_cast<const uint4 *>(pb + OFF_W2)[k * kMmaThreads + threadIdx.x];
#pragma unroll
        for (int k = 0; k < NH * NH / 8 / kMmaThreads; ++k) {
            const int e = 8 * (k * kMmaThreads + threadIdx.x);
            *reinterpret_cast<uint4 *>(w2s + e / NH * kW2Row + e % NH) = q[k];
        }
    } else {
#pragma unroll 8
        for (int e = threadIdx.x; e < NH * NH; e += kMmaThreads) w2s[e / NH * kW2Row + e % NH] = pb[OFF_W2 + e];
    }
#pragma unroll
    for (int e = threadIdx.x; e < NH * NI; e += kMmaThreads) w1[(e / NI) >> 1][e % NI][(e / NI) & 1] = __bfloat162float(pb[e]);
    if (threadIdx.x < NH) {
        const int u = threadIdx.x;
        w1[u >> 1][NI][u & 1] = __bfloat162float(pb[OFF_B1 + u]);
        b2s[u] = __bfloat162float(pb[OFF_B2 + u]);
        w3s[u] = __bfloat162float(pb[OFF_W3 + u]);
        if (u == 0) b3s = __bfloat162float(pb[OFF_B3]);
    }
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const int g = lane >> 2, tig = lane & 3;
    const unsigned *w2 = reinterpret_cast<const unsigned *>(w2s) + g * (kW2Row / 2) + tig;  // BF16 pairs, input fastest
    const long long ntile = (n + 15) / 16;
    const long long warps = (long long)gridDim.x * (blockDim.x >> 5);
    for (long long tile = blockIdx.x * (long long)(blockDim.x >> 5) + (threadIdx.x >> 5); tile < ntile;
         tile += warps) {
        const long long s0 = tile * 16 + g, s1 = s0 + 8;
        f32x2 xb[2][NI];  // rows g and g + 8, each input in both halves
#pragma unroll
        for (int k = 0; k < NI; ++k) {
            const float a = s0 < n ? x[s0 * NI + k] : 0.f, b = s1 < n ? x[s1 * NI + k] : 0.f;
            xb[0][k] = pack2(a, a);
            xb[1][k] = pack2(b, b);
        }
        float acc[8][4];
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
            const float2 b = *reinterpret_cast<const float2 *>(b2s + 8 * nt + 2 * tig);
            acc[nt][0] = acc[nt][2] = b.x;
            acc[nt][1] = acc[nt][3] = b.y;
        }
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {
            // this lane's first-layer units 16 ks + 2 tig + {0, 1} and 8 further;
            // A registers: row g k lo, row g + 8 k lo, row g k hi, row g + 8 k hi
            unsigned A[3][4];
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const float4 *wp = reinterpret_cast<const float4 *>(&w1[8 * ks + 4 * q + tig][0][0]);
                const float4 wa = wp[0], wb = wp[1], wc = wp[2];
                const f32x2 w[NI] = {pack2(wa.x, wa.y), pack2(wa.z, wa.w), pack2(wb.x, wb.y), pack2(wb.z, wb.w),
                                     pack2(wc.x, wc.y)};
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    f32x2 a = pack2(wc.z, wc.w);
#pragma unroll
                    for (int k = 0; k < NI; ++k) a = fma2(w[k], xb[r][k], a);
                    f32x2 h = tanh2(a);
                    // three BF16 terms of the pair
#pragma unroll
                    for (int t = 0; t < 3; ++t) {
                        const float2 v = unpack2(h);
                        const unsigned u = pack_bf16(v.x, v.y);
                        A[t][r + 2 * q] = u;
                        if (t < 2)
                            h = fma2(pack2(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u)),
                                     pack2(-1.f, -1.f), h);
                    }
                }
            }
#pragma unroll
            for (int nt = 0; nt < 8; ++nt) {
                // B column = output unit 8 nt + g
                const unsigned b0 = w2[8 * nt * (kW2Row / 2) + 8 * ks], b1 = w2[8 * nt * (kW2Row / 2) + 8 * ks + 4];
                mma_bf16_16816(acc[nt], A[2], b0, b1);
                mma_bf16_16816(acc[nt], A[1], b0, b1);
                mma_bf16_16816(acc[nt], A[0], b0, b1);
            }
        }
        f32x2 p0 = pack2(0.f, 0.f), p1 = p0;
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
            const float2 w = *reinterpret_cast<const float2 *>(w3s + 8 * nt + 2 * tig);
            p0 = fma2(pack2(w.x, w.y), tanh2(pack2(acc[nt][0], acc[nt][1])), p0);
            p1 = fma2(pack2(w.x, w.y), tanh2(pack2(acc[nt][2], acc[nt][3])), p1);
        }
        float o0 = unpack2(p0).x + unpack2(p0).y, o1 = unpack2(p1).x + unpack2(p1).y;
        o0 += __shfl_xor_sync(0xffffffffu, o0, 1);
        o0 += __shfl_xor_sync(0xffffffffu, o0, 2);
        o1 += __shfl_xor_sync(0xffffffffu, o1, 1);
        o1 += __shfl_xor_sync(0xffffffffu, o1, 2);
        if (tig == 0) {
            float out0 = __fadd_rn(o0, b3s), out1 = __fadd_rn(o1, b3s);
            if (residual) {  // the network predicts log-DCF + log density (radius 2)
                out0 = __fsub_rn(out0, unpack2(xb[0][1]).x);
                out1 = __fsub_rn(out1, unpack2(xb[1][1]).x);
            }
            if (s0 < n) y[s0] = exp_out ? __fmul_rn(scale, expf(out0)) : out0;
            if (s1 < n) y[s1] = exp_out ? __fmul_rn(scale, expf(out1)) : out1;
        }
    }
}

// Forward and reverse pass of the (optionally weighted) mean squared error
// (1/n) sum_s c_s (y_s - t_s)^2 and its gradient, tiles of 64 samples: the
// three 64 x 64 x 64 products of a tile (W2 h1, W2^T d2, d2 h1^T) from shared
// memory, a 4 x 4 block per thread, in FP32; the gradient stays in registers
// from tile to tile and leaves as one partial per CTA.  Activations and deltas
// are held unit-major ([unit][sample], rows of kRow floats, so that 8 lanes on
// 8 rows cover the banks).
// Bound: FP32 issue (0.8 M FMA and 8192 tanh a tile), then the latency of one
// tile.  16,384 samples: 92 us for the gradient kernel (64 CTAs, activations
// and deltas through memory) and 29 us for the pass before it, 31 us so; the
// whole step with Adam 124 -> 37 us.
constexpr int kTile = 64;              // samples per tile
constexpr int kRow = kTile + 4;        // floats per shared row
constexpr int kStepThreads = 256;      // 16 x 16 blocks of 4 x 4
constexpr int kStepSmem = (4 * NH * kRow + kTile * NI + 2 * kTile + NH * NI + 3 * NH + 4) * 4;
static_assert(NH == 64 && kTile == 64, "16 x 16 threads of 4 x 4 outputs");

__device__ __forceinline__ void outer4(float (&c)[4][4], const float4 a, const float4 b)
{
    const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) c[i][j] = fmaf(av[i], bv[j], c[i][j]);
}

__global__ void __launch_bounds__(kStepThreads, 2) mlp_step_kernel(const __nv_bfloat16 *__restrict__ pb,
                                                                   const float *__restrict__ x,
                                                                   const float *__restrict__ t,
                                                                   const float *__restrict__ cw, long long n,
                                                                   float *__restrict__ partials,
                                                                   float *__restrict__ loss_part)
{
    extern __shared__ float4 sm4[];
    float *w2 = reinterpret_cast<float *>(sm4);  // [j][i]
    float *w2t = w2 + NH * kRow;                 // [i][j]
    float *h1 = w2t + NH * kRow;                 // [i][s]
    float *d2 = h1 + NH * kRow;                  // [j][s]
    float *xs = d2 + NH * kRow;                  // [s][NI]
    float *ts = xs + kTile * NI;                 // targets
    float *cs = ts + kTile;                      // sample weights (0 past the batch)
    float *w1 = cs + kTile;                      // [i][NI]
    float *b1 = w1 + NH * NI, *b2 = b1 + NH, *w3 = b2 + NH, *b3 = w3 + NH;
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    for (int p = tid; p < NP; p += kStepThreads) {
        const float v = __bfloat162float(pb[p]);
        if (p < OFF_B1) w1[p] = v;
        else if (p < OFF_W2) b1[p - OFF_B1] = v;
        else if (p < OFF_B2) {
            const int j = (p - OFF_W2) / NH, i = (p - OFF_W2) % NH;
            w2[j * kRow + i] = v;
            w2t[i * kRow + j] = v;
        } else if (p < OFF_W3) b2[p - OFF_B2] = v;
        else if (p < OFF_B3) w3[p - OFF_W3] = v;
        else b3[0] = v;
    }
    const float inv_n = 1.f / (float)n;
    // gradients of this thread: W2[ty + 16 a][tx + 16 b]; W1 and b1 of units
    // 4 tx + k, W3 and b2 of units 4 tx + k (over its samples), b3, loss
    float g2[4][4] = {}, g1[4][NI] = {}, gb1[4] = {}, gw3[4] = {}, gb2[4] = {}, gb3 = 0.f, lsum = 0.f;
    const long long ntile = (n + kTile - 1) / kTile;
    for (long long tile = blockIdx.x; tile < ntile; tile += gridDim.x) {
        const long long s0 = tile * kTile;
        __syncthreads();  // tables staged; the last tile's rows no longer read
        for (int e = tid; e < kTile * NI; e += kStepThreads) xs[e] = s0 * NI + e < n * NI ? x[s0 * NI + e] : 0.f;
        if (tid < kTile) {
            const bool in = s0 + tid < n;
            ts[tid] = in ? t[s0 + tid] : 0.f;
            cs[tid] = in ? (cw ? cw[s0 + tid] : 1.f) : 0.f;
        }
        __syncthreads();
        {  // first layer: sample tid % 64, units 16 (tid / 64) + k
            const int s = tid & 63, i0 = (tid >> 6) * 16;
            float xv[NI];
#pragma unroll
            for (int k = 0; k < NI; ++k) xv[k] = xs[s * NI + k];
#pragma unroll 4
            for (int i = i0; i < i0 + 16; ++i) {
                float a = b1[i];
#pragma unroll
                for (int k = 0; k < NI; ++k) a = fmaf(w1[i * NI + k], xv[k], a);
                h1[i * kRow + s] = tanhf(a);
            }
        }
        __syncthreads();
        {  // second layer and output: samples 4 ty + i, units 4 tx + j
            float a[4][4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) a[i][j] = b2[4 * tx + j];
#pragma unroll 8
            for (int k = 0; k < NH; ++k)
                outer4(a, *reinterpret_cast<const float4 *>(h1 + k * kRow + 4 * ty),
                       *reinterpret_cast<const float4 *>(w2t + k * kRow + 4 * tx));
            const float4 wv = *reinterpret_cast<const float4 *>(w3 + 4 * tx);
            const float w[4] = {wv.x, wv.y, wv.z, wv.w};
            float dy[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float o = 0.f;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    a[i][j] = tanhf(a[i][j]);
                    o = fmaf(w[j], a[i][j], o);
                }
#pragma unroll
                for (int d = 1; d < 16; d <<= 1) o += __shfl_xor_sync(0xffffffffu, o, d);
                const float r = (o + b3[0]) - ts[4 * ty + i], c = cs[4 * ty + i];
                dy[i] = 2.f * c * r * inv_n;
                if (tx == 0) {
                    lsum = fmaf(c * r, r, lsum);
                    gb3 += dy[i];
                }
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                float v[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    gw3[j] = fmaf(dy[i], a[i][j], gw3[j]);
                    v[i] = dy[i] * w[j] * (1.f - a[i][j] * a[i][j]);
                    gb2[j] += v[i];
                }
                *reinterpret_cast<float4 *>(d2 + (4 * tx + j) * kRow + 4 * ty) = make_float4(v[0], v[1], v[2], v[3]);
            }
        }
        __syncthreads();
        {  // first layer's deltas: samples 4 ty + i, units 4 tx + j
            float a[4][4] = {};
#pragma unroll 8
            for (int k = 0; k < NH; ++k)
                outer4(a, *reinterpret_cast<const float4 *>(d2 + k * kRow + 4 * ty),
                       *reinterpret_cast<const float4 *>(w2 + k * kRow + 4 * tx));
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float4 hv = *reinterpret_cast<const float4 *>(h1 + (4 * tx + j) * kRow + 4 * ty);
                const float h[4] = {hv.x, hv.y, hv.z, hv.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float d = a[i][j] * (1.f - h[i] * h[i]);
                    gb1[j] += d;
#pragma unroll
                    for (int k = 0; k < NI; ++k) g1[j][k] = fmaf(d, xs[(4 * ty + i) * NI + k], g1[j][k]);
                }
            }
        }
        // W2's gradient: rows ty + 16 a of d2, rows tx + 16 b of h1
#pragma unroll 4
        for (int s = 0; s < kTile; s += 4) {
            float4 dv[4], hv[4];
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                dv[a] = *reinterpret_cast<const float4 *>(d2 + (ty + 16 * a) * kRow + s);
                hv[a] = *reinterpret_cast<const float4 *>(h1 + (tx + 16 * a) * kRow + s);
            }
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    g2[a][b] = fmaf(dv[a].x, hv[b].x, g2[a][b]);
                    g2[a][b] = fmaf(dv[a].y, hv[b].y, g2[a][b]);
                    g2[a][b] = fmaf(dv[a].z, hv[b].z, g2[a][b]);
                    g2[a][b] = fmaf(dv[a].w, hv[b].w, g2[a][b]);
                }
        }
    }
    float *out = partials + (size_t)blockIdx.x * NP;
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) out[OFF_W2 + (ty + 16 * a) * NH + tx + 16 * b] = g2[a][b];
    // the rest over the 16 ty: the warp's two by a shuffle, the 8 warps in
    // shared memory ([warp][unit][W1 row, b1, W3, b2], then b3 and loss)
    constexpr int NV = NI + 3;
    __syncthreads();
    float *red = w2;
    float *rows = red + 8 * NH * NV;
    const int warp = tid >> 5;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        float v[NV];
#pragma unroll
        for (int k = 0; k < NI; ++k) v[k] = g1[j][k];
        v[NI] = gb1[j];
        v[NI + 1] = gw3[j];
        v[NI + 2] = gb2[j];
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            v[k] += __shfl_xor_sync(0xffffffffu, v[k], 16);
            if ((tid & 16) == 0) red[(warp * NH + 4 * tx + j) * NV + k] = v[k];
        }
    }
    gb3 += __shfl_xor_sync(0xffffffffu, gb3, 16);
    lsum += __shfl_xor_sync(0xffffffffu, lsum, 16);
    if ((tid & 31) == 0) {
        rows[2 * warp] = gb3;
        rows[2 * warp + 1] = lsum;
    }
    __syncthreads();
    for (int e = tid; e < NH * NV; e += kStepThreads) {
        const int u = e / NV, k = e % NV;
        float v = 0.f;
#pragma unroll
        for (int q = 0; q < 8; ++q) v += red[(q * NH + u) * NV + k];
        out[k < NI ? OFF_W1 + u * NI + k : k == NI ? OFF_B1 + u : k == NI + 1 ? OFF_W3 + u : OFF_B2 + u] = v;
    }
    if (tid < 2) {
        float v = 0.f;
        for (int q = 0; q < 8; ++q) v += rows[2 * q + tid];
        if (tid == 0) out[OFF_B3] = v;
        else loss_part[blockIdx.x] = v;
    }
}

// Sum of the CTAs' partial gradients, 32 parameters per CTA: thread (slice,
// parameter) sums every 8th partial, then the 8 slices in order.  The last CTA
// sums the loss.  (One thread per
// parameter over 64 partials: 8 us; 256 partials so: 7 us.)
__global__ void __launch_bounds__(256) mlp_reduce_kernel(const float *__restrict__ partials, int nparts,
                                                         const float *__restrict__ loss_part, float inv_n, float *grad,
                                                         float *loss)
{
    __shared__ float part[8][33];
    const int lane = threadIdx.x & 31, slice = threadIdx.x >> 5;
    const bool is_loss = blockIdx.x == gridDim.x - 1;
    const int p = blockIdx.x * 32 + lane;
    float a = 0.f;
    if (is_loss) {
        for (int b = slice * 32 + lane; b < nparts; b += 256) a += loss_part[b];
    } else if (p < NP) {
#pragma unroll 4
        for (int b = slice; b < nparts; b += 8) a += partials[(size_t)b * NP + p];
    }
    part[slice][lane] = a;
    __syncthreads();
    if (slice == 0) {
        float v = 0.f;
#pragma unroll
        for (int q = 0; q < 8; ++q) v += part[q][lane];
        if (is_loss) {
#pragma unroll
            for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
            if (lane == 0 && loss) *loss = v * inv_n;
        } else if (p < NP) {
            grad[p] = v;
        }
    }
}

__global__ void mlp_adam_kernel(float *master, __nv_bfloat16 *pb, const float *__restrict__ g, float *m, float *v,
                                int count, float lr, float b1, float b2, float eps, float c1, float c2)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float w = master[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    master[i] = w;
    pb[i] = __float2bfloat16_rn(w);
}

__global__ void to_bf16_kernel(const float *__restrict__ a, __nv_bfloat16 *b, int count)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < count) b[i] = __float2bfloat16_rn(a[i]);
}

int sm_count_mlp()
{
    int dev = 0, n = 132;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return n;
}

// FR_MLP_SIMT=1: the forward pass on the FP32 CUDA cores (A/B measurements).
bool mlp_use_simt()
{
    const char *e = std::getenv("FR_MLP_SIMT");
    return e && std::atoi(e) != 0;
}

// CTAs of the training step: one per tile up to two per SM.
int step_blocks(size_t n)
{
    return (int)std::min<long long>((long long)((n + kTile - 1) / kTile), 2ll * sm_count_mlp());
}

}  // namespace

size_t mlp_workspace_bytes(size_t n)
{
    // a partial gradient and loss per CTA
    return (size_t)step_blocks(std::max<size_t>(n, 1)) * (NP + 1) * 4 + 256;
}

int mlp_forward_run(const void *d_params, const float *d_x, size_t n, int exp_out, int residual, float scale,
                    float *d_y, cudaStream_t s)
{
    if (n == 0) return FR_OK;
    const int blocks = (int)std::max<long long>(1, std::min<long long>(((long long)n + kFwdThreads - 1) / kFwdThreads,
                                                                       (long long)sm_count_mlp() * 16));
    if (mlp_use_simt()) {
        mlp_forward_kernel<<<blocks, kFwdThreads, 0, s>>>(static_cast<const __nv_bfloat16 *>(d_params), d_x,
                                                          (long long)n, exp_out, residual, scale, d_y);
        FR_CHECK_LAUNCH("mlp_forward_kernel");
        return FR_OK;
    }
    const long long tiles = ((long long)n + 15) / 16;
    const int mblocks = (int)std::max<long long>(
        1, std::min<long long>((tiles + kMmaThreads / 32 - 1) / (kMmaThreads / 32), (long long)sm_count_mlp() * 4));
    mlp_forward_mma_kernel<<<mblocks, kMmaThreads, 0, s>>>(static_cast<const __nv_bfloat16 *>(d_params), d_x,
                                                          (long long)n, exp_out, residual, scale, d_y);
    FR_CHECK_LAUNCH("mlp_forward_mma_kernel");
    return FR_OK;
}

int mlp_backward_run(const void *d_params, const float *d_x, const float *d_t, const float *d_w, size_t n, void *ws,
                     float *d_grad, float *d_loss, cudaStream_t s)
{
    if (n == 0) return fail(FR_ERR_INVALID_ARGUMENT, "empty batch");
    const int nb = step_blocks(n);
    float *partials = static_cast<float *>(ws);
    float *loss_part = partials + (size_t)nb * NP;
    FR_CUDA(cudaFuncSetAttribute(mlp_step_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kStepSmem));
    mlp_step_kernel<<<nb, kStepThreads, kStepSmem, s>>>(static_cast<const __nv_bfloat16 *>(d_params), d_x, d_t, d_w,
                                                        (long long)n, partials, loss_part);
    FR_CHECK_LAUNCH("mlp_step_kernel");
    mlp_reduce_kernel<<<(NP + 31) / 32 + 1, 256, 0, s>>>(partials, nb, loss_part, 1.f / (float)n, d_grad, d_loss);
    FR_CHECK_LAUNCH("mlp_reduce_kernel");
    return FR_OK;
}

int mlp_adam_run(float *d_master, void *d_params, const float *d_grad, float *d_m, float *d_v, int count, float lr,
                 float beta1, float beta2, float eps, int step, cudaStream_t s)
{
    if (count <= 0 || step < 1) return fail(FR_ERR_INVALID_ARGUMENT, "count > 0 and step >= 1");
    const float c1 = 1.f - powf(beta1, (float)step), c2 = 1.f - powf(beta2, (float)step);
    mlp_adam_kernel<<<(count + 255) / 256, 256, 0, s>>>(d_master, static_cast<__nv_bfloat16 *>(d_params), d_grad, d_m,
                                                        d_v, count, lr, beta1, beta2, eps, c1, c2);
    FR_CHECK_LAUNCH("mlp_adam_kernel");
    return FR_OK;
}

int to_bf16_run(const float *d_a, void *d_b, int count, cudaStream_t s)
{
    if (count <= 0) return FR_OK;
    to_bf16_kernel<<<(count + 255) / 256, 256, 0, s>>>(d_a, static_cast<__nv_bfloat16 *>(d_b), count);
    FR_CHECK_LAUNCH("to_bf16_kernel");
    return FR_OK;
}

}  // namespace fr
