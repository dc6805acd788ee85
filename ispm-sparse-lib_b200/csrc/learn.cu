// Learned drop tolerances for the approximate inverse: per-row features and
// a small MLP (32 -> 64 -> 64 -> 2) trained and run on the GPU.
//
// The reference picks one global drop tolerance for fastainv_sym by a
// golden-section search that costs a full build and solve per probe
// (fastainv/droptol-tuning.h:4-103).  Here a per-row network predicts, from
// local matrix features, the drop tolerance of each row of the factor and a
// diagonal rescale of that row (applied through fastainv_sym_ex); the
// caller keeps the plain build as the fallback and the yardstick.
//
// Network: y = W3 relu(W2 relu(W1 x + b1) + b2) + b3 with BF16 weights and
// inputs and FP32 accumulation.  Layers 1 and 2 (and the weight gradients of
// both) run on the tensor cores with mma.sync m16n8k16 (BF16 in, FP32
// accumulate): at 12.5 kflop per 64-byte feature row the network is
// bandwidth-bound, far below the point where tcgen05's larger tiles would
// pay.  Layer 3 (two outputs) runs on the FP32 cores.  Rounding points, which
// the CPU oracle reproduces: x, W1, W2, W3 and the layer-1 activations are
// BF16; the layer-2 activations stay FP32 for layer 3; in the backward pass
// the layer-2 and layer-1 activation gradients are rounded to BF16 where they
// feed a tensor-core product (dH1 = dH2 W2, dW2 = dH2^T H1, dW1 = dH1^T X)
// and kept FP32 for the bias gradients and dW3.
//
// Training is deterministic: each CTA accumulates its rows' gradients in a
// fixed order and writes one partial per CTA; a second kernel adds the
// partials in a fixed order; Adam runs on FP32 master weights.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstddef>
#include <cstdint>
#include <cstring>
#include <memory>
#include <mutex>
#include <vector>

#include "cuda_util.cuh"

namespace ispm {
namespace {

constexpr int kIn = 32, kH = 64, kOut = 2;
constexpr int kW1 = 0, kB1 = kW1 + kH * kIn, kW2 = kB1 + kH, kB2 = kW2 + kH * kH,
              kW3 = kB2 + kH, kB3 = kW3 + kOut * kH, kParams = kB3 + kOut;
constexpr int kPart = kParams + 1;  // + loss
static_assert(kW2 % 4 == 0, "the weight matrices are read in 16-byte words");
constexpr int kFwdCtas = 5;         // forward CTAs an SM holds (96 registers a thread)
constexpr int kFwdThreads = 128;    // forward: 4 warps, 32 rows a warp and step
constexpr int kWarps = 8, kThreads = 32 * kWarps;
constexpr int kBlockRows = 128;     // training: rows per CTA step, 16 per warp
constexpr int kLd1 = kIn + 8;       // padded row lengths: the eight 16-byte rows of
constexpr int kLd2 = kH + 8;        // an ldmatrix land on distinct banks
constexpr int kSums = 8;            // per lane: halves of db2, dW3[0], dW3[1], db1

using bf16 = __nv_bfloat16;

struct Weights {
  bf16 w1[kH * kLd1];
  bf16 w2[kH * kLd2];
  float b1[kH], b2[kH], w3[kOut * kH], b3[kOut + 2];
};

struct TrainSmem {
  Weights w;
  bf16 x[2][kBlockRows * kLd1];  // this step's rows and the next one's
  bf16 h1[kBlockRows * kLd2];
  bf16 d2[kBlockRows * kLd2];
  bf16 d1[kBlockRows * kLd2];
};

__device__ __forceinline__ uint32_t pack2(float lo, float hi)
{
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t *>(&v);
}

__device__ __forceinline__ float lo_f(uint32_t v)
{
  return __uint_as_float(v << 16);
}

__device__ __forceinline__ float hi_f(uint32_t v) { return __uint_as_float(v & 0xffff0000u); }

__device__ __forceinline__ void st32(bf16 *p, uint32_t v)
{
  *reinterpret_cast<uint32_t *>(p) = v;
}

__device__ __forceinline__ uint32_t smem_addr(const void *p)
{
  return (uint32_t)__cvta_generic_to_shared(p);
}

// Four 8x8 BF16 blocks, one row address per lane (lanes 8q .. 8q+7: block q).
__device__ __forceinline__ void ldm4(uint32_t (&r)[4], const bf16 *p)
{
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(smem_addr(p)));
}

__device__ __forceinline__ void ldm4t(uint32_t (&r)[4], const bf16 *p)
{
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(smem_addr(p)));
}

// D += A B, m16n8k16, BF16 inputs, FP32 accumulators.
__device__ __forceinline__ void mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0,
                                    uint32_t b1)
{
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
      "{%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint2 pack4(const float4 &v)
{
  return make_uint2(pack2(v.x, v.y), pack2(v.z, v.w));
}

// Weights into shared memory (BF16-rounded), 16 bytes of the master copy a load.
__device__ void load_weights(Weights &s, const float *__restrict__ prm)
{
  const float4 *w1 = reinterpret_cast<const float4 *>(prm + kW1);
  const float4 *w2 = reinterpret_cast<const float4 *>(prm + kW2);
#pragma unroll 4
  for (int i = threadIdx.x; i < kH * kIn / 4; i += blockDim.x)
    *reinterpret_cast<uint2 *>(s.w1 + (i / (kIn / 4)) * kLd1 + i % (kIn / 4) * 4) =
        pack4(__ldg(w1 + i));
#pragma unroll 4
  for (int i = threadIdx.x; i < kH * kH / 4; i += blockDim.x)
    *reinterpret_cast<uint2 *>(s.w2 + (i / (kH / 4)) * kLd2 + i % (kH / 4) * 4) =
        pack4(__ldg(w2 + i));
  for (int i = threadIdx.x; i < kH; i += blockDim.x) {
    s.b1[i] = __ldg(prm + kB1 + i);
    s.b2[i] = __ldg(prm + kB2 + i);
  }
  for (int i = threadIdx.x; i < kOut * kH; i += blockDim.x)
    s.w3[i] = __bfloat162float(__float2bfloat16_rn(__ldg(prm + kW3 + i)));
  if (threadIdx.x < kOut)
    s.b3[threadIdx.x] = __ldg(prm + kB3 + threadIdx.x);
}

// Sum over the 8 lanes sharing threadID_in_group (lane bits 2..4).
__device__ __forceinline__ float sum_g(float v)
{
  v += __shfl_xor_sync(0xffffffffu, v, 4);
  v += __shfl_xor_sync(0xffffffffu, v, 8);
  v += __shfl_xor_sync(0xffffffffu, v, 16);
  return v;
}

// Eight such sums at once: lane g (its bits 2..4) returns the sum of v[g].
// Halving the set at each step takes 7 shuffles where sum_g takes 24.
__device__ __forceinline__ float sum8_g(const float (&v)[8])
{
  const int lane = threadIdx.x & 31;
  float a[4], b[2];
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const bool hi = lane & 16;
    a[k] = (hi ? v[k + 4] : v[k]) + __shfl_xor_sync(0xffffffffu, hi ? v[k] : v[k + 4], 16);
  }
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const bool hi = lane & 8;
    b[k] = (hi ? a[k + 2] : a[k]) + __shfl_xor_sync(0xffffffffu, hi ? a[k] : a[k + 2], 8);
  }
  const bool hi = lane & 4;
  return (hi ? b[1] : b[0]) + __shfl_xor_sync(0xffffffffu, hi ? b[0] : b[1], 4);
}

// Forward pass, 32 rows (two 16-row tiles) a warp and step, so every weight
// fragment read from shared memory serves two products; the layer-2
// activations go into the two outputs as they come and are never kept.
// Bound by the issue of mma.sync and the fragment reads (512,000 rows: 31 us,
// 39 us with one tile a step and 32-bit fragment loads; its 72 bytes a row
// would take 6 us).  The next step's rows are loaded a step ahead.
__global__ void __launch_bounds__(kFwdThreads, kFwdCtas)
    mlp_forward_kernel(const float *__restrict__ prm, const bf16 *__restrict__ X,
                       float2 *__restrict__ Y, long long M)
{
  __shared__ __align__(16) Weights s;
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, w = threadIdx.x >> 5;
  const long long step = (long long)gridDim.x * (kFwdThreads / 32) * 32;
  uint32_t xn[2][2][4];  // the next step's rows: [tile][k-step]
  auto load_rows = [&](long long r0) {
#pragma unroll
    for (int m = 0; m < 2; m++)
#pragma unroll
      for (int q = 0; q < 2; q++) {
        const long long r = r0 + 16 * m + 8 * q + g;
        const unsigned *px = reinterpret_cast<const unsigned *>(X + r * kIn) + t;
#pragma unroll
        for (int kk = 0; kk < 2; kk++) {
          xn[m][kk][q] = r < M ? __ldg(px + kk * 8) : 0u;
          xn[m][kk][q + 2] = r < M ? __ldg(px + kk * 8 + 4) : 0u;
        }
      }
  };
  const long long first = ((long long)blockIdx.x * (kFwdThreads / 32) + w) * 32;
  pdl_wait();
  load_rows(first);
  load_weights(s, prm);
  __syncthreads();
  // B fragments of a weight matrix stored [out][in]: rows 8j .. 8j+7, 32 columns
  const bf16 *w1p = s.w1 + (lane & 7) * kLd1 + (lane >> 3) * 8;
  const bf16 *w2p = s.w2 + (lane & 7) * kLd2 + (lane >> 3) * 8;
  for (long long r0 = first; r0 < M; r0 += step) {
    uint32_t xa[2][2][4];
#pragma unroll
    for (int m = 0; m < 2; m++)
#pragma unroll
      for (int kk = 0; kk < 2; kk++)
#pragma unroll
        for (int e = 0; e < 4; e++)
          xa[m][kk][e] = xn[m][kk][e];
    load_rows(r0 + step);
    // layer 1 -> relu -> BF16 A fragments of layer 2
    uint32_t ha[2][4][4];
#pragma unroll
    for (int j = 0; j < 8; j++) {
      uint32_t bw[4];
      ldm4(bw, w1p + 8 * j * kLd1);
      const float2 bias = *reinterpret_cast<const float2 *>(s.b1 + 8 * j + 2 * t);
#pragma unroll
      for (int m = 0; m < 2; m++) {
        float h[4] = {bias.x, bias.y, bias.x, bias.y};
        mma(h, xa[m][0], bw[0], bw[1]);
        mma(h, xa[m][1], bw[2], bw[3]);
        ha[m][j >> 1][(j & 1) * 2 + 0] = pack2(fmaxf(h[0], 0.f), fmaxf(h[1], 0.f));
        ha[m][j >> 1][(j & 1) * 2 + 1] = pack2(fmaxf(h[2], 0.f), fmaxf(h[3], 0.f));
      }
    }
    // layer 2, its activations straight into layer 3 on the FP32 cores
    float y[2][2][kOut];  // [tile][row half][output]
#pragma unroll
    for (int m = 0; m < 2; m++)
#pragma unroll
      for (int q = 0; q < 2; q++)
        y[m][q][0] = y[m][q][1] = 0.f;
#pragma unroll
    for (int j = 0; j < 8; j++) {
      uint32_t b0[4], b1[4];
      ldm4(b0, w2p + 8 * j * kLd2);
      ldm4(b1, w2p + 8 * j * kLd2 + 32);
      const int c = 8 * j + 2 * t;
      const float2 bias = *reinterpret_cast<const float2 *>(s.b2 + c);
      const float2 wa = *reinterpret_cast<const float2 *>(s.w3 + c);
      const float2 wb = *reinterpret_cast<const float2 *>(s.w3 + kH + c);
#pragma unroll
      for (int m = 0; m < 2; m++) {
        float h[4] = {bias.x, bias.y, bias.x, bias.y};
        mma(h, ha[m][0], b0[0], b0[1]);
        mma(h, ha[m][1], b0[2], b0[3]);
        mma(h, ha[m][2], b1[0], b1[1]);
        mma(h, ha[m][3], b1[2], b1[3]);
#pragma unroll
        for (int q = 0; q < 2; q++) {
          const float r0v = fmaxf(h[2 * q], 0.f), r1v = fmaxf(h[2 * q + 1], 0.f);
          y[m][q][0] = fmaf(r1v, wa.y, fmaf(r0v, wa.x, y[m][q][0]));
          y[m][q][1] = fmaf(r1v, wb.y, fmaf(r0v, wb.x, y[m][q][1]));
        }
      }
    }
#pragma unroll
    for (int m = 0; m < 2; m++)
#pragma unroll
      for (int q = 0; q < 2; q++) {
#pragma unroll
        for (int o = 0; o < kOut; o++) {
          float v = y[m][q][o];
          v += __shfl_xor_sync(0xffffffffu, v, 1);
          v += __shfl_xor_sync(0xffffffffu, v, 2);
          y[m][q][o] = v + s.b3[o];
        }
        const long long r = r0 + 16 * m + 8 * q + g;
        if (t == 0 && r < M)
          Y[r] = make_float2(y[m][q][0], y[m][q][1]);
      }
  }
  pdl_trigger();
}

// One warp's 16 rows of a training step: forward, loss, backward up to the
// activation gradients, which it leaves (BF16, row-major) beside h1 for the
// weight gradients.  Rows >= M contribute nothing.
__device__ __forceinline__ void train_tile(TrainSmem &s, const bf16 *x, const float2 *__restrict__ T,
                                           const float2 *__restrict__ Wt, long long r0, long long M,
                                           float scale, int lr0, float (&sums)[kSums],
                                           float (&tail)[3])
{
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const Weights &w = s.w;
  const long long ra = r0 + g, rb = r0 + g + 8;
  const bool va = ra < M, vb = rb < M;
  // targets and weights early: their latency hides behind the products
  float2 ta = make_float2(0.f, 0.f), tb = ta, wa = make_float2(1.f, 1.f), wb = wa;
  if (va) {
    ta = __ldg(T + ra);
    if (Wt)
      wa = __ldg(Wt + ra);
  }
  if (vb) {
    tb = __ldg(T + rb);
    if (Wt)
      wb = __ldg(Wt + rb);
  }
  // X fragments (K = 32: two k-steps)
  uint32_t xa[2][4];
  const bf16 *xp = x + (lr0 + (lane & 15)) * kLd1 + (lane >> 4) * 8;
  ldm4(xa[0], xp);
  ldm4(xa[1], xp + 16);
  // layer 1 -> relu -> BF16 A fragments of layer 2
  uint32_t ha[4][4];
  const bf16 *w1p = w.w1 + (lane & 7) * kLd1 + (lane >> 3) * 8;
#pragma unroll
  for (int j = 0; j < 8; j++) {
    uint32_t bw[4];
    ldm4(bw, w1p + 8 * j * kLd1);
    const float2 bias = *reinterpret_cast<const float2 *>(w.b1 + 8 * j + 2 * t);
    float h[4] = {bias.x, bias.y, bias.x, bias.y};
    mma(h, xa[0], bw[0], bw[1]);
    mma(h, xa[1], bw[2], bw[3]);
    const uint32_t p01 = pack2(fmaxf(h[0], 0.f), fmaxf(h[1], 0.f));
    const uint32_t p23 = pack2(fmaxf(h[2], 0.f), fmaxf(h[3], 0.f));
    ha[j >> 1][(j & 1) * 2 + 0] = p01;
    ha[j >> 1][(j & 1) * 2 + 1] = p23;
    const int c = 8 * j + 2 * t;
    st32(s.h1 + (lr0 + g) * kLd2 + c, p01);
    st32(s.h1 + (lr0 + g + 8) * kLd2 + c, p23);
  }
  // layer 2 (pre-activations), then layer 3 on the FP32 cores
  float h2[8][4];
  const bf16 *w2p = w.w2 + (lane & 7) * kLd2 + (lane >> 3) * 8;
  float ya[kOut] = {0.f, 0.f}, yb[kOut] = {0.f, 0.f};
#pragma unroll
  for (int j = 0; j < 8; j++) {
    uint32_t b0[4], b1[4];
    ldm4(b0, w2p + 8 * j * kLd2);
    ldm4(b1, w2p + 8 * j * kLd2 + 32);
    const int c = 8 * j + 2 * t;
    const float2 bias = *reinterpret_cast<const float2 *>(w.b2 + c);
    h2[j][0] = bias.x, h2[j][1] = bias.y, h2[j][2] = bias.x, h2[j][3] = bias.y;
    mma(h2[j], ha[0], b0[0], b0[1]);
    mma(h2[j], ha[1], b0[2], b0[3]);
    mma(h2[j], ha[2], b1[0], b1[1]);
    mma(h2[j], ha[3], b1[2], b1[3]);
#pragma unroll
    for (int o = 0; o < kOut; o++) {
      const float2 wo = *reinterpret_cast<const float2 *>(w.w3 + o * kH + c);
      ya[o] = fmaf(fmaxf(h2[j][1], 0.f), wo.y, fmaf(fmaxf(h2[j][0], 0.f), wo.x, ya[o]));
      yb[o] = fmaf(fmaxf(h2[j][3], 0.f), wo.y, fmaf(fmaxf(h2[j][2], 0.f), wo.x, yb[o]));
    }
  }
#pragma unroll
  for (int o = 0; o < kOut; o++) {
    ya[o] += __shfl_xor_sync(0xffffffffu, ya[o], 1);
    ya[o] += __shfl_xor_sync(0xffffffffu, ya[o], 2);
    yb[o] += __shfl_xor_sync(0xffffffffu, yb[o], 1);
    yb[o] += __shfl_xor_sync(0xffffffffu, yb[o], 2);
    ya[o] += w.b3[o];
    yb[o] += w.b3[o];
  }
  // dL/dy for L = sum_rows sum_o w_o (y_o - t_o)^2 * scale
  float dya[kOut] = {0.f, 0.f}, dyb[kOut] = {0.f, 0.f}, loss = 0.f;
  if (va) {
    const float e0 = ya[0] - ta.x, e1 = ya[1] - ta.y;
    dya[0] = 2.f * scale * wa.x * e0;
    dya[1] = 2.f * scale * wa.y * e1;
    loss += scale * (wa.x * e0 * e0 + wa.y * e1 * e1);
  }
  if (vb) {
    const float e0 = yb[0] - tb.x, e1 = yb[1] - tb.y;
    dyb[0] = 2.f * scale * wb.x * e0;
    dyb[1] = 2.f * scale * wb.y * e1;
    loss += scale * (wb.x * e0 * e0 + wb.y * e1 * e1);
  }
  // every t-lane holds the same values; the lanes with t = 0 are summed
  tail[0] += dya[0] + dyb[0];
  tail[1] += dya[1] + dyb[1];
  tail[2] += loss;
  // dW3 = dy^T relu(h2); dH2 = (dy W3) * [h2 > 0]; db2
  uint32_t da[4][4];
#pragma unroll
  for (int hf = 0; hf < 2; hf++) {
    float s0[8], s1[8], sb[8];
#pragma unroll
    for (int jj = 0; jj < 4; jj++) {
      const int j = 4 * hf + jj, c = 8 * j + 2 * t;
      const float2 w30 = *reinterpret_cast<const float2 *>(w.w3 + c);
      const float2 w31 = *reinterpret_cast<const float2 *>(w.w3 + kH + c);
      float d[4];
#pragma unroll
      for (int e = 0; e < 4; e++) {
        const float dy0 = e < 2 ? dya[0] : dyb[0], dy1 = e < 2 ? dya[1] : dyb[1];
        d[e] = h2[j][e] > 0.f ? fmaf(dy0, e & 1 ? w30.y : w30.x, dy1 * (e & 1 ? w31.y : w31.x))
                              : 0.f;
      }
#pragma unroll
      for (int e2 = 0; e2 < 2; e2++) {
        const float r0v = fmaxf(h2[j][e2], 0.f), r1v = fmaxf(h2[j][e2 + 2], 0.f);
        s0[2 * jj + e2] = fmaf(dya[0], r0v, dyb[0] * r1v);
        s1[2 * jj + e2] = fmaf(dya[1], r0v, dyb[1] * r1v);
        sb[2 * jj + e2] = d[e2] + d[e2 + 2];
      }
      const uint32_t p01 = pack2(d[0], d[1]), p23 = pack2(d[2], d[3]);
      da[j >> 1][(j & 1) * 2 + 0] = p01;
      da[j >> 1][(j & 1) * 2 + 1] = p23;
      st32(s.d2 + (lr0 + g) * kLd2 + c, p01);
      st32(s.d2 + (lr0 + g + 8) * kLd2 + c, p23);
    }
    sums[hf] += sum8_g(sb);
    sums[2 + hf] += sum8_g(s0);
    sums[4 + hf] += sum8_g(s1);
  }
  // dH1 = (dH2 W2) * [h1 > 0]; db1 (W2 is stored [k][n] for this product:
  // transposed fragments)
  const bf16 *w2t = w.w2 + lane * kLd2;
#pragma unroll
  for (int hf = 0; hf < 2; hf++) {
    float sb[8];
#pragma unroll
    for (int jj = 0; jj < 4; jj++) {
      const int j = 4 * hf + jj, c = 8 * j + 2 * t;
      float d[4] = {0.f, 0.f, 0.f, 0.f};
      uint32_t b0[4], b1[4];
      ldm4t(b0, w2t + 8 * j);
      ldm4t(b1, w2t + 32 * kLd2 + 8 * j);
      mma(d, da[0], b0[0], b0[1]);
      mma(d, da[1], b0[2], b0[3]);
      mma(d, da[2], b1[0], b1[1]);
      mma(d, da[3], b1[2], b1[3]);
      // h1 of these positions: A fragment of layer-2 k-step j/2, half j&1
      const uint32_t hv01 = ha[j >> 1][(j & 1) * 2 + 0], hv23 = ha[j >> 1][(j & 1) * 2 + 1];
      if (!(lo_f(hv01) > 0.f)) d[0] = 0.f;
      if (!(hi_f(hv01) > 0.f)) d[1] = 0.f;
      if (!(lo_f(hv23) > 0.f)) d[2] = 0.f;
      if (!(hi_f(hv23) > 0.f)) d[3] = 0.f;
      sb[2 * jj] = d[0] + d[2];
      sb[2 * jj + 1] = d[1] + d[3];
      st32(s.d1 + (lr0 + g) * kLd2 + c, pack2(d[0], d[1]));
      st32(s.d1 + (lr0 + g + 8) * kLd2 + c, pack2(d[2], d[3]));
    }
    sums[6 + hf] += sum8_g(sb);
  }
}

// Rows r0 .. r0 + kBlockRows - 1 of X into shared memory (asynchronous; rows
// past M read as zero): 16 bytes a copy when X is 16-byte aligned, else 4.
__device__ __forceinline__ void stage_rows(bf16 *dst, const bf16 *__restrict__ X, long long r0,
                                           long long M, bool al16)
{
  if (al16) {
    for (int i = threadIdx.x; i < kBlockRows * (kIn / 8); i += kThreads) {
      const int r = i / (kIn / 8), c = i % (kIn / 8) * 8;
      const bool in = r0 + r < M;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(
                       smem_addr(dst + r * kLd1 + c)),
                   "l"(X + (in ? (r0 + r) * kIn + c : 0)), "r"(in ? 16 : 0));
    }
  } else {
    for (int i = threadIdx.x; i < kBlockRows * (kIn / 2); i += kThreads) {
      const int r = i / (kIn / 2), c = i % (kIn / 2) * 2;
      const bool in = r0 + r < M;
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(
                       smem_addr(dst + r * kLd1 + c)),
                   "l"(X + (in ? (r0 + r) * kIn + c : 0)), "r"(in ? 4 : 0));
    }
  }
  asm volatile("cp.async.commit_group;\n");
}

// Loss and gradient partials of one CTA (part[blockIdx.x][kPart]).
//
// Latency-bound at the training loop's minibatch (65,536 rows are 3.5 steps an
// SM): eight warps a CTA and two CTAs an SM, each warp one 16-row tile a step;
// the next step's rows arrive by asynchronous copy meanwhile.  Activations
// and their gradients are staged row-major with 32-bit stores and read back
// as transposed fragments (ldmatrix.trans), the bias and dW3 sums stay in
// registers (eight a lane) until the end.  65,536 rows: 24 us, 38 us with four
// warps of two tiles, 16-bit staging stores and a shuffle sum per column.
__global__ void __launch_bounds__(kThreads, 2)
    mlp_train_kernel(const float *__restrict__ prm, const bf16 *__restrict__ X,
                     const float2 *__restrict__ T, const float2 *__restrict__ Wt, long long M,
                     float scale, int al16, float *__restrict__ part)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  TrainSmem &s = *reinterpret_cast<TrainSmem *>(smem_raw);
  const long long first = (long long)blockIdx.x * kBlockRows;
  const long long step = (long long)gridDim.x * kBlockRows;
  pdl_wait();
  stage_rows(s.x[0], X, first, M, al16);
  load_weights(s.w, prm);
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, w = threadIdx.x >> 5;
  // weight gradients: warp w owns output rows 16 (w & 3) .. + 15 and, of
  // them, half w >> 2 of the columns
  const int m0 = 16 * (w & 3), nh = w >> 2;
  float acc2[4][4], acc1[2][4];
#pragma unroll
  for (int j = 0; j < 4; j++)
#pragma unroll
    for (int e = 0; e < 4; e++) {
      acc2[j][e] = 0.f;
      if (j < 2)
        acc1[j][e] = 0.f;
    }
  float sums[kSums] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, tail[3] = {0.f, 0.f, 0.f};
  int buf = 0;
  for (long long r0 = first; r0 < M; r0 += step, buf ^= 1) {
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();  // x[buf] has landed; the last step's reads are over
    if (r0 + step < M)
      stage_rows(s.x[buf ^ 1], X, r0 + step, M, al16);
    train_tile(s, s.x[buf], T, Wt, r0 + 16 * w, M, scale, 16 * w, sums, tail);
    __syncthreads();
    // dW2 += dH2^T H1, dW1 += dH1^T X
    const int ar = (lane & 7) + (lane >> 4) * 8, ac = m0 + ((lane >> 3) & 1) * 8;
    const int br = lane & 15, bc = (lane >> 4) * 8;
#pragma unroll
    for (int kk = 0; kk < kBlockRows / 16; kk++) {
      uint32_t a[4], b[4];
      ldm4t(a, s.d2 + (16 * kk + ar) * kLd2 + ac);
#pragma unroll
      for (int j = 0; j < 4; j += 2) {
        ldm4t(b, s.h1 + (16 * kk + br) * kLd2 + 32 * nh + 8 * j + bc);
        mma(acc2[j], a, b[0], b[1]);
        mma(acc2[j + 1], a, b[2], b[3]);
      }
      ldm4t(a, s.d1 + (16 * kk + ar) * kLd2 + ac);
      ldm4t(b, s.x[buf] + (16 * kk + br) * kLd1 + 16 * nh + bc);
      mma(acc1[0], a, b[0], b[1]);
      mma(acc1[1], a, b[2], b[3]);
    }
  }
  pdl_trigger();
  float *out = part + (size_t)blockIdx.x * kPart;
#pragma unroll
  for (int j = 0; j < 4; j++) {
    float *q = out + kW2 + (m0 + g) * kH + 32 * nh + 8 * j + 2 * t;
    q[0] = acc2[j][0], q[1] = acc2[j][1];
    q[8 * kH] = acc2[j][2], q[8 * kH + 1] = acc2[j][3];
  }
#pragma unroll
  for (int j = 0; j < 2; j++) {
    float *q = out + kW1 + (m0 + g) * kIn + 16 * nh + 8 * j + 2 * t;
    q[0] = acc1[j][0], q[1] = acc1[j][1];
    q[8 * kIn] = acc1[j][2], q[8 * kIn + 1] = acc1[j][3];
  }
  // the warps' sums in warp order
  __syncthreads();
  float *red = reinterpret_cast<float *>(s.h1);  // [kWarps][kSums * 32 + 3]
  constexpr int kRed = kSums * 32 + 3;
#pragma unroll
  for (int k = 0; k < kSums; k++)
    red[w * kRed + 32 * k + lane] = sums[k];
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const float v = sum_g(tail[k]);
    if (lane == 0)
      red[w * kRed + kSums * 32 + k] = v;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < kRed; i += kThreads) {
    float v = 0.f;
    for (int ww = 0; ww < kWarps; ww++)
      v += red[ww * kRed + i];
    int dst;
    if (i >= kSums * 32) {
      const int k = i - kSums * 32;
      dst = k < kOut ? kB3 + k : kParams;  // the loss last
    } else {
      // sum k of lane (g, t): column 8 (4 (k & 1) + g / 2) + 2 t + (g & 1)
      const int k = i >> 5, gg = (i >> 2) & 7, tt = i & 3;
      const int c = 8 * (4 * (k & 1) + (gg >> 1)) + 2 * tt + (gg & 1);
      dst = (k < 2 ? kB2 : k < 4 ? kW3 : k < 6 ? kW3 + kH : kB1) + c;
    }
    out[dst] = v;
  }
}

// grad[p] = sum over CTAs of part[cta][p].  32 parameters a CTA; warp w adds
// CTAs w, w + 8, ... in order (coalesced rows, eight loads in flight), then
// the eight sums are added in warp order: the same result every time.  One
// thread a parameter over all partials took 15.4 us for 296 of them.
constexpr int kReduceWarps = 8;
__global__ void __launch_bounds__(32 * kReduceWarps)
    mlp_reduce_kernel(const float *__restrict__ part, int n_cta, float *__restrict__ grad)
{
  __shared__ float sh[kReduceWarps][32];
  pdl_wait();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, p = blockIdx.x * 32 + lane;
  float v = 0.f;
  if (p < kPart) {
#pragma unroll 8
    for (int c = w; c < n_cta; c += kReduceWarps)
      v += __ldcg(part + (size_t)c * kPart + p);
  }
  sh[w][lane] = v;
  __syncthreads();
  if (w == 0 && p < kPart) {
    v = sh[0][lane];
#pragma unroll
    for (int k = 1; k < kReduceWarps; k++)
      v += sh[k][lane];
    grad[p] = v;
  }
}

__global__ void mlp_adam_kernel(float *__restrict__ prm, float *__restrict__ m,
                                float *__restrict__ v, const float *__restrict__ grad, float lr,
                                float b1, float b2, float eps, float c1, float c2, float wd)
{
  pdl_wait();
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= kParams)
    return;
  const float gr = grad[p] + wd * prm[p];
  const float mm = b1 * m[p] + (1.f - b1) * gr;
  const float vv = b2 * v[p] + (1.f - b2) * gr * gr;
  m[p] = mm;
  v[p] = vv;
  prm[p] -= lr * (mm / c1) / (sqrtf(vv / c2) + eps);
}

// ---- per-row features ------------------------------------------------------

constexpr int kFeat = 32;

// Feature row of matrix row i (CSR, FP64 values):
//  0: log(a_ii) / 8             1: sum_{j != i} |a_ij| / a_ii
//  2..27: |a_ij| / a_ii of the 26 neighbours (dz, dy, dx) in {-1,0,1}^3 \ 0,
//         lexicographic, located through the grid dimensions (nx, ny); with
//         nx = 0 the off-diagonal entries in column order
//  28: 1 for a row with more than 7 entries (27-point stencil), else 0
//  29: log(max |a_ij| / min |a_ij|) / 8 over the off-diagonal entries
//  30: row length / 27          31: 1
//
// A CTA's rows are one run of the CSR: it copies the run's columns and values
// into shared memory (coalesced, asynchronous) and two lanes then walk each
// row there; the feature rows are assembled in shared memory too and
// leave in 128-byte stores.  A run longer than the buffer (rows of more than
// 28 entries on average) is walked in global memory instead, by the same code.
// Bound by HBM (12 bytes an entry, 64 a row) and, close behind, by issue: the
// neighbour's place comes from comparisons, not divisions, and one reciprocal
// serves the row.  80^3 27-point matrix: 74 us (issue slots 64% busy, two
// lanes a row for occupancy); one thread a row straight on the CSR, with
// 64-bit divisions, took 164 us.
constexpr int kFeatRows = 128;                 // rows a CTA
constexpr int kFeatCap = kFeatRows * 28;       // entries the buffer holds
constexpr int kFeatLd = kFeat + 2;             // halfwords: rows on distinct banks
struct FeatSmem {
  double v[kFeatCap];
  int ci[kFeatCap];
  bf16 f[kFeatRows * kFeatLd];
};

// Grid of a box stencil: the column offsets at which the neighbour's plane and
// line change.  I holds every sum below (int where nx ny is under 2^29).
template <class I> struct FeatGrid {
  I nx, plane, z0, z1, z2, z3;
  __device__ FeatGrid(int nx_, int ny_)
      : nx(nx_), plane((I)nx_ * ny_), z0(-(plane + nx + 1)), z1(z0 + plane), z2(z1 + plane),
        z3(z2 + plane)
  {
  }
  // Feature slot 0 .. 25 of the neighbour at column offset d, or -1.
  __device__ int slot(I d) const
  {
    const bool in_z = d >= z0 && d < z3;
    const int dz = d < z1 ? 0 : d < z2 ? 1 : 2;
    const I rem = d + (d < z1 ? plane : d < z2 ? I(0) : -plane);  // in (-nx - 2, plane)
    const bool in_y = rem >= z1 && rem < 2 * nx - 1;
    const int dy = rem < -1 ? 0 : rem < nx - 1 ? 1 : 2;
    const I dx = rem + (rem < -1 ? nx : rem < nx - 1 ? I(0) : -nx);
    const int q = dz * 9 + dy * 3 + (int)dx + 1;
    return in_z && in_y && dx >= -1 && dx <= 1 ? q - (q >= 13) : -1;
  }
};

struct RowSums {
  double off = 0.0, mx = 0.0, mn = HUGE_VAL;
  int n = 0;
};

// Entries first, first + STEP, ... of a row: their ratios to the diagonal d
// into f (by its reciprocal, or by division where that would lose digits) and
// the sums of their magnitudes.  own_at: the diagonal's entry (STEP 2).
template <class I, int STEP, bool DIV, class Cp, class Vp>
__device__ __forceinline__ RowSums feature_entries(int i, int first, int len, int own_at, Cp c,
                                                   Vp x, const FeatGrid<I> &grid, double d,
                                                   bf16 *f)
{
  RowSums s;
  int seen = 0;
  const double rd = DIV ? 0.0 : 1.0 / d;
#pragma unroll 4
  for (int e = first; e < len; e += STEP) {
    const int col = c[e];
    const double a = fabs(x[e]);
    const bool own = col == i, some = !own && a > 0.0;  // (a NaN is left out of the sums)
    if (some) {
      s.off += a;
      s.mx = a > s.mx ? a : s.mx;
      s.mn = a < s.mn ? a : s.mn;
      s.n++;
    }
    int k;
    if (grid.nx > 0) {
      k = grid.slot((I)col - (I)i);
    } else {
      k = STEP == 2 ? e - (own_at >= 0 && e > own_at) : seen;  // its place among the others
      k = k < 26 ? k : -1;
      seen += !own;
    }
    if (k >= 0 && !own)
      f[2 + k] = __float2bfloat16_rn((float)(DIV ? a / d : a * rd));
  }
  return s;
}

// One row by two neighbouring lanes (h = 0, 1): columns c and values x, len of
// them, into f.  Sorted columns: each lane takes every other entry.  Others
// (a column may then come twice, and its last entry counts): lane 0 alone.
template <class I, class Cp, class Vp>
__device__ __forceinline__ void feature_row(int i, int len, int h, Cp c, Vp x, int nx, int ny,
                                            bf16 *f)
{
  int own_at = -1, sorted = 1;
#pragma unroll 4
  for (int e = h; e < len; e += 2) {
    const int col = c[e];
    own_at = col == i ? e : own_at;
    sorted &= e + 1 >= len || col < c[e + 1];
  }
  own_at = max(own_at, __shfl_xor_sync(0xffffffffu, own_at, 1));
  sorted &= __shfl_xor_sync(0xffffffffu, sorted, 1);
  const double aii = own_at >= 0 ? x[own_at] : 0.0;
  const double d = aii > 0.0 ? aii : 1.0;
  const FeatGrid<I> grid(nx, ny);
  RowSums s;
  if (sorted && d > 1e-300 && d < 1e300)
    s = feature_entries<I, 2, false>(i, h, len, own_at, c, x, grid, d, f);
  else if (h == 0)
    s = feature_entries<I, 1, true>(i, 0, len, own_at, c, x, grid, d, f);
  s.off += __shfl_xor_sync(0xffffffffu, s.off, 1);
  s.mx = fmax(s.mx, __shfl_xor_sync(0xffffffffu, s.mx, 1));
  s.mn = fmin(s.mn, __shfl_xor_sync(0xffffffffu, s.mn, 1));
  s.n += __shfl_xor_sync(0xffffffffu, s.n, 1);
  // the two logarithms, one a lane
  const float lg = (float)(log(h ? s.mx / s.mn : d) / 8.0);
  if (h == 0) {
    f[0] = __float2bfloat16_rn(lg);
    f[1] = __float2bfloat16_rn((float)(s.off / d));
    f[28] = __float2bfloat16_rn(len > 7 ? 1.f : 0.f);
  } else {
    f[29] = __float2bfloat16_rn(s.n >= 2 ? lg : 0.f);
    f[30] = __float2bfloat16_rn((float)len / 27.f);
    f[31] = __float2bfloat16_rn(1.f);
  }
}

template <class I>
__global__ void __launch_bounds__(2 * kFeatRows, 4)
    row_features_kernel(int n, const int *__restrict__ rp, const int *__restrict__ ci,
                        const double *__restrict__ v, int nx, int ny, bf16 *__restrict__ out)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  FeatSmem &s = *reinterpret_cast<FeatSmem *>(smem_raw);
  constexpr int kT = 2 * kFeatRows;
  pdl_wait();
  const int tid = threadIdx.x, r0 = blockIdx.x * kFeatRows, rows = min(kFeatRows, n - r0);
  const int first = __ldg(rp + r0), count = __ldg(rp + r0 + rows) - first;
  const bool staged = count <= kFeatCap;
  if (staged) {
    const double *gv = v + first;
    const int *gc = ci + first;
    const uint32_t sv = smem_addr(s.v), sc = smem_addr(s.ci);
#pragma unroll 4
    for (int k = tid; k < count; k += kT) {
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sv + 8 * k), "l"(gv + k));
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(sc + 4 * k), "l"(gc + k));
    }
    asm volatile("cp.async.commit_group;\n");
  }
  uint32_t *words = reinterpret_cast<uint32_t *>(s.f);
  for (int k = tid; k < rows * (kFeatLd / 2); k += kT)
    words[k] = 0u;
  // two lanes a row; a lane pair past the end walks an empty row of its own
  const int r = tid >> 1, h = tid & 1, i = r0 + r;
  const int e0 = r < rows ? __ldg(rp + i) : first;
  const int len = r < rows ? __ldg(rp + i + 1) - e0 : 0;
  bf16 *f = s.f + r * kFeatLd;
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  __syncthreads();
  if (staged)
    feature_row<I>(i, len, h, s.ci + (e0 - first), s.v + (e0 - first), nx, ny, f);
  else
    feature_row<I>(i, len, h, ci + e0, v + e0, nx, ny, f);
  pdl_trigger();
  __syncthreads();
  uint32_t *o = reinterpret_cast<uint32_t *>(out + (size_t)r0 * kFeat);
  for (int k = tid; k < rows * (kFeat / 2); k += kT)
    o[k] = words[k / (kFeat / 2) * (kFeatLd / 2) + k % (kFeat / 2)];
}

int train_grid(long long M)
{
  const long long blocks = (M + kBlockRows - 1) / kBlockRows;
  return (int)std::max(1LL, std::min(blocks, (long long)device_sm_count() * 2));
}

// Forward: CTAs that stay resident walk the rows in strides.
int fwd_grid(long long M)
{
  const long long blocks = (M + kFwdThreads - 1) / kFwdThreads;
  return (int)std::max(1LL, std::min(blocks, (long long)device_sm_count() * kFwdCtas));
}

int set_smem_attrs()
{
  // (a kernel's limit is per device)
  static std::atomic<unsigned long long> done{0};
  int dev = 0;
  ISPM_CUDA_TRY(cudaGetDevice(&dev));
  const unsigned long long bit = dev < 64 ? 1ull << dev : 0;
  if (done.load() & bit)
    return ISPM_OK;
  ISPM_CUDA_TRY(cudaFuncSetAttribute(mlp_train_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)sizeof(TrainSmem)));
  ISPM_CUDA_TRY(cudaFuncSetAttribute(row_features_kernel<int>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)sizeof(FeatSmem)));
  ISPM_CUDA_TRY(cudaFuncSetAttribute(row_features_kernel<long long>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)sizeof(FeatSmem)));
  done.fetch_or(bit);
  return ISPM_OK;
}

}  // namespace
}  // namespace ispm

struct ispm_mlp {
  float *prm = nullptr, *m = nullptr, *v = nullptr, *grad = nullptr, *part = nullptr;
  mutable std::mutex host_mu;
  mutable std::vector<float> host;  // results on their way to the caller
  mutable float *pinned = nullptr;
  mutable int copies = 0;
  // Where the next copy lands (host_mu held).  A pinned block saves a copy 5 us
  // but costs a process's only object 3 ms (2.6 to make, 0.5 to free), more than
  // all else a short-lived one does (0.4 ms to make, 0.4 its first step, 0.6 to
  // free): it is made once the copies have cost as much without it.
  float *landing() const
  {
    constexpr int kPinAfter = 600;
    if (copies < kPinAfter && ++copies == kPinAfter) {
      // (another thread may be capturing a graph, which an allocation must not end)
      cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
      cudaThreadExchangeStreamCaptureMode(&mode);
      if (cudaMallocHost(&pinned, host.size() * sizeof(float)) != cudaSuccess) {
        cudaGetLastError();
        pinned = nullptr;
      }
      cudaThreadExchangeStreamCaptureMode(&mode);
    }
    return pinned ? pinned : host.data();
  }
  int part_cta = 0;
  int step = 0;
  ~ispm_mlp()
  {
    if (pinned)
      cudaFreeHost(pinned);
    for (float *p : {prm, part})  // (m, v and grad are in prm's block)
      if (p)
        cudaFree(p);
  }
};

using namespace ispm;

extern "C" {

int ispm_mlp_n_params(void) { return kParams; }

int ispm_mlp_create(const float *init_params, ispm_mlp **out)
{
  clear_error();
  if (!out || !init_params)
    return fail(ISPM_ERR_INVALID, "NULL argument");
  *out = nullptr;
  std::unique_ptr<ispm_mlp> h(new (std::nothrow) ispm_mlp);
  if (!h)
    return fail(ISPM_ERR_NOMEM, "host allocation");
  // (part, 7.7 MB, waits for a training step: with it an object takes 0.5 ms to
  // make, not 0.1, which a prediction never needs)
  constexpr size_t each = (kPart + 63) / 64 * 64;
  if (cudaMalloc(&h->prm, sizeof(float) * 4 * each) != cudaSuccess) {
    cudaGetLastError();
    h->prm = nullptr;
    return fail(ISPM_ERR_NOMEM, "cudaMalloc");
  }
  h->m = h->prm + each;
  h->v = h->m + each;
  h->grad = h->v + each;
  ISPM_CUDA_TRY(cudaMemset(h->prm, 0, sizeof(float) * 4 * each));
  ISPM_CUDA_TRY(cudaMemcpy(h->prm, init_params, sizeof(float) * kParams, cudaMemcpyHostToDevice));
  try {
    h->host.resize(kPart);
  } catch (const std::bad_alloc &) {
    return fail(ISPM_ERR_NOMEM, "host allocation");
  }
  if (int e = set_smem_attrs())
    return e;
  *out = h.release();
  return ISPM_OK;
}

int ispm_mlp_get_params(const ispm_mlp *m, float *host_out)
{
  clear_error();
  if (!m || !host_out)
    return fail(ISPM_ERR_INVALID, "NULL argument");
  std::lock_guard<std::mutex> lock(m->host_mu);
  float *at = m->landing();
  ISPM_CUDA_TRY(cudaMemcpyAsync(at, m->prm, sizeof(float) * kParams, cudaMemcpyDeviceToHost, 0));
  ISPM_CUDA_TRY(cudaStreamSynchronize(0));
  memcpy(host_out, at, sizeof(float) * kParams);
  return ISPM_OK;
}

int ispm_mlp_set_params(ispm_mlp *m, const float *host_in)
{
  clear_error();
  if (!m || !host_in)
    return fail(ISPM_ERR_INVALID, "NULL argument");
  ISPM_CUDA_TRY(cudaMemcpy(m->prm, host_in, sizeof(float) * kParams, cudaMemcpyHostToDevice));
  ISPM_CUDA_TRY(cudaMemset(m->m, 0, sizeof(float) * kPart));
  ISPM_CUDA_TRY(cudaMemset(m->v, 0, sizeof(float) * kPart));
  m->step = 0;
  return ISPM_OK;
}

int ispm_mlp_forward(const ispm_mlp *m, long long n_rows, const void *feat_bf16, float *out,
                     void *stream)
{
  clear_error();
  if (!m || n_rows < 0 || (n_rows && (!feat_bf16 || !out)))
    return fail(ISPM_ERR_INVALID, "bad arguments");
  if (!aligned(feat_bf16, 4) || !aligned(out, 8))
    return fail(ISPM_ERR_INVALID, "features must be 4-byte, outputs 8-byte aligned");
  if (n_rows == 0)
    return ISPM_OK;
  ISPM_CUDA_TRY(launch_kernel(mlp_forward_kernel, dim3(fwd_grid(n_rows)), dim3(kFwdThreads), 0,
                              (cudaStream_t)stream, true, (const float *)m->prm,
                              (const bf16 *)feat_bf16, (float2 *)out, n_rows));
  ISPM_CUDA_TRY(cudaPeekAtLastError());
  return ISPM_OK;
}

int ispm_mlp_loss_grad(ispm_mlp *m, long long n_rows, const void *feat_bf16,
                       const float *target, const float *weight, float *grad_out,
                       double *loss_out, void *stream)
{
  clear_error();
  if (!m || n_rows <= 0 || !feat_bf16 || !target)
    return fail(ISPM_ERR_INVALID, "bad arguments");
  if (!aligned(feat_bf16, 4) || !aligned(target, 8) || (weight && !aligned(weight, 8)))
    return fail(ISPM_ERR_INVALID, "misaligned features / targets / weights");
  if (int e = set_smem_attrs())
    return e;
  const int grid = train_grid(n_rows);
  if (grid > m->part_cta) {
    if (m->part)
      cudaFree(m->part);
    m->part = nullptr;
    m->part_cta = 0;
    if (cudaMalloc(&m->part, sizeof(float) * kPart * grid) != cudaSuccess) {
      cudaGetLastError();
      m->part = nullptr;
      return fail(ISPM_ERR_NOMEM, "cudaMalloc");
    }
    m->part_cta = grid;
  }
  cudaStream_t s = (cudaStream_t)stream;
  // (programmatic launches: each kernel is set up while the one before it ends
  // and waits on the device for its results)
  ISPM_CUDA_TRY(launch_kernel(mlp_train_kernel, dim3(grid), dim3(kThreads), sizeof(TrainSmem), s,
                              true, (const float *)m->prm, (const bf16 *)feat_bf16,
                              (const float2 *)target, (const float2 *)weight, n_rows,
                              1.0f / (float)n_rows, (int)aligned(feat_bf16, 16), m->part));
  ISPM_CUDA_TRY(cudaPeekAtLastError());
  ISPM_CUDA_TRY(launch_kernel(mlp_reduce_kernel, dim3((kPart + 31) / 32), dim3(32 * kReduceWarps), 0,
                              s, true, (const float *)m->part, grid, m->grad));
  ISPM_CUDA_TRY(cudaPeekAtLastError());
  if (grad_out || loss_out) {  // one copy: the loss sits behind the gradient
    std::lock_guard<std::mutex> lock(m->host_mu);
    const size_t from = grad_out ? 0 : kParams;
    float *at = m->landing();
    ISPM_CUDA_TRY(cudaMemcpyAsync(at + from, m->grad + from, sizeof(float) * (kPart - from),
                                  cudaMemcpyDeviceToHost, s));
    ISPM_CUDA_TRY(cudaStreamSynchronize(s));
    if (grad_out)
      memcpy(grad_out, at, sizeof(float) * kParams);
    if (loss_out)
      *loss_out = at[kParams];
  }
  return ISPM_OK;
}

int ispm_mlp_adam_step(ispm_mlp *m, float lr, float beta1, float beta2, float eps,
                       float weight_decay, void *stream)
{
  clear_error();
  if (!m || !(lr > 0) || !(beta1 >= 0 && beta1 < 1) || !(beta2 >= 0 && beta2 < 1))
    return fail(ISPM_ERR_INVALID, "bad Adam parameters");
  m->step++;
  const float c1 = 1.f - std::pow(beta1, (float)m->step);
  const float c2 = 1.f - std::pow(beta2, (float)m->step);
  ISPM_CUDA_TRY(launch_kernel(mlp_adam_kernel, dim3((kParams + 255) / 256), dim3(256), 0,
                              (cudaStream_t)stream, true, m->prm, m->m, m->v,
                              (const float *)m->grad, lr, beta1, beta2, eps, c1, c2,
                              weight_decay));
  ISPM_CUDA_TRY(cudaPeekAtLastError());
  return ISPM_OK;
}

void ispm_mlp_free(ispm_mlp *m) { delete m; }

int ispm_row_features(int n, const int *row_ptr, const int *cols, const double *vals, int nx,
                      int ny, void *out_bf16, void *stream)
{
  clear_error();
  if (n < 0 || (n && (!row_ptr || !cols || !vals || !out_bf16)) || nx < 0 || ny < 0 ||
      (nx > 0) != (ny > 0))
    return fail(ISPM_ERR_INVALID, "bad arguments");
  if (!aligned(out_bf16, 4))
    return fail(ISPM_ERR_INVALID, "features must be 4-byte aligned");
  if (n == 0)
    return ISPM_OK;
  if (int e = set_smem_attrs())
    return e;
  const auto kernel = (long long)nx * ny < (1LL << 29) ? row_features_kernel<int>
                                                       : row_features_kernel<long long>;
  ISPM_CUDA_TRY(launch_kernel(kernel, dim3((n + kFeatRows - 1) / kFeatRows), dim3(2 * kFeatRows),
                              sizeof(FeatSmem), (cudaStream_t)stream, true, n, row_ptr, cols, vals,
                              nx, ny, (bf16 *)out_bf16));
  ISPM_CUDA_TRY(cudaPeekAtLastError());
  return ISPM_OK;
}

}  // extern "C"
