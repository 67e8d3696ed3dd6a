// Tensor-core inference of the learned WENO weights.
//
// The network maps a stencil normalised to its local range (the reference's
// normalize convention, dynamics_rk.h:42-53, WenoLimiter.h:85-96) to the five
// nonlinear weights of the left edge; the right edge uses the mirrored stencil
// (the right-edge weights of a stencil are the left-edge weights of its mirror
// image, WenoLimiter.h:383-387 vs 406-410):
//
//   x(9) -> relu(W1 bf(x) + b1) -> bf -> relu(W2 h1 + b2) -> bf -> W3 h2 + b3 -> softmax
//
// bf() rounds to bfloat16; weights are used rounded to bfloat16, biases and
// accumulation are FP32.  One warp evaluates 32 stencils and their mirrors
// (64 rows, four 16-row tiles) with mma.sync m16n8k16 BF16 -> FP32; each
// layer's accumulator fragment is the next layer's A-operand fragment after a
// fused relu + bfloat16 conversion, so activations never leave registers.
#pragma once

#include <cuda_bf16.h>

#include <cstdint>

namespace pu {
namespace mlp {
constexpr int NIN = 9, NH = 32, NOUT = 5;
constexpr int OFF_W1 = 0;
constexpr int OFF_B1 = OFF_W1 + NH * NIN;
constexpr int OFF_W2 = OFF_B1 + NH;
constexpr int OFF_B2 = OFF_W2 + NH * NH;
constexpr int OFF_W3 = OFF_B2 + NH;
constexpr int OFF_B3 = OFF_W3 + NOUT * NH;
constexpr int NPARAM = OFF_B3 + NOUT;   // 1541
// Operand fragments of the network, in shared memory while a kernel runs: ten
// groups of 16 bytes per lane (28 bf16x2 operand words, 10 FP32 biases, 2
// unused words), group by group over the 32 lanes.
constexpr int FRAG_GROUPS = 10, FRAG_WORDS = 4 * FRAG_GROUPS;
constexpr int FRAG_BYTES = 32 * FRAG_WORDS * 4;
// Per-warp shared memory: 64 input rows of 16 bf16 (2 KB), then the logits
// column by column with a 68-float stride (5 x 68 floats), bank-conflict
// free for the fragment-layout stores and the per-lane reads.
constexpr int LOGIT_STRIDE = 68;
constexpr int WARP_SMEM_BYTES = 64 * 32 + 5 * LOGIT_STRIDE * 4;

__host__ __device__ inline bool is_bias(int p) {
  return (p >= OFF_B1 && p < OFF_W2) || (p >= OFF_B2 && p < OFF_W3) || p >= OFF_B3;
}
}  // namespace mlp

__device__ __forceinline__ float bf16_round(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

__device__ __forceinline__ unsigned long long splitmix64(unsigned long long z) {
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

// (s - min) / (max - min); all zeros when the range is <= 1e-20 (the
// reference's normalize keeps scale = 1 there, WenoLimiter.h:85-96).
// Returns the largest normalised jump between neighbouring entries (every
// operation rounded by itself: the jump decides between the network and the
// limiter, and all callers must decide alike).
__device__ __forceinline__ float normalize9(const float (&s)[9], float (&x)[9]) {
  float mn = s[0], mx = s[0];
#pragma unroll
  for (int m = 1; m < 9; m++) {
    mn = fminf(mn, s[m]);
    mx = fmaxf(mx, s[m]);
  }
  const float rng = mx - mn;
  const float r = rng > 1e-20f ? 1.f / rng : 0.f;
#pragma unroll
  for (int m = 0; m < 9; m++) x[m] = __fmul_rn(s[m] - mn, r);
  float jmp = 0.f;
#pragma unroll
  for (int m = 0; m < 8; m++) jmp = fmaxf(jmp, fabsf(__fsub_rn(x[m + 1], x[m])));
  return jmp;
}

__device__ __forceinline__ uint32_t bf16_bits(float x) {
  __nv_bfloat16 b = __float2bfloat16_rn(x);
  return uint32_t(*reinterpret_cast<unsigned short *>(&b));
}

// Per-lane operand fragments of mma.m16n8k16 (B is K x N, K = layer input,
// N = layer output; bfloat16 pairs, lower k in the low half).  Groups of four
// words: 0-1 W1's four output tiles, 2-5 W2's output tiles (both K halves of
// each), 6 W3, 7-8 b2, 9 b3 (FP32 bits).
static __global__ void k_mlp_frags(const float *__restrict__ theta, uint32_t *__restrict__ frags) {
  using namespace mlp;
  const int lane = threadIdx.x;
  if (lane >= 32) return;
  const int g = lane >> 2, t = lane & 3;
  // Input columns 9 and 10 are constant 1: W1's columns there carry the
  // layer-1 bias split into a bfloat16 pair (b1 = hi + lo to about 2^-17).
  auto W1 = [&](int o, int i) {
    if (i < NIN) return theta[OFF_W1 + o * NIN + i];
    const float b = theta[OFF_B1 + o], hi = __bfloat162float(__float2bfloat16_rn(b));
    return i == NIN ? hi : (i == NIN + 1 ? b - hi : 0.f);
  };
  auto W2 = [&](int o, int i) { return theta[OFF_W2 + o * NH + i]; };
  auto W3 = [&](int o, int i) { return o < NOUT ? theta[OFF_W3 + o * NH + i] : 0.f; };
  auto pk = [](float lo, float hi) { return bf16_bits(lo) | (bf16_bits(hi) << 16); };
  int w = 0;
  auto put = [&](uint32_t v) {
    frags[((w >> 2) * 32 + lane) * 4 + (w & 3)] = v;
    w++;
  };
  for (int n = 0; n < 4; n++) {
    put(pk(W1(8 * n + g, 2 * t), W1(8 * n + g, 2 * t + 1)));
    put(pk(W1(8 * n + g, 2 * t + 8), W1(8 * n + g, 2 * t + 9)));
  }
  for (int n = 0; n < 4; n++)
    for (int s = 0; s < 2; s++) {
      put(pk(W2(8 * n + g, 16 * s + 2 * t), W2(8 * n + g, 16 * s + 2 * t + 1)));
      put(pk(W2(8 * n + g, 16 * s + 2 * t + 8), W2(8 * n + g, 16 * s + 2 * t + 9)));
    }
  for (int s = 0; s < 2; s++) {
    put(pk(W3(g, 16 * s + 2 * t), W3(g, 16 * s + 2 * t + 1)));
    put(pk(W3(g, 16 * s + 2 * t + 8), W3(g, 16 * s + 2 * t + 9)));
  }
  for (int n = 0; n < 4; n++) {
    put(__float_as_uint(theta[OFF_B2 + 8 * n + 2 * t]));
    put(__float_as_uint(theta[OFF_B2 + 8 * n + 2 * t + 1]));
  }
  put(__float_as_uint(2 * t < NOUT ? theta[OFF_B3 + 2 * t] : 0.f));
  put(__float_as_uint(2 * t + 1 < NOUT ? theta[OFF_B3 + 2 * t + 1] : 0.f));
  put(0u);
  put(0u);
}

// The fragments into shared memory, by asynchronous copies of the block's nt
// threads; frags_landed waits for a thread's own (the caller synchronises).
__device__ __forceinline__ void load_frags(const uint32_t *frags, uint4 *sF, int nt) {
  for (int e = threadIdx.x; e < mlp::FRAG_GROUPS * 32; e += nt)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(sF + e))),
                 "l"(reinterpret_cast<const uint4 *>(frags) + e)
                 : "memory");
}
__device__ __forceinline__ void frags_landed() { asm volatile("cp.async.wait_all;" ::: "memory"); }

__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1,
                                         const float (&c)[4]) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%10,%11,%12,%13};\n"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(c[0]), "f"(c[1]), "f"(c[2]),
        "f"(c[3]));
}

// relu, then round to a bfloat16 pair: low half <- lo, high half <- hi.
__device__ __forceinline__ uint32_t relu_bf16x2(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.relu.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}
__device__ __forceinline__ uint32_t bf16x2(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}

// Input fragment k-step s of the next layer from output tiles 2s (d0), 2s+1 (d1).
__device__ __forceinline__ void acc_to_a(const float (&d0)[4], const float (&d1)[4], uint32_t (&a)[4]) {
  a[0] = relu_bf16x2(d0[0], d0[1]);
  a[1] = relu_bf16x2(d0[2], d0[3]);
  a[2] = relu_bf16x2(d1[0], d1[1]);
  a[3] = relu_bf16x2(d1[2], d1[3]);
}

// One warp evaluates the network on the 32 normalised stencils held by its
// lanes and on their mirror images.  sW: per-warp scratch of WARP_SMEM_BYTES
// (16-byte aligned).  Input row r occupies 16-byte chunks 2r and 2r+1 with
// the halves swapped when bit 2 of r is set, so the row stores and the
// ldmatrix phases hit 8 distinct bank groups.  Returns each lane's left-edge
// weights and the right-edge weights of its stencil.  All 32 lanes must call it.
//
// The four 16-row tiles go through each layer together: a tile's chain of
// fourteen MMAs and the conversions between them is bound by their latency,
// four of them interleave, and a layer's operands (sF) are read once per warp
// call instead of staying in 38 registers (128x128x64 boundary layer: k_xy 640
// -> 576 us, the z march 414 -> 398 us per launch).
__device__ __forceinline__ int row_chunk(int r, int half) { return 2 * r + (half ^ ((r >> 2) & 1)); }

__device__ __forceinline__ void mlp_warp_weights(const uint4 *sF, uint32_t *sW, const float (&x)[9], float (&wl)[5],
                                                 float (&wr)[5]) {
  using mlp::LOGIT_STRIDE;
  const int lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  uint4 *rows = reinterpret_cast<uint4 *>(sW);
  float *sZ = reinterpret_cast<float *>(sW + 64 * 8);   // [5][LOGIT_STRIDE]
  const uint32_t one = 0x3F80u;   // bfloat16 1.0 in input column 10 (column 9 is the high half of word 4)
  rows[row_chunk(lane, 0)] =
      make_uint4(bf16x2(x[0], x[1]), bf16x2(x[2], x[3]), bf16x2(x[4], x[5]), bf16x2(x[6], x[7]));
  rows[row_chunk(lane, 1)] = make_uint4(bf16x2(x[8], 1.f), one, 0u, 0u);
  rows[row_chunk(32 + lane, 0)] =
      make_uint4(bf16x2(x[8], x[7]), bf16x2(x[6], x[5]), bf16x2(x[4], x[3]), bf16x2(x[2], x[1]));
  rows[row_chunk(32 + lane, 1)] = make_uint4(bf16x2(x[0], 1.f), one, 0u, 0u);
  __syncwarp();
  const uint4 *F = sF + lane;
  uint32_t a2[4][2][4], a3[4][2][4];
  {
    uint32_t a[4][4];
#pragma unroll
    for (int T = 0; T < 4; T++) {
      const uint4 *src = rows + row_chunk(16 * T + (lane & 15), lane >> 4);
      const unsigned addr = static_cast<unsigned>(__cvta_generic_to_shared(src));
      asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                   : "=r"(a[T][0]), "=r"(a[T][1]), "=r"(a[T][2]), "=r"(a[T][3])
                   : "r"(addr)
                   : "memory");
    }
    const float zero[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int s = 0; s < 2; s++) {
      const uint4 w = F[32 * s];
#pragma unroll
      for (int T = 0; T < 4; T++) {
        float d0[4], d1[4];
        mma_bf16(d0, a[T], w.x, w.y, zero);
        mma_bf16(d1, a[T], w.z, w.w, zero);
        acc_to_a(d0, d1, a2[T][s]);
      }
    }
  }
#pragma unroll
  for (int s = 0; s < 2; s++) {
    const uint4 w0 = F[32 * (2 + 2 * s)], w1 = F[32 * (3 + 2 * s)], b = F[32 * (7 + s)];
    const float c0[4] = {__uint_as_float(b.x), __uint_as_float(b.y), __uint_as_float(b.x), __uint_as_float(b.y)};
    const float c1[4] = {__uint_as_float(b.z), __uint_as_float(b.w), __uint_as_float(b.z), __uint_as_float(b.w)};
#pragma unroll
    for (int T = 0; T < 4; T++) {
      float d0[4], d1[4];
      mma_bf16(d0, a2[T][0], w0.x, w0.y, c0);
      mma_bf16(d1, a2[T][0], w1.x, w1.y, c1);
      mma_bf16(d0, a2[T][1], w0.z, w0.w, d0);
      mma_bf16(d1, a2[T][1], w1.z, w1.w, d1);
      acc_to_a(d0, d1, a3[T][s]);
    }
  }
  {
    const uint4 w = F[32 * 6], b = F[32 * 9];
    const float c[4] = {__uint_as_float(b.x), __uint_as_float(b.y), __uint_as_float(b.x), __uint_as_float(b.y)};
#pragma unroll
    for (int T = 0; T < 4; T++) {
      float d3[4];
      mma_bf16(d3, a3[T][0], w.x, w.y, c);
      mma_bf16(d3, a3[T][1], w.z, w.w, d3);
      const int r0 = 16 * T + g, r1 = r0 + 8;
      if (2 * t < 5) {
        sZ[2 * t * LOGIT_STRIDE + r0] = d3[0];
        sZ[2 * t * LOGIT_STRIDE + r1] = d3[2];
      }
      if (2 * t + 1 < 5) {
        sZ[(2 * t + 1) * LOGIT_STRIDE + r0] = d3[1];
        sZ[(2 * t + 1) * LOGIT_STRIDE + r1] = d3[3];
      }
    }
  }
  __syncwarp();
  float zl[5], zr[5];
#pragma unroll
  for (int k = 0; k < 5; k++) {
    zl[k] = sZ[k * LOGIT_STRIDE + lane];
    zr[k] = sZ[k * LOGIT_STRIDE + 32 + lane];
  }
  __syncwarp();   // the scratch is free for the next call
  float ml = zl[0], mr = zr[0];
#pragma unroll
  for (int k = 1; k < 5; k++) {
    ml = fmaxf(ml, zl[k]);
    mr = fmaxf(mr, zr[k]);
  }
  float sl = 0.f, sr = 0.f;
#pragma unroll
  for (int k = 0; k < 5; k++) {
    zl[k] = __expf(zl[k] - ml);
    zr[k] = __expf(zr[k] - mr);
    sl += zl[k];
    sr += zr[k];
  }
  const float il = __frcp_rn(sl), ir = __frcp_rn(sr);
#pragma unroll
  for (int k = 0; k < 5; k++) {
    wl[k] = zl[k] * il;
    wr[4 - k] = zr[k] * ir;   // the mirror's left weights, reversed, are the right-edge weights
  }
}

}  // namespace pu
