// Training and checking of the learned WENO weights (the network and its
// tensor-core inference are in mlp_infer.cuh).  The plain limiter's weights
// are the training targets and the fallback.  Contents:
//   k_harvest         -- sample stencils of a state and their plain weights
//   k_mlp_prepare     -- bfloat16-rounded copy of the FP32 master parameters
//   k_mlp_fwd_bwd     -- forward + backward of a batch tile, per-block gradient
//   k_mlp_update      -- deterministic sum of the per-block gradients, Adam
//                        update of the FP32 master parameters
//   k_mlp_eval        -- forward only (SIMT), for checks
//   k_mlp_eval_mma    -- tensor-core forward of a stencil list, for checks
#pragma once

#include <cstdint>

#include "dycore_kernels.cuh"
#include "mlp_infer.cuh"

namespace pu {
namespace mlp {
constexpr int TB = 128;                 // samples and threads per training block
constexpr int TW = TB / 32;             // warps per training block
// Rows of the per-sample tiles: 16-byte aligned, one 16-byte bank group apart.
constexpr int TBP = TB + 4;
constexpr int TROWS = 2 * NH;           // the largest pair of tiles (gradient and input of layer 2)
constexpr int WP = NH + 4;              // padded weight rows
constexpr int RSTRIDE = NH * WP + NH;   // one warp's gradient of one layer, rows padded, then the biases
// Shared-memory layout of the training kernel (floats).
constexpr int SM_W1T = 0;                       // [NIN][WP]   W1 transposed
constexpr int SM_W2 = SM_W1T + NIN * WP;        // [NH][NH]
constexpr int SM_W2T = SM_W2 + NH * NH;         // [NH][WP]    W2 transposed
constexpr int SM_W3 = SM_W2T + NH * WP;         // [NOUT][NH]
constexpr int SM_W3T = SM_W3 + NOUT * NH;       // [NH][8]     W3 transposed, columns from NOUT on zero
constexpr int SM_B1 = SM_W3T + NH * 8, SM_B2 = SM_B1 + NH, SM_B3 = SM_B2 + NH;   // B3 [8]
constexpr int SM_TILE = SM_B3 + 8;              // [TROWS][TBP]; the warps' gradients between phases
constexpr int SM_FLOATS = SM_TILE + TROWS * TBP;
static_assert(TW * RSTRIDE <= TROWS * TBP, "the warps' gradients exceed the tile");
static_assert(SM_FLOATS * 4 <= 48 * 1024, "training block exceeds the default shared memory");
static_assert(SM_W2 % 4 == 0 && SM_W2T % 4 == 0 && SM_W3 % 4 == 0 && SM_W3T % 4 == 0 && SM_TILE % 4 == 0, "alignment");
}  // namespace mlp

// ---------------------------------------------------------------------------
// Harvest: n samples of (normalised stencil, plain left-edge weights) from the
// state s.  Each sample draws a field, a direction and a cell from a
// counter-based generator; stencils touching immersed cells, or reaching the
// z walls, are redrawn (the dycore never uses the learned weights there).
// ---------------------------------------------------------------------------
template <class R, int NTR>
__global__ void k_harvest(const Grid<R> G, const R *__restrict__ s, long n, unsigned long long seed, long offset,
                          float *__restrict__ xs, float *__restrict__ ts) {
  const long q = long(blockIdx.x) * blockDim.x + threadIdx.x;
  if (q >= n) return;
  constexpr int F = 6 + NTR;
  const int nx = G.nx, ny = G.ny, nz = G.nz;
  const int ndir = G.sim2d ? 2 : 3;
  float st[9];
  for (int attempt = 0; attempt < 64; attempt++) {
    unsigned long long r = splitmix64(seed * 0x100000001B3ull + (unsigned long long)(offset + q) * 64 + attempt);
    const int f = int((r & 0xFFFF) % F);
    int dir = int(((r >> 16) & 0xFF) % ndir);
    if (G.sim2d && dir == 1) dir = 2;
    const int i = int(((r >> 24) & 0xFFFFF) % nx);
    const int j = int(((r >> 44) & 0xFFFFF) % ny);
    unsigned long long r2 = splitmix64(r);
    int k = int(r2 % nz);
    if (dir == 2) {
      if (nz < 2 * HS + 3) continue;
      k = HS + 1 + int(r2 % (nz - 2 * HS - 2));
    }
    if ((dir == 0 && G.bc_x != BC_PERIODIC) || (dir == 1 && G.bc_y != BC_PERIODIC)) {
      // precursor boundaries: keep the stencil inside the domain
      if (dir == 0 && (i < HS || i >= nx - HS)) continue;
      if (dir == 1 && (j < HS || j >= ny - HS)) continue;
    }
    bool ok = true;
    for (int m = 0; m < 9 && ok; m++) {
      int ii = i, jj = j, kk = k;
      if (dir == 0) ii = wrapi(i + m - 4, nx);
      else if (dir == 1) jj = wrapi(j + m - 4, ny);
      else kk = k + m - 4;
      const size_t idx = (size_t(kk) * ny + jj) * nx + ii;
      if (G.flags && (__ldg(G.flags + idx) & (FLAG_IMM | FLAG_ANY10))) ok = false;
      R w[F];
      prims<R, NTR>(G, s, idx, kk, w);
      st[m] = float(w[f]);
    }
    if (ok) break;
  }
  float x[9], wt[5];
  normalize9(st, x);
  weno9_left_weights(st, wt);
#pragma unroll
  for (int m = 0; m < 9; m++) xs[q * 9 + m] = x[m];
#pragma unroll
  for (int k = 0; k < 5; k++) ts[q * 5 + k] = wt[k];
}

// ---------------------------------------------------------------------------
// Training.
// ---------------------------------------------------------------------------
static __global__ void k_mlp_prepare(const float *__restrict__ theta, float *__restrict__ wq) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p < mlp::NPARAM) wq[p] = mlp::is_bias(p) ? theta[p] : bf16_round(theta[p]);
}

// Sample index of batch slot q at step `step`, uniform over the dataset.
__device__ __forceinline__ long batch_sample(unsigned long long seed, long step, long q, long ndata) {
  return long(splitmix64(seed ^ (0xA24BAED4963EE407ull * (unsigned long long)(step + 1)) ^ (unsigned long long)q) %
              (unsigned long long)ndata);
}

// acc[q] += W[row][2q..2q+1] * x for the 32 outputs of one weight row (16-byte
// aligned, the same address in every lane).
__device__ __forceinline__ void axpy32(float2 (&acc)[16], const float *row, float x) {
  const float2 xx = make_float2(x, x);
#pragma unroll
  for (int q = 0; q < 8; q++) {
    const float4 w = *reinterpret_cast<const float4 *>(row + 4 * q);
    acc[2 * q] = __ffma2_rn(make_float2(w.x, w.y), xx, acc[2 * q]);
    acc[2 * q + 1] = __ffma2_rn(make_float2(w.z, w.w), xx, acc[2 * q + 1]);
  }
}

// The gradient of one layer over a warp's 32 samples: this lane's NU x NV
// outputs sum_s A[tu + 8 i][s] B[tv + 4 j][s] and the row sums of A, from
// tiles with TBP samples a row.  Even and odd samples accumulate apart (one
// packed multiply-add takes two samples).  Each of the NU + NV 16-byte loads
// of a step reads 8 (A) or 4 (B) neighbouring rows: no bank conflict.
// Results go to the warp's block of R: rows of stride WP, then the row sums.
template <int NU, int NV, int ROWS_A, int ROWS_B>
__device__ __forceinline__ void warp_grad(const float *A, const float *B, float *R) {
  using namespace mlp;
  const int lane = threadIdx.x & 31, tu = lane >> 2, tv = lane & 3, s0 = (threadIdx.x >> 5) * 32;
  float2 acc[NU][NV], row[NU];
#pragma unroll
  for (int i = 0; i < NU; i++) {
    row[i] = make_float2(0.f, 0.f);
#pragma unroll
    for (int j = 0; j < NV; j++) acc[i][j] = make_float2(0.f, 0.f);
  }
#pragma unroll 2
  for (int s = s0; s < s0 + 32; s += 4) {
    float4 a[NU];
#pragma unroll
    for (int i = 0; i < NU; i++) {
      a[i] = *reinterpret_cast<const float4 *>(A + (tu + 8 * i) * TBP + s);
      row[i] = __fadd2_rn(row[i], make_float2(a[i].x, a[i].y));
      row[i] = __fadd2_rn(row[i], make_float2(a[i].z, a[i].w));
    }
#pragma unroll
    for (int j = 0; j < NV; j++) {
      const float4 b = *reinterpret_cast<const float4 *>(B + (tv + 4 * j) * TBP + s);
#pragma unroll
      for (int i = 0; i < NU; i++) {
        acc[i][j] = __ffma2_rn(make_float2(a[i].x, a[i].y), make_float2(b.x, b.y), acc[i][j]);
        acc[i][j] = __ffma2_rn(make_float2(a[i].z, a[i].w), make_float2(b.z, b.w), acc[i][j]);
      }
    }
  }
  __syncthreads();   // every warp has read the tiles, which R overlays
  R += (threadIdx.x >> 5) * RSTRIDE;
#pragma unroll
  for (int i = 0; i < NU; i++) {
    const int u = tu + 8 * i;
#pragma unroll
    for (int j = 0; j < NV; j++) {
      const int v = tv + 4 * j;
      if (u < ROWS_A && v < ROWS_B) R[u * WP + v] = acc[i][j].x + acc[i][j].y;
    }
    if (tv == 0 && u < ROWS_A) R[NH * WP + u] = row[i].x + row[i].y;
  }
  __syncthreads();
}

// The block's gradient of one layer from its warps', in a fixed order.
template <int ROWS_A, int ROWS_B>
__device__ __forceinline__ void block_grad(const float *R, float *w_out, float *b_out) {
  using namespace mlp;
  auto total = [&](int e) {
    float s = R[e];
#pragma unroll
    for (int g = 1; g < TW; g++) s += R[g * RSTRIDE + e];
    return s;
  };
  for (int p = threadIdx.x; p < ROWS_A * ROWS_B; p += TB) w_out[p] = total((p / ROWS_B) * WP + p % ROWS_B);
  if (threadIdx.x < ROWS_A) b_out[threadIdx.x] = total(NH * WP + threadIdx.x);
  __syncthreads();
}

// Forward and backward of TB samples per block, one per thread; writes the
// block's gradient sum (NPARAM values) and loss sum to partial[blockIdx.x].
//
// Per sample ~4,200 FP32 multiply-adds on a few KB of weights: bound by the
// multiply-add pipe and by shared-memory reads.  The layers run two outputs
// per packed multiply-add from 16-byte weight reads (each layer's weights
// kept in the orientation its pass walks); the weight gradients are products
// of per-sample tiles in shared memory, 4 x 8 outputs per lane in registers,
// the block's samples split over its warps.  One tile buffer serves the three
// layers in turn, so four blocks fit an SM.  Training at batch 65536: 43 us
// per step (this kernel and k_mlp_update; 39 us when launched to overlap)
// against 265 us with one thread per
// parameter walking the block's 256 samples (one block per SM, two
// shared-memory reads per multiply-add) and three kernels after it.
static __global__ void __launch_bounds__(mlp::TB, 4) k_mlp_fwd_bwd(const float *wq,
                                                                   const float *__restrict__ xs,
                                                                   const float *__restrict__ ts, long ndata, long step,
                                                                   unsigned long long seed, int batch, int sequential,
                                                                   float *__restrict__ partial) {
  using namespace mlp;
  extern __shared__ __align__(16) float sm[];
  const int tid = threadIdx.x;
  next_kernel_may_start();
  const long qb = long(blockIdx.x) * TB + tid;
  const bool live = qb < batch;
  float x[NIN], t[NOUT];
  // The samples are gathered before the last step's update has to be done.
  {
    const long smp = !live ? 0 : (sequential ? qb : batch_sample(seed, step, qb, ndata));
#pragma unroll
    for (int m = 0; m < NIN; m++) x[m] = live ? bf16_round(xs[smp * NIN + m]) : 0.f;
#pragma unroll
    for (int k = 0; k < NOUT; k++) t[k] = live ? ts[smp * NOUT + k] : 0.f;
  }
  previous_done();
  for (int p = tid; p < NPARAM; p += TB) {
    const float w = wq[p];
    if (p < OFF_B1) sm[SM_W1T + (p % NIN) * WP + p / NIN] = w;
    else if (p < OFF_W2) sm[SM_B1 + p - OFF_B1] = w;
    else if (p < OFF_B2) {
      const int q = p - OFF_W2;
      sm[SM_W2 + q] = w;
      sm[SM_W2T + (q % NH) * WP + q / NH] = w;
    } else if (p < OFF_W3) sm[SM_B2 + p - OFF_B2] = w;
    else if (p < OFF_B3) {
      const int q = p - OFF_W3;
      sm[SM_W3 + q] = w;
      sm[SM_W3T + (q % NH) * 8 + q / NH] = w;
    } else sm[SM_B3 + p - OFF_B3] = w;
  }
  if (tid < NH) {
#pragma unroll
    for (int k = NOUT; k < 8; k++) sm[SM_W3T + tid * 8 + k] = 0.f;
  }
  if (tid >= NOUT && tid < 8) sm[SM_B3 + tid] = 0.f;
  __syncthreads();

  float h1[NH], h2[NH];
  unsigned m1 = 0, m2 = 0;
  auto hidden = [&](const float2 (&a)[16], float (&h)[NH], unsigned &mask) {
#pragma unroll
    for (int q = 0; q < 16; q++) {
      if (a[q].x > 0.f) mask |= 1u << (2 * q);
      if (a[q].y > 0.f) mask |= 2u << (2 * q);
      h[2 * q] = bf16_round(fmaxf(a[q].x, 0.f));
      h[2 * q + 1] = bf16_round(fmaxf(a[q].y, 0.f));
    }
  };
  {
    float2 a[16];
#pragma unroll
    for (int q = 0; q < 16; q++) a[q] = *reinterpret_cast<const float2 *>(sm + SM_B1 + 2 * q);
#pragma unroll
    for (int m = 0; m < NIN; m++) axpy32(a, sm + SM_W1T + m * WP, x[m]);
    hidden(a, h1, m1);
  }
  {
    float2 a[16];
#pragma unroll
    for (int q = 0; q < 16; q++) a[q] = *reinterpret_cast<const float2 *>(sm + SM_B2 + 2 * q);
#pragma unroll
    for (int v = 0; v < NH; v++) axpy32(a, sm + SM_W2T + v * WP, h1[v]);
    hidden(a, h2, m2);
  }
  float z[NOUT], zmax, se = 0.f, loss = 0.f;
  {
    float2 a0 = *reinterpret_cast<const float2 *>(sm + SM_B3), a1 = *reinterpret_cast<const float2 *>(sm + SM_B3 + 2),
           a2 = *reinterpret_cast<const float2 *>(sm + SM_B3 + 4);
#pragma unroll
    for (int u = 0; u < NH; u++) {
      const float4 w = *reinterpret_cast<const float4 *>(sm + SM_W3T + u * 8);
      const float2 w2 = *reinterpret_cast<const float2 *>(sm + SM_W3T + u * 8 + 4), hh = make_float2(h2[u], h2[u]);
      a0 = __ffma2_rn(make_float2(w.x, w.y), hh, a0);
      a1 = __ffma2_rn(make_float2(w.z, w.w), hh, a1);
      a2 = __ffma2_rn(w2, hh, a2);
    }
    z[0] = a0.x, z[1] = a0.y, z[2] = a1.x, z[3] = a1.y, z[4] = a2.x;
  }
  zmax = fmaxf(fmaxf(fmaxf(fmaxf(fmaxf(-3.0e38f, z[0]), z[1]), z[2]), z[3]), z[4]);
#pragma unroll
  for (int k = 0; k < NOUT; k++) {
    z[k] = expf(z[k] - zmax);
    se += z[k];
  }
  const float inv_b = 1.f / float(batch);
#pragma unroll
  for (int k = 0; k < NOUT; k++) {
    const float p = z[k] / se;
    if (live && t[k] > 0.f) loss -= t[k] * logf(fmaxf(p, 1e-30f));
    z[k] = live ? (p - t[k]) * inv_b : 0.f;   // dz
  }

  float *T = sm + SM_TILE;
  float *out = partial + size_t(blockIdx.x) * (NPARAM + 1);
  // Layer 3: dz (rows 0..7) against h2 (rows 8..39).
#pragma unroll
  for (int k = 0; k < 8; k++) T[k * TBP + tid] = k < NOUT ? z[k < NOUT ? k : 0] : 0.f;
#pragma unroll
  for (int u = 0; u < NH; u++) T[(8 + u) * TBP + tid] = h2[u];
  // da2 = (W3^T dz) * [a2 > 0]
  float d2[NH];
  {
    float2 a[16];
#pragma unroll
    for (int q = 0; q < 16; q++) a[q] = make_float2(0.f, 0.f);
#pragma unroll
    for (int k = 0; k < NOUT; k++) axpy32(a, sm + SM_W3 + k * NH, z[k]);
#pragma unroll
    for (int q = 0; q < 16; q++) {
      d2[2 * q] = ((m2 >> (2 * q)) & 1u) ? a[q].x : 0.f;
      d2[2 * q + 1] = ((m2 >> (2 * q + 1)) & 1u) ? a[q].y : 0.f;
    }
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, o);
  __syncthreads();
  warp_grad<1, 8, NOUT, NH>(T, T + 8 * TBP, T);
  block_grad<NOUT, NH>(T, out + OFF_W3, out + OFF_B3);
  // Layer 2: da2 (rows 0..31) against h1 (rows 32..63); the warps' losses go
  // along in the rows' padding.
#pragma unroll
  for (int u = 0; u < NH; u++) {
    T[u * TBP + tid] = d2[u];
    T[(NH + u) * TBP + tid] = h1[u];
  }
  if ((tid & 31) == 0) T[(tid >> 5) * TBP + TB] = loss;
  // da1 = (W2^T da2) * [a1 > 0]
  float2 g1[16];
#pragma unroll
  for (int q = 0; q < 16; q++) g1[q] = make_float2(0.f, 0.f);
#pragma unroll
  for (int u = 0; u < NH; u++) axpy32(g1, sm + SM_W2 + u * NH, d2[u]);
#pragma unroll
  for (int q = 0; q < 16; q++) {
    if (!((m1 >> (2 * q)) & 1u)) g1[q].x = 0.f;
    if (!((m1 >> (2 * q + 1)) & 1u)) g1[q].y = 0.f;
  }
  __syncthreads();
  if (tid == 0) {
    float L = 0.f;
#pragma unroll
    for (int g = 0; g < TW; g++) L += T[g * TBP + TB];
    out[NPARAM] = L;
  }
  warp_grad<4, 8, NH, NH>(T, T + NH * TBP, T);
  block_grad<NH, NH>(T, out + OFF_W2, out + OFF_B2);
  // Layer 1: da1 (rows 0..31) against x (rows 32..40, three unused rows after).
#pragma unroll
  for (int q = 0; q < 16; q++) {
    T[2 * q * TBP + tid] = g1[q].x;
    T[(2 * q + 1) * TBP + tid] = g1[q].y;
  }
#pragma unroll
  for (int m = 0; m < 12; m++) T[(NH + m) * TBP + tid] = m < NIN ? x[m < NIN ? m : 0] : 0.f;
  __syncthreads();
  warp_grad<4, 3, NH, NIN>(T, T + NH * TBP, T);
  block_grad<NH, NIN>(T, out + OFF_W1, out + OFF_B1);
}

// grad[p] = sum over blocks of partial[b][p] in FP64 and a fixed order
// (deterministic).  A block takes 32 parameters, its 32 warps the rows b, b +
// 32, ..., so that a few loads per thread cover the batch's partials.
// ADAM: then the Adam update of the FP32 master parameters and the bfloat16
// copy the next step reads (the loss slot has none).
template <bool ADAM>
__global__ void __launch_bounds__(1024) k_mlp_update(const float *partial, int nblocks, float *grad, float *theta,
                                                     float *mom, float *var, float *wq, float lr, float b1, float b2,
                                                     float eps, float bc1, float bc2) {
  __shared__ double sums[32][33];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int p = blockIdx.x * 32 + lane;
  next_kernel_may_start();
  previous_done();
  double acc = 0.0;
  if (p <= mlp::NPARAM) {
#pragma unroll 8
    for (int b = warp; b < nblocks; b += 32) acc += partial[size_t(b) * (mlp::NPARAM + 1) + p];
  }
  sums[warp][lane] = acc;
  __syncthreads();
  if (warp != 0 || p > mlp::NPARAM) return;
#pragma unroll
  for (int w = 1; w < 32; w++) acc += sums[w][lane];
  const float g = float(acc);
  grad[p] = g;
  if (!ADAM || p >= mlp::NPARAM) return;
  const float mm = b1 * mom[p] + (1.f - b1) * g;
  const float vv = b2 * var[p] + (1.f - b2) * g * g;
  mom[p] = mm;
  var[p] = vv;
  const float th = theta[p] - lr * (mm / bc1) / (sqrtf(vv / bc2) + eps);
  theta[p] = th;
  wq[p] = mlp::is_bias(p) ? th : bf16_round(th);
}

// Forward only, one sample per thread (checks and statistics).
static __global__ void __launch_bounds__(256) k_mlp_eval(const float *__restrict__ wq, const float *__restrict__ xs, long n,
                                                  float *__restrict__ out) {
  using namespace mlp;
  __shared__ float W[NPARAM];
  for (int p = threadIdx.x; p < NPARAM; p += blockDim.x) W[p] = wq[p];
  __syncthreads();
  const long q = long(blockIdx.x) * blockDim.x + threadIdx.x;
  if (q >= n) return;
  float x[NIN], h1[NH], h2[NH], z[NOUT];
#pragma unroll
  for (int m = 0; m < NIN; m++) x[m] = bf16_round(xs[q * NIN + m]);
#pragma unroll
  for (int u = 0; u < NH; u++) {
    float a = W[OFF_B1 + u];
#pragma unroll
    for (int m = 0; m < NIN; m++) a = fmaf(W[OFF_W1 + u * NIN + m], x[m], a);
    h1[u] = bf16_round(fmaxf(a, 0.f));
  }
#pragma unroll
  for (int u = 0; u < NH; u++) {
    float a = W[OFF_B2 + u];
#pragma unroll
    for (int v = 0; v < NH; v++) a = fmaf(W[OFF_W2 + u * NH + v], h1[v], a);
    h2[u] = bf16_round(fmaxf(a, 0.f));
  }
  float zmax = -3.0e38f, se = 0.f;
#pragma unroll
  for (int k = 0; k < NOUT; k++) {
    float a = W[OFF_B3 + k];
#pragma unroll
    for (int u = 0; u < NH; u++) a = fmaf(W[OFF_W3 + k * NH + u], h2[u], a);
    z[k] = a;
    zmax = fmaxf(zmax, a);
  }
#pragma unroll
  for (int k = 0; k < NOUT; k++) {
    z[k] = expf(z[k] - zmax);
    se += z[k];
  }
#pragma unroll
  for (int k = 0; k < NOUT; k++) out[q * NOUT + k] = z[k] / se;
}

// Test entry: tensor-core evaluation of n stencils (already normalised),
// returning the left weights and the mirrored-stencil (right-edge) weights.
static __global__ void __launch_bounds__(128) k_mlp_eval_mma(const uint32_t *__restrict__ frags, const float *__restrict__ xs,
                                                      long n, float *__restrict__ wl_out, float *__restrict__ wr_out) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint4 *sF = reinterpret_cast<uint4 *>(smem_raw);
  uint32_t *sW = reinterpret_cast<uint32_t *>(smem_raw + mlp::FRAG_BYTES + warp * mlp::WARP_SMEM_BYTES);
  load_frags(frags, sF, blockDim.x);
  frags_landed();
  __syncthreads();
  const long q = (long(blockIdx.x) * (blockDim.x >> 5) + warp) * 32 + lane;
  float x[9], wl[5], wr[5];
#pragma unroll
  for (int m = 0; m < 9; m++) x[m] = q < n ? xs[q * 9 + m] : 0.f;
  mlp_warp_weights(sF, sW, x, wl, wr);
  if (q < n) {
#pragma unroll
    for (int k = 0; k < 5; k++) {
      wl_out[q * 5 + k] = wl[k];
      wr_out[q * 5 + k] = wr[k];
    }
  }
}

}  // namespace pu
