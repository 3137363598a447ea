// Fused kernels of the neural operator (learned.cu) for networks of ordinary width.
//
// A pointwise step of the network is a contraction over at most 64 channels plus 16 modes per grid point:
// 4 FP32 multiply-adds per byte that must move, so HBM bounds it and not the arithmetic.  These kernels
// therefore do each step in one pass over the activations: channel mix, spectral term, bias, activation
// (or its derivative) and the bias gradients' partial sums, in FP32 FMAs (packed two to an instruction,
// fma.rn.f32x2) with the weights broadcast from shared memory.  The weight gradients contract over the grid:
// each reads its two fields once, and one kernel adds the blocks' sums of all of them.
//
// Measured (loss and gradients, width 32, 16 modes, 4 layers): 512 x 512 grid, batch 4, 12.2 ms as separate
// products and elementwise kernels (113 launches), 3.5 ms so (38 launches); 64 x 64 grid, batch 16, 1.56 -> 0.85 ms.
#pragma once
#include "common.h"

namespace b200 {
namespace neural {

constexpr int kTile = 256;       // grid points per block
constexpr int kPwThreads = 128;  // two halves of 64 threads: a thread has 4 points (64 apart) and its half's 16 outputs
constexpr int kModes = 16;       // modes per direction, zero-padded

__device__ __forceinline__ float gelu(float x) { return 0.5f * x * (1.f + erff(x * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_grad(float x) {
  return 0.5f * (1.f + erff(x * 0.70710678118654752f)) + x * 0.39894228040143268f * expf(-0.5f * x * x);
}

__device__ __forceinline__ unsigned long long pack2(float x, float y) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ float2 unpack2(unsigned long long v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ void fma2(unsigned long long &d, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
// The 4 points x 16 outputs of a thread, outputs in pairs.
struct Acc {
  unsigned long long v[4][8];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int o = 0; o < 8; ++o) v[u][o] = 0ull;
  }
  __device__ __forceinline__ float get(int u, int o) const {
    const float2 f = unpack2(v[u][o >> 1]);
    return o & 1 ? f.y : f.x;
  }
};
// acc(u, o) += w[o] x[u]; w 16-byte aligned shared memory, the same for every lane.  A uniform 16-byte shared
// load takes the port as long as four of 4 bytes, so 4 points share each: 20 cycles of the port per channel
// and warp for 64 multiply-adds a lane (34 with 2 points and 32 outputs, which bounded pw_kernel at 245 us).
__device__ __forceinline__ void axpy4(Acc &acc, const float *w, const float (&x)[4]) {
  ulonglong2 ww[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) ww[q] = reinterpret_cast<const ulonglong2 *>(w)[q];
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const unsigned long long xx = pack2(x[u], x[u]);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      fma2(acc.v[u][2 * q], ww[q].x, xx);
      fma2(acc.v[u][2 * q + 1], ww[q].y, xx);
    }
  }
}
// acc += W^T X over `channels` rows of the staged tile X ([channel][kTile]) with weights [channel][ldw]
__device__ __forceinline__ void mix16(Acc &acc, const float *X, const float *W, int ldw, int channels, int t) {
#pragma unroll 2
  for (int c = 0; c < channels; ++c) {
    float x[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) x[u] = X[c * kTile + t + 64 * u];
    axpy4(acc, W + c * ldw, x);
  }
}

// a thread's 4 points of its outputs O0..O1-1 to the rows of a [O1 - O0][kTile] tile
template <int O0 = 0, int O1 = 16>
__device__ __forceinline__ void acc_to_tile(const Acc &acc, float *tile, int t) {
#pragma unroll
  for (int o = O0; o < O1; o += 2)
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const float2 f = unpack2(acc.v[u][o >> 1]);
      tile[(o - O0) * kTile + t + 64 * u] = f.x;
      tile[(o + 1 - O0) * kTile + t + 64 * u] = f.y;
    }
}

// Partial sums of a bias gradient over the block's points from the tile R ([channel][kTile]): part[c * stride]
// gets channel c < nc (the blocks' sums are added in order afterwards).
__device__ __forceinline__ void tile_sums(const float *R, int nc, float *part, size_t stride) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __syncthreads();
  for (int c = warp; c < nc; c += kPwThreads / 32) {
    float s = 0.f;
#pragma unroll
    for (int q = 0; q < kTile / 32; ++q) s += R[c * kTile + lane + 32 * q];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) part[c * stride] = s;
  }
}

// Stage `channels` rows of `width` points (from point p0 of fields of P points; zeros past P) in shared memory
// with asynchronous copies, so that a block has its whole tile in flight at once (plain loads in the channel
// loop left 12 KB in flight per SM, and pw_kernel at 360 us where 90 are due to its bytes): 16 bytes each when
// the fields allow it, 4 otherwise.
template <int WIDTH>
__device__ __forceinline__ void stage_tile(float *dst, const float *src, int channels, int P, int p0) {
  const uint32_t d0 = (uint32_t)__cvta_generic_to_shared(dst);
  if ((P & 3) == 0 && ((uintptr_t)src & 15) == 0 && p0 + WIDTH <= P) {
    for (int e = threadIdx.x; e < channels * (WIDTH / 4); e += kPwThreads) {
      const int c = e / (WIDTH / 4), q = e % (WIDTH / 4);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d0 + 16u * (uint32_t)e),
                   "l"(src + (size_t)c * P + p0 + 4 * q)
                   : "memory");
    }
  } else {
    for (int e = threadIdx.x; e < channels * WIDTH; e += kPwThreads) {
      const int c = e / WIDTH, q = e % WIDTH;
      const bool in = p0 + q < P;
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d0 + 4u * (uint32_t)e),
                   "l"(src + (in ? (size_t)c * P + p0 + q : 0)), "r"(in ? 4 : 0)
                   : "memory");
    }
  }
}
__device__ __forceinline__ void stage_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void stage_wait() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

struct PwArgs {
  const float *X;        // input, batch x Ci x P
  int Ci, Co, N, P;
  const float *Wt;       // weight of (output o, input c) at o * wo + c * wc
  int wo, wc;
  const float *T2;       // spectral weights, batch x Co x N x M (null: no spectral term)
  const float *Sp;       // N x kModes sine basis, zero past M
  int M;
  const float *bias;     // Co (null: none)
  const float *Ug;       // multiply the result by gelu'(Ug) (null: no)
  float *U;              // the result before the activation (null: not wanted)
  float *V;              // the result, through gelu when act
  int act;
  float *part;           // partial bias-gradient sums of the result, [Co][blocks] (null: none)
};

// out(o, p) = sum_c Wt(o, c) X(c, p) + sum_m T2(o, i, m) S(j, m) + bias(o) at the grid points p = i N + j of
// sample blockIdx.y, outputs [32 z, 32 (z+1)) for z = blockIdx.z.  The spectral term enters as M further inputs
// S(j, m) whose weights belong to the point's image row.
//
// Bound: HBM, one read of X (and Ug), one write of U and V (512 x 512 grid, batch 4, width 32: 403 MB, 62 us), and
// beside it the issue slots of erff.  Measured there: 170 us forward, 196 us with gelu' in the backward pass,
// where the separate products and elementwise kernels of a layer took 740 us.
__global__ void __launch_bounds__(kPwThreads) pw_kernel(PwArgs a) {
  extern __shared__ __align__(16) float sm[];
  const int tid = threadIdx.x, t = tid & 63, half = tid >> 6;
  const int b = blockIdx.y, o0 = blockIdx.z * 32, p0 = blockIdx.x * kTile, no = min(32, a.Co - o0);
  float *Xs = sm;                                 // [max(Ci, 32)][kTile]: the input, then the result
  float *Gs = Xs + max(a.Ci, 32) * kTile;         // [32][kTile], with Ug
  float *W = Gs + (a.Ug ? 32 * kTile : 0);        // [Ci][32]
  float *T2 = W + a.Ci * 32;                      // [row][kModes][32]
  stage_tile<kTile>(Xs, a.X + (size_t)b * a.Ci * a.P, a.Ci, a.P, p0);
  if (a.Ug) stage_tile<kTile>(Gs, a.Ug + ((size_t)b * a.Co + o0) * a.P, no, a.P, p0);
  stage_commit();
  for (int e = tid; e < a.Ci * 32; e += kPwThreads) {
    // neighbouring threads take neighbouring weights
    const int c = a.wc == 1 ? e % a.Ci : e >> 5, o = a.wc == 1 ? e / a.Ci : e & 31;
    W[c * 32 + o] = o < no ? __ldg(a.Wt + (o0 + o) * a.wo + c * a.wc) : 0.f;
  }
  const int i0 = p0 / a.N, nrows = (min(p0 + kTile, a.P) - 1) / a.N - i0 + 1;
  if (a.T2)
    for (int e = tid; e < nrows * kModes * 32; e += kPwThreads) {
      const int m = e & 15, r = (e >> 4) % nrows, o = (e >> 4) / nrows;
      T2[(r * kModes + m) * 32 + o] =
          o < no && m < a.M ? __ldg(a.T2 + ((size_t)(b * a.Co + o0 + o) * a.N + i0 + r) * a.M + m) : 0.f;
    }
  Acc acc;
#pragma unroll
  for (int o = 0; o < 16; o += 2) {
    const int q = 16 * half + o;
    const float b0 = a.bias && q < no ? __ldg(a.bias + o0 + q) : 0.f, b1 = a.bias && q + 1 < no ? __ldg(a.bias + o0 + q + 1) : 0.f;
#pragma unroll
    for (int u = 0; u < 4; ++u) acc.v[u][o >> 1] = pack2(b0, b1);
  }
  stage_wait();
  __syncthreads();
  mix16(acc, Xs, W + 16 * half, 32, a.Ci, t);
  if (a.T2) {
    const float *s[4];
    int row[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int p = min(p0 + t + 64 * u, a.P - 1), i = p / a.N;
      row[u] = i - i0;
      s[u] = a.Sp + (size_t)(p - i * a.N) * kModes;
    }
    if (nrows == 1) {
      for (int m = 0; m < a.M; m += 4) {
        float4 q[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) q[u] = __ldg(reinterpret_cast<const float4 *>(s[u] + m));
        const float x0[4] = {q[0].x, q[1].x, q[2].x, q[3].x}, x1[4] = {q[0].y, q[1].y, q[2].y, q[3].y};
        const float x2[4] = {q[0].z, q[1].z, q[2].z, q[3].z}, x3[4] = {q[0].w, q[1].w, q[2].w, q[3].w};
        axpy4(acc, T2 + m * 32 + 16 * half, x0);
        axpy4(acc, T2 + (m + 1) * 32 + 16 * half, x1);
        axpy4(acc, T2 + (m + 2) * 32 + 16 * half, x2);
        axpy4(acc, T2 + (m + 3) * 32 + 16 * half, x3);
      }
    } else {  // points of several image rows: each its own weights
      for (int m = 0; m < a.M; ++m)
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const ulonglong2 *w = reinterpret_cast<const ulonglong2 *>(T2 + (row[u] * kModes + m) * 32 + 16 * half);
          const float x = __ldg(s[u] + m);
          const unsigned long long xx = pack2(x, x);
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const ulonglong2 ww = w[q];
            fma2(acc.v[u][2 * q], ww.x, xx);
            fma2(acc.v[u][2 * q + 1], ww.y, xx);
          }
        }
    }
  }
  // The activation runs in a rolled loop over the results in shared memory: unrolled over a thread's 64
  // registers its code overflows the instruction cache (1.3 of 6 stall cycles per instruction).
  __syncthreads();  // the staged input is consumed
  float *R = Xs;    // [32][kTile]
  acc_to_tile(acc, R + 16 * half * kTile, t);
  float *mine = R + 16 * half * kTile + t;
  const float *ug = Gs + 16 * half * kTile + t;
  const size_t at0 = ((size_t)b * a.Co + o0 + 16 * half) * a.P + p0 + t;
  const int mo = min(16, no - 16 * half);
#pragma unroll 1
  for (int o = 0; o < mo; ++o) {
    const size_t at = at0 + (size_t)o * a.P;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const bool in = p0 + t + 64 * u < a.P;
      float x = mine[o * kTile + 64 * u];
      if (a.U && in) a.U[at + 64 * u] = x;
      if (a.Ug) x *= gelu_grad(ug[o * kTile + 64 * u]);
      if (a.act) x = gelu(x);
      if (in) a.V[at + 64 * u] = x;
      if (a.part) mine[o * kTile + 64 * u] = in ? x : 0.f;
    }
  }
  if (a.part) {
    const size_t blocks = (size_t)gridDim.x * gridDim.y;
    tile_sums(R, no, a.part + (size_t)o0 * blocks + (size_t)b * gridDim.x + blockIdx.x, blocks);
  }
}

// Projection, forward: Z = Q1 V + q1, H = gelu(Z), Y = Q2 H + q2 (at most 16 outputs), 32 hidden channels at a
// time (16 per half of the block; the halves' shares of Y meet at the end): V is read once, Z, H and Y are
// written once.  Z and H pass through shared memory 8 channels of a half at a time: three blocks fit an SM
// (with proj_bwd_kernel's, loss and gradients of 512 x 512, batch 4 take 3.60 ms instead of 3.76).
__global__ void __launch_bounds__(kPwThreads, 3) proj_fwd_kernel(const float *__restrict__ V, int W, int H, int K, int P,
                                                              const float *__restrict__ Q1, const float *__restrict__ q1,
                                                              const float *__restrict__ Q2, const float *__restrict__ q2,
                                                              float *Z, float *Hh, float *Y) {
  extern __shared__ __align__(16) float sm[];
  const int Hp = (H + 31) & ~31;
  float *Xs = sm;              // [W][kTile]
  float *Hs = Xs + W * kTile;  // [2][8][kTile]: Z then H of 8 channels per half; at the end the second half's share of Y
  float *w1 = Hs + 16 * kTile; // [W][Hp]
  float *w2 = w1 + W * Hp;     // [Hp][16]
  float *b1 = w2 + Hp * 16;    // [Hp]
  const int tid = threadIdx.x, t = tid & 63, half = tid >> 6, b = blockIdx.y, p0 = blockIdx.x * kTile;
  stage_tile<kTile>(Xs, V + (size_t)b * W * P, W, P, p0);
  stage_commit();
  for (int e = tid; e < W * Hp; e += kPwThreads) w1[e % W * Hp + e / W] = e / W < H ? Q1[e] : 0.f;
  for (int e = tid; e < Hp * 16; e += kPwThreads) w2[e] = e / 16 < H && e % 16 < K ? Q2[(e % 16) * H + e / 16] : 0.f;
  for (int e = tid; e < Hp; e += kPwThreads) b1[e] = e < H ? q1[e] : 0.f;
  stage_wait();
  __syncthreads();
  Acc y;
  y.zero();
  float *mine = Hs + 8 * half * kTile;  // a thread reads and writes its own points of its half's channels only
  for (int h0 = 16 * half; h0 < Hp; h0 += 32) {
    Acc z;
#pragma unroll
    for (int o = 0; o < 8; ++o)
#pragma unroll
      for (int u = 0; u < 4; ++u) z.v[u][o] = pack2(b1[h0 + 2 * o], b1[h0 + 2 * o + 1]);
    mix16(z, Xs, w1 + h0, Hp, W, t);
#pragma unroll
    for (int part = 0; part < 2; ++part) {
      const int h8 = h0 + 8 * part, mh = min(8, H - h8);
      if (part == 0) acc_to_tile<0, 8>(z, mine, t);
      else acc_to_tile<8, 16>(z, mine, t);
#pragma unroll 1
      for (int h = 0; h < mh; ++h) {
        const size_t at = ((size_t)b * H + h8 + h) * P + p0 + t;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          float *z1 = mine + h * kTile + t + 64 * u;
          const float x = *z1, g = gelu(x);
          *z1 = g;
          if (p0 + t + 64 * u < P) {
            Z[at + 64 * u] = x;
            Hh[at + 64 * u] = g;
          }
        }
      }
      mix16(y, mine, w2 + h8 * 16, 16, max(mh, 0), t);
    }
  }
  __syncthreads();
  if (half) acc_to_tile(y, Hs, t);
  __syncthreads();
  if (!half) {
#pragma unroll
    for (int k = 0; k < 16; ++k)
      if (k < K) {
        const float bk = q2[k];
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (p0 + t + 64 * u < P)
            Y[((size_t)b * K + k) * P + p0 + t + 64 * u] = (y.get(u, k) + Hs[k * kTile + t + 64 * u]) + bk;
      }
  }
}

// Loss, first stage: block (slice, k, b) sums y u and y y over its slice of the points.
constexpr int kLossSlice = 4096;
__global__ void __launch_bounds__(256) loss_part_kernel(const float *__restrict__ Y, const float *__restrict__ T, int K,
                                                        int P, float2 *part) {
  __shared__ float r1[8], r2[8];
  const int k = blockIdx.y, b = blockIdx.z;
  const size_t base = ((size_t)b * K + k) * P;
  const int p1 = min(P, (int)(blockIdx.x + 1) * kLossSlice);
  float yu = 0.f, yy = 0.f;
#pragma unroll 4
  for (int p = blockIdx.x * kLossSlice + threadIdx.x; p < p1; p += 256) {
    const float y = Y[base + p], u = T[base + p];
    yu = fmaf(y, u, yu);
    yy = fmaf(y, y, yy);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    yu += __shfl_xor_sync(0xffffffffu, yu, o);
    yy += __shfl_xor_sync(0xffffffffu, yy, o);
  }
  if ((threadIdx.x & 31) == 0) {
    r1[threadIdx.x >> 5] = yu;
    r2[threadIdx.x >> 5] = yy;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w) {
      yu += r1[w];
      yy += r2[w];
    }
    part[((size_t)b * K + k) * gridDim.x + blockIdx.x] = make_float2(yu, yy);
  }
}
// Second stage: loss_bk = 1 - (y.u)^2/(y.y), and dY = cu u + cy y over the block's slice (dY null, one block per (k, b):
// the loss alone).  Every block adds the slices' sums in their order for itself, which costs less than a launch between.
// dY is formed here and not in the backward pass: once the loss can be read, no kernel reads the caller's targets.
__global__ void __launch_bounds__(256) loss_final_kernel(const float2 *__restrict__ part, int slices, int K, int P,
                                                         float scale, const float *__restrict__ Y,
                                                         const float *__restrict__ T, float *loss_bk, float *dY) {
  __shared__ float2 sums[256], coef;
  const int e = blockIdx.z * K + blockIdx.y;
  float yu = 0.f, yy = 0.f;
  for (int s0 = 0; s0 < slices; s0 += 256) {
    if (s0 + (int)threadIdx.x < slices) sums[threadIdx.x] = __ldg(part + (size_t)e * slices + s0 + threadIdx.x);
    __syncthreads();
    if (threadIdx.x == 0)
#pragma unroll 8
      for (int s = 0; s < min(256, slices - s0); ++s) {
        yu += sums[s].x;
        yy += sums[s].y;
      }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    yy = fmaxf(yy, 1e-30f);
    if (blockIdx.x == 0) loss_bk[e] = 1.f - yu * yu / yy;
    coef = make_float2(-2.f * yu / yy * scale, 2.f * yu * yu / (yy * yy) * scale);
  }
  if (!dY) return;
  __syncthreads();
  const size_t base = (size_t)e * P;
  const float cu = coef.x, cy = coef.y;
  const int p1 = min(P, (int)(blockIdx.x + 1) * kLossSlice);
#pragma unroll 4
  for (int p = blockIdx.x * kLossSlice + threadIdx.x; p < p1; p += 256)
    dY[base + p] = cu * __ldg(T + base + p) + cy * __ldg(Y + base + p);
}

// Projection, backward: dH = Q2^T dY, dZ = dH gelu'(Z) (written for the gradient of Q1), dV = Q1^T dZ for at most 32
// channels per blockIdx.z, and the partial sums of dq2, dq1 (z = 0) and of dV.  Hidden channels go 32 at a time;
// gelu' replaces Z in place before dH is formed, so that one tile serves all three and three blocks fit an SM.
__global__ void __launch_bounds__(kPwThreads, 3) proj_bwd_kernel(const float *__restrict__ dY, const float *__restrict__ Z,
                                                              int W, int H, int K, int P, const float *__restrict__ Q1,
                                                              const float *__restrict__ Q2, float *dZ, float *dV,
                                                              float *part_k, float *part_h, float *part_w) {
  extern __shared__ __align__(16) float sm[];
  const int Hp = (H + 31) & ~31, c0 = blockIdx.z * 32, nc = min(32, W - c0);
  float *Zs = sm;                  // [32][kTile]: Z of the group, then gelu'(Z), then dZ; at the end dV
  float *Ys = Zs + 32 * kTile;     // [K][kTile]: dY
  float *w2 = Ys + K * kTile;      // [K][Hp]
  float *w1 = w2 + K * Hp;         // [Hp][32]
  const int tid = threadIdx.x, t = tid & 63, half = tid >> 6, b = blockIdx.y, p0 = blockIdx.x * kTile;
  const bool first = blockIdx.z == 0;
  const size_t blocks = (size_t)gridDim.x * gridDim.y, blk = (size_t)b * gridDim.x + blockIdx.x;
  stage_tile<kTile>(Zs, Z + (size_t)b * H * P, min(32, H), P, p0);
  stage_tile<kTile>(Ys, dY + (size_t)b * K * P, K, P, p0);  // zero past P
  stage_commit();
  for (int e = tid; e < K * Hp; e += kPwThreads) w2[e] = e % Hp < H ? Q2[(e / Hp) * H + e % Hp] : 0.f;
  for (int e = tid; e < Hp * 32; e += kPwThreads)
    w1[e] = (e >> 5) < H && (e & 31) < nc ? Q1[(e >> 5) * W + c0 + (e & 31)] : 0.f;
  stage_wait();
  if (first) tile_sums(Ys, K, part_k + blk, blocks);
  Acc g;
  g.zero();
  float *zh = Zs + 16 * half * kTile + t;
  for (int g0 = 0; g0 < H; g0 += 32) {
    stage_wait();
    __syncthreads();
    const int h0 = g0 + 16 * half, mh = min(16, H - h0);
    // a thread's own points and channels: no barrier
#pragma unroll 1
    for (int h = 0; h < mh; ++h)
#pragma unroll
      for (int u = 0; u < 4; ++u) zh[h * kTile + 64 * u] = gelu_grad(zh[h * kTile + 64 * u]);
    {
      Acc d;
      d.zero();
      mix16(d, Ys, w2 + h0, Hp, K, t);
#pragma unroll
      for (int h = 0; h < 16; ++h)
        if (h < mh) {
          const size_t at = ((size_t)b * H + h0 + h) * P + p0 + t;
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const float x = d.get(u, h) * zh[h * kTile + 64 * u];  // dY = 0 past P
            zh[h * kTile + 64 * u] = x;
            if (first && p0 + t + 64 * u < P) dZ[at + 64 * u] = x;
          }
        }
    }
    const int mg = min(32, H - g0);
    if (first) tile_sums(Zs, mg, part_h + (size_t)g0 * blocks + blk, blocks);
    else __syncthreads();
    mix16(g, Zs, w1 + g0 * 32 + 16 * half, 32, mg, t);
    __syncthreads();
    if (g0 + 32 < H) {
      stage_tile<kTile>(Zs, Z + ((size_t)b * H + g0 + 32) * P, min(32, H - g0 - 32), P, p0);
      stage_commit();
    }
  }
  acc_to_tile(g, Zs + 16 * half * kTile, t);
#pragma unroll 2
  for (int o = 0; o < min(16, nc - 16 * half); ++o) {
    const size_t at = ((size_t)b * W + c0 + 16 * half + o) * P + p0 + t;
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (p0 + t + 64 * u < P) dV[at + 64 * u] = zh[o * kTile + 64 * u];  // zero past P
  }
  tile_sums(Zs, nc, part_w + (size_t)c0 * blocks + blk, blocks);
}

// C[z] (M x M) = S^T X[z] S for the fields z = blockIdx.x of N x N points, 128 columns per block (blockIdx.y): the
// rows stream through a ring of shared-memory stages (32 rows of X and of S each), each warp forms T1 = S^T X
// over its rows with four columns per lane (they share the loads of S), the warps' shares are added in order,
// and the block multiplies by S.  The blocks of a field leave their shares in work, and the last to finish adds
// them in order (count: one zeroed word per field, zero again afterwards).  Bound: HBM, one read of X.
// 128 fields of 512 x 512: 56 us (134 MB, 21 us); with loads into registers instead of the stages 130 to 186 us.
constexpr int kModeThreads = 256;
constexpr int kModeCols = 128;
constexpr int kModeWarps = kModeThreads / 32;
constexpr int kModeRows = 32;    // rows of a stage
constexpr int kModeStages = 3;
constexpr int kModeStage = kModeRows * (kModeCols + kModes);  // floats of a stage
constexpr size_t kModeSmem = sizeof(float) * kModeStages * kModeStage;
__global__ void __launch_bounds__(kModeThreads, 2) modes_kernel(const float *__restrict__ X, const float *__restrict__ Sp,
                                                                int N, int M, float *C, float *work, unsigned *count) {
  extern __shared__ __align__(16) float sm[];  // the stages; then the warps' shares of T1, half of them at a time
  static_assert(kModeWarps / 2 * kModes * kModeCols <= kModeStages * kModeStage, "T1 shares fit the stages");
  __shared__ int last;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int j0 = blockIdx.y * kModeCols, nst = (N + kModeRows - 1) / kModeRows;
  const float *F = X + (size_t)blockIdx.x * N * N;
  const uint32_t sm0 = (uint32_t)__cvta_generic_to_shared(sm);
  const bool wide = (N & 3) == 0 && ((uintptr_t)X & 15) == 0;
  auto load = [&](int st) {
    if (st < nst) {
      const int i0 = st * kModeRows;
      const uint32_t xs = sm0 + 4u * (uint32_t)(st % kModeStages * kModeStage), ss = xs + 4u * kModeRows * kModeCols;
      if (wide) {
        for (int e = tid; e < kModeRows * kModeCols / 4; e += kModeThreads) {
          const int i = i0 + (e >> 5), j = j0 + 4 * (e & 31);
          const bool in = i < N && j < N;
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(xs + 16u * (uint32_t)e),
                       "l"(F + (in ? (size_t)i * N + j : 0)), "r"(in ? 16 : 0)
                       : "memory");
        }
      } else {
        for (int e = tid; e < kModeRows * kModeCols; e += kModeThreads) {
          const int i = i0 + (e >> 7), j = j0 + (e & 127);
          const bool in = i < N && j < N;
          asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(xs + 4u * (uint32_t)e),
                       "l"(F + (in ? (size_t)i * N + j : 0)), "r"(in ? 4 : 0)
                       : "memory");
        }
      }
      if (tid < kModeRows * kModes / 4) {
        const int i = i0 + (tid >> 2);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(ss + 16u * (uint32_t)tid),
                     "l"(Sp + (i < N ? (size_t)i * kModes + 4 * (tid & 3) : 0)), "r"(i < N ? 16 : 0)
                     : "memory");
      }
    }
    stage_commit();
  };
  unsigned long long acc[4][kModes / 2];
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int q = 0; q < kModes / 2; ++q) acc[u][q] = 0ull;
#pragma unroll
  for (int st = 0; st < kModeStages - 1; ++st) load(st);
  for (int st = 0; st < nst; ++st) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kModeStages - 2) : "memory");
    __syncthreads();  // stage st has landed, stage st - 1 is consumed
    load(st + kModeStages - 1);
    const float *xs = sm + st % kModeStages * kModeStage, *ss = xs + kModeRows * kModeCols;
#pragma unroll
    for (int r = 0; r < kModeRows / kModeWarps; ++r) {
      const int row = r * kModeWarps + warp;
      const float4 x = *reinterpret_cast<const float4 *>(xs + row * kModeCols + 4 * lane);
      const unsigned long long xx[4] = {pack2(x.x, x.x), pack2(x.y, x.y), pack2(x.z, x.z), pack2(x.w, x.w)};
#pragma unroll
      for (int q = 0; q < kModes / 4; ++q) {
        const ulonglong2 s2 = reinterpret_cast<const ulonglong2 *>(ss + row * kModes)[q];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          fma2(acc[u][2 * q], s2.x, xx[u]);
          fma2(acc[u][2 * q + 1], s2.y, xx[u]);
        }
      }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  // T1 of the 128 columns: warps 4..7 leave theirs, warps 0..3 add theirs, then the four sums in order
  auto row4 = [&](int w, int q) { return reinterpret_cast<float4 *>(sm + (w * kModes + q) * kModeCols + 4 * lane); };
  auto value = [&](int q, int u) {
    const float2 f = unpack2(acc[u][q >> 1]);
    return q & 1 ? f.y : f.x;
  };
  if (warp >= kModeWarps / 2)
#pragma unroll
    for (int q = 0; q < kModes; ++q)
      *row4(warp - kModeWarps / 2, q) = make_float4(value(q, 0), value(q, 1), value(q, 2), value(q, 3));
  __syncthreads();
  if (warp < kModeWarps / 2)
#pragma unroll
    for (int q = 0; q < kModes; ++q) {
      float4 v = *row4(warp, q);
      v.x += value(q, 0);
      v.y += value(q, 1);
      v.z += value(q, 2);
      v.w += value(q, 3);
      *row4(warp, q) = v;
    }
  __syncthreads();
  for (int e = tid; e < kModes * kModeCols; e += kModeThreads) {
    float s = sm[e];
#pragma unroll
    for (int h = 1; h < kModeWarps / 2; ++h) s += sm[h * kModes * kModeCols + e];
    sm[e] = s;
  }
  __syncthreads();
  const int k = tid >> 4, m = tid & 15, jn = min(kModeCols, N - j0);
  float part[4] = {0.f, 0.f, 0.f, 0.f};
  for (int j = 0; j < jn; j += 4) {
    const float4 v = *reinterpret_cast<const float4 *>(sm + k * kModeCols + j);  // zeros past N
    const float *s = Sp + (size_t)(j0 + j) * kModes + m;
    part[0] = fmaf(v.x, __ldg(s), part[0]);
    if (j + 1 < jn) part[1] = fmaf(v.y, __ldg(s + kModes), part[1]);
    if (j + 2 < jn) part[2] = fmaf(v.z, __ldg(s + 2 * kModes), part[2]);
    if (j + 3 < jn) part[3] = fmaf(v.w, __ldg(s + 3 * kModes), part[3]);
  }
  const float total = (part[0] + part[1]) + (part[2] + part[3]);
  float *out = C + (size_t)blockIdx.x * M * M + k * M + m;
  const bool mine = k < M && m < M;
  if (gridDim.y == 1) {
    if (mine) *out = total;
    return;
  }
  float *w = work + (size_t)blockIdx.x * gridDim.y * kModeThreads;
  w[(size_t)blockIdx.y * kModeThreads + tid] = total;
  __threadfence();
  __syncthreads();
  if (tid == 0) last = atomicAdd(count + blockIdx.x, 1u) == gridDim.y - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  float s = 0.f;
#pragma unroll 4
  for (unsigned q = 0; q < gridDim.y; ++q) s += __ldcg(w + (size_t)q * kModeThreads + tid);
  if (mine) *out = s;
  if (tid == 0) count[blockIdx.x] = 0;
}

// Per-mode channel mix and the first half of the way back to the grid, one block per (channel x, sample b), one
// thread per mode q = (k, m): D(q) = sum_y R(...) in(b, y, q) with R(o, c, q) at (o W + c) M2 + q (transposed = 0:
// x = o, y = c, forward; 1: x = c, y = o, backward), then T2(b, x, i, m) = sum_k S(i, k) D(k, m) for every image
// row i.  Blocks past W B form dR(o, c, q) = sum_b dD(b, o, q) C(b, c, q) instead (backward only).
__global__ void __launch_bounds__(256) mode_mix_kernel(const float *__restrict__ R, const float *__restrict__ in,
                                                       const float *__restrict__ Sp, float *T2, int B, int W, int N, int M,
                                                       int transposed, const float *__restrict__ C, float *dR) {
  __shared__ float D[kModes * kModes];
  const int M2 = M * M, q = threadIdx.x;
  int x = blockIdx.x;
  if (x < W * B) {
    const int b = x / W;
    x %= W;
    float acc = 0.f;
    if (q < M2) {
#pragma unroll 16
      for (int y = 0; y < W; ++y)
        acc = fmaf(__ldg(R + ((size_t)(transposed ? y * W + x : x * W + y)) * M2 + q),
                   __ldg(in + ((size_t)b * W + y) * M2 + q), acc);
      D[q] = acc;
    }
    __syncthreads();
    float *out = T2 + ((size_t)b * W + x) * N * M;
    const int m = q & 15;
    if (m < M) {
      float d[kModes];
#pragma unroll
      for (int k = 0; k < kModes; ++k) d[k] = k < M ? D[k * M + m] : 0.f;
#pragma unroll 4
      for (int i = q >> 4; i < N; i += 16) {
        const float4 *s = reinterpret_cast<const float4 *>(Sp + (size_t)i * kModes);
        float t = 0.f;
#pragma unroll
        for (int k = 0; k < kModes; k += 4) {
          const float4 v = __ldg(s + k / 4);
          t = fmaf(v.x, d[k], t);
          t = fmaf(v.y, d[k + 1], t);
          t = fmaf(v.z, d[k + 2], t);
          t = fmaf(v.w, d[k + 3], t);
        }
        out[i * M + m] = t;
      }
    }
    return;
  }
  if (q >= M2) return;
  x -= W * B;  // o W + c
  const int o = x / W, c = x % W;
  float s = 0.f;
#pragma unroll 4
  for (int b = 0; b < B; ++b)
    s = fmaf(__ldg(in + ((size_t)b * W + o) * M2 + q), __ldg(C + ((size_t)b * W + c) * M2 + q), s);
  dR[(size_t)x * M2 + q] = s;
}

// Bias gradients from the blocks' partial sums: block s sums row s of part and stores it at grads[off].
struct BiasRows {
  int count;                 // tensors
  int first[20];             // first row of each
  int blocks[20];            // partial sums per row
  long long at[20];          // element of the first partial sum of each
  long long off[20];         // offset in the gradient array
};
__global__ void __launch_bounds__(128) bias_rows_kernel(const float *__restrict__ part, BiasRows r, float *grads) {
  __shared__ float red[128];
  int t = 0;
  while (t + 1 < r.count && (int)blockIdx.x >= r.first[t + 1]) ++t;
  const int c = blockIdx.x - r.first[t], n = r.blocks[t];
  const float *p = part + r.at[t] + (size_t)c * n;
  float s = 0.f;
  for (int e = threadIdx.x; e < n; e += 128) s += p[e];
  red[threadIdx.x] = s;
  __syncthreads();
  for (int w = 64; w > 0; w >>= 1) {
    if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) grads[r.off[t] + c] = red[0];
}

// Weight gradients C[i][j] = sum over the batch and the points of A[b][i][p] B[b][j][p].  A block takes 32 rows of A
// and 8 NV of B over its share of the 64-point chunks (blockIdx.x: tile of the output, blockIdx.y: share), staged by
// asynchronous copies in a ring of kGradStages chunks.  Each of the four warps takes 16 of the 64 points; lane
// (gi, gj) = (lane / 8, lane % 8) holds rows gi + 4 u and columns gj + 8 v (rows 68 floats apart: the loads of four
// points of eight rows hit distinct banks), even and odd points in the halves of packed FP32 FMAs.  The block's
// sums go to part[tile][share][i][j]; grad_final_kernel adds the shares of every tensor in a fixed order.
// Bound: HBM (32 x 32 over 4 x 512^2 points: 268 MB, 42 us) and FP32 FMAs (30 us).
// Measured there 69 us, a split-depth tensor-core product with its own sum 165 (3-product TF32); 64 x 32 130 against
// 294, 32 x 3 33 against 128; the sums of all seven gradients 10 us in one launch against 14 each.
constexpr int kGradThreads = 128, kGradPoints = 64, kGradLd = kGradPoints + 4, kGradStages = 4, kGradCtasPerSm = 3;
__host__ __device__ constexpr size_t grad_smem(int nv) {
  return sizeof(float) * (size_t)kGradStages * (32 + 8 * nv) * kGradLd;
}
template <int NV>
__global__ void __launch_bounds__(kGradThreads) grad_kernel(const float *__restrict__ A, int ma, const float *__restrict__ B,
                                                          int mb, int batch, int P, int vec, float *part) {
  extern __shared__ __align__(16) float gsm[];
  constexpr int kRows = 32 + 8 * NV, kStage = kRows * kGradLd;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, gi = lane >> 3, gj = lane & 7;
  const int jt = (mb + 8 * NV - 1) / (8 * NV), i0 = blockIdx.x / jt * 32, j0 = blockIdx.x % jt * (8 * NV);
  const int ra = min(32, ma - i0), rb = min(8 * NV, mb - j0);
  const int per = (P + kGradPoints - 1) / kGradPoints;  // chunks of a field
  const long long total = (long long)batch * per;
  const long long c0 = total * blockIdx.y / gridDim.y, c1 = total * (blockIdx.y + 1) / gridDim.y;
  const int n = (int)(c1 - c0);
  for (int e = tid; e < kGradStages * kStage; e += kGradThreads) gsm[e] = 0.f;  // rows past ra, rb stay zero
  __syncthreads();
  int b = (int)(c0 / per), c = (int)(c0 - (long long)b * per);  // the next chunk to stage
  auto load = [&](int st) {
    if (st < n) {
      const uint32_t d = (uint32_t)__cvta_generic_to_shared(gsm + st % kGradStages * kStage);
      const int p0 = c * kGradPoints;
      const float *a = A + ((size_t)b * ma + i0) * P + p0, *x = B + ((size_t)b * mb + j0) * P + p0;
      if (vec) {
#pragma unroll
        for (int e = tid; e < kRows * (kGradPoints / 4); e += kGradThreads) {
          const int r = e / (kGradPoints / 4), q = 4 * (e % (kGradPoints / 4)), rr = r < 32 ? r : r - 32;
          if (rr < (r < 32 ? ra : rb)) {
            const bool in = p0 + q < P;
            const float *src = (r < 32 ? a : x) + (size_t)rr * P + (in ? q : 0);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d + 4u * (uint32_t)(r * kGradLd + q)),
                         "l"(src), "r"(in ? 16 : 0)
                         : "memory");
          }
        }
      } else {
        for (int e = tid; e < kRows * kGradPoints; e += kGradThreads) {
          const int r = e / kGradPoints, q = e % kGradPoints, rr = r < 32 ? r : r - 32;
          if (rr < (r < 32 ? ra : rb)) {
            const bool in = p0 + q < P;
            const float *src = (r < 32 ? a : x) + (size_t)rr * P + (in ? q : 0);
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d + 4u * (uint32_t)(r * kGradLd + q)),
                         "l"(src), "r"(in ? 4 : 0)
                         : "memory");
          }
        }
      }
      if (++c == per) {
        c = 0;
        ++b;
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  unsigned long long acc[8][NV];
#pragma unroll
  for (int u = 0; u < 8; ++u)
#pragma unroll
    for (int v = 0; v < NV; ++v) acc[u][v] = 0ull;
#pragma unroll
  for (int st = 0; st < kGradStages - 1; ++st) load(st);
  for (int st = 0; st < n; ++st) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kGradStages - 2) : "memory");
    __syncthreads();  // chunk st has landed, chunk st - 1 is consumed
    load(st + kGradStages - 1);
    const float *s = gsm + st % kGradStages * kStage + 16 * warp;
#pragma unroll
    for (int q = 0; q < 16; q += 4) {
      ulonglong2 bv[NV];
#pragma unroll
      for (int v = 0; v < NV; ++v) bv[v] = *reinterpret_cast<const ulonglong2 *>(s + (32 + gj + 8 * v) * kGradLd + q);
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const ulonglong2 av = *reinterpret_cast<const ulonglong2 *>(s + (gi + 4 * u) * kGradLd + q);
#pragma unroll
        for (int v = 0; v < NV; ++v) {
          fma2(acc[u][v], av.x, bv[v].x);
          fma2(acc[u][v], av.y, bv[v].y);
        }
      }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  constexpr int kOut = 32 * 8 * NV;  // four warps' sums fit the ring: 4 kOut <= kGradStages kStage
#pragma unroll
  for (int u = 0; u < 8; ++u)
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      const float2 h = unpack2(acc[u][v]);
      gsm[warp * kOut + (gi + 4 * u) * (8 * NV) + gj + 8 * v] = h.x + h.y;
    }
  __syncthreads();
  float *out = part + ((size_t)blockIdx.x * gridDim.y + blockIdx.y) * kOut;
  for (int e = tid; e < kOut; e += kGradThreads)
    out[e] = (gsm[e] + gsm[kOut + e]) + (gsm[2 * kOut + e] + gsm[3 * kOut + e]);
}

// A tensor's partial sums: output (i, j) of tile t at part[at + ((t * shares + share) * 32 + i % 32) * cols + j % cols],
// to grads[off + i * si + j * sj].
struct GradTensor {
  int first;          // first block of grad_final_kernel
  int ma, mb, cols, shares, si, sj;
  long long at, off;
};
struct GradTable {
  int count;
  GradTensor t[20];
};
// A block takes 32 consecutive outputs of a tile; its 8 warps every eighth share, eight loads in flight.
__global__ void __launch_bounds__(256) grad_final_kernel(const float *__restrict__ part, const __grid_constant__ GradTable tab,
                                                         float *grads) {
  __shared__ float red[8][32];
  int k = 0;
  while (k + 1 < tab.count && (int)blockIdx.x >= tab.t[k + 1].first) ++k;
  const GradTensor &t = tab.t[k];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, outs = 32 * t.cols;
  const int e0 = (blockIdx.x - t.first) * 32 + lane, tile = e0 / outs, e = e0 - tile * outs;
  const float *p = part + t.at + (size_t)tile * t.shares * outs + e;
  float acc = 0.f;
  for (int s0 = warp; s0 < t.shares; s0 += 64) {
    float v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] = s0 + 8 * u < t.shares ? __ldcg(p + (size_t)(s0 + 8 * u) * outs) : 0.f;
#pragma unroll
    for (int u = 0; u < 8; ++u) acc += v[u];
  }
  red[warp][lane] = acc;
  __syncthreads();
  if (warp != 0) return;
#pragma unroll
  for (int w = 1; w < 8; ++w) acc += red[w][lane];
  const int jt = (t.mb + t.cols - 1) / t.cols, i = tile / jt * 32 + e / t.cols, j = tile % jt * t.cols + e % t.cols;
  if (i < t.ma && j < t.mb) grads[t.off + (long long)i * t.si + (long long)j * t.sj] = acc;
}

}  // namespace neural
}  // namespace b200
