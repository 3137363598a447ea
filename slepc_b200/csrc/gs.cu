// Fused classical Gram-Schmidt with DGKS refinement for sm_100a: one cooperative launch per column.
//
// Replaces the BV Gram-Schmidt path of SLEPc:
//   BVOrthogonalizeGS (src/sys/classes/bv/interface/bvorthog.c:145-217)
//   BVOrthogonalizeCGS1 (bvorthog.c:91-132) with BVDotColumnInc (:32-47),
//   BVMultColumn (bvops.c:165), BV_SquareRoot / BV_SquareSum / BV_AddCoefficients
//   (include/slepc/private/bvimpl.h:121-141, 289-415)
// whose GPU form (bvcuda.cu:204-264, 45-60, 420-548) issues a cuBLAS gemv per
// half-pass plus 2-4 synchronous device-to-host scalar copies per pass.
//
// gs_column_kernel runs every pass of a column.  A pass is any combination of
//   UPDATE  w <- w - V(:,0:jb) coef        (the second half of CGS pass p)
//   SCALE   w <- w * scale                 (BVOrthonormalizeColumn's 1/norm)
//   DOT     c <- [V(:,0:jb)^T w', w'^T w'] (the first half of CGS pass p+1)
// in one streaming read of V; fusing the update of pass p with the dot of pass
// p+1 reads V three times for a column refined once, where a gemv per half-pass
// reads it four times.  After a DOT the CTAs meet at a grid barrier, every CTA
// sums the per-CTA dots in the same fixed order and takes the DGKS decision of
// BVOrthogonalizeGS for itself (the same bits everywhere), so the next pass
// starts without a launch and without another exchange.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <atomic>

#include "common.h"
#include "kernels.h"

namespace b200 {
namespace {

constexpr int kConsumerWarps = 8;                // warps that compute
constexpr int kConsumers = kConsumerWarps * 32;  // 256 consumer threads
constexpr int kThreads = kConsumers + 32;        // + one producer warp issuing the tile loads
constexpr int kPartCols = 32;                    // most basis columns a consumer lane holds in registers
constexpr int kMaxStages = 8;
constexpr double kDefTol = 10.0 * 2.220446049250313e-16;  // BV deftol = 10*PETSC_MACHINE_EPSILON (bvfunc.c:184)
constexpr size_t kStageBudget = 192 * 1024;      // bytes of all stages together

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n"
      " .reg .pred p;\n"
      " mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(done)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return done != 0;
}
// Bounded wait: after kSpinLimit polls, or once another wait of the CTA has given up, it sets *gave_up
// and returns; the caller goes on (every thread keeps meeting the CTA's barriers) and the column ends
// with an error.
__device__ __forceinline__ void mbar_wait_bounded(uint64_t *bar, uint32_t parity, volatile int *gave_up) {
  if (mbar_try_wait(bar, parity)) return;
  for (long long it = 0; it < kSpinLimit && !*gave_up; ++it)
    if (mbar_try_wait(bar, parity)) return;
  *gave_up = 1;
}
// 2-D tile load through a tensor map: box at (x = first row, y = first column).
__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *tmap, int x, int y, uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
          smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(tmap)), "r"(x), "r"(y), "r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// Barrier `id` over `threads` threads of the CTA (the warps that share a group of rows).
__device__ __forceinline__ void group_sync(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  return v;
}

// Lane l < CPW returns the sum over the lanes of acc[l]: a halving exchange, 31 shuffles for 32 columns
// where a tree per column takes 160.
template <int CPW>
__device__ __forceinline__ double lane_column_sums(const double (&acc)[CPW], int lane) {
  double v[32];
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = i < CPW ? acc[i < CPW ? i : 0] : 0.0;
#pragma unroll
  for (int half = 16; half > 0; half >>= 1) {
#pragma unroll
    for (int i = 0; i < half; ++i) {
      const bool up = (lane & half) != 0;
      const double keep = up ? v[i + half] : v[i], send = up ? v[i] : v[i + half];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, half);
    }
  }
  return v[0];
}

// Lane l returns the sum over the lanes of d[l / 8]: two halving exchanges and a tree, 6 shuffles for four
// columns (the shuffles, not the additions, bound a short dot: 20 a tree each).
__device__ __forceinline__ double quad_sum(const double (&d)[4], int lane) {
  const bool up = (lane & 16) != 0, odd = (lane & 8) != 0;
  const double a0 = up ? d[2] : d[0], a1 = up ? d[3] : d[1], b0 = up ? d[0] : d[2], b1 = up ? d[1] : d[3];
  const double e0 = a0 + __shfl_xor_sync(0xffffffffu, b0, 16), e1 = a1 + __shfl_xor_sync(0xffffffffu, b1, 16);
  double v = (odd ? e1 : e0) + __shfl_xor_sync(0xffffffffu, odd ? e0 : e1, 8);
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

struct ColumnParams {
  GsPassArgs a;
  GsState *st;
  double *cnew;
  double *partials;  // two buffers of G x (jb + 1) per-CTA dots, by parity of the pass
  double eta;
  double deftol;
  int fresh;         // start of a run: the control block's counters and halt flag are replaced (not its error bits)
  int plain_dot;     // plain BVDotVec: one DOT, no decision
  int parts;         // warps that share a group of 32 rows (1, 2, 4, 8): each owns 1/parts of the columns
  int stages;
  int nchunks;
};

// State of the DGKS machine of one column, kept by every CTA (all CTAs hold the same values).
struct Decision {
  int stage, pass, action, lindep, err;
  double onrm, nrm, scale;
};

// BVOrthogonalizeGS's "finish a pass" logic (bvorthog.c:176-187, 209-214).  Returns true if the dot
// just reduced is already the dot of the next pass (have_next) and that pass is to be taken.
__device__ bool finish_pass(Decision &d, const ColumnParams &p, double onrm, double nrm, bool have_next) {
  const bool refine = d.pass < 3 && nrm != 0.0 && fabs(nrm) < p.eta * fabs(onrm);
  if (refine) {
    d.stage = kStageDotOfPass;
    if (!have_next) d.action = kActUpdate | kActDot;
    return have_next;
  }
  d.lindep = !(nrm != 0.0 && fabs(nrm) >= p.eta * fabs(onrm));
  d.nrm = nrm;
  d.scale = (p.a.normalize && nrm != 1.0 && nrm != 0.0) ? 1.0 / nrm : 1.0;
  d.action = (have_next ? 0 : kActUpdate) | (d.scale != 1.0 ? kActScale : 0);
  d.stage = kStageDone;
  return false;
}

// The decision after a DOT, run by one warp: cnew_s holds the reduced dots, coef_s gets the
// coefficients of the next UPDATE, hsum the accumulated ones (BV_AddCoefficients).
__device__ void decide(Decision &d, const ColumnParams &p, const double *cnew_s, double *coef_s, double *hsum,
                       int lane) {
  const int jb = p.a.jb;
  const double self = cnew_s[jb];
  if (d.stage == kStageExplicitNorm) {
    // BV_NormVecOrColumn: the norm of the updated vector
    if (!finish_pass(d, p, d.onrm, (self < 0.0) ? 0.0 : sqrt(self), true)) return;
  }
  double sum = 0.0;
  for (int i = lane; i < jb; i += 32) {
    const double c = cnew_s[i];
    coef_s[i] = c;
    hsum[i] = d.pass == 0 ? c : hsum[i] + c;
    sum = fma(c, c, sum);
  }
  sum = warp_sum(sum);  // BV_SquareSum
  d.pass += 1;
  if (p.a.column && !(self > -p.deftol)) d.err |= kDevErrInnerProduct;  // BV_SafeSqrt
  const double onrm = (self < 0.0) ? 0.0 : sqrt(self);
  const double t = onrm * onrm - sum;  // estimate |v'| from |v| (bvorthog.c:124-127)
  if (t > 0.0) {
    finish_pass(d, p, onrm, sqrt(t), false);
  } else {
    d.onrm = onrm;
    d.action = kActUpdate | kActDot;  // explicit norm of the updated vector next
    d.stage = kStageExplicitNorm;
  }
}

// Grid-wide barrier on one word: the CTAs' increments cancel in the low bits and flip the top bit once
// all have arrived, so the word carries over between launches of any grid size.  Every CTA is resident
// (cooperative launch).  Called by one thread per CTA between __syncthreads(); false after kSpinLimit
// polls.
__device__ __forceinline__ unsigned grid_arrive(unsigned *word, int G) {
  __threadfence();
  return atomicAdd(word, blockIdx.x == 0 ? 0x80000000u - (unsigned)(G - 1) : 1u);
}
__device__ __forceinline__ bool grid_wait(unsigned *word, unsigned arrived) {
  for (long long it = 0; it < kSpinLimit; ++it) {
    unsigned now;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(now) : "l"(word) : "memory");
    if ((now ^ arrived) & 0x80000000u) return true;
  }
  return false;
}

// One column.  Warps 0..7 consume, warp 8 produces.  The producer streams row chunks of the jb basis
// columns (one 2-D TMA tile load each) into a ring of shared-memory stages; full[s] completes when a
// tile has landed, empty[s] when the consumer warps have copied it into registers.  The chunk's rows
// form groups of 32, one row per lane; `parts` warps share a group, each holding its share of the
// columns (CPW, jb / parts rounded up to the instantiated sizes: fixed trip counts, the columns past jb
// are zeros that no load writes) of its lane's row in registers from the update to the dot, so a tile is
// read from shared memory once, the update needs no exchange for jb <= 32 (parts = 1) and otherwise one
// partial sum per warp and row behind a barrier of the group's warps alone, and the dots stay
// lane-private across all chunks.  What bounds it: HBM for large n (8 n (jb + 1) bytes per pass), the
// passes' latency for small n.
//   * Passes alternate direction over the chunks, so a pass finds in L2 what the one before read last.
//   * The pass that follows a DOT needs V again whatever is decided (unless the DOT was for an explicit
//     norm), so its first tiles are loaded while the grid barrier, the reduction and the decision run.
//   * w is read and written with plain loads and stores by the CTA that owns its rows (one chunk ahead);
//     only V, which the kernel does not write, goes through the async proxy.
// Measured (whole b200_bv_orthonormalize_column calls, refined columns, against five launches of a pass
// kernel that read each tile twice and shared a row among all eight warps): n = 2,097,152 j = 8 198 ->
// 144 us, j = 40 434 -> 359, j = 60 555 -> 523 (5.9 TB/s), j = 79 761 -> 658 (6.2 TB/s); n = 262,144
// j = 60 135 -> 106; n = 10,000 j = 20 62 -> 55.  Alternating direction is worth 10% at n = 262,144
// j = 60 and nothing at n = 2,097,152.  Trip counts taken from jb at run time instead of CPW: 636 us at
// j = 60 (588 instructions per warp and tile, 150 so).
template <int CPW>
__global__ void __launch_bounds__(kThreads, 1) gs_column_kernel(ColumnParams p, const __grid_constant__ CUtensorMap tmap) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t full[kMaxStages], empty[kMaxStages];
  __shared__ __align__(16) double coef_s[kConsumerWarps * CPW];  // zero past jb
  __shared__ double cnew_s[kMaxCols + 1], hsum[kMaxCols + 1];
  __shared__ double red[kConsumerWarps][kMaxCols + 1];
  __shared__ double upd[2][kConsumerWarps][32];  // partial update sums, by parity of the chunk
  __shared__ Decision dsh;
  __shared__ volatile int gave_up;
  __shared__ int grid_ok;
  // Launched as a programmatic dependent of the previous kernel in the stream: wait until that
  // grid has finished and its writes (the control block, w) are visible, then let the next kernel
  // be launched at once (its CTAs take each SM as this grid's CTA leaves it).
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" :::);
  const GsPassArgs &a = p.a;
  GsState *st = p.st;
  if (a.step >= 0 && !p.fresh && st->halt && st->halt_step < a.step) return;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool producer = warp == kConsumerWarps;
  const int G = gridDim.x, S = p.stages, jb = a.jb, parts = p.parts;
  const int CH = kConsumers / parts;
  const uint32_t tile_bytes = (uint32_t)CH * (uint32_t)jb * 8u;                          // what a load brings
  const uint32_t stage_bytes = (uint32_t)CH * (uint32_t)(parts * CPW) * 8u;  // with the zero columns past jb
  unsigned char *stage_base = smem_raw + ((128u - (smem_u32(smem_raw) & 127u)) & 127u);
  if (tid == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], kConsumerWarps);
    }
    fence_mbar_init();
    gave_up = 0;
    dsh = Decision{kStageDotOfPass, 0, kActDot, 0, 0, 0.0, 0.0, 1.0};
  }
  for (int i = tid; i < kConsumerWarps * CPW; i += kThreads) coef_s[i] = 0.0;
  for (int s = 0; s < S; ++s) {
    double *pad = reinterpret_cast<double *>(stage_base + (size_t)s * stage_bytes) + (size_t)CH * jb;
    for (int i = tid; i < CH * (parts * CPW - jb); i += kThreads) pad[i] = 0.0;
  }
  __syncthreads();

  const int nmine = (p.nchunks > (int)blockIdx.x) ? (p.nchunks - 1 - (int)blockIdx.x) / G + 1 : 0;
  double *Vw = a.V + (size_t)a.wcol * a.ld;
  // this warp's group of rows and share of the columns
  const int group = warp / parts, part = warp % parts;
  const int c0 = part * CPW;
  const int ldp = jb + 1;

  int tile = 0;        // tiles issued (producer) or consumed (consumers) so far
  int ahead = 0;       // producer: tiles of the coming pass that are already issued
  unsigned npass = 0;
  unsigned long long bytes = 0;
  bool ok = true;
  for (int pass = 0;; ++pass) {
    const int action = dsh.action;
    const bool do_update = (action & kActUpdate) != 0, do_dot = (action & kActDot) != 0;
    const bool do_scale = (action & kActScale) != 0;
    const bool rewrite = do_update || do_scale;
    const bool tiles = (do_update || do_dot) && jb > 0;
    const bool next_tiles = tiles && do_dot && dsh.stage == kStageDotOfPass && !p.plain_dot;
    const double scale = do_scale ? dsh.scale : 1.0;
    // chunk i of the pass, in the pass's direction
    auto chunk_row = [&](int i, int ps) {
      const int k = (ps & 1) ? nmine - 1 - i : i;
      return ((long long)blockIdx.x + (long long)k * G) * CH;
    };
    if (producer) {
      if (lane == 0 && tiles) {
        const int total = nmine + (next_tiles ? min(S, nmine) : 0);
        for (int i = ahead; i < total; ++i, ++tile) {
          const int s = tile % S;
          if (tile >= S) mbar_wait_bounded(&empty[s], (uint32_t)(((tile / S) - 1) & 1), &gave_up);
          if (gave_up) break;
          const bool next = i >= nmine;
          mbar_arrive_expect_tx(&full[s], tile_bytes);
          tma_load_2d(stage_base + (size_t)s * stage_bytes, &tmap, (int)chunk_row(next ? i - nmine : i, pass + (next ? 1 : 0)),
                      0, &full[s]);
        }
        ahead = total - nmine;
      }
      __syncwarp();
    } else {
      double acc[CPW], self = 0.0;
#pragma unroll
      for (int t = 0; t < CPW; ++t) acc[t] = 0.0;
      const int lrow = group * 32 + lane;
      auto load_w = [&](int i) {
        const long long row = chunk_row(i, pass) + lrow;
        return (i < nmine && row < a.n) ? __ldcg(Vw + row) : 0.0;
      };
      double wnext = load_w(0);
      for (int i = 0; i < nmine; ++i) {
        const long long row = chunk_row(i, pass) + lrow;
        double wv = wnext;
        wnext = load_w(i + 1);
        double v[CPW];
        if (tiles) {
          const int s = tile % S;
          mbar_wait_bounded(&full[s], (uint32_t)((tile / S) & 1), &gave_up);
          const double *Vs = reinterpret_cast<const double *>(stage_base + (size_t)s * stage_bytes) + (size_t)c0 * CH + lrow;
#pragma unroll
          for (int t = 0; t < CPW; ++t) v[t] = Vs[t * CH];
          __syncwarp();
          if (lane == 0) mbar_arrive(&empty[s]);  // copied out: the next tile load may overwrite it
          ++tile;
        }
        if (do_update) {
          double tot = 0.0;
          if (tiles) {
            double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
            const double2 *cf = reinterpret_cast<const double2 *>(coef_s + c0);
#pragma unroll
            for (int t = 0; t < CPW; t += 4) {
              const double2 ca = cf[t / 2], cb = cf[t / 2 + 1];
              s0 = fma(v[t], ca.x, s0);
              s1 = fma(v[t + 1], ca.y, s1);
              s2 = fma(v[t + 2], cb.x, s2);
              s3 = fma(v[t + 3], cb.y, s3);
            }
            tot = (s0 + s1) + (s2 + s3);
          }
          if (parts > 1) {
            double(*up)[32] = upd[i & 1];
            up[warp][lane] = tot;
            group_sync(1 + group, parts * 32);
            tot = 0.0;
            for (int r = 0; r < parts; ++r) tot += up[group * parts + r][lane];  // the same order in every warp
          }
          wv -= tot;
        }
        if (rewrite) {
          if (do_scale) wv *= scale;
          if (part == 0 && row < a.n) Vw[row] = wv;
        }
        if (do_dot) {
          if (tiles) {
#pragma unroll
            for (int t = 0; t < CPW; ++t) acc[t] = fma(v[t], wv, acc[t]);
          }
          if (part == 0) self = fma(wv, wv, self);
        }
      }
      if (do_dot) {
        const double mine = lane_column_sums(acc, lane);
        if (lane < CPW && c0 + lane < jb) red[group][c0 + lane] = mine;
        self = warp_sum(self);
        if (part == 0 && lane == 0) red[group][jb] = self;
      }
    }
    ++npass;
    // algorithmic traffic of this pass: streamed columns + w read, w written back if changed
    bytes += (unsigned long long)a.n * 8ull * ((tiles ? jb : 0) + 1 + (rewrite ? 1 : 0));
    if (!do_dot) break;
    __syncthreads();
    double *pb = p.partials + (size_t)(pass & 1) * G * ldp;
    const int groups = kConsumerWarps / parts;
    for (int c = tid; c <= jb; c += kThreads) {
      double sacc = 0.0;
      for (int g = 0; g < groups; ++g) sacc += red[g][c];
      __stcg(pb + (size_t)blockIdx.x * ldp + c, sacc);
    }
    __syncthreads();
    if (tid == 0) {
      const unsigned arrived = grid_arrive(&st->ticket, G);
      // a plain dot is reduced by CTA 0 alone
      grid_ok = (p.plain_dot && blockIdx.x != 0) || grid_wait(&st->ticket, arrived);
      __threadfence();
    }
    __syncthreads();
    ok = grid_ok != 0;
    if (!ok || (p.plain_dot && blockIdx.x != 0)) break;
    // Fixed-order sum over the CTAs: warp w adds CTAs w, w + 8, ... with one column per lane (32
    // independent coalesced loads in flight per warp and column group), then the warps in order.
    if (!producer) {
      for (int c = lane; c <= jb; c += 32) {
        double sacc = 0.0;
#pragma unroll 8
        for (int b = warp; b < G; b += kConsumerWarps) sacc += __ldcg(pb + (size_t)b * ldp + c);
        red[warp][c] = sacc;
      }
    }
    __syncthreads();
    if (warp == 0) {
      for (int c = lane; c <= jb; c += 32) {
        double sacc = 0.0;
#pragma unroll
        for (int w = 0; w < kConsumerWarps; ++w) sacc += red[w][c];
        cnew_s[c] = sacc;
      }
      __syncwarp();
      if (!p.plain_dot) {
        Decision d = dsh;
        decide(d, p, cnew_s, coef_s, hsum, lane);
        __syncwarp();
        if (lane == 0) dsh = d;
      }
    }
    __syncthreads();
    if (p.plain_dot || dsh.action == kActNone || gave_up) break;
  }

  __syncthreads();
  if (blockIdx.x == 0) {
    if (p.plain_dot) {
      if (ok)
        for (int c = tid; c <= jb; c += kThreads) p.cnew[c] = cnew_s[c];
    } else if (ok && dsh.stage == kStageDone) {
      const Decision &d = dsh;
      if (a.hacc) {
        for (int c = tid; c < jb; c += kThreads) a.hacc[c] = hsum[c];
        if (tid == 0) a.hacc[jb] = d.lindep ? 0.0 : d.nrm;  // BV_SetValue(bv,k,k,h,...)
      }
      if (tid == 0) {
        if (a.T) {
          a.T[a.step] = jb > 0 ? hsum[jb - 1] : 0.0;
          a.T[a.ldt + a.step] = d.lindep ? 0.0 : d.nrm;
        }
        st->beta_out = d.nrm;
        st->lindep = d.lindep;
        st->halt = d.lindep && a.step >= 0;
        st->halt_step = a.step;
      }
    }
    if (tid == 0) {
      if (dsh.err) atomicOr(&st->err, dsh.err);
      st->bytes = (p.fresh ? 0 : st->bytes) + bytes;
      st->passes = (p.fresh ? 0 : st->passes) + (int)npass;
    }
  }
  if (!ok || gave_up) {
    // report, and let the copies still in flight land (bounded) before the CTA leaves
    if (tid == 0) atomicOr(&st->err, (int)kDevErrTimeout);
    if (producer && lane == 0)
      for (int t = tile > S ? tile - S : 0; t < tile; ++t)
        for (long long it = 0; it < kSpinLimit && !mbar_try_wait(&full[t % S], (uint32_t)((t / S) & 1)); ++it) {
        }
  }
}

// ---------------------------------------------------------------- a whole Lanczos run in one launch
//
// BVMatLanczos for a basis that fits the chip's shared memory: every CTA owns a contiguous range of
// 32-row slices of the sliced-ELL operator and keeps its rows of all the run's basis columns in shared
// memory, so a column costs no launch and no basis traffic: SpMV of its rows, then the passes of
// gs_column_kernel with the same DGKS decisions, an exchange of the CTAs' dots after each DOT and a
// barrier when the new column is complete.  Two forms:
//   * gs_cluster_run_kernel, the smallest: one 16-CTA cluster, the exchanges and the gathered x through
//     distributed shared memory;
//   * gs_run_kernel: up to one CTA per SM, the exchanges and x through L2.
// What bounds both is a chain of latencies (exchange, decision, SpMV gathers), and beside it the issue
// slots: a phase is a few hundred instructions per warp, so the loops keep their indices in 32 bits, take
// no divisions and give every warp one share.
// Measured (BVMatLanczos on 2-D Laplacians, whole calls; column by column / one CTA per SM / one cluster):
// n = 3,660 columns 0..30 583 / 356 / 232 us; n = 10,000 columns 16..32 373 / 221 / 195; n = 14,400 columns
// 0..20 428 / 254 / 192; n = 40,000 columns 0..40 1,030 / 612 / -; n = 65,000 columns 0..20 508 / 319 / -.
// So the cluster runs wherever its shared memory holds the basis, then one CTA per SM wherever that does.
constexpr int kRunWarps = 16;
constexpr int kRunThreads = kRunWarps * 32;
constexpr int kRunCached = 8;                   // entries per row of the operator held in registers
constexpr size_t kRunSmem = 184 * 1024;         // shared memory for the basis rows, w and its partial updates

struct RunParams {
  double *V;
  int ld, n, k, m;
  double *coefbuf;  // column j + 1 of the coefficient buffer gets the coefficients of column j + 1
  int ldc;
  double *T;
  int ldt;
  GsState *st;
  ulonglong2 *slots;         // two buffers of G x (jb + 1) {partial dot, epoch}
  unsigned long long epoch;  // epochs of this run start above it (no earlier run on these slots used them)
  double eta, deftol;
  int nslices, spc;          // slices of the operator, slices per CTA
  const long long *off;
  const int *width;
  const int *cols;
};

// What the passes of a run share with the CTA's threads.
struct RunPass {
  int action, lindep;
  double scale, nrm;
};

// sum over c < nc of v[c R] coef[c]; coef 16-byte aligned
__device__ __forceinline__ double run_row_sum(const double *v, int R, const double *coef, int nc) {
  double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
  int c = 0;
#pragma unroll 2
  for (; c + 4 <= nc; c += 4, v += 4 * R) {
    const double2 ca = *reinterpret_cast<const double2 *>(coef + c), cb = *reinterpret_cast<const double2 *>(coef + c + 2);
    s0 = fma(v[0], ca.x, s0);
    s1 = fma(v[R], ca.y, s1);
    s2 = fma(v[2 * R], cb.x, s2);
    s3 = fma(v[3 * R], cb.y, s3);
  }
  for (; c < nc; ++c, v += R) s0 = fma(v[0], coef[c], s0);
  return (s0 + s1) + (s2 + s3);
}

// UPDATE and SCALE of the CTA's rows.  With parts = 1 << lp warps to a slice (lp > 0: at most 16 slices a
// CTA, one share per warp) the parts of the columns meet in ups; with one warp to a slice a lane finishes
// its row by itself.
__device__ __forceinline__ void run_update(const double *Vs, double *ws, double *ups, const double *coef, int jb, int R,
                                           int spc, int lp, int slice, int part, bool update, double scale) {
  const int lane = threadIdx.x & 31;
  if (lp > 0) {
    if (update) {
      if (part < (1 << lp)) {
        const int q = (((jb + (1 << lp) - 1) >> lp) + 1) & ~1, c0 = part * q;  // even: aligned coefficient pairs
        ups[part * R + 32 * slice + lane] =
            run_row_sum(Vs + c0 * R + 32 * slice + lane, R, coef + c0, min(q, jb - c0));
      }
      __syncthreads();
    }
    for (int r = threadIdx.x; r < R; r += kRunThreads) {
      double tot = 0.0;
      if (update)
        for (int q = 0; q < (1 << lp); ++q) tot += ups[q * R + r];
      ws[r] = (ws[r] - tot) * scale;
    }
  } else {
    for (int s = slice; s < spc; s += kRunWarps) {
      const int r = 32 * s + lane;
      const double tot = update ? run_row_sum(Vs + r, R, coef, jb) : 0.0;
      ws[r] = (ws[r] - tot) * scale;
    }
  }
  __syncthreads();
}

// Lane l returns column 4 cg + l / 8 of the dots of w with the basis columns (column jb is w itself) over
// the rows [ra, rb) of the CTA.
__device__ __forceinline__ double run_dot4(const double *Vs, const double *ws, int jb, int R, int cg, int ra, int rb) {
  const int lane = threadIdx.x & 31;
  const double *v[4];
  double d[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
  for (int q = 0; q < 4; ++q) v[q] = 4 * cg + q < jb ? Vs + (4 * cg + q) * R : ws;
#pragma unroll 2
  for (int r = ra + lane; r < rb; r += 32) {
    const double wv = ws[r];
#pragma unroll
    for (int q = 0; q < 4; ++q) d[q] = fma(v[q][r], wv, d[q]);
  }
  return quad_sum(d, lane);
}

// The decision after an exchange, by warp 0 (d stays in its registers), published for the CTA.
__device__ __forceinline__ void run_decide(Decision &d, const ColumnParams &cp, const double *cnew_s, double *coef_s,
                                           double *hsum, RunPass *pass) {
  const int lane = threadIdx.x & 31;
  decide(d, cp, cnew_s, coef_s, hsum, lane);
  if (lane == 0) {
    pass->action = d.action;
    pass->scale = d.scale;
    if (d.stage == kStageDone) {
      pass->lindep = d.lindep;
      pass->nrm = d.nrm;
    }
  }
}

// The outputs of a finished column: coefficients, alpha and beta, error bits.
__device__ __forceinline__ void run_column_out(const RunParams &p, int j, const double *hsum, const RunPass &pass) {
  const int jb = j + 1;
  double *h = p.coefbuf + (size_t)jb * p.ldc;
  for (int c = threadIdx.x; c < jb; c += kRunThreads) h[c] = hsum[c];
  if (threadIdx.x == 0) {
    const double beta = pass.lindep ? 0.0 : pass.nrm;
    h[jb] = beta;
    p.T[j] = hsum[jb - 1];
    p.T[p.ldt + j] = beta;
  }
}

// {value, epoch} of one CTA's partial dot.  The pair is stored and loaded as one 16-byte access (single-copy
// atomic for .b128), so a reader that finds the epoch it waits for has the value too: the exchange after a
// DOT needs neither a fence nor an arrival counter.
__device__ __forceinline__ void slot_store(ulonglong2 *slot, double v, unsigned long long epoch) {
  asm volatile("{\n .reg .b128 q;\n mov.b128 q, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], q;\n}\n" ::"l"(slot),
               "l"(__double_as_longlong(v)), "l"(epoch)
               : "memory");
}
__device__ __forceinline__ ulonglong2 slot_load(const ulonglong2 *slot) {
  ulonglong2 r;
  asm volatile("{\n .reg .b128 q;\n ld.relaxed.gpu.global.b128 q, [%2];\n mov.b128 {%0, %1}, q;\n}\n"
               : "=l"(r.x), "=l"(r.y)
               : "l"(slot)
               : "memory");
  return r;
}

template <typename VT>
__global__ void __launch_bounds__(kRunThreads, 1) gs_run_kernel(RunParams p, const VT *__restrict__ sval) {
  extern __shared__ __align__(16) double run_smem[];
  __shared__ __align__(16) double coef_s[kMaxCols + 1];
  __shared__ double cnew_s[kMaxCols + 1], hsum[kMaxCols + 1];
  __shared__ double red[kRunWarps][kMaxCols + 1];
  __shared__ RunPass ps;
  __shared__ int grid_ok;
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" :::);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int G = gridDim.x, n = p.n, spc = p.spc, R = 32 * spc;
  const int r0 = blockIdx.x * R, rows = min(R, n - r0);
  const int lp = 31 - __clz(kRunWarps / spc);  // parts of the columns in an update: 1 << lp warps to a slice
  // a warp's slice and share of the columns; with lp = 0 it owns whole slices, and past spc none
  const int slice = lp ? warp % spc : warp, part = lp ? warp / spc : 0;
  double *ws = run_smem;       // w of the CTA's rows
  double *ups = ws + R;        // partial updates [part][row]
  double *Vs = ups + (R << lp);  // basis columns [column][row]
  for (int c = 0; c <= p.k; ++c)
    for (int r = tid; r < R; r += kRunThreads) Vs[c * R + r] = r < rows ? p.V[(size_t)c * p.ld + r0 + r] : 0.0;
  // the operator's entries of this lane's row: the first kRunCached stay in registers for the run
  const int sl = blockIdx.x * spc + warp;
  const bool has_slice = warp < spc && sl < p.nslices;
  const int wid = has_slice ? p.width[sl] : 0;
  const long long base = has_slice ? p.off[sl] + lane : 0;
  int cc[kRunCached];
  VT aa[kRunCached];
#pragma unroll
  for (int u = 0; u < kRunCached; ++u) {
    cc[u] = u < wid ? p.cols[base + 32ll * u] : -1;
    aa[u] = u < wid ? sval[base + 32ll * u] : VT(0);
  }
  if (tid == 0) grid_ok = 1;
  unsigned target = 0;
  // Grid barrier: the arrivals of all CTAs bring the word to the next multiple of G.  False (for the whole
  // CTA) after kSpinLimit polls.
  auto grid_sync = [&]() -> bool {
    target += (unsigned)G;
    __syncthreads();
    if (tid == 0) {
      asm volatile("fence.acq_rel.gpu;\n red.relaxed.gpu.global.add.u32 [%0], 1;" ::"l"(&p.st->run_ticket) : "memory");
      int ok = 0;
      for (long long it = 0; it < kSpinLimit && !ok; ++it) {
        unsigned now;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(now) : "l"(&p.st->run_ticket) : "memory");
        ok = (int)(now - target) >= 0;
      }
      grid_ok = ok;
    }
    __syncthreads();
    return grid_ok != 0;
  };

  ColumnParams cp;  // what the decision reads
  cp.eta = p.eta;
  cp.deftol = p.deftol;
  cp.a.normalize = 1;
  cp.a.column = 1;
  Decision d;
  unsigned npass = 0;
  unsigned long long epoch = p.epoch, bytes = 0;
  bool ok = true;
  int halt = 0, halt_step = -1, errs = 0;
  double beta = 0.0;
  for (int j = p.k; j < p.m && ok && !halt; ++j) {
    const int jb = j + 1, ldp = jb + 1;
    const double *x = p.V + (size_t)j * p.ld;  // written by every CTA: read through L2
    if (warp < spc) {
      double sacc = 0.0;
      double xv[kRunCached];
#pragma unroll
      for (int u = 0; u < kRunCached; ++u) xv[u] = cc[u] >= 0 ? __ldcg(x + cc[u]) : 0.0;
#pragma unroll
      for (int u = 0; u < kRunCached; ++u)
        if (cc[u] >= 0) sacc = __dadd_rn(sacc, __dmul_rn((double)aa[u], xv[u]));
      for (int u = kRunCached; u < wid; ++u) {
        const int c = p.cols[base + 32ll * u];
        if (c >= 0) sacc = __dadd_rn(sacc, __dmul_rn((double)sval[base + 32ll * u], __ldcg(x + c)));
      }
      ws[32 * warp + lane] = sacc;  // rows past n have no entries
    }
    d = Decision{kStageDotOfPass, 0, kActDot, 0, 0, 0.0, 0.0, 1.0};
    cp.a.jb = jb;
    int action = kActDot;
    double scale = 1.0;
    __syncthreads();
    for (;;) {
      const bool update = (action & kActUpdate) != 0, rewrite = (action & (kActUpdate | kActScale)) != 0;
      const bool dot = (action & kActDot) != 0;
      ++npass;
      bytes += (unsigned long long)n * 8ull * ((update || dot ? jb : 0) + 1 + (rewrite ? 1 : 0));
      if (rewrite) run_update(Vs, ws, ups, coef_s, jb, R, spc, lp, slice, part, update, scale);
      if (!dot) break;
      ulonglong2 *pb = p.slots + (size_t)(epoch & 1) * G * ldp;
      ++epoch;
      for (int cg = warp; 4 * cg <= jb; cg += kRunWarps) {
        const double mine = run_dot4(Vs, ws, jb, R, cg, 0, R);
        const int c = 4 * cg + (lane >> 3);
        if ((lane & 7) == 0 && c <= jb) slot_store(pb + blockIdx.x * ldp + c, mine, epoch);
      }
      // Fixed-order sum over the CTAs: warp w adds CTAs w, w + 16, ... with one column per lane, up to eight
      // loads in flight, each repeated until it brings this exchange's epoch.
      bool arrived = true;
      for (int c = lane; c <= jb; c += 32) {
        double sacc = 0.0;
        for (int b0 = warp; b0 < G; b0 += 8 * kRunWarps) {
          ulonglong2 r[8];
#pragma unroll
          for (int u = 0; u < 8; ++u)
            if (b0 + u * kRunWarps < G) r[u] = slot_load(pb + (b0 + u * kRunWarps) * ldp + c);
#pragma unroll
          for (int u = 0; u < 8; ++u)
            if (b0 + u * kRunWarps < G) {
              for (long long it = 0; r[u].y != epoch && arrived; ++it) {
                r[u] = slot_load(pb + (b0 + u * kRunWarps) * ldp + c);
                if (it >= kSpinLimit) arrived = false;
              }
              sacc += __longlong_as_double(r[u].x);
            }
        }
        red[warp][c] = sacc;
      }
      if (!arrived) grid_ok = 0;
      __syncthreads();
      ok = grid_ok != 0;
      if (!ok) break;
      if (warp == 0) {
        for (int c = lane; c <= jb; c += 32) {
          double t[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) t[q] = (red[q][c] + red[q + 4][c]) + (red[q + 8][c] + red[q + 12][c]);
          cnew_s[c] = (t[0] + t[1]) + (t[2] + t[3]);
        }
        __syncwarp();
        run_decide(d, cp, cnew_s, coef_s, hsum, &ps);
        errs |= d.err;
      }
      __syncthreads();
      action = ps.action;
      scale = ps.scale;
      if (action == kActNone) break;
    }
    if (!ok) break;
    // the new column: into the basis rows of this CTA and into V, where every CTA gathers it
    double *vn = p.V + (size_t)jb * p.ld + r0;
    for (int r = tid; r < R; r += kRunThreads) {
      Vs[jb * R + r] = ws[r];
      if (r < rows) __stcg(vn + r, ws[r]);
    }
    beta = ps.nrm;
    if (blockIdx.x == 0) run_column_out(p, j, hsum, ps);
    if (ps.lindep) {
      halt = 1;
      halt_step = j;
    } else if (j + 1 < p.m) {
      ok = grid_sync();
    }
  }
  if (tid == 0) {
    if (!ok) atomicOr(&p.st->err, (int)kDevErrTimeout);
    if (blockIdx.x == 0 && ok) {
      if (errs) atomicOr(&p.st->err, errs);
      p.st->beta_out = beta;
      p.st->lindep = halt;
      p.st->halt = halt;
      p.st->halt_step = halt_step;
      p.st->passes = (int)npass;
      p.st->bytes = bytes;
    }
    // the last CTA to leave clears the barrier word for the next run
    __threadfence();
    if (atomicAdd(&p.st->run_exit, 1u) == (unsigned)(G - 1)) {
      p.st->run_ticket = 0;
      p.st->run_exit = 0;
    }
  }
}

// ---- the cluster form
constexpr int kClusterCtas = 16;
constexpr int kRowParts = 2;       // the rows of a dot are split in two, so that a short basis feeds all warps
constexpr int kClusterSlices = 2;  // slices of the operator a warp applies

__device__ __forceinline__ uint32_t cluster_map(uint32_t addr, uint32_t cta) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(cta));
  return r;
}
__device__ __forceinline__ double cluster_load(uint32_t addr) {
  double v;
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(addr) : "memory");
  return v;
}
// Store to another CTA's shared memory that counts its bytes on that CTA's mbarrier: the receiver's wait
// for the bytes is the whole exchange (a store followed by the cluster barrier takes twice as long).
__device__ __forceinline__ void cluster_store_tx(uint32_t addr, double v, uint32_t bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(addr),
               "l"(__double_as_longlong(v)), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void cluster_sync() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Shared doubles of a CTA: basis rows, w, partial updates, dot exchange.
__host__ __device__ inline size_t cluster_run_doubles(int spc, int m) {
  const int parts = spc <= kRunWarps / 2 ? kRunWarps / spc : 1;
  return (size_t)32 * spc * (m + 1 + 1 + parts) + (size_t)2 * kClusterCtas * kRowParts * (m + 1);
}

template <typename VT>
__global__ void __launch_bounds__(kRunThreads, 1) gs_cluster_run_kernel(RunParams p, const VT *__restrict__ sval) {
  extern __shared__ __align__(16) double run_smem[];
  __shared__ __align__(16) double coef_s[kMaxCols + 1];
  __shared__ double cnew_s[kMaxCols + 1], hsum[kMaxCols + 1];
  __shared__ __align__(8) uint64_t bars[2];  // bytes of an exchange, by its parity
  __shared__ RunPass ps;
  __shared__ volatile int gave_up, stop;
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" :::);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n = p.n, spc = p.spc, R = 32 * spc, rank = blockIdx.x;
  const int r0 = rank * R, rows = min(R, n - r0);  // negative for a CTA past the last row
  const int lp = spc <= kRunWarps / 2 ? 31 - __clz(kRunWarps / spc) : 0;
  const int slice = lp ? warp % spc : warp, part = lp ? warp / spc : 0;
  double *Vs = run_smem;                  // basis rows [column][row]
  double *ws = Vs + (p.m + 1) * R;        // w of the CTA's rows
  double *xch = ws + R;                   // two buffers of [CTA and row part][column] dots
  double *ups = xch + 2 * kClusterCtas * kRowParts * (p.m + 1);  // partial updates [part][row]
  if (tid == 0) {
    mbar_init(&bars[0], 1);
    mbar_init(&bars[1], 1);
    fence_mbar_init();
    gave_up = 0;
    stop = 0;
  }
  for (int c = 0; c <= p.k; ++c)
    for (int r = tid; r < R; r += kRunThreads) Vs[c * R + r] = r < rows ? p.V[(size_t)c * p.ld + r0 + r] : 0.0;
  // the operator's entries of this lane's rows (slices warp and warp + 16 of the CTA): the first kRunCached
  // of a row stay in registers for the run, a column as the cluster address of its basis row
  const uint32_t vs0 = smem_u32(Vs);
  uint32_t ca[kClusterSlices][kRunCached];
  VT aa[kClusterSlices][kRunCached];
  int wid[kClusterSlices];
  long long base[kClusterSlices];
  auto address = [&](int c) { return c >= 0 ? cluster_map(vs0 + 8u * (uint32_t)(c % R), (uint32_t)(c / R)) : 0u; };
#pragma unroll
  for (int h = 0; h < kClusterSlices; ++h) {
    const int ls = warp + h * kRunWarps, sl = rank * spc + ls;
    const bool has = ls < spc && sl < p.nslices;
    wid[h] = has ? p.width[sl] : 0;
    base[h] = has ? p.off[sl] + lane : 0;
#pragma unroll
    for (int u = 0; u < kRunCached; ++u) {
      ca[h][u] = u < wid[h] ? address(p.cols[base[h] + 32ll * u]) : 0u;
      aa[h][u] = u < wid[h] ? sval[base[h] + 32ll * u] : VT(0);
    }
  }
  ColumnParams cp;  // what the decision reads
  cp.eta = p.eta;
  cp.deftol = p.deftol;
  cp.a.normalize = 1;
  cp.a.column = 1;
  Decision d;
  unsigned npass = 0, exchange = 0;
  unsigned long long bytes = 0;
  int halt = 0, halt_step = -1, errs = 0;
  double beta = 0.0;
  cluster_sync();  // every CTA's basis rows are loaded and its mbarriers live
  for (int j = p.k; j < p.m && !halt; ++j) {
    const int jb = j + 1, ldp = jb + 1;
    const uint32_t xoff = 8u * (uint32_t)j * (uint32_t)R;  // column j of any CTA's basis rows
#pragma unroll
    for (int h = 0; h < kClusterSlices; ++h) {
      const int ls = warp + h * kRunWarps;
      if (ls < spc) {
        double xv[kRunCached], sacc = 0.0;
#pragma unroll
        for (int u = 0; u < kRunCached; ++u) xv[u] = ca[h][u] ? cluster_load(ca[h][u] + xoff) : 0.0;
#pragma unroll
        for (int u = 0; u < kRunCached; ++u)
          if (ca[h][u]) sacc = __dadd_rn(sacc, __dmul_rn((double)aa[h][u], xv[u]));
        for (int u = kRunCached; u < wid[h]; ++u) {
          const uint32_t a = address(p.cols[base[h] + 32ll * u]);
          if (a) sacc = __dadd_rn(sacc, __dmul_rn((double)sval[base[h] + 32ll * u], cluster_load(a + xoff)));
        }
        ws[32 * ls + lane] = sacc;  // rows past n have no entries
      }
    }
    d = Decision{kStageDotOfPass, 0, kActDot, 0, 0, 0.0, 0.0, 1.0};
    cp.a.jb = jb;
    int action = kActDot;
    double scale = 1.0;
    __syncthreads();
    for (;;) {
      const bool update = (action & kActUpdate) != 0, rewrite = (action & (kActUpdate | kActScale)) != 0;
      const bool dot = (action & kActDot) != 0;
      ++npass;
      bytes += (unsigned long long)n * 8ull * ((update || dot ? jb : 0) + 1 + (rewrite ? 1 : 0));
      if (rewrite) run_update(Vs, ws, ups, coef_s, jb, R, spc, lp, slice, part, update, scale);
      if (!dot) break;
      // (four columns, half of the rows) shares over the warps; each sum goes to every CTA of the cluster
      const int buf = exchange & 1;
      double *xb = xch + buf * kClusterCtas * kRowParts * (p.m + 1);
      if (tid == 0) mbar_arrive_expect_tx(&bars[buf], (uint32_t)(kClusterCtas * kRowParts * ldp * 8));
      const uint32_t bar = smem_u32(&bars[buf]);
      for (int it = warp; 4 * (it / kRowParts) <= jb; it += kRunWarps) {
        const int cg = it / kRowParts, rp = it % kRowParts;
        const double mine = run_dot4(Vs, ws, jb, R, cg, rp ? 32 * (spc / 2) : 0, rp ? R : 32 * (spc / 2));
        const int c = 4 * cg + (lane >> 3);
        if (c <= jb) {
          const uint32_t slot = smem_u32(xb + (rank * kRowParts + rp) * (p.m + 1) + c);
#pragma unroll
          for (int t = 0; t < kClusterCtas / 8; ++t) {
            const uint32_t to = (lane & 7) + 8 * t;
            cluster_store_tx(cluster_map(slot, to), mine, cluster_map(bar, to));
          }
        }
      }
      if (warp == 0) {
        mbar_wait_bounded(&bars[buf], (exchange >> 1) & 1, &gave_up);
        for (int c = lane; c <= jb; c += 32) {
          const double *x = xb + c;
          double t[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
          for (int b = 0; b < kClusterCtas * kRowParts; ++b) t[b & 3] += x[b * (p.m + 1)];
          cnew_s[c] = (t[0] + t[1]) + (t[2] + t[3]);
        }
        __syncwarp();
        run_decide(d, cp, cnew_s, coef_s, hsum, &ps);
        errs |= d.err;
      }
      ++exchange;
      __syncthreads();
      action = ps.action;
      scale = ps.scale;
      if (action == kActNone || gave_up) break;
    }
    // the new column: into the basis rows, where the cluster gathers it, and into V
    double *vn = p.V + (size_t)jb * p.ld + r0;
    for (int r = tid; r < R; r += kRunThreads) {
      Vs[jb * R + r] = ws[r];
      if (r < rows) vn[r] = ws[r];
    }
    beta = ps.nrm;
    if (rank == 0) run_column_out(p, j, hsum, ps);
    if (ps.lindep) {
      halt = 1;
      halt_step = j;
    }
    // a CTA that gave up a wait stops the whole cluster here, so that none sends to a CTA that has left
    if (gave_up && tid < kClusterCtas)
      asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(cluster_map(smem_u32((const void *)&stop), tid)), "r"(1) : "memory");
    cluster_sync();  // column j + 1 is complete; after the last column, no CTA leaves while another reads it
    if (stop) break;
  }
  if (tid == 0 && gave_up) atomicOr(&p.st->err, (int)kDevErrTimeout);
  if (rank == 0 && tid == 0) {
    if (errs) atomicOr(&p.st->err, errs);
    p.st->beta_out = beta;
    p.st->lindep = halt;
    p.st->halt = halt;
    p.st->halt_step = halt_step;
    p.st->passes = (int)npass;
    p.st->bytes = bytes;
  }
}

PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
    void *ptr = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      ptr = nullptr;
    return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(ptr);
  }();
  return fn;
}

// Tensor map over the basis: dim 0 = rows (n, contiguous), dim 1 = columns (stride ld), box rows x cols.
cudaError_t make_tmap(CUtensorMap *tm, const GsPassArgs &a, int rows, int cols) {
  memset(tm, 0, sizeof(*tm));
  if (cols <= 0) return cudaSuccess;  // no tile load in this column
  PFN_cuTensorMapEncodeTiled_v12000 enc = encode_fn();
  if (!enc) return cudaErrorNotSupported;
  const cuuint64_t dims[2] = {(cuuint64_t)a.n, (cuuint64_t)a.total_cols};
  const cuuint64_t strides[1] = {(cuuint64_t)a.ld * sizeof(double)};
  const cuuint32_t box[2] = {(cuuint32_t)rows, (cuuint32_t)cols};
  const cuuint32_t estr[2] = {1, 1};
  CUresult r = enc(tm, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 2, (void *)a.V, dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

// Warps that share a group of rows: the fewest whose lanes can hold the columns (32 doubles of the row
// and as many dots).  More warps with fewer columns each cost a barrier and smaller tiles: n = 2,097,152
// j = 50 takes 424 us with 32 columns a lane, 564 with 24 or 16; j = 79 658, 659 and 1002.
int column_parts(int jb) {
  int parts = 1;
  while (parts < kConsumerWarps && jb > parts * kPartCols) parts *= 2;
  return parts;
}

template <int CPW>
cudaError_t launch_column_t(ColumnParams &p, int G, cudaStream_t stream) {
  const GsPassArgs &a = p.a;
  const int CH = kConsumers / p.parts;
  const size_t stage = (size_t)CH * p.parts * CPW * sizeof(double);
  p.stages = (int)(kStageBudget / stage);
  if (p.stages > kMaxStages) p.stages = kMaxStages;
  CUtensorMap tm;
  cudaError_t e = make_tmap(&tm, a, CH, a.jb);
  if (e != cudaSuccess) return e;
  if ((e = allow_max_dynamic_smem(gs_column_kernel<CPW>)) != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)G);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = stage * p.stages + 128;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  // The CTAs meet at grid barriers: all of them are resident or none, also beside another stream's launches
  // (columns and runs of two bases on two streams at once keep their bits).
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  e = cudaLaunchKernelEx(&cfg, gs_column_kernel<CPW>, p, tm);
  count_launch();
  return e;
}

cudaError_t launch_column(const GsPassArgs &a, const GsWork &w, double eta, int fresh, int plain_dot,
                          cudaStream_t stream) {
  if (a.jb < 0 || a.jb >= kMaxCols) return cudaErrorInvalidValue;
  ColumnParams p;
  p.a = a;
  p.st = w.st;
  p.cnew = w.cnew;
  p.partials = w.partials;
  p.eta = eta;
  p.deftol = kDefTol;
  p.fresh = fresh;
  p.plain_dot = plain_dot;
  p.parts = column_parts(a.jb);
  const int CH = kConsumers / p.parts;
  p.nchunks = (a.n + CH - 1) / CH;
  int G = w.num_sms < w.max_ctas ? w.num_sms : w.max_ctas;
  if (G > p.nchunks) G = p.nchunks;
  const int q = (a.jb + p.parts - 1) / p.parts;  // columns per warp
  if (q <= 4) return launch_column_t<4>(p, G, stream);
  if (q <= 8) return launch_column_t<8>(p, G, stream);
  if (q <= 12) return launch_column_t<12>(p, G, stream);
  if (q <= 16) return launch_column_t<16>(p, G, stream);
  if (q <= 20) return launch_column_t<20>(p, G, stream);
  if (q <= 24) return launch_column_t<24>(p, G, stream);
  if (q <= 28) return launch_column_t<28>(p, G, stream);
  return launch_column_t<32>(p, G, stream);
}

template <typename VT>
cudaError_t launch_run(RunParams &p, const void *vals, int G, size_t smem, cudaStream_t stream) {
  cudaError_t e = allow_max_dynamic_smem(gs_run_kernel<VT>);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)G);
  cfg.blockDim = dim3(kRunThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  e = cudaLaunchKernelEx(&cfg, gs_run_kernel<VT>, p, static_cast<const VT *>(vals));
  count_launch();
  return e;
}

// The cluster form where one fits; cudaErrorNotSupported otherwise.
template <typename VT>
cudaError_t launch_cluster_run(RunParams &p, const void *vals, cudaStream_t stream) {
  const int spc = (p.nslices + kClusterCtas - 1) / kClusterCtas;
  if (spc > kClusterSlices * kRunWarps) return cudaErrorNotSupported;
  const size_t smem = sizeof(double) * cluster_run_doubles(spc, p.m);
  // device limits, once per device: dynamic shared memory and whether a 16-CTA cluster of that size exists
  static std::atomic<int> most[64];
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorNotSupported;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(kClusterCtas);
  cfg.blockDim = dim3(kRunThreads);
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = kClusterCtas;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  int limit = most[dev].load(std::memory_order_acquire);
  if (limit == 0) {
    limit = -1;
    cudaFuncAttributes fa;
    int clusters = 0;
    if (cudaFuncSetAttribute(gs_cluster_run_kernel<VT>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
        allow_max_dynamic_smem(gs_cluster_run_kernel<VT>) == cudaSuccess &&
        cudaFuncGetAttributes(&fa, gs_cluster_run_kernel<VT>) == cudaSuccess) {
      cfg.dynamicSmemBytes = (size_t)fa.maxDynamicSharedSizeBytes;
      cfg.numAttrs = 1;
      if (cudaOccupancyMaxActiveClusters(&clusters, gs_cluster_run_kernel<VT>, &cfg) == cudaSuccess && clusters > 0)
        limit = fa.maxDynamicSharedSizeBytes;
    }
    cudaGetLastError();
    most[dev].store(limit, std::memory_order_release);
  }
  if (limit < 0 || smem > (size_t)limit) return cudaErrorNotSupported;
  p.spc = spc;
  cfg.dynamicSmemBytes = smem;
  cfg.numAttrs = 2;
  e = cudaLaunchKernelEx(&cfg, gs_cluster_run_kernel<VT>, p, static_cast<const VT *>(vals));
  count_launch();
  return e;
}

__global__ void gs_reset_kernel(GsState *st) {
  GsState h;
  memset(&h, 0, sizeof(h));
  h.halt_step = -1;
  *st = h;
}

// out[0] = the norm, out[1] = the lindep flag, out[2] = the device error bits of the last column
// orthogonalisation (read back once for a block of columns)
__global__ void gs_record_kernel(const GsState *__restrict__ st, double *out) {
  out[0] = st->beta_out;
  out[1] = (double)st->lindep;
  out[2] = (double)st->err;
}

}  // namespace

cudaError_t gs_state_reset(const GsWork &w, cudaStream_t stream) {
  gs_reset_kernel<<<1, 1, 0, stream>>>(w.st);
  count_launch();
  return cudaGetLastError();
}

cudaError_t gs_orthogonalize_launch(const GsPassArgs &a, const GsWork &w, double eta, bool fresh,
                                    cudaStream_t stream) {
  return launch_column(a, w, eta, fresh ? 1 : 0, 0, stream);
}

cudaError_t gs_run_launch(const GsRunArgs &a, const SpmvSell &S, bool f32, const GsWork &w, double eta,
                          unsigned long long epoch, cudaStream_t stream) {
  if (!w.slots || S.nrest > 0 || S.nslices <= 0 || a.m >= kMaxCols) return cudaErrorNotSupported;
  RunParams p;
  p.V = a.V;
  p.ld = a.ld;
  p.n = a.n;
  p.k = a.k;
  p.m = a.m;
  p.coefbuf = a.coefbuf;
  p.ldc = a.ldc;
  p.T = a.T;
  p.ldt = a.ldt;
  p.st = w.st;
  p.slots = w.slots;
  p.epoch = epoch;
  p.eta = eta;
  p.deftol = kDefTol;
  p.nslices = S.nslices;
  p.off = S.off;
  p.width = S.width;
  p.cols = S.cols;
  cudaError_t e = f32 ? launch_cluster_run<float>(p, S.vals, stream) : launch_cluster_run<double>(p, S.vals, stream);
  if (e != cudaErrorNotSupported) return e;
  const int ctas = w.num_sms < w.max_ctas ? w.num_sms : w.max_ctas;
  const int spc = (S.nslices + ctas - 1) / ctas;
  if (spc > kRunWarps) return cudaErrorNotSupported;
  const int R = 32 * spc, parts = kRunWarps / spc;
  const size_t smem = sizeof(double) * (size_t)R * (1 + parts + a.m + 1);
  if (smem > kRunSmem) return cudaErrorNotSupported;
  p.spc = spc;
  const int G = (S.nslices + spc - 1) / spc;
  return f32 ? launch_run<float>(p, S.vals, G, smem, stream) : launch_run<double>(p, S.vals, G, smem, stream);
}

cudaError_t gs_record_launch(const GsWork &w, double *out, cudaStream_t stream) {
  gs_record_kernel<<<1, 1, 0, stream>>>(w.st, out);
  count_launch();
  return cudaGetLastError();
}

cudaError_t gs_dot_launch(const GsPassArgs &a, const GsWork &w, cudaStream_t stream) {
  return launch_column(a, w, 0.0, 0, 1, stream);
}

}  // namespace b200
