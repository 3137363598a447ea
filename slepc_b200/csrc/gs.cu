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

#include "common.h"
#include "kernels.h"

namespace b200 {
namespace {

constexpr int kConsumerWarps = 8;                // warps that compute
constexpr int kConsumers = kConsumerWarps * 32;  // 256 consumer threads
constexpr int kThreads = kConsumers + 32;        // + one producer warp issuing the tile loads
constexpr int kPartCols = 32;                    // most basis columns a consumer lane holds in registers
constexpr int kMaxStages = 8;
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

struct ColumnParams {
  GsPassArgs a;
  GsState *st;
  double *cnew;
  double *partials;  // two buffers of G x (jb + 1) per-CTA dots, by parity of the pass
  double eta;
  double deftol;     // BV deftol = 10*PETSC_MACHINE_EPSILON (bvfunc.c:184)
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
  attr[0].id = cudaLaunchAttributeCooperative;  // the CTAs meet at grid barriers
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
  p.deftol = 10.0 * 2.220446049250313e-16;
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

cudaError_t gs_record_launch(const GsWork &w, double *out, cudaStream_t stream) {
  gs_record_kernel<<<1, 1, 0, stream>>>(w.st, out);
  count_launch();
  return cudaGetLastError();
}

cudaError_t gs_dot_launch(const GsPassArgs &a, const GsWork &w, cudaStream_t stream) {
  return launch_column(a, w, 0.0, 0, 1, stream);
}

}  // namespace b200
