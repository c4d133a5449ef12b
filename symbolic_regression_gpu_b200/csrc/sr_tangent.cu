// sr_tangent.cu — forward-mode (tangent) gradient of the population MSE with
// respect to the constants of expressions with at most kMaxTangentConsts
// constants.  (No reference counterpart: the reference evaluates MSE only.)
//
//   tan_kernel<DPT, MAXW, MINB>
//                       the interpreter's work decomposition (a producer
//                       thread streaming X spans into shared memory and
//                       folding span results, warps claiming expressions of a
//                       group) with, beside each datapoint's value T, one
//                       tangent row t_c = d T / d constant c per constant, in
//                       the warp's shared memory.  Per instruction the warp
//                       computes the operator's value and local partials and
//                       moves the tangents forward:
//                         t_c = dT * t_c  for the constants under the
//                                          accumulator (mask A),
//                         t_c = db * t_c  for the constants under the operand
//                                          b (mask B: the constant itself, or
//                                          a spilled subtree, whose rows
//                                          stayed where they were),
//                       and a constant that enters (a leaf or operand b)
//                       starts at t_c = 1.  The masks come from the host (one
//                       word per instruction: A, B and a constant-load flag);
//                       instructions with A = B = 0 compute no partials.
//                       At the end of a tile d MSE / d c gets sum over
//                       datapoints of seed * t_c, seed = 2 (pred - y) for valid
//                       datapoints (0 otherwise): each lane's DPT products in
//                       FP32, FP64 across lanes, tiles and spans.  No tape, no
//                       second pass.
//
// Zero rule (the mirror of the reverse sweep's "a zero adjoint times anything
// is zero"): a zero partial times anything is zero (t_c = dT == 0 ? 0 :
// dT * t_c), and the final product is zero where the seed is zero.  An
// expression is a tree, so each constant reaches the result along one path
// and the two rules give the same zeros: whichever of an infinite and a zero
// factor lies nearer the result decides, in both modes, between NaN and 0.
// Constants outside a mask are never multiplied, so an infinite partial off
// a constant's path (sqrt'(0) in a branch without that constant) does not
// reach its tangent.
//
// Values and partials are those of the reverse-mode kernel (sr_grad_ops.cuh
// formulas, the forward interpreter's routines), so the MSE equals the
// forward pass's up to summation order and the gradients differ from the
// reverse mode only by the order of the FP32 products along each path.
#include <cuda_runtime.h>
#include <stdint.h>

#include "sr_adjoint.hpp"
#include "sr_kernels.hpp"
#include "sr_partials.cuh"

namespace sr {
namespace {

// t = d == 0 ? 0 : d * t
template <int DPT>
__device__ __forceinline__ void kill_mul(float (&t)[DPT], const float (&d)[DPT]) {
#pragma unroll
  for (int k = 0; k < DPT; k += 2) {
    const float2 r = __fmul2_rn(make_float2(d[k], d[k + 1]), make_float2(t[k], t[k + 1]));
    t[k] = (d[k] == 0.0f) ? 0.0f : r.x;
    t[k + 1] = (d[k + 1] == 0.0f) ? 0.0f : r.y;
  }
}

// The tangents of the constants under one operand of an instruction times the
// operator's partial by it.  These constants are the ones of a subtree, so they
// are neighbours: `mask` is one run of bits and their rows follow one another.
// Constants that enter here (`fresh`: a constant leaf, a constant operand b)
// start from lane c's `tinit` (1, or a folded subtree's derivative by constant
// c); rows of an operator whose partial is exactly 1 stay as they are, and -1
// negates them.  A partial that is zero somewhere in the lane takes the zero
// rule's selects, out of line; the others need none.
template <int DPT>
__device__ __noinline__ void tan_rows_zero(float *row, int n, const float *d) {
  float f[DPT];
#pragma unroll
  for (int k = 0; k < DPT; ++k) f[k] = d[k];
#pragma unroll 1
  for (int c = 0; c < n; ++c, row += 32 * DPT) {
    float tv[DPT];
    lds_vec<DPT>(row, 0, tv);
    kill_mul<DPT>(tv, f);
    sts_vec<DPT>(row, 0, tv);
  }
}
template <int DPT>
__device__ __forceinline__ void tan_rows(float *tan, uint32_t mask, int lane, int kind,
                                         float (&d)[DPT], bool fresh, float tinit) {
  if (kind == kDOne && !fresh) return;
  const int c0 = __ffs(mask) - 1, n = __popc(mask);
  float *row = tan + c0 * (32 * DPT) + lane * 4;
  if (fresh) {
    float *q = row;
#pragma unroll 1
    for (int c = 0; c < n; ++c, q += 32 * DPT) {
      float t0 = __shfl_sync(0xffffffffu, tinit, c0 + c), tv[DPT];
      if (kind == kDNeg) t0 = -t0;
#pragma unroll
      for (int k = 0; k < DPT; ++k) tv[k] = t0;
      sts_vec<DPT>(q, 0, tv);
    }
    if (kind != kDGen) return;
  }
  if (kind == kDNeg) {
#pragma unroll
    for (int k = 0; k < DPT; ++k) d[k] = -1.0f;
  }
  if (min_abs<DPT>(d) > 0.0f) {
#pragma unroll 1
    for (int c = 0; c < n; ++c, row += 32 * DPT) {
      float tv[DPT];
      lds_vec<DPT>(row, 0, tv);
#pragma unroll
      for (int k = 0; k < DPT; k += 2) {
        const float2 r = __fmul2_rn(make_float2(d[k], d[k + 1]), make_float2(tv[k], tv[k + 1]));
        tv[k] = r.x;
        tv[k + 1] = r.y;
      }
      sts_vec<DPT>(row, 0, tv);
    }
  } else {
    float f[DPT];
#pragma unroll
    for (int k = 0; k < DPT; ++k) f[k] = d[k];
    tan_rows_zero<DPT>(row, n, f);
  }
}

// One program over the warp's tile: values in T (registers), tangents in the
// warp's shared-memory rows tan[c][TILE] (c = constant index).  A spilled
// subtree's tangents stay in their rows: the instructions that follow it (up to
// the one that takes it back as operand b) belong to other subtrees, whose
// constants are other constants, so they never write its rows; the instruction
// that consumes it multiplies them by db in place.
template <int DPT>
__device__ __forceinline__ void run_tangent_program(const Instr *__restrict__ code, int len,
                                                    const float *xs, int xrs,
                                                    const SpillStack &st, int lane, float *tan,
                                                    float tinit, float (&T)[DPT]) {
  uint4 ins = ldg_instr(code);
  for (int i = 0; i < len; ++i) {
    // The code buffer ends with a padding entry, so this prefetch of the next
    // entry is always in bounds.
    const uint4 nxt = ldg_instr(code + i + 1);
    // Word and masks are the same in every lane; the reductions say so to the
    // compiler (uniform registers).
    const uint32_t w = __reduce_or_sync(0xffffffffu, ins.x);
    const uint32_t m = __reduce_or_sync(0xffffffffu, ins.w);
    const uint32_t A = m & 0xFFu, B = (m >> 8) & 0xFFu;
    if (w & (kLoadBit | kSpillBit)) {
      if (instr_spill(w)) spill_store<DPT>(st, instr_spill_slot(w), lane, T);
      if (instr_load(w))
        load_leaf<DPT, false>(instr_leaf_kind(w), ins.y, T, xs, xrs, lane, nullptr, 0, 0);
    }
    float b[DPT], dT[DPT], db[DPT];
    const uint32_t bk = instr_b_kind(w);
    if (bk != kBNone) load_operand<DPT, false>(bk, ins.z, b, xs, xrs, st, lane, nullptr, 0, 0);
    const uint32_t d = instr_dispatch(w);
    int dk = kDOne, bkn = kDOne;
    if (d & kDLinear) {
      // + - * as the interpreter's fused multiply-adds, with its values.
      if (d & kDMul) {
        dk = bkn = kDGen;
#pragma unroll
        for (int k = 0; k < DPT; k += 2) {
          const float2 t = make_float2(T[k], T[k + 1]), u = make_float2(b[k], b[k + 1]);
          const float2 r = __fmul2_rn(t, u);
          dT[k] = u.x;
          dT[k + 1] = u.y;
          db[k] = t.x;
          db[k + 1] = t.y;
          T[k] = r.x;
          T[k + 1] = r.y;
        }
      } else {
        const float st_ = (d & kDRSub) ? -1.0f : 1.0f;
        if (d & kDRSub) dk = kDNeg;
        if (d & kDSub) bkn = kDNeg;
        if (d & kDSub) {
#pragma unroll
          for (int k = 0; k < DPT; ++k) b[k] = -b[k];
        }
#pragma unroll
        for (int k = 0; k < DPT; k += 2) {
          const float2 r = __ffma2_rn(make_float2(T[k], T[k + 1]), make_float2(st_, st_),
                                      make_float2(b[k], b[k + 1]));
          T[k] = r.x;
          T[k + 1] = r.y;
        }
      }
    } else {
      tan_apply<DPT, false>(instr_op(w), (A | B) != 0, T, b, dT, db, dk, bkn);
    }
    if (A) tan_rows<DPT>(tan, A, lane, dk, dT, (m & kTanLoadConst) != 0, tinit);
    if (B) tan_rows<DPT>(tan, B, lane, bkn, db, bk == kBC, tinit);
    ins = nxt;
  }
}

// MAXW / MINB: at most MAXW evaluating warps, at least MINB resident blocks
// per SM.
template <int DPT, int MAXW, int MINB>
__global__ void __launch_bounds__((MAXW + 1) * 32, MINB) tan_kernel(const TanArgs a) {
  constexpr int TILE = 32 * DPT;
  const EvalArgs &p = a.e;
  const int K = a.K;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int W = p.W;
  const int rows = p.V + 1;
  const int span = p.span;
  float *xbuf = reinterpret_cast<float *>(smem_raw);
  float *sreg = xbuf + static_cast<size_t>(kBufs) * rows * span;
  float *tans = sreg + static_cast<size_t>(W) * p.s_smem * TILE;  // [W][K][TILE]
  double *gsm = reinterpret_cast<double *>(tans + static_cast<size_t>(W) * K * TILE);  // [W][K][32]
  float *csm = reinterpret_cast<float *>(gsm + static_cast<size_t>(W) * K * 32);  // [W][K][32]
  ItemDesc *desc = reinterpret_cast<ItemDesc *>(csm + static_cast<size_t>(W) * K * 32);
  uint64_t *full = reinterpret_cast<uint64_t *>(desc + kBufs);
  uint64_t *empty = full + kBufs;
  SpanPart *part = reinterpret_cast<SpanPart *>(empty + kBufs);
  GroupAcc *gacc = reinterpret_cast<GroupAcc *>(part + kBufs * p.G);
  double *gpart = reinterpret_cast<double *>(gacc + p.G);  // [kBufs][G][K]
  double *ggacc = gpart + static_cast<size_t>(kBufs) * p.G * K;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kBufs; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], static_cast<uint32_t>(W));
    }
    mbar_init_fence();
  }
  __syncthreads();

  const int k_spans = p.span_per_item;
  const int n_items = p.n_groups * ((p.n_spans + k_spans - 1) / k_spans);
  if (warp == W) {
    run_producer<true>(lane, p.n_groups, n_items, k_spans, p.n_spans, p.work_counter, p.error, p.X,
                         nullptr, rows, p.ldx, rows, span, span, xbuf, desc, full, empty,
                         FoldArgs{part, gacc, p.partial, p.G, a.n_valid, a.n_valid, K, gpart, ggacc,
                                  a.gout, a.gout_off, a.const_cnt, a.C});
    return;
  }

  SpillStack st;  // value spill slots
  st.ss = sreg + static_cast<size_t>(warp) * p.s_smem * TILE;
  st.gs = p.spill + (static_cast<size_t>(blockIdx.x) * W + warp) *
                        static_cast<size_t>(p.smax - p.s_smem) * TILE;
  st.s_smem = p.s_smem;
  float *tan = tans + static_cast<size_t>(warp) * K * TILE;
  double *gl = gsm + static_cast<size_t>(warp) * K * 32 + lane;  // per-lane gradient sums
  float *half = csm + static_cast<size_t>(warp) * K * 32 + lane;  // of a pair's first tile
  const int tiles = span / TILE;
  uint32_t buf = 0, phase = 0;
  for (;;) {
    if (!mbar_wait(&full[buf], phase, p.error)) return;
    const ItemDesc d = desc[buf];
    if (d.item < 0) return;
    const float *xb = xbuf + static_cast<size_t>(buf) * rows * span;
    const int64_t dp_span = static_cast<int64_t>(d.span) * span;
    for (;;) {
      int j = 0;
      if (lane == 0) j = atomicAdd(&desc[buf].claim, 1);
      j = __shfl_sync(0xffffffffu, j, 0);
      if (j >= p.G) break;
      const int e = p.group_expr[static_cast<int64_t>(d.group) * p.G + j];
      if (e < 0) break;  // groups are padded at their end only
      const Instr *code = p.code + p.code_off[e];
      const int len = p.code_len[e];
      const int nconst = min(a.const_cnt[e], K);
      // Lane c holds what the tangent of constant c starts from.
      const float tinit = lane < nconst ? __ldg(a.tinit + a.const_off[e] + lane) : 1.0f;
      double acc = 0.0;
      int cnt = 0;
      for (int c = 0; c < nconst; ++c) gl[c * 32] = 0.0;
      for (int t = 0; t < tiles; ++t) {
        const int64_t dp0 = dp_span + static_cast<int64_t>(t) * TILE;
        if (dp0 >= p.N) break;  // tail of the last span
        const float *xs = xb + t * TILE;
        float T[DPT];
        run_tangent_program<DPT>(code, len, xs, span, st, lane, tan, tinit, T);
        float y[DPT], sd[DPT];
        lds_vec<DPT>(xs + p.V * span, lane, y);
        const bool full_tile = dp0 + TILE <= p.N;  // warp-uniform
        float dfs[DPT], dsq[DPT];
#pragma unroll
        for (int k = 0; k < DPT; k += 2) {
          const float2 df2 = __fadd2_rn(make_float2(T[k], T[k + 1]), make_float2(-y[k], -y[k + 1]));
          const float2 sq2 = __fmul2_rn(df2, df2);
          dfs[k] = df2.x;
          dfs[k + 1] = df2.y;
          dsq[k] = sq2.x;
          dsq[k + 1] = sq2.y;
        }
        const int before = cnt;
        add_squares<DPT>(T, dsq, full_tile, dp0, lane, p.N, acc, cnt);
#pragma unroll
        for (int k = 0; k < DPT; ++k) sd[k] = 2.0f * dfs[k];
        if (cnt - before != DPT) {
#pragma unroll
          for (int k = 0; k < DPT; ++k) {
            const bool valid =
                (full_tile || dp0 + (k / 4) * 128 + lane * 4 + (k % 4) < p.N) && isfinite(T[k]);
            sd[k] = valid ? sd[k] : 0.0f;
          }
        }
        // d MSE / d c (times the count): seed * t_c, zero where the seed is;
        // each lane adds its products of a pair of tiles (2 DPT) in order in
        // FP32, FP64 from there on (an FP32 lane sum overflows only for products
        // beyond ~4e37).  Spans hold whole pairs; the last one may lack its
        // second tile.
        const bool odd = (t & 1) != 0;
        const bool pair_end = odd || dp0 + TILE >= p.N;
        const bool seeded = min_abs<DPT>(sd) > 0.0f;
#pragma unroll 1
        for (int cc = 0; cc < nconst; ++cc) {
          float tv[DPT];
          lds_vec<DPT>(tan + cc * TILE, lane, tv);
#pragma unroll
          for (int k = 0; k < DPT; k += 2) {
            const float2 r = __fmul2_rn(make_float2(sd[k], sd[k + 1]), make_float2(tv[k], tv[k + 1]));
            tv[k] = r.x;
            tv[k + 1] = r.y;
          }
          if (!seeded) {
#pragma unroll
            for (int k = 0; k < DPT; ++k) tv[k] = sd[k] == 0.0f ? 0.0f : tv[k];
          }
          float g = odd ? __fadd_rn(half[cc * 32], tv[0]) : tv[0];
#pragma unroll
          for (int k = 1; k < DPT; ++k) g = __fadd_rn(g, tv[k]);
          if (pair_end)
            gl[cc * 32] += static_cast<double>(g);
          else
            half[cc * 32] = g;
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        acc += __shfl_xor_sync(0xffffffffu, acc, o);
        cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
      }
      double *gp = gpart + (static_cast<size_t>(buf) * p.G + j) * K;
      for (int cc = 0; cc < K; ++cc) {
        double g = cc < nconst ? gl[cc * 32] : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) g += __shfl_xor_sync(0xffffffffu, g, o);
        if (lane == 0) gp[cc] = g;
      }
      if (lane == 0) part[static_cast<size_t>(buf) * p.G + j] = SpanPart{acc, cnt, e};
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[buf]);
    if (++buf == kBufs) {
      buf = 0;
      phase ^= 1u;
    }
  }
}

// Folded constant subtrees of a gradient launch, one thread each: the value
// and, constant by constant, the derivative from the constant up to the root,
// through the tangent kernel's own operators and zero rule (the rows of these
// constants would hold the same products at the subtree's root), and the
// partials met on the way.  A subtree's work is that of a few datapoints; the
// launch over all of them is latency-bound: one thread's chain of operators, once per
// constant (91 us from cold caches for 4,096 trees with 1 to 8 constants).
constexpr int kMaxFoldDepth = 40;  // values waiting in a subtree of 64 tokens
__global__ void __launch_bounds__(64)
    fold_grad_kernel(const GradFold *__restrict__ items, const uint2 *__restrict__ tokens, int n,
                     const float *__restrict__ consts, const int4 *__restrict__ cinfo,
                     float *__restrict__ tinit, float *__restrict__ path) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const GradFold it = items[i];
  float val[kMaxFoldDepth], tan[kMaxFoldDepth];
  bool on[kMaxFoldDepth];  // the constant lies under it
  for (int j = 0; j < it.nc; ++j) {
    const int64_t cj = it.c0 + j;
    const int4 info = cinfo[cj];
    int sp = 0, seen = 0, step = info.y;
    for (uint32_t k = it.len; k-- > 0;) {
      const uint32_t op = tokens[it.first + k].x;
      if (op == 0) {
        const int idx = it.nc - 1 - seen++;
        val[sp] = consts[it.c0 + idx];
        tan[sp] = 1.0f;
        on[sp] = idx == j;
        ++sp;
        continue;
      }
      const int a = --sp;
      const int b = op < 10 ? --sp : a;
      float T[2] = {val[a], val[a]}, B[2] = {val[b], val[b]};
      float dT[2], dB[2];
      int kt, kb;
      tan_apply<2, true>(op, true, T, B, dT, dB, kt, kb);
      const bool under_b = op < 10 && on[b];
      const bool under = on[a] || under_b;
      if (under) {
        float t[2] = {under_b ? tan[b] : tan[a], 0.0f};
        t[1] = t[0];
        const int kind = under_b ? kb : kt;
        float d = kind == kDOne ? 1.0f : -1.0f;
        if (kind == kDGen) {
          d = under_b ? dB[0] : dT[0];
          if (under_b)
            kill_mul<2>(t, dB);
          else
            kill_mul<2>(t, dT);
        } else if (kind == kDNeg) {
          t[0] = -t[0];
        }
        path[info.x + --step] = d;
        tan[sp] = t[0];
      }
      on[sp] = under;
      val[sp] = T[0];
      ++sp;
    }
    tinit[cj] = tan[0];
    if (j == 0) *it.dst = __float_as_uint(val[0]);
  }
}

// mse and grad of the expressions of one tangent launch: one warp per
// expression, the span groups over its lanes (see finalize_dd_kernel), their
// double-double MSE sums and FP64 gradient sums added over the warp in a fixed
// order; the FP64 sums themselves go to sums ((sum, count) per expression) and
// gsum (per constant).  Up to kMaxTangentConsts constants are summed together
// so that their loads overlap.
__global__ void __launch_bounds__(256)
    tan_finalize_kernel(const double2 *__restrict__ partial, const double *__restrict__ gout,
                        int n_groups, int64_t C, const int32_t *__restrict__ exprs,
                        int n_exprs, const int64_t *__restrict__ const_off,
                        const int64_t *__restrict__ gout_off,
                        const int32_t *__restrict__ const_cnt, int K, float *__restrict__ mse,
                        float *__restrict__ grad, double *__restrict__ gsum,
                        double2 *__restrict__ sums, SequenceEnd end) {
  end_sequence(end);
  const int q = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (q >= n_exprs) return;  // warp-uniform
  const int e = exprs[q];
  const int nc = min(const_cnt[e], K);
  const int64_t o = const_off[e], og = gout_off[e];
  double hi = 0.0, lo = 0.0, cnt = 0.0;
  double g[kMaxTangentConsts];
#pragma unroll
  for (int c = 0; c < kMaxTangentConsts; ++c) g[c] = 0.0;
  for (int k = lane; k < n_groups; k += 32) {
    const double2 *pp = partial + 2 * (static_cast<int64_t>(k) * n_exprs + q);
    const double2 v = pp[0];
    dd_add(hi, lo, v.x);
    dd_add(hi, lo, v.y);
    cnt += pp[1].x;
    const double *gk = gout + static_cast<int64_t>(k) * C + og;
#pragma unroll
    for (int c = 0; c < kMaxTangentConsts; ++c)
      if (c < nc) g[c] += gk[c];
  }
  dd_warp_sum(hi, lo, cnt);
  cnt = __shfl_sync(0xffffffffu, cnt, 0);
#pragma unroll
  for (int c = 0; c < kMaxTangentConsts; ++c) {
    if (c >= nc) break;
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) g[c] += __shfl_xor_sync(0xffffffffu, g[c], d);
    if (lane == 0) {
      gsum[o + c] = g[c];
      grad[o + c] = (cnt > 0.0) ? static_cast<float>(g[c] / cnt) : qnan();
    }
  }
  if (lane == 0) {
    const double s = isfinite(hi) ? __dadd_rn(hi, lo) : hi;
    mse[e] = (cnt > 0.0) ? static_cast<float>(s / cnt) : qnan();
    sums[e] = make_double2(s, cnt);
  }
}

template <int DPT, int MAXW, int MINB>
const void *tan_fn() {
  return reinterpret_cast<const void *>(&tan_kernel<DPT, MAXW, MINB>);
}

// Launch shapes: 4 datapoints per thread, one block per SM with as many
// evaluating warps as the register file holds beside the producer warp: 31 (64
// registers per thread) for up to 4 tangent rows, 27 (72) for more, as far as
// their tangent rows fit in shared memory.  The kernel lives on resident warps:
// 8 datapoints per thread and 19 or 15 warps issued on 61 and 53 % of the cycles
// (dependent chains, instruction fetches), these on 83 and 75 %, which outweighs
// a quarter more instructions: 4,096 x 262,144 19.8 -> 18.9 ms, 1,000 x 20,001
// 0.65 -> 0.55 ms a pass.  Widths of 2, 4, 6 and 8 rows in four launches give
// 18.4 and 0.59 ms; 3, 5 and 8 18.7 and 0.56.
constexpr int kTanDpt = 4;
constexpr int tan_max_warps(int K) { return K <= 4 ? 31 : 27; }
const void *select_tan(int K) {
  return K <= 4 ? tan_fn<kTanDpt, 31, 1>() : tan_fn<kTanDpt, 27, 1>();
}

}  // namespace

int tan_dpt() { return kTanDpt; }
int tan_warps(int K) { return tan_max_warps(K); }

size_t tan_smem_bytes(int K, int W, int V, int s_smem, int span, int G) {
  const size_t tile = 32u * static_cast<size_t>(kTanDpt);
  return (static_cast<size_t>(kBufs) * (V + 1) * span +
          static_cast<size_t>(W) * (s_smem + K) * tile) * sizeof(float) +
         static_cast<size_t>(W) * K * 32 * (sizeof(double) + sizeof(float)) +
         kBufs * sizeof(ItemDesc) + 2 * kBufs * sizeof(uint64_t) +
         static_cast<size_t>(G) * (kBufs * sizeof(SpanPart) + sizeof(GroupAcc)) +
         static_cast<size_t>(G) * K * (kBufs + 1) * sizeof(double);
}

cudaError_t tan_configure(int K, size_t smem, int W, int *blocks_per_sm) {
  const void *fn = select_tan(K);
  if (W < 1 || W > tan_max_warps(K)) return cudaErrorInvalidValue;
  const cudaError_t err = raise_smem_limit(fn, smem);
  if (err != cudaSuccess) return err;
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, fn, (W + 1) * 32, smem);
}

cudaError_t tan_set_smem_limit(int K, size_t smem) {
  return raise_smem_limit(select_tan(K), smem);
}

cudaError_t launch_tangent(const TanArgs &args, int blocks, size_t smem, cudaStream_t stream) {
  if (args.K < 1 || args.K > kMaxTangentConsts) return cudaErrorInvalidValue;
  const void *fn = select_tan(args.K);
  if (args.e.W < 1 || args.e.W > tan_max_warps(args.K)) return cudaErrorInvalidValue;
  void *params[] = {const_cast<TanArgs *>(&args)};
  return cudaLaunchKernel(fn, dim3(blocks), dim3((args.e.W + 1) * 32), params, smem, stream);
}

cudaError_t launch_fold_grad(const GradFold *items, const uint2 *tokens, int n,
                             const float *consts, const int4 *cinfo, float *tinit, float *path,
                             cudaStream_t stream) {
  if (n <= 0) return cudaSuccess;
  fold_grad_kernel<<<(n + 63) / 64, 64, 0, stream>>>(items, tokens, n, consts, cinfo, tinit, path);
  return cudaGetLastError();
}

cudaError_t launch_tan_finalize(const double2 *partial, const double *gout, int n_groups,
                                int64_t C, const int32_t *exprs, int n_exprs,
                                const int64_t *const_off, const int64_t *gout_off,
                                const int32_t *const_cnt, int K,
                                float *mse, float *grad, double *gsum, double2 *sums,
                                SequenceEnd end, cudaStream_t stream) {
  if (n_exprs <= 0) return cudaSuccess;
  tan_finalize_kernel<<<(n_exprs + 7) / 8, 256, 0, stream>>>(
      partial, gout, n_groups, C, exprs, n_exprs, const_off, gout_off, const_cnt, K, mse, grad,
      gsum, sums, end);
  return cudaGetLastError();
}

}  // namespace sr
