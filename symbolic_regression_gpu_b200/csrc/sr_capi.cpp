// sr_capi.cpp — the C ABI (sr_eval.h): context lifecycle, dataset upload,
// population compilation / planning / upload, launches and read-back
// (gradients and Adam: sr_capi_grad.cpp; the FP64 reference, the device
// generation loop, microbenchmarks, detection and host-only helpers:
// sr_capi_tools.cpp; shared helpers: sr_capi_internal.hpp).
//
// Reference counterpart: evaluate_gpu_mse (src/cleaned/cl_gpu_eval.cu:332-564)
// and evaluate_gpu_simple (src/cleaned/cl_gpu_simple.cu:187-310).  Where the
// reference synchronises after every copy and kernel and exits the process
// on a CUDA error, this runtime compiles on host threads, issues pinned
// asynchronous copies and all kernels back to back on one stream, waits once,
// and reports failures as status codes.
#include <cuda_runtime.h>

#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <fstream>
#include <numeric>
#include <sstream>
#include <thread>

#include "sr_adjoint.hpp"
#include "sr_capi_internal.hpp"
#include "sr_context.hpp"
#include "sr_detect_gpu.hpp"
#include "sr_evolve.hpp"
#include "sr_kernels.hpp"
#include "sr_trace.hpp"

using sr::Instr;
using sr::ProgramSet;
using namespace sr::capi;

namespace sr {
namespace capi {

double now_ms() {
  using namespace std::chrono;
  return duration<double, std::milli>(steady_clock::now().time_since_epoch()).count();
}

// Milliseconds between two events, 0 when either was never recorded (the
// device-resident paths skip the upload pair).  cudaEventElapsedTime reports
// that case as an error that would otherwise stay as the thread's last error
// and surface at the next launch check, so it is consumed here.
float elapsed_ms(cudaEvent_t a, cudaEvent_t b) {
  float ms = 0.f;
  if (cudaEventElapsedTime(&ms, a, b) != cudaSuccess) {
    cudaGetLastError();
    return 0.f;
  }
  return ms;
}

sr_status cuda_fail(sr_context *ctx, cudaError_t e, const char *what) {
  const sr_status s = (e == cudaErrorMemoryAllocation) ? SR_ERR_OUT_OF_MEMORY : SR_ERR_CUDA;
  cudaGetLastError();  // reported here; a non-sticky error must not fail the next call's launch check
  return ctx->fail(s, std::string(what) + ": " + cudaGetErrorString(e));
}

int host_threads(const sr_context *ctx) {
  int t = ctx->opts.host_threads;
  if (t <= 0) t = static_cast<int>(std::thread::hardware_concurrency());
  return std::max(1, std::min(t, 64));
}

int64_t round_up(int64_t a, int64_t b) { return (a + b - 1) / b * b; }

sr_status check_population(sr_context *ctx, const sr_population *pop) {
  if (!pop) return ctx->fail(SR_ERR_INVALID_ARGUMENT, "population is NULL");
  if (pop->num_exprs < 0) return ctx->fail(SR_ERR_INVALID_ARGUMENT, "num_exprs < 0");
  if (pop->num_exprs == 0) return SR_OK;
  if (!pop->tokens || !pop->values || !pop->offsets)
    return ctx->fail(SR_ERR_INVALID_ARGUMENT, "population arrays must not be NULL");
  if (pop->offsets[0] != 0) return ctx->fail(SR_ERR_INVALID_ARGUMENT, "offsets[0] must be 0");
  for (int i = 0; i < pop->num_exprs; ++i) {
    const int64_t len = pop->offsets[i + 1] - pop->offsets[i];
    if (len <= 0)
      return ctx->fail(SR_ERR_MALFORMED_EXPRESSION,
                       "expression " + std::to_string(i) + " is empty");
    if (len > SR_MAX_TOKENS)
      return ctx->fail(SR_ERR_EXPRESSION_TOO_LONG,
                       "expression " + std::to_string(i) + " has " + std::to_string(len) +
                           " tokens (max " + std::to_string(SR_MAX_TOKENS) + ")");
  }
  return SR_OK;
}

// Compile expressions [0, E) of a CSR population into ps (pinned staging).
// With `share` equal expressions are compiled once and folded subtrees and
// derived rows collapse to leaves; fold_constants (gradient and cached programs)
// folds constant subtrees alone.  Folded subtrees, there and under kHintFold hints,
// are added to ctx->folds.
sr_status compile_set(sr_context *ctx, int E, const int32_t *tok, const double *val,
                      const int64_t *off, const int32_t *hints, ProgramSet &ps,
                      const sr::Sharing *share, bool fold_constants) {
  SR_TRACE("sr: compile");
  ps.E = E;
  ps.cost.assign(static_cast<size_t>(E), 0.f);
  ps.n_const.assign(static_cast<size_t>(E), 0);
  ps.smax = 0;
  ps.n_instr = 0;
  ps.n_tokens = ps.n_executed = 0;
  ps.sfu_per_dp = ps.fp32_per_dp = 0.0;
  ps.n_derived = 0;
  // About 20 ns a token, and tens of microseconds to wake the workers: chunks
  // of 2,500 tokens or more, one thread below two of them.
  const int64_t n_tok = E > 0 ? off[E] - off[0] : 0;
  const int nt = static_cast<int>(
      std::max<int64_t>(1, std::min<int64_t>({host_threads(ctx), E, n_tok / 2500})));
  struct Chunk {
    std::vector<Instr> code;
    std::vector<sr::FoldSet::Ref> folds;  // loc and first relative to the chunk
    std::vector<uint2> fold_tokens;
    sr_status st = SR_OK;
    std::string msg;
    int64_t bad = -1, in_profile = 0;
    bool refs = false;
  };
  std::vector<Chunk> chunks(static_cast<size_t>(nt));
  std::vector<sr::ExprInfo> infos(static_cast<size_t>(E));
  std::vector<int32_t> reps(share ? static_cast<size_t>(E) : 0);
  const auto compile_chunk = [&](int ci) {
    Chunk &c = chunks[static_cast<size_t>(ci)];
    const int64_t x0 = static_cast<int64_t>(E) * ci / nt, x1 = static_cast<int64_t>(E) * (ci + 1) / nt;
    c.code.reserve(static_cast<size_t>((off[x1] - off[x0]) * 2 / 3 + 8));
    std::vector<int32_t> marks(share || fold_constants ? SR_MAX_TOKENS : 0);
    std::vector<sr::FoldRef> refs;
    for (int64_t x = x0; x < x1; ++x) {
      sr::ExprInfo &info = infos[static_cast<size_t>(x)];
      const int len = static_cast<int>(off[x + 1] - off[x]);
      const int32_t *h = hints ? hints + off[x] : nullptr;
      if (share) {
        const int r = share->rep(static_cast<int>(x));
        reps[static_cast<size_t>(x)] = r;
        if (r == x && share->mark(static_cast<int>(x), marks.data())) h = marks.data();
        if (r != x) {
          info.n_tokens = len;
          continue;
        }
      }
      if (fold_constants && sr::mark_constant_subtrees(tok + off[x], len, marks.data())) {
        if (h) sr::merge_hints(h, len, marks.data());
        h = marks.data();
      }
      const int64_t i0 = static_cast<int64_t>(c.code.size());
      refs.clear();
      const sr_status s = sr::compile_expression(tok + off[x], val + off[x], len, ctx->V, h, c.code,
                                                 info, &c.msg, ctx->V + 1, &refs);
      if (s != SR_OK) {
        c.st = s;
        c.bad = x;
        return;
      }
      for (const sr::FoldRef &f : refs) {
        const int64_t t0 = off[x] + f.tok;
        uint32_t n = 0;
        int32_t c0 = 0, nc = 0;
        for (int32_t k = 0; k < f.tok; ++k) c0 += tok[off[x] + k] == SR_TOK_CONST ? 1 : 0;
        for (int need = 1; need > 0; ++n) {
          const int t = tok[t0 + n];
          nc += t == SR_TOK_CONST ? 1 : 0;
          need += t <= 0 ? -1 : (sr::is_binary_token(t) ? 1 : 0);
          uint2 w{static_cast<uint32_t>(t), 0u};
          const float v = static_cast<float>(val[t0 + n]);
          if (t == SR_TOK_CONST) std::memcpy(&w.y, &v, sizeof v);
          c.fold_tokens.push_back(w);
        }
        c.folds.push_back(sr::FoldSet::Ref{&ps, (i0 << 1) + f.loc,
                                           static_cast<uint32_t>(c.fold_tokens.size()) - n, n,
                                           static_cast<int32_t>(x), c0, nc});
      }
    }
    for (Instr &in : c.code) {
      in.w = sr::with_dispatch(in.w);
      c.in_profile += sr::in_protected_profile(sr::instr_op(in.w)) ? 1 : 0;
      c.refs = c.refs || (sr::instr_load(in.w) && sr::instr_leaf_kind(in.w) == sr::kLeafR) ||
               sr::instr_b_kind(in.w) == sr::kBR;
    }
  };
  ctx->workers.run(nt, nt, compile_chunk);
  int64_t total = 0;
  for (const Chunk &c : chunks) {
    if (c.st != SR_OK)
      return ctx->fail(c.st, "expression " + std::to_string(c.bad) + ": " + c.msg);
    total += static_cast<int64_t>(c.code.size());
  }
  SR_TRY_CUDA(ctx, ps.layout_host(static_cast<size_t>(total + 1), static_cast<size_t>(E)));
  int64_t pos = 0;
  ps.n_instr_protected = 0;
  ps.cache_refs = false;
  for (const Chunk &c : chunks) {
    const uint32_t t0 = static_cast<uint32_t>(ctx->folds.tokens.size());
    for (sr::FoldSet::Ref r : c.folds) {
      r.loc += pos << 1;
      r.first += t0;
      ctx->folds.refs.push_back(r);
    }
    ctx->folds.tokens.insert(ctx->folds.tokens.end(), c.fold_tokens.begin(), c.fold_tokens.end());
    std::memcpy(ps.h_code.p + pos, c.code.data(), c.code.size() * sizeof(Instr));
    pos += static_cast<int64_t>(c.code.size());
    ps.n_instr_protected += c.in_profile;
    ps.cache_refs = ps.cache_refs || c.refs;
  }
  ps.h_code.p[total] = Instr{0, 0, 0, 0};  // prefetch padding
  ps.n_listed = E;
  int64_t o = 0;
  for (int x = 0; x < E; ++x) {
    const auto &in = infos[static_cast<size_t>(x)];
    ps.h_off.p[x] = o;
    ps.h_len.p[x] = in.n_instr;
    o += in.n_instr;
    ps.cost[static_cast<size_t>(x)] = in.cost;
    ps.n_const[static_cast<size_t>(x)] = in.n_const;
    ps.smax = std::max(ps.smax, in.need);
    ps.n_tokens += in.n_tokens;
    ps.n_executed += in.n_executed;
    ps.sfu_per_dp += in.sfu_ops;
    ps.fp32_per_dp += in.fp32_ops;
    if (share) {
      ps.h_row.p[x] = reps[static_cast<size_t>(x)];
      if (reps[static_cast<size_t>(x)] != x) --ps.n_listed;
    }
  }
  ps.shared = ps.n_listed < E;
  ps.n_instr = total;
  return SR_OK;
}

// Copies the folded subtrees collected by compile_set and has the device
// compute them into the (uploaded) programs.
static sr_status upload_folds(sr_context *ctx) {
  sr::FoldSet &f = ctx->folds;
  if (f.refs.empty()) return SR_OK;
  const size_t ib = f.refs.size() * sizeof(sr::FoldItem), tb = f.tokens.size() * sizeof(uint2);
  SR_TRY_CUDA(ctx, f.h_pack.ensure(ib + tb));
  SR_TRY_CUDA(ctx, f.pack.ensure(ib + tb));
  auto *items = reinterpret_cast<sr::FoldItem *>(f.h_pack.p);
  for (size_t i = 0; i < f.refs.size(); ++i) {
    const sr::FoldSet::Ref &r = f.refs[i];
    Instr *in = r.set->code.p + (r.loc >> 1);
    items[i] = sr::FoldItem{r.first, r.len, (r.loc & 1) ? &in->b : &in->a};
  }
  std::memcpy(f.h_pack.p + ib, f.tokens.data(), tb);
  ctx->prep_stats.h2d_bytes += static_cast<int64_t>(ib + tb);
  SR_TRY_CUDA(ctx, cudaMemcpyAsync(f.pack.p, f.h_pack.p, ib + tb, cudaMemcpyHostToDevice,
                                   ctx->stream));
  SR_TRY_CUDA(ctx, sr::launch_fold(reinterpret_cast<const sr::FoldItem *>(f.pack.p),
                                   reinterpret_cast<const uint2 *>(f.pack.p + ib),
                                   static_cast<int>(f.refs.size()), ctx->stream));
  return SR_OK;
}

// Derived rows of a population whose programs spill at most `slots` values, at
// most: what 512-datapoint spans, twice buffered, leave of shared memory beside
// the spill slots of 31 warps (31 KB a slot) and the span sums.  More rows leave
// 256-datapoint spans, whose items cost what the rows save (batched population,
// interpreter at the time: no rows 42.9 ms, 16 rows 37.7, 32 rows at 256
// datapoints 37.5; 24 rows with two of the three spill slots it needs, the other
// in global scratch, 46.9).  A bounded part of the device's memory too.
static int derived_row_limit(const sr_context *ctx, int slots) {
  const int fit = (ctx->max_smem - 9 * 1024 - slots * 31 * 1024) / 4096;
  int r = std::min(sr::kMaxDerivedRows, fit - (ctx->V + 1));
  const double row = static_cast<double>(ctx->ldx) * sizeof(float);
  const double room = std::min(1073741824.0, static_cast<double>(ctx->device_memory) / 16.0);
  r = std::min(r, static_cast<int>(room / row));
  return r < 4 ? 0 : r;
}

// Whether finding shared work pays.  The search and the two more kernels cost
// about 0.15 ms and 4 ns a token; the evaluation, 0.28 ms per 1e9 tokens x
// datapoints, becomes a quarter shorter, 0.07 ps a token and datapoint: even at
// 60,000 datapoints for the tokens' part, and 3e9 leaves room for the rest.
// A call without and with it, us:
//   1,000 ramped trees x 100k    660 / 750       1,500 bred x 200k   1,689 / 1,629
//   500 ramped x 400k          1,017 / 1,080     5,000 bred x 100k   2,941 / 2,876
//   1,500 ramped x 200k        1,465 / 1,460     1,500 bred x 400k   3,113 / 2,697
//   500 long x 200k            1,039 / 1,034     5,000 long x 200k   8,990 / 7,440
static bool sharing_pays(const sr_context *ctx, const sr_population *pop) {
  const double tokens = static_cast<double>(pop->offsets[pop->num_exprs]);
  return tokens * (static_cast<double>(ctx->N) - 60000.0) >= 3e9;
}

// Batched programs with the shared work found (sh, or null) taken out: compiled,
// planned and uploaded.
static sr_status prepare_programs(sr_context *ctx, const sr_population *pop, sr::Sharing *sh) {
  const int E = pop->num_exprs;
  const double tc0 = now_ms();
  SR_TRY(compile_set(ctx, E, pop->tokens, pop->values, pop->offsets, nullptr, ctx->main, sh));
  // Programs of long expressions can need a fourth spill slot: fewer rows then.
  if (sh && ctx->main.smax > 3 &&
      static_cast<int>(sh->rows().size()) > derived_row_limit(ctx, 4)) {
    sh->keep_rows(derived_row_limit(ctx, 4));
    ctx->folds.refs.clear();
    ctx->folds.tokens.clear();
    SR_TRY(compile_set(ctx, E, pop->tokens, pop->values, pop->offsets, nullptr, ctx->main, sh));
  }
  if (sh && !sh->rows().empty()) {
    std::vector<int32_t> tok, hints;
    std::vector<double> val;
    std::vector<int64_t> off{0};
    for (const auto &r : sh->rows()) {
      tok.insert(tok.end(), pop->tokens + r.tok, pop->tokens + r.tok + r.size);
      val.insert(val.end(), pop->values + r.tok, pop->values + r.tok + r.size);
      hints.resize(tok.size());
      sh->mark_row(r, hints.data() + off.back());
      off.push_back(static_cast<int64_t>(tok.size()));
    }
    const int R = static_cast<int>(sh->rows().size());
    SR_TRY(compile_set(ctx, R, tok.data(), val.data(), off.data(), hints.data(), ctx->rows));
    for (int r = 0; r < R; ++r) ctx->rows.h_row.p[r] = r;
    SR_TRY(plan_set(ctx, ctx->rows, true, 8, sr::kMaxWarps));
    SR_TRY(upload_set(ctx, ctx->rows, true));
    ctx->main.n_derived = R;
  }
  ctx->prep_stats.host_compile_time_ms += now_ms() - tc0;
  return prepare_main_shape(ctx, true, false);
}

// Batched programs, shared work found and taken out where that pays.
static sr_status prepare_batched(sr_context *ctx, const sr_population *pop, bool with_rows) {
  const double tc0 = now_ms();
  sr::Sharing &sh = ctx->sharing;
  ctx->rows.plan = sr::Plan{};
  bool share = sharing_pays(ctx, pop);
  if (share) {
    SR_TRACE("sr: share");
    share = sh.find(pop->num_exprs, pop->tokens, pop->values, pop->offsets,
                    with_rows ? derived_row_limit(ctx, 3) : 0, ctx->workers, host_threads(ctx));
    // Rows are an option: without the memory for them they are evaluated in
    // place like everything else.
    if (share && !sh.rows().empty() &&
        ctx->derived.ensure(sh.rows().size() * static_cast<size_t>(ctx->ldx)) != cudaSuccess) {
      cudaGetLastError();
      sh.drop_rows();
    }
  }
  ctx->prep_stats.host_compile_time_ms = now_ms() - tc0;
  sr_status st = prepare_programs(ctx, pop, share ? &sh : nullptr);
  // derived_row_limit counts the spill slots of the shapes chosen here; a shape
  // given from outside may leave the rows no shared memory.
  if (st == SR_ERR_UNSUPPORTED && share && !sh.rows().empty()) {
    SR_TRY_CUDA(ctx, cudaStreamSynchronize(ctx->stream));  // the rows' upload
    ctx->last_error.clear();
    ctx->folds.refs.clear();
    ctx->folds.tokens.clear();
    sh.drop_rows();
    st = prepare_programs(ctx, pop, &sh);
  }
  SR_TRY(st);
  const int64_t row_tokens = ctx->main.n_derived > 0 ? ctx->rows.n_executed : 0;
  ctx->prep_stats.node_evals = ctx->main.n_tokens * ctx->N;
  ctx->prep_stats.node_evals_executed = (ctx->main.n_executed + row_tokens) * ctx->N;
  return SR_OK;
}

// Operator profile of a compiled set (the evaluation launches; prediction
// launches always use kOpsAll).
// Shortest datapoint span the planner shrinks to for occupancy.
constexpr int64_t kMinSpan = 256;

bool protected_profile(const ProgramSet &ps) {
  return ps.n_instr > 0 &&
         static_cast<double>(ps.n_instr_protected) >= sr::kProtectedShare * ps.n_instr;
}

// The listed expressions in decreasing cost, equal ones in index order: a
// counting sort over half units of cost (all costs are multiples of one; those
// above the last bucket, far beyond any program that differs in rank, keep
// index order).
static void cost_order(const ProgramSet &ps, sr::GroupRec *order) {
  const std::vector<float> &cost = ps.cost;
  const auto listed = [&](int x) { return !ps.shared || ps.h_row.p[x] == x; };
  const auto rec = [&](int x) { return sr::GroupRec{x, ps.h_len.p[x], ps.h_off.p[x]}; };
  if (ps.E < 1024) {  // fewer than the buckets' own cost
    int n = 0;
    for (int x = 0; x < ps.E; ++x)
      if (listed(x)) order[n++] = rec(x);
    std::stable_sort(order, order + n, [&](const sr::GroupRec &a, const sr::GroupRec &b) {
      return cost[static_cast<size_t>(a.e)] > cost[static_cast<size_t>(b.e)];
    });
    return;
  }
  constexpr int kBuckets = 1 << 14;
  std::vector<int32_t> start(kBuckets + 1, 0);
  const auto bucket = [&](int x) {
    return kBuckets - 1 -
           static_cast<int>(std::min(2.0f * cost[static_cast<size_t>(x)], kBuckets - 1.0f));
  };
  for (int x = 0; x < ps.E; ++x)
    if (listed(x)) ++start[static_cast<size_t>(bucket(x)) + 1];
  for (int b = 0; b < kBuckets; ++b) start[static_cast<size_t>(b) + 1] += start[static_cast<size_t>(b)];
  for (int x = 0; x < ps.E; ++x)
    if (listed(x)) order[start[static_cast<size_t>(bucket(x))]++] = rec(x);
}

// Size class of a launch, from its 256-datapoint tiles of expressions per SM:
// 0 below 120, 1 below 600, 2 below 6,000, 3 above.  A small launch wants every
// warp of every SM at work on one expression and one tile: groups of one
// expression per warp and 256-datapoint spans, in blocks of 8 warps at first,
// then in the wide ones (500 expressions x 1,000 datapoints 86 -> 34 us, 1,000 x
// 10,000 186 -> 112 us against groups of 124).  A middle one takes groups of two
// expressions per warp, so that the last groups balance over the SMs (1,000 x
// 100,000 720 -> 517 us, 4,000 x 30,000 853 -> 638 us); a large one reuses each
// staged span for four (1,531 x 250,007: 2,172 us with two, 2,165 us).  Timed on
// expressions of 2 to 7 variables around each line.
int launch_size(const sr_context *ctx, int E) {
  const double tiles = static_cast<double>(E) * static_cast<double>((ctx->N + 255) / 256);
  const double per_sm = tiles / std::max(ctx->num_sms, 1);
  return per_sm < 120.0 ? 0 : (per_sm < 600.0 ? 1 : (per_sm < 6000.0 ? 2 : 3));
}

// interp_configure with its answer kept (the shared-memory limit it raises is
// raised again by the launch).
static cudaError_t resident_blocks(sr_context *ctx, int dpt, bool pred, int ops, bool general,
                                   size_t smem, int W, int *bps) {
  const std::array<int64_t, 6> key{dpt, pred, ops, general, static_cast<int64_t>(smem), W};
  const auto it = ctx->occupancy.find(key);
  if (it != ctx->occupancy.end()) {
    *bps = it->second;
    return cudaSuccess;
  }
  const cudaError_t e = sr::interp_configure(dpt, pred, ops, general, smem, W, bps);
  if (e == cudaSuccess) {
    if (ctx->occupancy.size() >= 1024) ctx->occupancy.clear();
    ctx->occupancy.emplace(key, *bps);
  }
  return e;
}

// Launch shape: groups of G cost-sorted expressions x spans of datapoints.
// `split`: spill slots per warp kept in shared memory (-1 = the default for
// the dpt); the deeper slots live in per-warp global scratch.  `per_warp`:
// expressions per group and evaluating warp (a group of G = W x per_warp
// expressions shares each staged X span), 0 to choose it, and the span, by the
// launch's size.
sr_status plan_set(sr_context *ctx, ProgramSet &ps, bool pred, int dpt, int W, int split,
                   int per_warp, int span_target) {
  sr::Plan p;
  p.dpt = dpt;
  p.W = W;
  p.ops = (!pred && protected_profile(ps)) ? sr::kOpsProtected : sr::kOpsAll;
  p.smax = std::max(ps.smax, 0);
  const int slots = sr::smem_spill_slots(dpt);
  p.s_smem = std::min(p.smax, split >= 0 ? split : slots);
  p.general = !pred && (ps.cache_refs || p.s_smem < p.smax);
  const int64_t tile = 32 * dpt;
  const int E = ps.n_listed;
  const int rows = ctx->V + ps.n_derived;  // besides y
  const bool by_size = per_warp <= 0;
  if (by_size) {
    const int size = launch_size(ctx, E);
    per_warp = size <= 1 ? 1 : (size == 2 ? 2 : 4);
    if (size <= 1) span_target = static_cast<int>(std::max<int64_t>(tile, kMinSpan));
    // Derived rows fill shared memory: spans of 512 at most, and at a middle
    // size twice the expressions for them.
    if (ps.n_derived > 0 && span_target > 512) {
      span_target = 512;
      per_warp = 4;
    }
  }
  p.G = std::max(1, W * per_warp);
  p.n_groups = (E + p.G - 1) / p.G;
  const size_t max_smem = static_cast<size_t>(ctx->max_smem);
  // Span: the target, shrunk to the data and to the shared-memory budget.
  int64_t span = std::min<int64_t>(span_target, std::max<int64_t>(tile, round_up(ctx->N, tile)));
  auto smem_at = [&](int64_t sp) {
    return sr::interp_smem_bytes(dpt, W, rows, p.s_smem, static_cast<int>(sp), p.G, pred);
  };
  while (span > tile && smem_at(span) > max_smem) span = std::max<int64_t>(tile, (span / 2) / tile * tile);
  if (smem_at(span) > max_smem)
    return ctx->fail(SR_ERR_UNSUPPORTED, "launch shape needs " + std::to_string(smem_at(span)) +
                                             " bytes of shared memory");
  // Then, while the span's shared memory (the X buffers grow with the
  // variable count) rather than the registers limits the resident blocks,
  // halve it: more resident warps pay for more, shorter work items
  // (9 variables, 8 datapoints x 8 warps: 2 -> 3 blocks per SM at 512).
  int bps = 0;
  SR_TRY_CUDA(ctx, resident_blocks(ctx, dpt, pred, p.ops, p.general, smem_at(span), W, &bps));
  while (span / 2 >= std::max<int64_t>(tile, kMinSpan) && (span / 2) % tile == 0) {
    int bps_half = 0;
    SR_TRY_CUDA(ctx, resident_blocks(ctx, dpt, pred, p.ops, p.general, smem_at(span / 2), W,
                                     &bps_half));
    if (bps_half <= bps) break;
    span /= 2;
    bps = bps_half;
  }
  // The kernel walks a span tile by tile: it must hold whole tiles.
  if (span % tile != 0) return ctx->fail(SR_ERR_UNSUPPORTED, "span is not a multiple of the tile");
  p.span = static_cast<int>(span);
  p.smem = smem_at(p.span);
  p.n_spans = (ctx->N == 0 || E == 0) ? 0 : static_cast<int>((ctx->N + span - 1) / span);
  // Spans per work item: as many as keep about 32 items of 32 expressions
  // per SM (up to 32 spans), so the per-(span group, expression) entries stay
  // small while the items still balance over the SMs; counted in units of 32
  // expressions, so that larger groups (more warps per block) do not cut the
  // span range into more span groups.  The result does not depend on this
  // choice (the spans' sums are added as double-doubles).
  p.k_spans = 1;
  if (!pred && p.n_spans > 0) {
    const int64_t units = (static_cast<int64_t>(E) + 31) / 32;
    const int64_t per_sm = static_cast<int64_t>(p.n_spans) * units /
                           (32 * static_cast<int64_t>(std::max(ctx->num_sms, 1)));
    p.k_spans = static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(32, per_sm)));
  }
  // One FP64 (sum as hi + lo, count) per (span group, expression): 32 B x E
  // x span groups.  It is sized against the device's memory (the allocation
  // itself reports SR_ERR_OUT_OF_MEMORY when the free memory is short).
  if (!pred) {
    const double need = static_cast<double>(p.n_span_groups()) * ps.E * 32.0;
    if (need > 0.9 * static_cast<double>(ctx->device_memory))
      return ctx->fail(SR_ERR_UNSUPPORTED,
                       "partial-sum buffer (" + std::to_string(static_cast<int64_t>(need)) +
                           " bytes) exceeds the device memory; split the population or the "
                           "datapoints");
  }
  if (bps <= 0) return ctx->fail(SR_ERR_UNSUPPORTED, "launch shape does not fit on an SM");
  const int64_t resident = static_cast<int64_t>(bps) * ctx->num_sms;
  // Few single-span items per resident block in a shape given from outside:
  // shorter spans give more, smaller items and a shorter tail.
  if (!pred && !by_size && p.k_spans == 1) {
    while (p.items() < 16 * resident && p.span / 2 >= std::max<int64_t>(tile, 256) &&
           (p.span / 2) % tile == 0) {
      p.span /= 2;
      p.n_spans = static_cast<int>((ctx->N + p.span - 1) / p.span);
    }
    p.smem = smem_at(p.span);
  }
  p.blocks = static_cast<int>(std::min<int64_t>(resident, std::max<int64_t>(p.items(), 1)));
  // Global scratch for the spill slots that do not fit in shared memory.
  const size_t spill_floats = static_cast<size_t>(p.blocks) * W *
                              static_cast<size_t>(p.smax - p.s_smem) * static_cast<size_t>(tile);
  if (spill_floats > 0) SR_TRY_CUDA(ctx, ctx->spill.ensure(spill_floats));
  // Group table: expressions in decreasing modelled cost, G per group, so
  // every group holds similar work and hands out its largest first.
  if (p.G > sr::kMaxGroup) return ctx->fail(SR_ERR_UNSUPPORTED, "expression group too large");
  cost_order(ps, ps.h_group.p);
  for (int64_t k = ps.n_listed; k < static_cast<int64_t>(p.n_groups) * p.G; ++k)
    ps.h_group.p[k] = sr::GroupRec{-1, 0, 0};
  ps.plan = p;
  return SR_OK;
}

sr_status upload_groups(sr_context *ctx, ProgramSet &ps) {
  SR_TRACE("sr: upload groups");
  const size_t ng = static_cast<size_t>(std::max(ps.plan.n_groups * ps.plan.G, 1));
  ctx->prep_stats.h2d_bytes += static_cast<int64_t>(ng * sizeof(sr::GroupRec));
  SR_TRY_CUDA(ctx, cudaMemcpyAsync(ps.group.p, ps.h_group.p, ng * sizeof(sr::GroupRec),
                                   cudaMemcpyHostToDevice, ctx->stream));
  return SR_OK;
}

sr_status upload_set(sr_context *ctx, ProgramSet &ps, bool groups) {
  SR_TRACE("sr: upload");
  SR_TRY_CUDA(ctx, ps.layout_device(static_cast<size_t>(ps.n_instr + 1), static_cast<size_t>(ps.E)));
  const size_t ng = groups ? static_cast<size_t>(ps.plan.n_groups) * ps.plan.G : 0;
  const size_t bytes = static_cast<size_t>(
      reinterpret_cast<unsigned char *>(ps.h_group.p + ng) - ps.h_pack.p);
  ctx->prep_stats.h2d_bytes += static_cast<int64_t>(bytes);
  SR_TRY_CUDA(ctx, cudaMemcpyAsync(ps.pack.p, ps.h_pack.p, bytes, cudaMemcpyHostToDevice,
                                   ctx->stream));
  return SR_OK;
}

// Work counters at zero, by a memset where the last sequence has not left them
// so.  counters_used follows what has been enqueued for execution: on a stream
// that its owner is capturing the memset goes into the capture, whose replays
// meet whatever ran before them, and the flag stays set.
static sr_status zero_counters(sr_context *ctx) {
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  SR_TRY_CUDA(ctx, cudaStreamIsCapturing(ctx->stream, &capture));
  ctx->outer_capture = capture != cudaStreamCaptureStatusNone;
  if (ctx->outer_capture || ctx->counters_used)
    SR_TRY_CUDA(ctx, cudaMemsetAsync(ctx->d_counter, 0, sr::kCounters * sizeof(int32_t),
                                     ctx->stream));
  ctx->counters_used = ctx->outer_capture;
  return SR_OK;
}

sr_status begin_sequence(sr_context *ctx) {
  if (ctx->capturing) return SR_OK;  // the launch of the graph sees to it
  SR_TRY(zero_counters(ctx));
  ctx->counters_used = true;
  return SR_OK;
}

void finish_sequence(sr_context *ctx) {
  if (!ctx->capturing && !ctx->outer_capture) ctx->counters_used = false;
}

sr::SequenceEnd sequence_end(sr_context *ctx) {
  sr::SequenceEnd e;
  e.counters = ctx->d_counter;
  e.n_counters = sr::kCounters;
  e.error = ctx->d_error;
  e.error_out = reinterpret_cast<int32_t *>(ctx->mse.p) + ctx->E;
  return e;
}

sr::EvalArgs make_args(sr_context *ctx, ProgramSet &ps, int32_t *counter) {
  sr::EvalArgs a{};
  a.X = ctx->X.p;
  a.ldx = ctx->ldx;
  a.N = ctx->N;
  a.code = ps.code.p;
  a.code_off = ps.off.p;
  a.code_len = ps.len.p;
  a.groups = ps.group.p;
  a.partial = ctx->partial.p;
  a.work_counter = counter;
  a.error = ctx->d_error;
  a.cache = ctx->cache_vals.p;
  a.ldc = ctx->ldx;
  a.V = ctx->V;
  a.E = ps.E;
  a.derived = ctx->derived.p;
  a.n_derived = ps.n_derived;
  a.n_listed = ps.n_listed;
  a.W = ps.plan.W;
  a.smax = ps.plan.smax;
  a.G = ps.plan.G;
  a.n_groups = ps.plan.n_groups;
  a.span = ps.plan.span;
  a.n_spans = ps.plan.n_spans;
  a.spill = ctx->spill.p;
  a.s_smem = ps.plan.s_smem;
  a.span_per_item = ps.plan.k_spans;
  return a;
}

sr_status launch_set(sr_context *ctx, ProgramSet &ps, bool pred, int32_t *counter,
                     float *pred_out, int64_t ldp, const int32_t *pred_row) {
  if (ps.plan.items() == 0) return SR_OK;
  sr::EvalArgs a = make_args(ctx, ps, counter);
  a.pred = pred_out;
  a.ldp = ldp;
  a.pred_row = pred_row;
  SR_TRY_CUDA(ctx, sr::launch_interp(ps.plan.dpt, pred, ps.plan.ops, ps.plan.general, a,
                                     ps.plan.blocks, ps.plan.smem,
                                     ctx->stream));
  return SR_OK;
}

// Derived rows of the prepared population, if it has any.
static sr_status launch_rows(sr_context *ctx) {
  if (ctx->main.n_derived == 0) return SR_OK;
  return launch_set(ctx, ctx->rows, true, ctx->d_counter + 1, ctx->derived.p, ctx->ldx,
                    ctx->rows.row.p);
}

// ---- launch-shape tuning ---------------------------------------------------

std::string tune_key(const sr_context *ctx, const ProgramSet &ps) {
  const int lg_n = ctx->N > 0 ? static_cast<int>(std::log2(static_cast<double>(ctx->N))) : 0;
  const int lg_e = ps.E > 0 ? static_cast<int>(std::log2(static_cast<double>(ps.E))) : 0;
  const double mean_instr = ps.E > 0 ? static_cast<double>(ps.n_instr) / ps.E : 0.0;
  std::ostringstream k;
  const bool prot = protected_profile(ps);
  k << ctx->device_name << "|V" << ctx->V << "|N" << lg_n << "|E" << lg_e << "|I"
    << static_cast<int>(std::lround(std::log2(1.0 + mean_instr) * 4.0)) << "|S" << ps.smax
    << "|P" << (prot ? sr::kOpsProtected : sr::kOpsAll);
  if (ps.n_derived > 0) k << "|R" << ps.n_derived;
  return k.str();
}

void load_tune_cache(sr_context *ctx) {
  ctx->tune_loaded = true;
  if (!ctx->opts.tune_cache_path) return;
  std::ifstream f(ctx->opts.tune_cache_path);
  if (!f) return;
  // Format: one entry per line:  "key": [dpt, W, split, per_warp],  (the last
  // two optional)
  std::string line;
  while (std::getline(f, line)) {
    const size_t q0 = line.find('"'), q1 = line.find('"', q0 + 1);
    const size_t b0 = line.find('[', q1), b1 = line.find(']', b0);
    if (q0 == std::string::npos || q1 == std::string::npos || b0 == std::string::npos ||
        b1 == std::string::npos)
      continue;
    int dpt = 0, w = 0, split = -1, per_warp = 4;
    const int n = std::sscanf(line.c_str() + b0, "[%d, %d, %d, %d]", &dpt, &w, &split, &per_warp);
    if (n >= 2 && (dpt == 4 || dpt == 8 || dpt == 16) && w >= 1 && w <= sr::kMaxInterpWarps &&
        split >= -1 && split <= sr::kMaxSpillSlots && per_warp >= 1 && per_warp <= 16)
      ctx->tuned[line.substr(q0 + 1, q1 - q0 - 1)] = {dpt, w, n >= 3 ? split : -1,
                                                       n >= 4 ? per_warp : 4};
  }
}

void save_tune_cache(const sr_context *ctx) {
  if (!ctx->opts.tune_cache_path) return;
  std::ofstream f(ctx->opts.tune_cache_path, std::ios::trunc);
  if (!f) return;
  f << "{\n";
  size_t i = 0;
  for (const auto &kv : ctx->tuned) {
    f << "  \"" << kv.first << "\": [" << kv.second.dpt << ", " << kv.second.W << ", "
      << kv.second.split << ", " << kv.second.per_warp << "]"
      << (++i < ctx->tuned.size() ? "," : "") << "\n";
  }
  f << "}\n";
}

// Milliseconds of two launches of the prepared main set in the given shape
// (after one warm-up launch); a negative value when the shape does not fit.
static sr_status time_shape(sr_context *ctx, int dpt, int W, int split, int per_warp,
                            float *ms_out) {
  *ms_out = -1.f;
  if (plan_set(ctx, ctx->main, false, dpt, W, split, per_warp) != SR_OK) {
    ctx->last_error.clear();
    return SR_OK;
  }
  SR_TRY(upload_groups(ctx, ctx->main));
  SR_TRY_CUDA(ctx, ctx->partial.ensure(static_cast<size_t>(std::max<int64_t>(
                       2 * static_cast<int64_t>(ctx->main.plan.n_span_groups()) * ctx->main.E,
                       1))));
  cudaEvent_t a = ctx->ev[4], b = ctx->ev[5];
  float t_sum = 0.f;
  for (int rep = 0; rep < 3; ++rep) {
    SR_TRY(begin_sequence(ctx));
    SR_TRY_CUDA(ctx, cudaEventRecord(a, ctx->stream));
    SR_TRY(launch_set(ctx, ctx->main, false, ctx->d_counter, nullptr, 0, nullptr));
    SR_TRY_CUDA(ctx, cudaEventRecord(b, ctx->stream));
    SR_TRY_CUDA(ctx, cudaEventSynchronize(b));
    const float ms = elapsed_ms(a, b);
    if (rep > 0) t_sum += ms;  // the first run warms up
  }
  *ms_out = t_sum;
  return SR_OK;
}

// Times candidate shapes on the prepared population and keeps the fastest:
// first datapoints per thread x warps per block with the default spill split,
// then, for programs that spill, other splits of the spill slots between
// shared memory and global scratch for the winning shape (fewer slots in
// shared memory can fit more blocks per SM; more keep the deeper slots out
// of L2), then the expressions per group (2, 4 or 8 per warp: larger groups
// reuse each staged X span more, smaller ones balance better).
sr_status autotune_main(sr_context *ctx, const std::string &key) {
  SR_TRACE("sr: autotune");
  static const int kCand[][2] = {{16, 8}, {16, 16}, {8, 8}, {8, 15}, {8, 31}, {4, 8}, {4, 16}};
  float best = 1e30f;
  sr_context::TunedShape win{8, 8, -1, 4};
  for (const auto &c : kCand) {
    float ms = 0.f;
    SR_TRY(time_shape(ctx, c[0], c[1], -1, 4, &ms));
    if (ms >= 0.f && ms < best) {
      best = ms;
      win = {c[0], c[1], -1, 4};
    }
  }
  const int smax = ctx->main.smax;
  if (smax > 0) {
    const int rule = std::min(smax, sr::smem_spill_slots(win.dpt));
    int tried[4] = {rule, -1, -1, -1};
    int n_tried = 1;
    for (const int split : {0, rule / 2, smax}) {
      if (split > sr::kMaxSpillSlots || std::find(tried, tried + n_tried, split) != tried + n_tried)
        continue;
      tried[n_tried++] = split;
      float ms = 0.f;
      SR_TRY(time_shape(ctx, win.dpt, win.W, split, 4, &ms));
      if (ms >= 0.f && ms < best) {
        best = ms;
        win.split = split;
      }
    }
  }
  for (const int per_warp : {2, 8}) {
    float ms = 0.f;
    SR_TRY(time_shape(ctx, win.dpt, win.W, win.split, per_warp, &ms));
    if (ms >= 0.f && ms < best) {
      best = ms;
      win.per_warp = per_warp;
    }
  }
  ctx->tuned[key] = win;
  save_tune_cache(ctx);
  return SR_OK;
}

sr_status prepare_main_shape(sr_context *ctx, bool allow_tune, bool on_device) {
  ProgramSet &ps = ctx->main;
  int dpt = ctx->opts.dpt, W = ctx->opts.warps_per_block, split = -1, per_warp = 0;
  if (dpt == 0 || W == 0) {
    if (!ctx->tune_loaded) load_tune_cache(ctx);
    const std::string key = tune_key(ctx, ps);
    auto it = ctx->tuned.find(key);
    if (it == ctx->tuned.end() && allow_tune && ctx->opts.autotune && ps.E > 0 && ctx->N > 0) {
      if (!on_device) {
        SR_TRY(upload_set(ctx, ps, false));
        SR_TRY(upload_folds(ctx));
        SR_TRY(begin_sequence(ctx));
        SR_TRY(launch_rows(ctx));
        on_device = true;
      }
      SR_TRY(autotune_main(ctx, key));
      it = ctx->tuned.find(key);
    }
    // Untuned defaults: 8 datapoints x 31 warps (one 1,024-thread block per
    // SM) for the protected profile, 8 x 8 (3 blocks per SM) where the wide
    // block's shared memory would not fit even at the shortest span (many
    // variables); 4 x 16 for populations over every operator, whose larger
    // dispatch switch fits the instruction cache better at 4 datapoints
    // (150 -> 82 ms on 4,000 all-operator expressions x 1M datapoints); 8
    // warps for small launches (launch_size).
    const bool prot = protected_profile(ps);
    const bool have = it != ctx->tuned.end();
    int wide = 8;
    if (prot) {
      const int s_smem = std::min(std::max(ps.smax, 0), sr::smem_spill_slots(8));
      const int W = sr::kMaxInterpWarps;
      if (sr::interp_smem_bytes(8, W, ctx->V + ps.n_derived, s_smem, 32 * 8 * 2, W * 4, false) <=
          static_cast<size_t>(ctx->max_smem))
        wide = W;
    }
    const int tdpt = have ? it->second.dpt : (prot ? 8 : 4);
    const bool small = launch_size(ctx, ps.n_listed) == 0;
    const int tw = have ? it->second.W : (small ? 8 : (prot ? wide : 16));
    // the tuned split belongs to the tuned shape only
    if (have && (dpt == 0 || dpt == tdpt) && (W == 0 || W == tw)) {
      split = it->second.split;
      per_warp = it->second.per_warp;
    }
    if (dpt == 0) dpt = W > sr::kMaxWarps ? 8 : tdpt;
    if (W == 0) W = tw;
  }
  if (ctx->opts.smem_spill_slots >= 0) split = ctx->opts.smem_spill_slots;
  SR_TRY(plan_set(ctx, ps, false, dpt, W, split, per_warp));
  if (on_device) {
    SR_TRY(upload_groups(ctx, ps));
  } else {
    SR_TRY(upload_set(ctx, ps, true));
    SR_TRY(upload_folds(ctx));
  }
  SR_TRY_CUDA(ctx, ctx->partial.ensure(static_cast<size_t>(std::max<int64_t>(
                       2 * static_cast<int64_t>(ps.plan.n_span_groups()) * ps.E, 1))));
  return SR_OK;
}

}  // namespace capi
}  // namespace sr

// ============================================================================
// Record timing event k on the context stream.  While sr_launch captures a
// graph the event is recorded as an external event, which makes it an
// event-record node of the graph (a plain record would only mark a capture
// dependency); outside capture that flag is not accepted.
cudaError_t sr::capi::record_event(sr_context *ctx, int k) {
  return ctx->capturing ? cudaEventRecordWithFlags(ctx->ev[k], ctx->stream, cudaEventRecordExternal)
                        : cudaEventRecord(ctx->ev[k], ctx->stream);
}

// Forget the prepared launch (and its captured graph, whose kernel arguments
// point into buffers that the next prepare / set_data may move).
void sr::capi::reset_prepared(sr_context *ctx) {
  ctx->mode = sr::Mode::kNone;
  ctx->folds.refs.clear();
  ctx->folds.tokens.clear();
  ctx->launched = false;
  ctx->cache.rollback();  // subtrees of a launch that never ran hold no values
  if (ctx->graph_exec) {
    cudaGraphExecDestroy(ctx->graph_exec);
    ctx->graph_exec = nullptr;
  }
  ctx->graph_launches = 0;
}

// Derived rows are an option: a call that fails for want of memory (and drops
// the prepared launch anyway) gives theirs back and tries once more.
bool sr::capi::give_back_rows(sr_context *ctx, sr_status st) {
  if (st != SR_ERR_OUT_OF_MEMORY || !ctx->derived.p) return false;
  if (cudaStreamSynchronize(ctx->stream) != cudaSuccess) return false;
  reset_prepared(ctx);
  ctx->derived.release();
  ctx->last_error.clear();
  return true;
}

// Drop the dataset, the cache built on it and every prepared launch.
void sr::capi::invalidate_data(sr_context *ctx) {
  reset_prepared(ctx);
  ctx->cache.clear();  // cached subtree values belong to the old data
  ctx->V = -1;
  ctx->N = 0;
}

extern "C" {

int32_t sr_abi_version(void) { return SR_ABI_VERSION; }

sr_status sr_inject_allocation_failure(int64_t n) {
  if (n < 0) return SR_ERR_INVALID_ARGUMENT;
  sr::alloc_fault_countdown().store(n);
  return SR_OK;
}

const char *sr_status_string(sr_status s) {
  switch (s) {
    case SR_OK: return "ok";
    case SR_ERR_INVALID_ARGUMENT: return "invalid argument";
    case SR_ERR_BAD_TOKEN: return "unknown token";
    case SR_ERR_MALFORMED_EXPRESSION: return "malformed expression";
    case SR_ERR_EXPRESSION_TOO_LONG: return "expression too long";
    case SR_ERR_NO_DATA: return "no dataset on the device";
    case SR_ERR_CUDA: return "CUDA error";
    case SR_ERR_OUT_OF_MEMORY: return "out of memory";
    case SR_ERR_DEVICE_TIMEOUT: return "device wait timed out";
    case SR_ERR_DEVICE_CHECK: return "device bounds check failed";
    case SR_ERR_UNSUPPORTED: return "unsupported";
    case SR_ERR_NO_DEVICE: return "no CUDA device";
    case SR_ERR_TOO_MANY_VARS: return "too many variables";
  }
  return "unknown status";
}

const char *sr_last_error(const sr_context *ctx) {
  return ctx ? ctx->last_error.c_str() : "";
}

sr_status sr_options_init(sr_options *o) {
  if (!o) return SR_ERR_INVALID_ARGUMENT;
  std::memset(o, 0, sizeof *o);
  o->device = -1;
  o->cache_capacity = 2048;
  o->min_subtree_size = 3;
  o->min_subtree_freq = 10;
  o->dpt = 0;
  o->warps_per_block = 0;
  o->autotune = 0;
  o->use_graphs = 0;
  o->host_threads = 0;
  o->tune_cache_path = nullptr;
  o->stream = nullptr;
  o->smem_spill_slots = -1;
  return SR_OK;
}

sr_status sr_create(const sr_options *opts, sr_context **out) {
  if (!out) return SR_ERR_INVALID_ARGUMENT;
  *out = nullptr;
  sr_options o;
  if (opts) o = *opts;
  else sr_options_init(&o);
  if (o.dpt != 0 && o.dpt != 4 && o.dpt != 8 && o.dpt != 16) return SR_ERR_INVALID_ARGUMENT;
  if (o.warps_per_block < 0 || o.warps_per_block > sr::kMaxInterpWarps) return SR_ERR_INVALID_ARGUMENT;
  // More than 16 warps per block exist only at 8 datapoints per thread.
  if (o.warps_per_block > sr::kMaxWarps && o.dpt != 0 && o.dpt != 8) return SR_ERR_INVALID_ARGUMENT;
  if (o.smem_spill_slots < -1 || o.smem_spill_slots > sr::kMaxSpillSlots)
    return SR_ERR_INVALID_ARGUMENT;
  if (o.cache_capacity < 0 || o.min_subtree_size < 1 || o.min_subtree_freq < 1)
    return SR_ERR_INVALID_ARGUMENT;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev <= 0) {
    cudaGetLastError();
    return SR_ERR_NO_DEVICE;
  }
  int dev = o.device;
  if (dev < 0 && cudaGetDevice(&dev) != cudaSuccess) return SR_ERR_NO_DEVICE;
  if (dev >= ndev) return SR_ERR_INVALID_ARGUMENT;
  auto *ctx = new sr_context();
  ctx->opts = o;
  ctx->device = dev;
  DeviceScope scope(dev);
  cudaDeviceProp prop{};
  if (cudaGetDeviceProperties(&prop, dev) != cudaSuccess || prop.major < 10) {
    delete ctx;
    return SR_ERR_NO_DEVICE;  // this build carries sm_100a code only
  }
  ctx->num_sms = prop.multiProcessorCount;
  ctx->device_memory = prop.totalGlobalMem;
  ctx->max_smem = static_cast<int>(prop.sharedMemPerBlockOptin);
  ctx->sm_smem = static_cast<int>(prop.sharedMemPerMultiprocessor);
  ctx->block_smem = static_cast<int>(prop.reservedSharedMemPerBlock);
  ctx->device_name = prop.name;
  ctx->cache.capacity = o.cache_capacity;
  cudaError_t e = cudaSuccess;
  if (o.stream) {
    ctx->stream = static_cast<cudaStream_t>(o.stream);
  } else {
    e = cudaStreamCreateWithFlags(&ctx->stream, cudaStreamNonBlocking);
    ctx->own_stream = (e == cudaSuccess);
  }
  if (e == cudaSuccess) e = cudaMalloc(&ctx->d_counter, sr::kCounters * sizeof(int32_t));
  if (e == cudaSuccess)
    e = cudaMemsetAsync(ctx->d_counter, 0, sr::kCounters * sizeof(int32_t), ctx->stream);
  if (e == cudaSuccess) e = cudaMalloc(&ctx->d_error, sizeof(int32_t));
  if (e == cudaSuccess) e = cudaMemsetAsync(ctx->d_error, 0, sizeof(int32_t), ctx->stream);
  if (e == cudaSuccess) e = cudaMallocHost(&ctx->h_error, sizeof(int32_t));
  for (int i = 0; i < 6 && e == cudaSuccess; ++i) e = cudaEventCreate(&ctx->ev[i]);
  if (e != cudaSuccess) {
    sr_destroy(ctx);
    return e == cudaErrorMemoryAllocation ? SR_ERR_OUT_OF_MEMORY : SR_ERR_CUDA;
  }
  *out = ctx;
  return SR_OK;
}

sr_status sr_destroy(sr_context *ctx) {
  if (!ctx) return SR_OK;
  DeviceScope scope(ctx->device);
  if (ctx->stream) cudaStreamSynchronize(ctx->stream);
  reset_prepared(ctx);
  for (auto &ev : ctx->ev)
    if (ev) cudaEventDestroy(ev);
  if (ctx->d_counter) cudaFree(ctx->d_counter);
  if (ctx->d_error) cudaFree(ctx->d_error);
  if (ctx->h_error) cudaFreeHost(ctx->h_error);
  if (ctx->own_stream && ctx->stream) cudaStreamDestroy(ctx->stream);
  delete ctx;  // device and pinned buffers are released by their owners
  return SR_OK;
}

static sr_status set_data_device(sr_context *ctx, const float *X_dev, int64_t ld, int32_t num_vars,
                                 int64_t num_dps) {
  SR_TRACE("sr_set_data_device");
  if (!ctx) return SR_ERR_INVALID_ARGUMENT;
  if (num_vars < 0 || num_dps < 0 || (num_dps > 0 && !X_dev) || ld < num_dps)
    return ctx->fail(SR_ERR_INVALID_ARGUMENT, "bad dataset arguments");
  if (num_vars > SR_MAX_VARS)
    return ctx->fail(SR_ERR_TOO_MANY_VARS, "num_vars " + std::to_string(num_vars) +
                                               " exceeds " + std::to_string(SR_MAX_VARS));
  DeviceScope scope(ctx->device);
  SR_TRY_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  // Done before X is touched: a failure below (allocation, copy) leaves the
  // context without data instead of holding launches that point into a
  // released or half-written X.
  invalidate_data(ctx);
  const int64_t ldx = std::max<int64_t>(sr::kDataAlign, round_up(num_dps, sr::kDataAlign));
  const size_t rows = static_cast<size_t>(num_vars) + 1;
  SR_TRY_CUDA(ctx, ctx->X.ensure(rows * static_cast<size_t>(ldx)));
  SR_TRY_CUDA(ctx, cudaMemsetAsync(ctx->X.p, 0, rows * ldx * sizeof(float), ctx->stream));
  if (num_dps > 0)
    SR_TRY_CUDA(ctx, cudaMemcpy2DAsync(ctx->X.p, ldx * sizeof(float), X_dev, ld * sizeof(float),
                                       num_dps * sizeof(float), rows, cudaMemcpyDeviceToDevice,
                                       ctx->stream));
  SR_TRY_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  ctx->ldx = ldx;
  ctx->V = num_vars;
  ctx->N = num_dps;
  return SR_OK;
}

sr_status sr_set_data_device(sr_context *ctx, const float *X_dev, int64_t ld, int32_t num_vars,
                             int64_t num_dps) {
  const sr_status st = set_data_device(ctx, X_dev, ld, num_vars, num_dps);
  return ctx && give_back_rows(ctx, st) ? set_data_device(ctx, X_dev, ld, num_vars, num_dps) : st;
}

static sr_status set_data_host(sr_context *ctx, const float *X, const float *const *rows_ptr,
                               int32_t num_vars, int64_t num_dps) {
  SR_TRACE("sr_set_data");
  if (!ctx) return SR_ERR_INVALID_ARGUMENT;
  if (num_vars < 0 || num_dps < 0 || (num_dps > 0 && !X && !rows_ptr))
    return ctx->fail(SR_ERR_INVALID_ARGUMENT, "bad dataset arguments");
  if (num_vars > SR_MAX_VARS)
    return ctx->fail(SR_ERR_TOO_MANY_VARS, "num_vars " + std::to_string(num_vars) +
                                               " exceeds " + std::to_string(SR_MAX_VARS));
  DeviceScope scope(ctx->device);
  SR_TRY_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  // Done before X is touched: a failure below (allocation, copy) leaves the
  // context without data instead of holding launches that point into a
  // released or half-written X.
  invalidate_data(ctx);
  const int64_t ldx = std::max<int64_t>(sr::kDataAlign, round_up(num_dps, sr::kDataAlign));
  const size_t rows = static_cast<size_t>(num_vars) + 1;
  SR_TRY_CUDA(ctx, ctx->X.ensure(rows * static_cast<size_t>(ldx)));
  SR_TRY_CUDA(ctx, cudaMemsetAsync(ctx->X.p, 0, rows * ldx * sizeof(float), ctx->stream));
  if (num_dps > 0) {
    if (X) {
      SR_TRY_CUDA(ctx, cudaMemcpy2DAsync(ctx->X.p, ldx * sizeof(float), X,
                                         num_dps * sizeof(float), num_dps * sizeof(float), rows,
                                         cudaMemcpyHostToDevice, ctx->stream));
    } else {
      for (size_t v = 0; v < rows; ++v) {
        if (!rows_ptr[v]) return ctx->fail(SR_ERR_INVALID_ARGUMENT, "data row is NULL");
        SR_TRY_CUDA(ctx, cudaMemcpyAsync(ctx->X.p + v * ldx, rows_ptr[v], num_dps * sizeof(float),
                                         cudaMemcpyHostToDevice, ctx->stream));
      }
    }
  }
  SR_TRY_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  ctx->ldx = ldx;
  ctx->V = num_vars;
  ctx->N = num_dps;
  return SR_OK;
}

static sr_status set_data(sr_context *ctx, const float *X, const float *const *rows,
                          int32_t num_vars, int64_t num_dps) {
  const sr_status st = set_data_host(ctx, X, rows, num_vars, num_dps);
  return ctx && give_back_rows(ctx, st) ? set_data_host(ctx, X, rows, num_vars, num_dps) : st;
}

sr_status sr_set_data(sr_context *ctx, const float *X, int32_t num_vars, int64_t num_dps) {
  return set_data(ctx, X, nullptr, num_vars, num_dps);
}

sr_status sr_set_data_rows(sr_context *ctx, const float *const *rows, int32_t num_vars,
                           int64_t num_dps) {
  if (ctx && num_dps > 0 && !rows) return ctx->fail(SR_ERR_INVALID_ARGUMENT, "rows is NULL");
  return set_data(ctx, nullptr, rows, num_vars, num_dps);
}

}  // extern "C"

namespace sr {
namespace capi {

// ---- prepare --------------------------------------------------------------

sr_status prepare_plain(sr_context *ctx, const sr_population *pop) {
  SR_TRACE("sr: prepare plain");
  sr::PlainSet &ps = ctx->plain;
  const int E = pop->num_exprs;
  const int64_t T = pop->offsets[E];
  // Validate through the compiler (same rules as the batched path) and check
  // the raw stack depth against the plain kernel's local stack.
  std::vector<Instr> scratch;
  for (int x = 0; x < E; ++x) {
    const int64_t o = pop->offsets[x];
    const int len = static_cast<int>(pop->offsets[x + 1] - o);
    sr::ExprInfo info;
    std::string err;
    scratch.clear();
    const sr_status s = sr::compile_expression(pop->tokens + o, pop->values + o, len, ctx->V,
                                               nullptr, scratch, info, &err);
    if (s != SR_OK) return ctx->fail(s, "expression " + std::to_string(x) + ": " + err);
    int depth = 0, maxd = 0;
    for (int i = len - 1; i >= 0; --i) {
      const int t = pop->tokens[o + i];
      if (t <= 0) ++depth;
      else if (sr::is_binary_token(t)) --depth;
      maxd = std::max(maxd, depth);
    }
    if (maxd > sr::kPlainStack)
      return ctx->fail(SR_ERR_UNSUPPORTED, "expression " + std::to_string(x) +
                                               " exceeds the plain kernel's stack");
  }
  SR_TRY_CUDA(ctx, ps.h_tok.ensure(static_cast<size_t>(T)));
  SR_TRY_CUDA(ctx, ps.h_val.ensure(static_cast<size_t>(T)));
  SR_TRY_CUDA(ctx, ps.h_off.ensure(static_cast<size_t>(E)));
  SR_TRY_CUDA(ctx, ps.h_len.ensure(static_cast<size_t>(E)));
  for (int64_t i = 0; i < T; ++i) {
    const int t = pop->tokens[i];
    const double v = pop->values[i];
    ps.h_tok.p[i] = t;
    if (t == SR_TOK_VAR) {
      const bool ok = v > -2147483648.0 && v < 2147483648.0;
      const int vi = ok ? static_cast<int>(v) : -1;
      ps.h_val.p[i] = static_cast<float>((vi >= 0 && vi < ctx->V) ? vi : -1);
    } else {
      ps.h_val.p[i] = static_cast<float>(v);
    }
  }
  for (int x = 0; x < E; ++x) {
    ps.h_off.p[x] = pop->offsets[x];
    ps.h_len.p[x] = static_cast<int32_t>(pop->offsets[x + 1] - pop->offsets[x]);
  }
  SR_TRY_CUDA(ctx, ps.tok.ensure(static_cast<size_t>(T)));
  SR_TRY_CUDA(ctx, ps.val.ensure(static_cast<size_t>(T)));
  SR_TRY_CUDA(ctx, ps.off.ensure(static_cast<size_t>(E)));
  SR_TRY_CUDA(ctx, ps.len.ensure(static_cast<size_t>(E)));
  SR_TRY_CUDA(ctx, cudaMemcpyAsync(ps.tok.p, ps.h_tok.p, T * sizeof(int32_t),
                                   cudaMemcpyHostToDevice, ctx->stream));
  SR_TRY_CUDA(ctx, cudaMemcpyAsync(ps.val.p, ps.h_val.p, T * sizeof(float),
                                   cudaMemcpyHostToDevice, ctx->stream));
  SR_TRY_CUDA(ctx, cudaMemcpyAsync(ps.off.p, ps.h_off.p, E * sizeof(int64_t),
                                   cudaMemcpyHostToDevice, ctx->stream));
  SR_TRY_CUDA(ctx, cudaMemcpyAsync(ps.len.p, ps.h_len.p, E * sizeof(int32_t),
                                   cudaMemcpyHostToDevice, ctx->stream));
  ps.E = E;
  ctx->prep_stats.h2d_bytes += T * static_cast<int64_t>(sizeof(int32_t) + sizeof(float)) +
                               static_cast<int64_t>(E) * (sizeof(int64_t) + sizeof(int32_t));
  ps.n_dpblocks = static_cast<int>(std::min<int64_t>((ctx->N + 127) / 128, 256));
  SR_TRY_CUDA(ctx, ctx->partial.ensure(static_cast<size_t>(
                       std::max<int64_t>(static_cast<int64_t>(ps.n_dpblocks) * E, 1))));
  ctx->prep_stats.node_evals = T * ctx->N;
  ctx->prep_stats.node_evals_executed = T * ctx->N;
  return SR_OK;
}

// Common-subtree detection on the context's GPU: the same Detection as
// sr::detect_common_subtrees (groups largest first, stable in hash order).
sr_status detect_on_device(sr_context *ctx, int E, const int32_t *tok, const double *val,
                                  const int64_t *off, int min_size, int min_freq,
                                  sr::Detection &out) {
  SR_TRACE("sr: detect (device)");
  out = sr::Detection{};
  out.total_tokens = E > 0 ? off[E] - off[0] : 0;
  const int64_t T = out.total_tokens;
  if (E <= 0 || T <= 0) return SR_OK;
  if (T >= (1ll << 31)) return ctx->fail(SR_ERR_UNSUPPORTED, "population too large for device detection");
  sr::DetectBufs &b = ctx->det;
  cudaStream_t s = ctx->stream;
  const size_t n = static_cast<size_t>(T);
  SR_TRY_CUDA(ctx, cudaStreamSynchronize(s));  // buffers may grow
  SR_TRY_CUDA(ctx, b.tok.ensure(n));
  SR_TRY_CUDA(ctx, b.val.ensure(n));
  SR_TRY_CUDA(ctx, b.off.ensure(static_cast<size_t>(E) + 1));
  for (auto *buf : {&b.size, &b.pos_in, &b.pos_out, &b.run_count, &b.run_start, &b.rep, &b.gsize,
                    &b.vcount})
    SR_TRY_CUDA(ctx, buf->ensure(n));
  SR_TRY_CUDA(ctx, b.out3.ensure(3 * n));
  for (auto *buf : {&b.hash, &b.key_in, &b.key_out, &b.run_key}) SR_TRY_CUDA(ctx, buf->ensure(n));
  SR_TRY_CUDA(ctx, b.cand.ensure(n));
  SR_TRY_CUDA(ctx, b.mark.ensure(n));
  SR_TRY_CUDA(ctx, b.counters.ensure(2));
  SR_TRY_CUDA(ctx, b.covered.ensure(1));
  SR_TRY_CUDA(ctx, b.h_counters.ensure(2));
  SR_TRY_CUDA(ctx, b.h_covered.ensure(1));
  const size_t temp = std::max(sr::detect_scratch_sizes(T).temp_bytes,
                               sr::detect_scan_temp_bytes(static_cast<int>(T)));
  SR_TRY_CUDA(ctx, b.temp.ensure(std::max<size_t>(temp, 1)));
  SR_TRY_CUDA(ctx, cudaMemcpyAsync(b.tok.p, tok + off[0], n * sizeof(int32_t),
                                   cudaMemcpyHostToDevice, s));
  SR_TRY_CUDA(ctx, cudaMemcpyAsync(b.val.p, val + off[0], n * sizeof(double),
                                   cudaMemcpyHostToDevice, s));
  SR_TRY_CUDA(ctx, cudaMemcpyAsync(b.off.p, off, (static_cast<size_t>(E) + 1) * sizeof(int64_t),
                                   cudaMemcpyHostToDevice, s));
  sr::DetectArgs a{};
  a.tok = b.tok.p;
  a.val = b.val.p;
  a.off = b.off.p;
  a.E = E;
  a.T = T;
  a.min_size = min_size;
  a.min_freq = min_freq;
  a.size = b.size.p;
  a.hash = b.hash.p;
  a.cand = b.cand.p;
  a.mark = b.mark.p;
  a.pos_in = b.pos_in.p;
  a.pos_out = b.pos_out.p;
  a.key_in = b.key_in.p;
  a.key_out = b.key_out.p;
  a.run_key = b.run_key.p;
  a.run_count = b.run_count.p;
  a.run_start = b.run_start.p;
  a.rep = b.rep.p;
  a.gsize = b.gsize.p;
  a.vcount = b.vcount.p;
  a.n_sel = b.counters.p;
  a.n_runs = b.counters.p + 1;
  a.covered = b.covered.p;
  a.temp = b.temp.p;
  a.temp_bytes = b.temp.cap;
  auto read_counters = [&]() -> sr_status {
    SR_TRY_CUDA(ctx, cudaMemcpyAsync(b.h_counters.p, b.counters.p, 2 * sizeof(int32_t),
                                     cudaMemcpyDeviceToHost, s));
    SR_TRY_CUDA(ctx, cudaStreamSynchronize(s));
    return SR_OK;
  };
  SR_TRY_CUDA(ctx, cudaMemsetAsync(b.counters.p, 0, 2 * sizeof(int32_t), s));
  SR_TRY_CUDA(ctx, sr::detect_candidates(a, s));
  SR_TRY(read_counters());
  const int M = b.h_counters.p[0];
  SR_TRY_CUDA(ctx, sr::detect_groups(a, M, s));
  SR_TRY(read_counters());
  const int R = M > 0 ? b.h_counters.p[1] : 0;
  SR_TRY_CUDA(ctx, sr::detect_verify(a, R, s));
  SR_TRY_CUDA(ctx, sr::detect_frequent(a, R, b.out3.p, s));
  SR_TRY(read_counters());
  const int F = R > 0 ? b.h_counters.p[0] : 0;
  SR_TRY_CUDA(ctx, b.h_out3.ensure(static_cast<size_t>(3 * std::max(F, 1))));
  if (F > 0)
    SR_TRY_CUDA(ctx, cudaMemcpyAsync(b.h_out3.p, b.out3.p, 3 * static_cast<size_t>(F) * sizeof(int32_t),
                                     cudaMemcpyDeviceToHost, s));
  SR_TRY_CUDA(ctx, cudaMemcpyAsync(b.h_covered.p, b.covered.p, sizeof(unsigned long long),
                                   cudaMemcpyDeviceToHost, s));
  SR_TRY_CUDA(ctx, cudaStreamSynchronize(s));
  // Groups in hash order -> size descending, stable.
  std::vector<int> order(static_cast<size_t>(F));
  std::iota(order.begin(), order.end(), 0);
  const int32_t *o3 = b.h_out3.p;
  std::stable_sort(order.begin(), order.end(),
                   [&](int x, int y) { return o3[3 * x + 1] > o3[3 * y + 1]; });
  int64_t size_sum = 0;
  out.groups.reserve(static_cast<size_t>(F));
  for (int k : order) {
    const int64_t g = o3[3 * k] + off[0];  // absolute token index
    const int64_t *it = std::upper_bound(off, off + E + 1, g) - 1;
    const int32_t x = static_cast<int32_t>(it - off);
    out.groups.push_back(sr::Detection::Group{x, static_cast<int32_t>(g - off[x]), o3[3 * k + 1],
                                              o3[3 * k + 2]});
    size_sum += o3[3 * k + 1];
  }
  out.covered_tokens = static_cast<int64_t>(*b.h_covered.p);
  out.avg_subtree_size = F > 0 ? static_cast<double>(size_sum) / F : 0.0;
  out.coverage = T > 0 ? static_cast<double>(out.covered_tokens) / T : 0.0;
  return SR_OK;
}

sr_status prepare_cached(sr_context *ctx, const sr_population *pop, uint32_t flags) {
  SR_TRACE("sr: prepare cached");
  const int E = pop->num_exprs;
  const int64_t T = pop->offsets[E];
  // Validate first so that malformed input never reaches the cache.
  {
    std::vector<Instr> scratch;
    for (int x = 0; x < E; ++x) {
      const int64_t o = pop->offsets[x];
      sr::ExprInfo info;
      std::string err;
      scratch.clear();
      const sr_status s = sr::compile_expression(pop->tokens + o, pop->values + o,
                                                 static_cast<int>(pop->offsets[x + 1] - o), ctx->V,
                                                 nullptr, scratch, info, &err);
      if (s != SR_OK) return ctx->fail(s, "expression " + std::to_string(x) + ": " + err);
    }
  }
  if (flags & SR_EVAL_CLEAR_CACHE) ctx->cache.clear();
  const int threads = host_threads(ctx);
  const double t0 = now_ms();
  sr::Detection det;
  if (ctx->opts.device_detect) {
    SR_TRY(detect_on_device(ctx, E, pop->tokens, pop->values, pop->offsets,
                            ctx->opts.min_subtree_size, ctx->opts.min_subtree_freq, det));
  } else {
    SR_TRACE("sr: detect (host)");
    sr::detect_common_subtrees(E, pop->tokens, pop->values, pop->offsets,
                               ctx->opts.min_subtree_size, ctx->opts.min_subtree_freq, threads,
                               det);
  }
  ctx->prep_stats.detect_time_ms = now_ms() - t0;
  ctx->prep_stats.num_subtrees = static_cast<int32_t>(det.groups.size());
  ctx->prep_stats.avg_subtree_size = det.avg_subtree_size;
  ctx->prep_stats.coverage = det.coverage;

  // Cache update (reference cl_gpu_eval.cu:384-396): new keys get the next
  // free slot until the capacity is reached.  They stay pending until this
  // prepare's launch is enqueued (sr_launch commits them).
  ctx->cache.begin_pending();
  std::vector<int32_t> sub_tok;
  std::vector<double> sub_val;
  std::vector<int64_t> sub_off{0};
  std::vector<int32_t> sub_slot;
  for (const auto &g : det.groups) {
    const int32_t *t = pop->tokens + pop->offsets[g.expr] + g.pos;
    const double *v = pop->values + pop->offsets[g.expr] + g.pos;
    const uint64_t key = sr::flat_key(t, v, g.size);
    if (ctx->cache.slot_of.count(key)) continue;
    if (ctx->cache.used >= ctx->cache.capacity) continue;
    const int32_t slot = ctx->cache.used++;
    ctx->cache.slot_of.emplace(key, slot);
    ctx->cache.pending.push_back(key);
    sub_tok.insert(sub_tok.end(), t, t + g.size);
    sub_val.insert(sub_val.end(), v, v + g.size);
    sub_off.push_back(static_cast<int64_t>(sub_tok.size()));
    sub_slot.push_back(slot);
  }
  const int n_new = static_cast<int>(sub_slot.size());
  ctx->prep_stats.new_subtrees = n_new;
  ctx->prep_stats.cache_slots_used = ctx->cache.used;

  // Cache values live in [capacity][ldx]; allocated on first use.
  if (ctx->cache.capacity > 0)
    SR_TRY_CUDA(ctx, ctx->cache_vals.ensure(static_cast<size_t>(ctx->cache.capacity) * ctx->ldx));

  // Subtrees to evaluate into the cache this call.
  const double tc0 = now_ms();
  // Constant subtrees are folded in both sets (a cached one too, where it lies in
  // a larger subtree of constants or is one: a constant costs no load).
  SR_TRY(compile_set(ctx, n_new, sub_tok.data(), sub_val.data(), sub_off.data(), nullptr, ctx->sub,
                     nullptr, true));
  for (int k = 0; k < n_new; ++k) ctx->sub.h_row.p[k] = sub_slot[static_cast<size_t>(k)];
  if (n_new > 0) {
    SR_TRY(plan_set(ctx, ctx->sub, true, 8, sr::kMaxWarps));
    SR_TRY(upload_set(ctx, ctx->sub, true));
  } else {
    ctx->sub.plan = sr::Plan{};
  }

  // Skeletons (reference mark_cached_subtrees_from_state + skeleton rewrite,
  // cl_gpu_eval.cu:294-329, 433-459).
  ctx->hints.resize(static_cast<size_t>(T));
  sr::mark_cached_subtrees(E, pop->tokens, pop->values, pop->offsets, ctx->cache, threads,
                           ctx->hints.data());
  SR_TRY(compile_set(ctx, E, pop->tokens, pop->values, pop->offsets, ctx->hints.data(), ctx->main,
                     nullptr, true));
  ctx->prep_stats.host_compile_time_ms = now_ms() - tc0;
  SR_TRY(prepare_main_shape(ctx, false, false));
  ctx->prep_stats.node_evals = T * ctx->N;
  ctx->prep_stats.node_evals_executed = (ctx->main.n_executed + ctx->sub.n_executed) * ctx->N;
  return SR_OK;
}

}  // namespace capi
}  // namespace sr

extern "C" {

// One attempt; without derived rows (with_rows = false) after memory ran out.
static sr_status prepare_once(sr_context *ctx, const sr_population *pop, uint32_t flags,
                              bool with_rows) {
  SR_TRY_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  reset_prepared(ctx);
  ctx->prep_stats = sr_stats{};
  const int E = pop->num_exprs;
  ctx->E = E;
  if (E == 0) return SR_OK;
  // One entry more than expressions: the device error word travels behind the
  // results (SequenceEnd).
  SR_TRY_CUDA(ctx, ctx->mse.ensure(static_cast<size_t>(E) + 1));
  SR_TRY_CUDA(ctx, ctx->h_mse.ensure(static_cast<size_t>(E) + 1));
  SR_TRY_CUDA(ctx, cudaEventRecord(ctx->ev[4], ctx->stream));
  if (flags & SR_EVAL_GRADIENT) {
    SR_TRY(prepare_grad(ctx, pop, (flags & SR_EVAL_GRAD_RECOMPUTE) != 0,
                        (flags & SR_EVAL_GRAD_REVERSE) != 0));
    ctx->mode = sr::Mode::kGrad;
  } else if (flags & SR_EVAL_PLAIN) {
    SR_TRY(prepare_plain(ctx, pop));
    ctx->mode = sr::Mode::kPlain;
  } else if (flags & SR_EVAL_SUBTREE_CACHE) {
    SR_TRY(prepare_cached(ctx, pop, flags));
    ctx->mode = sr::Mode::kCached;
  } else {
    SR_TRY(prepare_batched(ctx, pop, with_rows));
    ctx->mode = sr::Mode::kBatched;
  }
  SR_TRY_CUDA(ctx, cudaEventRecord(ctx->ev[5], ctx->stream));
  return SR_OK;
}

sr_status sr_prepare(sr_context *ctx, const sr_population *pop, uint32_t flags) {
  SR_TRACE("sr_prepare");
  if (!ctx) return SR_ERR_INVALID_ARGUMENT;
  ctx->last_error.clear();
  SR_TRY(check_population(ctx, pop));
  if (ctx->V < 0) return ctx->fail(SR_ERR_NO_DATA, "no dataset: call sr_set_data first");
  DeviceScope scope(ctx->device);
  const sr_status st = prepare_once(ctx, pop, flags, true);
  return give_back_rows(ctx, st) ? prepare_once(ctx, pop, flags, false) : st;
}

// Where each expression's result is, when equal ones share an evaluation.
static const int32_t *representatives(const sr_context *ctx) {
  return ctx->mode == sr::Mode::kBatched && ctx->main.shared ? ctx->main.row.p : nullptr;
}

// Enqueue the prepared launch sequence on the context stream.
static sr_status enqueue_launch(sr_context *ctx, int *launches_out) {
  cudaStream_t s = ctx->stream;
  SR_TRY_CUDA(ctx, record_event(ctx, 0));
  int launches = 0;
  if (ctx->mode == sr::Mode::kGrad) {
    SR_TRY(launch_grad(ctx));
    launches = grad_launch_count(ctx->grad);
  } else if (ctx->mode == sr::Mode::kPlain) {
    SR_TRY_CUDA(ctx, record_event(ctx, 1));
    SR_TRY_CUDA(ctx, sr::launch_plain(ctx->plain.tok.p, ctx->plain.val.p, ctx->plain.off.p,
                                      ctx->plain.len.p, ctx->X.p, ctx->ldx, ctx->V, ctx->N,
                                      ctx->plain.E, ctx->partial.p, ctx->plain.n_dpblocks, s));
    launches += ctx->N > 0 ? 1 : 0;
    SR_TRY_CUDA(ctx, record_event(ctx, 2));
    SR_TRY_CUDA(ctx, sr::launch_finalize(ctx->partial.p, ctx->N > 0 ? ctx->plain.n_dpblocks : 0,
                                         ctx->E, ctx->mse.p, s));
    ++launches;
  } else {
    SR_TRY(begin_sequence(ctx));
    if (ctx->mode == sr::Mode::kCached && ctx->sub.plan.items() > 0) {
      SR_TRY(launch_set(ctx, ctx->sub, true, ctx->d_counter + 1, ctx->cache_vals.p, ctx->ldx,
                        ctx->sub.row.p));
      ++launches;
    }
    if (ctx->mode == sr::Mode::kBatched && ctx->main.n_derived > 0 && ctx->rows.plan.items() > 0) {
      SR_TRY(launch_rows(ctx));
      ++launches;
    }
    SR_TRY_CUDA(ctx, record_event(ctx, 1));
    if (ctx->main.plan.items() > 0) {
      SR_TRY(launch_set(ctx, ctx->main, false, ctx->d_counter, nullptr, 0, nullptr));
      ++launches;
    }
    SR_TRY_CUDA(ctx, record_event(ctx, 2));
    SR_TRY_CUDA(ctx, sr::launch_finalize_groups(ctx->partial.p, representatives(ctx),
                                                ctx->main.plan.n_span_groups(),
                                                ctx->E, ctx->mse.p, nullptr, sequence_end(ctx),
                                                s));
    finish_sequence(ctx);
    ++launches;
  }
  SR_TRY_CUDA(ctx, record_event(ctx, 3));
  *launches_out = launches;
  return SR_OK;
}

static sr_status launch_prepared(sr_context *ctx, bool allow_graph);

sr_status sr_launch(sr_context *ctx) { return launch_prepared(ctx, true); }

// allow_graph = false for one-shot evaluations (a graph pays off only when the
// prepared launch is replayed).
static sr_status launch_prepared(sr_context *ctx, bool allow_graph) {
  SR_TRACE("sr_launch");
  if (!ctx) return SR_ERR_INVALID_ARGUMENT;
  if (ctx->E == 0) return SR_OK;
  if (ctx->mode == sr::Mode::kNone) return ctx->fail(SR_ERR_INVALID_ARGUMENT, "nothing prepared");
  DeviceScope scope(ctx->device);
  cudaStream_t s = ctx->stream;
  int launches = 0;
  if (ctx->opts.use_graphs && (allow_graph || ctx->graph_exec)) {
    if (!ctx->graph_exec) {
      // Relaxed mode: the launchers set kernel attributes while capturing.
      SR_TRY_CUDA(ctx, cudaStreamBeginCapture(s, cudaStreamCaptureModeRelaxed));
      ctx->capturing = true;
      const sr_status st = enqueue_launch(ctx, &launches);
      ctx->capturing = false;
      cudaGraph_t graph = nullptr;
      const cudaError_t ce = cudaStreamEndCapture(s, &graph);
      if (st != SR_OK) {
        if (graph) cudaGraphDestroy(graph);
        return st;
      }
      SR_TRY_CUDA(ctx, ce);
      const cudaError_t ie = sr::alloc_fault_fires()
                                 ? cudaErrorMemoryAllocation
                                 : cudaGraphInstantiate(&ctx->graph_exec, graph, 0);
      cudaGraphDestroy(graph);
      if (ie != cudaSuccess) ctx->graph_exec = nullptr;
      SR_TRY_CUDA(ctx, ie);
      ctx->graph_launches = launches;
    }
    SR_TRY(zero_counters(ctx));  // the captured sequence only leaves them at zero
    SR_TRY_CUDA(ctx, cudaGraphLaunch(ctx->graph_exec, s));
    launches = ctx->graph_launches;
  } else {
    SR_TRY(enqueue_launch(ctx, &launches));
  }
  ctx->cache.commit();  // the subtree launch that writes the new cached values is enqueued
  ctx->timing_valid = true;
  ctx->launched = true;
  ctx->prep_stats.kernel_launches = launches;
  return SR_OK;
}

}  // extern "C"

namespace sr {
namespace capi {

sr_status check_device_error(sr_context *ctx) {
  if (*ctx->h_error == 0) return SR_OK;
  const int32_t code = *ctx->h_error;
  *ctx->h_error = 0;
  cudaMemsetAsync(ctx->d_error, 0, sizeof(int32_t), ctx->stream);
  cudaStreamSynchronize(ctx->stream);
  ctx->cache.clear();  // the failed launch may have left cached values unwritten
  if (code & sr::kDevErrTimeout)
    return ctx->fail(SR_ERR_DEVICE_TIMEOUT, "a device-side wait exceeded its time limit");
  return ctx->fail(SR_ERR_DEVICE_CHECK, "device bounds check failed");
}

void fill_stats(sr_context *ctx, sr_stats *st) {
  if (!st) return;
  *st = ctx->prep_stats;
  if (ctx->timing_valid) {
    st->gpu_kernel_time_ms = elapsed_ms(ctx->ev[0], ctx->ev[3]);
    st->eval_kernel_time_ms = elapsed_ms(ctx->ev[1], ctx->ev[2]);
    st->data_transfer_time_ms = elapsed_ms(ctx->ev[4], ctx->ev[5]);
  }
  if (ctx->mode == sr::Mode::kBatched || ctx->mode == sr::Mode::kCached) {
    st->declared_sfu_ops = ctx->main.sfu_per_dp * static_cast<double>(ctx->N);
    st->declared_fp32_ops = ctx->main.fp32_per_dp * static_cast<double>(ctx->N);
  }
  st->d2h_bytes += static_cast<int64_t>(ctx->E) * static_cast<int64_t>(sizeof(float)) +
                   static_cast<int64_t>(sizeof(int32_t));
  const sr::Plan &p = ctx->main.plan;
  st->dpt = p.dpt;
  st->warps_per_block = p.W;
  st->blocks = p.blocks;
  st->work_items = static_cast<int32_t>(p.items());
}

}  // namespace capi
}  // namespace sr

extern "C" {

sr_status sr_read_mse(sr_context *ctx, float *mse_out, sr_stats *stats) {
  SR_TRACE("sr_read_mse");
  if (!ctx) return SR_ERR_INVALID_ARGUMENT;
  if (ctx->E == 0) return SR_OK;
  if (ctx->mode == sr::Mode::kNone) return ctx->fail(SR_ERR_INVALID_ARGUMENT, "nothing launched");
  if (!mse_out) return ctx->fail(SR_ERR_INVALID_ARGUMENT, "mse_out is NULL");
  DeviceScope scope(ctx->device);
  // The error word comes with the results of a launch (the plain path raises none).
  const bool with_error = ctx->launched && ctx->mode != sr::Mode::kPlain;
  SR_TRY_CUDA(ctx, cudaMemcpyAsync(ctx->h_mse.p, ctx->mse.p,
                                   (ctx->E + (with_error ? 1 : 0)) * sizeof(float),
                                   cudaMemcpyDeviceToHost, ctx->stream));
  SR_TRY_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  if (with_error) {
    std::memcpy(ctx->h_error, ctx->h_mse.p + ctx->E, sizeof(int32_t));
    SR_TRY(check_device_error(ctx));
  }
  std::memcpy(mse_out, ctx->h_mse.p, ctx->E * sizeof(float));
  fill_stats(ctx, stats);
  return SR_OK;
}

sr_status sr_read_sums(sr_context *ctx, double *sum_out, double *count_out) {
  SR_TRACE("sr_read_sums");
  if (!ctx) return SR_ERR_INVALID_ARGUMENT;
  if (ctx->E == 0) return SR_OK;
  if (ctx->mode == sr::Mode::kNone) return ctx->fail(SR_ERR_INVALID_ARGUMENT, "nothing launched");
  if (!sum_out || !count_out)
    return ctx->fail(SR_ERR_INVALID_ARGUMENT, "sum_out / count_out is NULL");
  int n_spans = 0;
  switch (ctx->mode) {
    case sr::Mode::kPlain: n_spans = ctx->N > 0 ? ctx->plain.n_dpblocks : 0; break;
    case sr::Mode::kGrad: n_spans = ctx->grad.n_spans; break;
    default: n_spans = ctx->main.plan.n_span_groups(); break;
  }
  const int E = ctx->E;
  DeviceScope scope(ctx->device);
  SR_TRY_CUDA(ctx, cudaStreamSynchronize(ctx->stream));  // the buffers may grow
  SR_TRY_CUDA(ctx, ctx->sums.ensure(static_cast<size_t>(E)));
  SR_TRY_CUDA(ctx, ctx->h_sums.ensure(static_cast<size_t>(E)));
  if (ctx->mode == sr::Mode::kPlain)
    SR_TRY_CUDA(ctx, sr::launch_sums(ctx->partial.p, n_spans, E, ctx->sums.p, ctx->stream));
  else if (ctx->mode == sr::Mode::kGrad)
    ;  // the gradient finalize kernels wrote ctx->sums
  else
    SR_TRY_CUDA(ctx, sr::launch_finalize_groups(ctx->partial.p, representatives(ctx), n_spans, E, nullptr,
                                                ctx->sums.p, sr::SequenceEnd{}, ctx->stream));
  SR_TRY_CUDA(ctx, cudaMemcpyAsync(ctx->h_sums.p, ctx->sums.p, E * sizeof(double2),
                                   cudaMemcpyDeviceToHost, ctx->stream));
  SR_TRY_CUDA(ctx, cudaMemcpyAsync(ctx->h_error, ctx->d_error, sizeof(int32_t),
                                   cudaMemcpyDeviceToHost, ctx->stream));
  SR_TRY_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  SR_TRY(check_device_error(ctx));
  for (int e = 0; e < E; ++e) {
    sum_out[e] = ctx->h_sums.p[e].x;
    count_out[e] = ctx->h_sums.p[e].y;
  }
  return SR_OK;
}

sr_status sr_read_grad_sums(sr_context *ctx, double *grad_sum_out) {
  if (!ctx) return SR_ERR_INVALID_ARGUMENT;
  if (ctx->E == 0) return SR_OK;
  if (ctx->mode != sr::Mode::kGrad)
    return ctx->fail(SR_ERR_INVALID_ARGUMENT, "no gradient prepared (SR_EVAL_GRADIENT)");
  const int64_t C = ctx->grad.C;
  if (C == 0) return SR_OK;
  if (!grad_sum_out) return ctx->fail(SR_ERR_INVALID_ARGUMENT, "grad_sum_out is NULL");
  DeviceScope scope(ctx->device);
  SR_TRY_CUDA(ctx, cudaMemcpyAsync(grad_sum_out, ctx->grad.grad_acc.p, C * sizeof(double),
                                   cudaMemcpyDeviceToHost, ctx->stream));
  SR_TRY_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  return SR_OK;
}

sr_status sr_read_grad(sr_context *ctx, float *grad_out) {
  if (!ctx) return SR_ERR_INVALID_ARGUMENT;
  if (ctx->E == 0) return SR_OK;
  if (ctx->mode != sr::Mode::kGrad)
    return ctx->fail(SR_ERR_INVALID_ARGUMENT, "no gradient prepared (SR_EVAL_GRADIENT)");
  const int64_t C = ctx->grad.C;
  if (C == 0) return SR_OK;
  if (!grad_out) return ctx->fail(SR_ERR_INVALID_ARGUMENT, "grad_out is NULL");
  DeviceScope scope(ctx->device);
  SR_TRY_CUDA(ctx, cudaMemcpyAsync(grad_out, ctx->grad.grad.p, C * sizeof(float),
                                   cudaMemcpyDeviceToHost, ctx->stream));
  SR_TRY_CUDA(ctx, cudaMemcpyAsync(ctx->h_error, ctx->d_error, sizeof(int32_t),
                                   cudaMemcpyDeviceToHost, ctx->stream));
  SR_TRY_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  SR_TRY(check_device_error(ctx));
  ctx->prep_stats.d2h_bytes += C * static_cast<int64_t>(sizeof(float));
  return SR_OK;
}

sr_status sr_last_launch_times(sr_context *ctx, float *launch_ms, float *eval_kernel_ms) {
  if (!ctx) return SR_ERR_INVALID_ARGUMENT;
  if (!ctx->timing_valid) return ctx->fail(SR_ERR_INVALID_ARGUMENT, "no launch recorded");
  DeviceScope scope(ctx->device);
  SR_TRY_CUDA(ctx, cudaEventSynchronize(ctx->ev[3]));
  float a = 0.f, b = 0.f;
  SR_TRY_CUDA(ctx, cudaEventElapsedTime(&a, ctx->ev[0], ctx->ev[3]));
  SR_TRY_CUDA(ctx, cudaEventElapsedTime(&b, ctx->ev[1], ctx->ev[2]));
  if (launch_ms) *launch_ms = a;
  if (eval_kernel_ms) *eval_kernel_ms = b;
  return SR_OK;
}

sr_status sr_device_mse(sr_context *ctx, float **mse_dev) {
  if (!ctx || !mse_dev) return SR_ERR_INVALID_ARGUMENT;
  *mse_dev = ctx->mse.p;
  return SR_OK;
}

sr_status sr_eval_mse(sr_context *ctx, const sr_population *pop, uint32_t flags, float *mse_out,
                      sr_stats *stats) {
  SR_TRACE("sr_eval_mse");
  if (!ctx) return SR_ERR_INVALID_ARGUMENT;
  const double t0 = now_ms();
  SR_TRY(sr_prepare(ctx, pop, flags));
  if (pop->num_exprs == 0) {
    if (stats) *stats = sr_stats{};
    return SR_OK;
  }
  SR_TRY(launch_prepared(ctx, false));
  SR_TRY(sr_read_mse(ctx, mse_out, stats));
  if (stats) stats->total_eval_time_ms = now_ms() - t0;
  return SR_OK;
}

// Programs, shape and output buffer of a prediction launch.
static sr_status prepare_predictions(sr_context *ctx, const sr_population *pop) {
  const int E = pop->num_exprs;
  SR_TRY_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  reset_prepared(ctx);
  SR_TRY(compile_set(ctx, E, pop->tokens, pop->values, pop->offsets, nullptr, ctx->main));
  for (int x = 0; x < E; ++x) ctx->main.h_row.p[x] = x;
  int dpt = ctx->opts.dpt ? ctx->opts.dpt : 8;
  int W = ctx->opts.warps_per_block ? std::min(ctx->opts.warps_per_block, sr::kMaxWarps)
                                     : sr::kMaxWarps;
  SR_TRY(plan_set(ctx, ctx->main, true, dpt, W));
  SR_TRY(upload_set(ctx, ctx->main, true));
  SR_TRY_CUDA(ctx, ctx->pred.ensure(static_cast<size_t>(E) * ctx->ldx));
  return SR_OK;
}

sr_status sr_eval_predictions(sr_context *ctx, const sr_population *pop, int64_t dp_begin,
                              int64_t dp_count, float *pred_out) {
  SR_TRACE("sr_eval_predictions");
  if (!ctx) return SR_ERR_INVALID_ARGUMENT;
  ctx->last_error.clear();
  SR_TRY(check_population(ctx, pop));
  if (ctx->V < 0) return ctx->fail(SR_ERR_NO_DATA, "no dataset: call sr_set_data first");
  if (dp_begin < 0 || dp_count < 0 || dp_begin + dp_count > ctx->N)
    return ctx->fail(SR_ERR_INVALID_ARGUMENT, "datapoint range outside the dataset");
  if (pop->num_exprs == 0 || dp_count == 0) return SR_OK;
  if (!pred_out) return ctx->fail(SR_ERR_INVALID_ARGUMENT, "pred_out is NULL");
  const int E = pop->num_exprs;
  const double bytes = static_cast<double>(E) * ctx->ldx * sizeof(float);
  if (bytes > 16.0 * (1ull << 30))
    return ctx->fail(SR_ERR_UNSUPPORTED, "prediction buffer would exceed 16 GiB");
  DeviceScope scope(ctx->device);
  const sr_status st = prepare_predictions(ctx, pop);
  SR_TRY(give_back_rows(ctx, st) ? prepare_predictions(ctx, pop) : st);
  SR_TRY(begin_sequence(ctx));
  SR_TRY(launch_set(ctx, ctx->main, true, ctx->d_counter, ctx->pred.p, ctx->ldx, ctx->main.row.p));
  SR_TRY_CUDA(ctx, cudaMemcpy2DAsync(pred_out, dp_count * sizeof(float), ctx->pred.p + dp_begin,
                                     ctx->ldx * sizeof(float), dp_count * sizeof(float), E,
                                     cudaMemcpyDeviceToHost, ctx->stream));
  SR_TRY_CUDA(ctx, cudaMemcpyAsync(ctx->h_error, ctx->d_error, sizeof(int32_t),
                                   cudaMemcpyDeviceToHost, ctx->stream));
  SR_TRY_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  SR_TRY(check_device_error(ctx));
  return SR_OK;
}

sr_status sr_count_constants(const sr_population *pop, int64_t *const_offsets) {
  if (!pop || !const_offsets || pop->num_exprs < 0) return SR_ERR_INVALID_ARGUMENT;
  int64_t acc = 0;
  for (int x = 0; x < pop->num_exprs; ++x) {
    const_offsets[x] = acc;
    for (int64_t i = pop->offsets[x]; i < pop->offsets[x + 1]; ++i)
      acc += pop->tokens[i] == SR_TOK_CONST ? 1 : 0;
  }
  const_offsets[pop->num_exprs] = acc;
  return SR_OK;
}

}  // extern "C"
