// sr_partials.cuh — one instruction's value and local partials for both gradient
// modes: the hot operators of the protected set inline and two datapoints at a
// time, the others through the routines of sr_grad_ops.cuh.
#pragma once
#include "sr_device.cuh"
#include "sr_grad_ops.cuh"

namespace sr {
namespace {

// How a partial is known: exactly 1, exactly -1, or computed into dT / db.
enum : int { kDOne = 0, kDNeg = 1, kDGen = 2 };

// Operators outside the inline set: value and partials by the general
// routine; T, b, dT, db travel through the stack.
template <int DPT>
__device__ __noinline__ void tan_op_cold(uint32_t op, float *T, float *b, float *dT, float *db) {
  float t[DPT], bb[DPT], d1[DPT], d2[DPT];
#pragma unroll
  for (int k = 0; k < DPT; ++k) {
    t[k] = T[k];
    bb[k] = b[k];
    d1[k] = 0.0f;
    d2[k] = 0.0f;
  }
  apply_op_grad<DPT>(op, t, bb, d1, d2);
#pragma unroll
  for (int k = 0; k < DPT; ++k) {
    T[k] = t[k];
    dT[k] = d1[k];
    db[k] = d2[k];
  }
}

// sin / cos with their derivative for a lane holding an argument outside the
// fast reduction range (out of line, rare).
template <int DPT>
__device__ __noinline__ void tan_sincos_cold(float *T, float *dT, int q_offset) {
#pragma unroll
  for (int k = 0; k < DPT; ++k) {
    float s, c;
    sr_sincosf(T[k], &s, &c);
    T[k] = q_offset ? c : s;
    dT[k] = q_offset ? -s : c;
  }
}

// Division and reciprocal, two datapoints at a time where the lane's arguments
// are of middling magnitude, one by one out of line elsewhere: one short copy
// of each in the kernel's hot code (its instruction-cache misses were its second
// stall).
template <int DPT>
__device__ __noinline__ void div_cold(float *T, const float *b) {
#pragma unroll
  for (int k = 0; k < DPT; ++k) T[k] = __fdiv_rn(T[k], b[k]);
}
template <int DPT>
__device__ __noinline__ void rcp_cold(const float *b, float *r) {
#pragma unroll
  for (int k = 0; k < DPT; ++k) r[k] = __frcp_rn(b[k]);
}
// T = T / b and, for live instructions, r = 1 / b, from one approximate reciprocal
// and one range test (each on its own: 4,096 x 262,144 18.9 -> 18.2 ms, reverse
// mode 512 x 65,536 3.43 -> 3.34 ms).
template <int DPT>
__device__ __forceinline__ void div_rcp_wide(float (&T)[DPT], const float (&b)[DPT],
                                             float (&r)[DPT], bool live) {
  if (fmaxf(max_abs<DPT>(T), max_abs<DPT>(b)) <= kDivMax &&
      min_abs<DPT>(T) >= kDivMin && min_abs<DPT>(b) >= kDivMin) {
#pragma unroll
    for (int k = 0; k < DPT; k += 2) {
      float2 q = make_float2(T[k], T[k + 1]), s;
      div_rcp2_mid(q, make_float2(b[k], b[k + 1]), s);
      T[k] = q.x;
      T[k + 1] = q.y;
      r[k] = s.x;
      r[k + 1] = s.y;
    }
  } else {
    float t[DPT], u[DPT], q[DPT];
#pragma unroll
    for (int k = 0; k < DPT; ++k) {
      t[k] = T[k];
      u[k] = b[k];
    }
    div_cold<DPT>(t, u);
    if (live) rcp_cold<DPT>(u, q);
#pragma unroll
    for (int k = 0; k < DPT; ++k) {
      T[k] = t[k];
      r[k] = q[k];
    }
  }
}
template <int DPT>
__device__ __forceinline__ void rcp_wide(const float (&b)[DPT], float (&r)[DPT]) {
  if (max_abs<DPT>(b) <= kDivMax && min_abs<DPT>(b) >= kDivMin) {
#pragma unroll
    for (int k = 0; k < DPT; k += 2) {
      const float2 q = rcp2_mid(make_float2(b[k], b[k + 1]));
      r[k] = q.x;
      r[k + 1] = q.y;
    }
  } else {
    float u[DPT], q[DPT];
#pragma unroll
    for (int k = 0; k < DPT; ++k) u[k] = b[k];
    rcp_cold<DPT>(u, q);
#pragma unroll
    for (int k = 0; k < DPT; ++k) r[k] = q[k];
  }
}

// T = op(T, b) with the partials a gradient needs (only when `live`:
// instructions off every constant's path skip them).  dk / bk_: how dT / db
// are known.  The IEEE divisions and reciprocals of the protected division
// (both operand orders), the protected log's and sqrt|x|'s derivatives run
// in one shared loop each after the switch, so the code holds one copy of
// each (instruction-cache footprint).
template <int DPT, bool LINEAR>
__device__ __forceinline__ void tan_apply(uint32_t op, bool live, float (&T)[DPT],
                                          float (&b)[DPT], float (&dT)[DPT], float (&db)[DPT],
                                          int &dk, int &bk_) {
  dk = kDGen;
  bk_ = kDGen;
  // post bit 1: T = T / b; bit 2: the partials from 1 / b (when live).  For
  // these operators b holds the divisor (the protected denominator) or, for
  // the unary ones, the value to invert.
  int post = 0;
  if constexpr (LINEAR) {
    switch (op) {
      // + - * in paired FP32 instructions (each half correctly rounded, a - b
      // as a + (-b)): the forward interpreter's values.
      case 1:
#pragma unroll
        for (int k = 0; k < DPT; k += 2) {
          const float2 r = __fadd2_rn(make_float2(T[k], T[k + 1]), make_float2(b[k], b[k + 1]));
          T[k] = r.x;
          T[k + 1] = r.y;
        }
        dk = kDOne;
        bk_ = kDOne;
        return;
      case 2:
#pragma unroll
        for (int k = 0; k < DPT; k += 2) {
          const float2 r = __fadd2_rn(make_float2(T[k], T[k + 1]), make_float2(-b[k], -b[k + 1]));
          T[k] = r.x;
          T[k + 1] = r.y;
        }
        dk = kDOne;
        bk_ = kDNeg;
        return;
      case kOpReversed + 2:
#pragma unroll
        for (int k = 0; k < DPT; k += 2) {
          const float2 r = __fadd2_rn(make_float2(b[k], b[k + 1]), make_float2(-T[k], -T[k + 1]));
          T[k] = r.x;
          T[k + 1] = r.y;
        }
        dk = kDNeg;
        bk_ = kDOne;
        return;
      case 3:
#pragma unroll
        for (int k = 0; k < DPT; k += 2) {
          dT[k] = b[k];
          dT[k + 1] = b[k + 1];
          db[k] = T[k];
          db[k + 1] = T[k + 1];
          const float2 r = __fmul2_rn(make_float2(T[k], T[k + 1]), make_float2(b[k], b[k + 1]));
          T[k] = r.x;
          T[k + 1] = r.y;
        }
        return;
      default: break;
    }
  }
  switch (op) {
    case 0:
      dk = kDOne;
      break;
    case 8:  // T / protected(b)
#pragma unroll
      for (int k = 0; k < DPT; ++k) {
        db[k] = fabsf(b[k]) <= 1e-9f ? 0.0f : 1.0f;  // 0: the flat region
        b[k] = loose_denom(b[k]);
      }
      post = 1 | 2;
      break;
    case kOpReversed + 8:  // b / protected(T), as T' / b' with T' = b, b' = protected(T)
#pragma unroll
      for (int k = 0; k < DPT; ++k) {
        dT[k] = fabsf(T[k]) <= 1e-9f ? 0.0f : 1.0f;
        const float d = loose_denom(T[k]);
        T[k] = b[k];
        b[k] = d;
      }
      post = 1 | 2;
      break;
    case 10:
    case 11: {
      const int qoff = (op == 11) ? 1 : 0;
      if (!(max_abs<DPT>(T) <= kSinCosFastMax)) {
        float t_[DPT], d_[DPT];
#pragma unroll
        for (int k = 0; k < DPT; ++k) t_[k] = T[k];
        tan_sincos_cold<DPT>(t_, d_, qoff);
#pragma unroll
        for (int k = 0; k < DPT; ++k) {
          T[k] = t_[k];
          dT[k] = d_[k];
        }
      } else {
#pragma unroll
        for (int k = 0; k < DPT; k += 2) {
          SinCosParts p0, p1;
          sincos_parts2(make_float2(T[k], T[k + 1]), p0, p1);
          // sin with sin(-0) = -0, as sr_sincosf returns it
          const float s0 = T[k] == 0.0f ? T[k] : sincos_pick(p0, 0);
          const float s1 = T[k + 1] == 0.0f ? T[k + 1] : sincos_pick(p1, 0);
          const float c0 = sincos_pick(p0, 1), c1 = sincos_pick(p1, 1);
          T[k] = qoff ? c0 : s0;
          T[k + 1] = qoff ? c1 : s1;
          dT[k] = qoff ? -s0 : c0;
          dT[k + 1] = qoff ? -s1 : c1;
        }
      }
      break;
    }
    case kOpExpClamp:
#pragma unroll
      for (int k = 0; k < DPT; ++k) {
        const float x = T[k];
        const float o = expf(fminf(x, 80.0f));
        dT[k] = (x < 80.0f) ? o : 0.0f;
        T[k] = o;
      }
      break;
    case 22:  // protected log: -1e9 at 0, else log|x|; derivative 0 at 0, else 1/x
#pragma unroll
      for (int k = 0; k < DPT; ++k) b[k] = T[k];
      llog_wide<DPT>(T);
      post = 2;
      break;
    case 27:  // sqrt|x|: derivative 0 at 0, else sign(x) / (2 out)
#pragma unroll
      for (int k = 0; k < DPT; ++k) dT[k] = T[k];
      lsqrt_wide<DPT>(T);
#pragma unroll
      for (int k = 0; k < DPT; ++k) {
        const float x = dT[k];
        b[k] = x == 0.0f ? 1.0f : 2.0f * T[k];  // at 0: sign 0 times 1
        dT[k] = signf(x);                        // times 1 / (2 out) below
      }
      post = 2;
      break;
    default: {
      float t_[DPT], b_[DPT];
#pragma unroll
      for (int k = 0; k < DPT; ++k) {
        t_[k] = T[k];
        b_[k] = b[k];
      }
      if (live) {
        float d1[DPT], d2[DPT];
        tan_op_cold<DPT>(op, t_, b_, d1, d2);
#pragma unroll
        for (int k = 0; k < DPT; ++k) {
          dT[k] = d1[k];
          db[k] = d2[k];
        }
      } else {
        apply_op_cold<DPT>(op, t_, b_);
      }
#pragma unroll
      for (int k = 0; k < DPT; ++k) T[k] = t_[k];
      break;
    }
  }
  float rc[DPT];
  if (post & 1) {
    div_rcp_wide<DPT>(T, b, rc, live);
  } else if (post && live) {
    rcp_wide<DPT>(b, rc);
  }
  if (post && live) {
    // Partials from the reciprocal (the reverse-mode routines' formulas).
    if (op == 8) {  // d/dT = 1/den, d/db = -out/den (0 in the flat region)
#pragma unroll
      for (int k = 0; k < DPT; ++k) {
        db[k] = db[k] == 0.0f ? 0.0f : __fmul_rn(-T[k], rc[k]);
        dT[k] = rc[k];
      }
    } else if (op == kOpReversed + 8) {  // d/db = 1/den, d/dT = -out/den
#pragma unroll
      for (int k = 0; k < DPT; ++k) {
        dT[k] = dT[k] == 0.0f ? 0.0f : __fmul_rn(-T[k], rc[k]);
        db[k] = rc[k];
      }
    } else if (op == 22) {
#pragma unroll
      for (int k = 0; k < DPT; ++k) dT[k] = b[k] == 0.0f ? 0.0f : rc[k];
    } else {  // 27
#pragma unroll
      for (int k = 0; k < DPT; ++k) dT[k] = dT[k] * rc[k];
    }
  }
}

}  // namespace
}  // namespace sr
