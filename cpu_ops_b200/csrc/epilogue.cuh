// Device-side epilogue: D = chain(act(alpha * acc + beta * C)).
//
// Arithmetic contract (what the CPU library computes, element by element):
//   s32: alpha*acc + beta*C in wrap-around 32-bit arithmetic; C is not read
//        when beta == 0  (epilogue/linear_combination.h:33-38, integer branch)
//   f32: beta != 0 ? fma(beta, C, alpha*acc) : alpha*acc   (:27-31)
//   then Activation::kRelu (:85-87), then the chain ops in order
//   (epilogue/fusion.h:31-129, 136-166).
// Gelu/Silu are evaluated in f32 (silu_f32, gelu_f32); the CPU library itself mixes
// a polynomial vector form and a double-precision scalar form for them, so
// they are compared with a tolerance, never bit for bit.
#pragma once

#include "gemm_params.h"

namespace b200 {

// Gelu and Silu without branches.  An epilogue warp evaluates them for 32 independent elements
// and is one of four or eight warps on its SM, so what counts is that nothing keeps those 32
// chains from overlapping: IEEE division and tanhf compile to code with rarely taken branches,
// and one such branch per element made the chain run one element after the other:
// 2048 x 4096 x 2048 e4m3 with bias + SiLU 120.8 us (31.8 without a chain), 42.1 in this form;
// 512 x 2048 x 1024 21.3 -> 9.7, with GELU 20.8 -> 9.9.

// x == y (x > y) ? a : b as a select: the compiler makes a branch around a costly a or b otherwise.
__device__ __forceinline__ float select_equal(float x, float y, float a, float b) {
  float r;
  asm("{ .reg .pred p; setp.eq.f32 p, %1, %2; selp.f32 %0, %3, %4, p; }" : "=f"(r) : "f"(x), "f"(y), "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float select_greater(float x, float y, float a, float b) {
  float r;
  asm("{ .reg .pred p; setp.gt.f32 p, %1, %2; selp.f32 %0, %3, %4, p; }" : "=f"(r) : "f"(x), "f"(y), "f"(a), "f"(b));
  return r;
}

// a / d from an approximate reciprocal r of d (within an ulp), the quotient q = a r corrected by
// its exact remainder, q - r (d q - a) (Markstein, IBM J. Res. Dev. 34(1), 1990): the IEEE quotient's rounding
// but for near ties, for d in [0.25, 2^126] and a finite quotient.
__device__ __forceinline__ float quotient_f32(float a, float d) {
  const float r = __fdividef(1.0f, d);
  const float q = a * r;
  return __fmaf_rn(-r, __fmaf_rn(d, q, -a), q);
}

// v / (1 + exp(-v)), both sides of the division quartered, which keeps the whole range of the
// denominator within the reciprocal's.  Where it overflows (v < -88.7) the quotient is -0 (of
// -inf: NaN), and where it is 1 the quotient is v (inf has no remainder).  v times a reciprocal is a rounding
// shorter and was up to 0.4 ulp further off: 2048 x 4096 x 2048 + bias + SiLU 39.0 us, 42.1 in this form
// (512 x 2048 x 1024 9.7 in both).
__device__ __forceinline__ float silu_f32(float v) {
  const float d = __fmaf_rn(expf(-v), 0.25f, 0.25f);
  const float y = select_equal(d, 0.25f, v, 0.25f * quotient_f32(v, d));
  return select_equal(d, INFINITY, v * 0.0f, y);
}

// tanh form: 0.5 v (1 + tanh(u)) = v * sigmoid(2 u), from s = sigmoid(-|2 u|): v s below zero, and
// v - v s above, where the last rounding is all but the whole error.  1 + tanhf cancels below
// zero (nothing is left of it at v = -5), this does not; for v in [1, 6] the error against float64 is
// 2.5e-8 rms (with tanhf 3.3e-8, as v * sigmoid 4.3e-8).
__device__ __forceinline__ float gelu_f32(float v) {
  const float x = 2.0f * 0.7978845608028654f * (v + 0.044715f * v * v * v);
  const float t = expf(-fabsf(x));
  const float s = quotient_f32(t, 1.0f + t);
  const float above = select_equal(s, 0.0f, v, __fmaf_rn(-v, s, v));  // (no inf * 0)
  return select_greater(x, 0.0f, above, v * s);
}

template <bool kInt>
__device__ __forceinline__ uint32_t linear_combine_bits(const EpilogueParams& e, uint32_t acc,
                                                        uint32_t src) {
  if constexpr (kInt) {
    uint32_t v = e.alpha * acc;
    if (e.beta_nonzero) v += e.beta * src;
    if (e.activation == 1 && static_cast<int32_t>(v) < 0) v = 0;
    return v;
  } else {
    const float a = __uint_as_float(e.alpha), b = __uint_as_float(e.beta);
    float v = __fmul_rn(a, __uint_as_float(acc));
    if (e.beta_nonzero) v = __fmaf_rn(b, __uint_as_float(src), v);
    if (e.activation == 1) v = v < 0.0f ? 0.0f : v;
    return __float_as_uint(v);
  }
}

template <bool kInt>
__device__ __forceinline__ uint32_t apply_op_bits(const EpilogueOp& op, uint32_t x, int krow,
                                                  int kcol) {
  const int idx = op.index_by_krow ? krow : kcol;
  if constexpr (kInt) {
    int32_t v = static_cast<int32_t>(x);
    switch (op.opcode) {
      case kOpRelu: v = v < 0 ? 0 : v; break;
      case kOpClamp: {
        const int32_t lo = static_cast<int32_t>(op.lo), hi = static_cast<int32_t>(op.hi);
        v = v < lo ? lo : (hi < v ? hi : v);
        break;
      }
      case kOpBiasAdd:
        v = static_cast<int32_t>(static_cast<uint32_t>(v) +
                                 static_cast<uint32_t>(__ldg(static_cast<const int32_t*>(op.ptr) + idx)));
        break;
      case kOpScalePerRow:
      case kOpScalePerCol:
        v = static_cast<int32_t>(static_cast<uint32_t>(v) *
                                 static_cast<uint32_t>(__ldg(static_cast<const int32_t*>(op.ptr) + idx)));
        break;
      default: break;
    }
    return static_cast<uint32_t>(v);
  } else {
    float v = __uint_as_float(x);
    switch (op.opcode) {
      case kOpRelu: v = v < 0.0f ? 0.0f : v; break;
      case kOpClamp: {
        const float lo = __uint_as_float(op.lo), hi = __uint_as_float(op.hi);
        v = v < lo ? lo : (hi < v ? hi : v);
        break;
      }
      case kOpBiasAdd: v = __fadd_rn(v, __ldg(static_cast<const float*>(op.ptr) + idx)); break;
      case kOpScalePerRow:
      case kOpScalePerCol: v = __fmul_rn(v, __ldg(static_cast<const float*>(op.ptr) + idx)); break;
      case kOpGelu: v = gelu_f32(v); break;
      case kOpSilu: v = silu_f32(v); break;
      default: break;
    }
    return __float_as_uint(v);
  }
}

// One chain op on an N-column chunk of one accumulator row (registers r[0..N)).  The
// opcode is uniform over the kernel, so it is dispatched once per chunk, outside the
// element loop; a vector indexed by column is fetched in 16-byte loads (the same
// addresses in every lane: one broadcast transaction each), a vector indexed by row as
// one load.  Columns at or beyond `ncols` are computed on harmlessly and never stored.
// The arithmetic per element is exactly apply_op_bits'.
template <bool kInt, int N>
__device__ __forceinline__ void apply_op_chunk(const EpilogueOp& op, uint32_t (&r)[N], int krow,
                                               int kcol0, int ncols) {
  const int code = op.opcode;
  if (code == kOpBiasAdd || code == kOpScalePerRow || code == kOpScalePerCol) {
    uint32_t v[N];
    const uint32_t* vec = static_cast<const uint32_t*>(op.ptr);
    if (op.index_by_krow) {
      const uint32_t x = __ldg(vec + krow);
#pragma unroll
      for (int i = 0; i < N; ++i) v[i] = x;
    } else if (ncols == N && (reinterpret_cast<uintptr_t>(vec + kcol0) & 15u) == 0) {
#pragma unroll
      for (int i = 0; i < N; i += 4) {
        const uint4 q = __ldg(reinterpret_cast<const uint4*>(vec + kcol0 + i));
        v[i] = q.x; v[i + 1] = q.y; v[i + 2] = q.z; v[i + 3] = q.w;
      }
    } else {
#pragma unroll
      for (int i = 0; i < N; ++i) v[i] = i < ncols ? __ldg(vec + kcol0 + i) : 0u;
    }
    if constexpr (kInt) {
      if (code == kOpBiasAdd) {
#pragma unroll
        for (int i = 0; i < N; ++i) r[i] += v[i];
      } else {
#pragma unroll
        for (int i = 0; i < N; ++i) r[i] *= v[i];
      }
    } else {
      if (code == kOpBiasAdd) {
#pragma unroll
        for (int i = 0; i < N; ++i)
          r[i] = __float_as_uint(__fadd_rn(__uint_as_float(r[i]), __uint_as_float(v[i])));
      } else {
#pragma unroll
        for (int i = 0; i < N; ++i)
          r[i] = __float_as_uint(__fmul_rn(__uint_as_float(r[i]), __uint_as_float(v[i])));
      }
    }
  } else if (code == kOpRelu) {
#pragma unroll
    for (int i = 0; i < N; ++i) {
      if constexpr (kInt) {
        r[i] = static_cast<int32_t>(r[i]) < 0 ? 0u : r[i];
      } else {
        r[i] = __uint_as_float(r[i]) < 0.0f ? 0u : r[i];  // x < 0 ? +0.0f : x (NaN and -0.0 pass)
      }
    }
  } else if (code == kOpClamp) {
#pragma unroll
    for (int i = 0; i < N; ++i) {
      if constexpr (kInt) {
        const int32_t lo = static_cast<int32_t>(op.lo), hi = static_cast<int32_t>(op.hi);
        const int32_t x = static_cast<int32_t>(r[i]);
        r[i] = static_cast<uint32_t>(x < lo ? lo : (hi < x ? hi : x));
      } else {
        const float lo = __uint_as_float(op.lo), hi = __uint_as_float(op.hi);
        const float x = __uint_as_float(r[i]);
        r[i] = __float_as_uint(x < lo ? lo : (hi < x ? hi : x));
      }
    }
  } else if constexpr (!kInt) {
    if (code == kOpGelu) {
#pragma unroll
      for (int i = 0; i < N; ++i) r[i] = __float_as_uint(gelu_f32(__uint_as_float(r[i])));
    } else if (code == kOpSilu) {
#pragma unroll
      for (int i = 0; i < N; ++i) r[i] = __float_as_uint(silu_f32(__uint_as_float(r[i])));
    }
  }
}

// Reads every field of the epilogue parameters once.  Kernel parameters live in constant
// memory, and a field's first read on an SM misses the constant cache (measured: about
// 0.6 us).  The epilogue warps call this while they are still waiting for their first
// accumulator, so that the misses are not paid between the last MMA and the first store.
__device__ __forceinline__ void warm_epilogue_params(const EpilogueParams& e) {
  uint32_t sink = e.alpha ^ e.beta ^ static_cast<uint32_t>(e.beta_nonzero) ^ static_cast<uint32_t>(e.activation) ^
                  static_cast<uint32_t>(e.n_ops) ^ static_cast<uint32_t>(reinterpret_cast<uintptr_t>(e.D)) ^
                  static_cast<uint32_t>(reinterpret_cast<uintptr_t>(e.C)) ^ static_cast<uint32_t>(e.d_sr) ^
                  static_cast<uint32_t>(e.d_sc) ^ static_cast<uint32_t>(e.c_sr) ^ static_cast<uint32_t>(e.c_sc);
#pragma unroll
  for (int t = 0; t < kMaxOps; ++t)
    sink ^= static_cast<uint32_t>(e.ops[t].opcode) ^ static_cast<uint32_t>(reinterpret_cast<uintptr_t>(e.ops[t].ptr)) ^
            e.ops[t].lo ^ e.ops[t].hi;
  asm volatile("" ::"r"(sink));
}

// One element, all steps (used by the split-k reduce and k == 0 kernels).
template <bool kInt>
__device__ __forceinline__ uint32_t epilogue_element(const EpilogueParams& e, uint32_t acc,
                                                     int krow, int kcol) {
  uint32_t src = 0;
  if (e.beta_nonzero) {
    // plain load: C may alias D, which this kernel writes
    src = static_cast<const uint32_t*>(e.C)[krow * e.c_sr + kcol * e.c_sc];
  }
  uint32_t v = linear_combine_bits<kInt>(e, acc, src);
  for (int t = 0; t < e.n_ops; ++t) v = apply_op_bits<kInt>(e.ops[t], v, krow, kcol);
  return v;
}

}  // namespace b200
