// Element-wise part of the 16-bit kernels' epilogues: alpha, bias, activation on the accumulator values
// that a lane holds.
//
// It runs on the CUDA cores between the tensor-memory load and the store of every output, so on factors
// that write much it is the time of a tile.  Values go in pairs through the two-wide fp32 instructions
// (same roundings, half the issue slots), and the bias of a batch-first tile, one value per column, comes
// through shared memory: a lane converts its two values once and every lane reads four columns per
// broadcast load, instead of a shuffle and a conversion per value.  (1,768,192,4) fp16 with a bias, 25088
// rows, batch-first in block order: 82 -> 66 us (61 without a bias), with a GELU too 105 -> 83 us; split in
// the kernel (tc_bsfirst_d.cu), 12544 rows: 63 -> 55 us.
#pragma once

#include "common.cuh"

namespace ksmm {
namespace tc {

__device__ __forceinline__ uint64_t pack_f2(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack_f2(uint64_t v, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ uint64_t fma_f2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t mul_f2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// gelu_16bit (common.cuh) of two values, step by step the same
__device__ __forceinline__ void gelu_16bit_2(uint32_t& r0, uint32_t& r1) {
  const uint64_t x = pack_f2(__uint_as_float(r0), __uint_as_float(r1));
  float u0, u1;
  unpack_f2(mul_f2(x, x), u0, u1);
  const uint64_t u = pack_f2(fminf(u0, 49.f), fminf(u1, 49.f));
  uint64_t p = fma_f2(u, pack_f2(-3.2060774e-4f, -3.2060774e-4f), pack_f2(3.6819428e-2f, 3.6819428e-2f));
  p = fma_f2(p, u, pack_f2(7.9770428e-1f, 7.9770428e-1f));
  float z0, z1, t0, t1;
  unpack_f2(mul_f2(x, p), z0, z1);
  asm("tanh.approx.f32 %0, %1;" : "=f"(t0) : "f"(z0));
  asm("tanh.approx.f32 %0, %1;" : "=f"(t1) : "f"(z1));
  const uint64_t h = mul_f2(x, pack_f2(0.5f, 0.5f));
  float y0, y1;
  unpack_f2(fma_f2(h, pack_f2(t0, t1), h), y0, y1);
  r0 = __float_as_uint(y0);
  r1 = __float_as_uint(y1);
}

// Stages the bias of 64 16-bit output columns as floats at shared address dst: lane t converts elements
// e0 + 2 t and e0 + 2 t + 1, where they exist.  D > 1: column e goes to place (e % D) * (64 / D) + e / D, the
// order of D accumulators side by side.  The caller synchronises the warp before and after.
template <int D>
__device__ __forceinline__ void stage_bias_16(const void* bias, int64_t e0, bool exist, int dtype, uint32_t dst, int lane) {
  float b0 = 0.f, b1 = 0.f;
  if (exist) {
    const uint16_t* bp = static_cast<const uint16_t*>(bias) + e0 + 2 * lane;
    const uint32_t w = (reinterpret_cast<uintptr_t>(bp) & 3) == 0
                           ? *reinterpret_cast<const uint32_t*>(bp)
                           : (static_cast<uint32_t>(bp[0]) | (static_cast<uint32_t>(bp[1]) << 16));
    if (dtype == KSMM_BF16) {
      b0 = __uint_as_float(w << 16);
      b1 = __uint_as_float(w & 0xffff0000u);
    } else {
      b0 = __half2float(__ushort_as_half(static_cast<uint16_t>(w & 0xffffu)));
      b1 = __half2float(__ushort_as_half(static_cast<uint16_t>(w >> 16)));
    }
  }
  if constexpr (D == 1) {
    asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(dst + lane * 8), "f"(b0), "f"(b1) : "memory");
  } else {
    const uint32_t at = dst + ((2 * lane % D) * (64 / D) + 2 * lane / D) * 4;
    asm volatile("st.shared.f32 [%0], %1;" ::"r"(at), "f"(b0) : "memory");
    asm volatile("st.shared.f32 [%0], %1;" ::"r"(at + (64 / D) * 4), "f"(b1) : "memory");
  }
}

// r(e) = alpha * r(e) + bias[e] for N values e, bias staged at shared address src
template <int N, typename Ref>
__device__ __forceinline__ void scale_and_bias(Ref&& r, float alpha, uint32_t src) {
  const uint64_t al = pack_f2(alpha, alpha);
#pragma unroll
  for (int e = 0; e < N; e += 4) {
    float b[4], y[4];
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(b[0]), "=f"(b[1]), "=f"(b[2]), "=f"(b[3])
                 : "r"(src + e * 4)
                 : "memory");
#pragma unroll
    for (int q = 0; q < 4; q += 2) {
      unpack_f2(fma_f2(al, pack_f2(__uint_as_float(r(e + q)), __uint_as_float(r(e + q + 1))), pack_f2(b[q], b[q + 1])), y[q], y[q + 1]);
      r(e + q) = __float_as_uint(y[q]);
      r(e + q + 1) = __float_as_uint(y[q + 1]);
    }
  }
}

// the same with one bias value for all of them
template <int N, typename Ref>
__device__ __forceinline__ void scale_and_add(Ref&& r, float alpha, float bias) {
  const uint64_t al = pack_f2(alpha, alpha), bb = pack_f2(bias, bias);
#pragma unroll
  for (int e = 0; e < N; e += 2) {
    float y0, y1;
    unpack_f2(fma_f2(al, pack_f2(__uint_as_float(r(e)), __uint_as_float(r(e + 1))), bb), y0, y1);
    r(e) = __float_as_uint(y0);
    r(e + 1) = __float_as_uint(y1);
  }
}

// the activation of N values that are rounded to 16 bits (B16) or stay fp32
template <int N, bool B16, typename Ref>
__device__ __forceinline__ void activate(Ref&& r, int act) {
  if (act == KSMM_ACT_GELU) {
#pragma unroll
    for (int e = 0; e < N; e += 2) {
      if constexpr (B16) {
        gelu_16bit_2(r(e), r(e + 1));
      } else {
        r(e) = __float_as_uint(apply_activation(__uint_as_float(r(e)), 1));
        r(e + 1) = __float_as_uint(apply_activation(__uint_as_float(r(e + 1)), 1));
      }
    }
  } else if (act == KSMM_ACT_RELU) {
#pragma unroll
    for (int e = 0; e < N; ++e) r(e) = __float_as_uint(fmaxf(__uint_as_float(r(e)), 0.f));
  }
}

}  // namespace tc
}  // namespace ksmm
