// Per-tensor e4m3 quantisation of activations on the device: scale = amax / 448 (1 where the tensor is
// zero or holds a NaN), q = clamp(x / scale, -448, 448), the arithmetic of ksmm_b200.quantize_e4m3.
//
// Two launches and no host round trip: every CTA of the first leaves the largest |x| of its part (as
// bits, so that a NaN wins), every CTA of the second takes the maximum of those partial results, at
// most kParts, and quantises; its first CTA stores the scale, which the factor's kernel reads on the
// device.  The second has a transposing form: a batch-first input lands batch-last, which is how a
// factor that no batch-first kernel covers gets its input without a layout conversion.
//
// 12544 x 768 bf16 (19 MB in, 10 MB out): 9 + 13 us, against 90 us for the eight element-wise launches
// and the device-to-host copy of the scale that they replace; the whole layer of two factors 377 -> 92 us.
//
// The kernels start before the one ahead of them has finished (grid_dep_wait), so none of their loads may
// be of the read-only kind (__ldg, const __restrict__): the compiler may move those above the wait.
#include "backward.h"
#include "common.cuh"
#include "tc_host.h"
#include "tc_ptx.cuh"

namespace ksmm {
namespace {

using tc::grid_dep_launch;
using tc::grid_dep_wait;

__device__ __forceinline__ uint32_t abs_bits(float v) { return __float_as_uint(v) & 0x7fffffffu; }

// the maximum over the block's threads, in every thread
__device__ __forceinline__ uint32_t block_max(uint32_t m) {
  __shared__ uint32_t warp_max[8];
  m = __reduce_max_sync(0xffffffffu, m);
  if ((threadIdx.x & 31) == 0) warp_max[threadIdx.x >> 5] = m;
  __syncthreads();
  m = warp_max[threadIdx.x & 7];
  return __reduce_max_sync(0xffffffffu, m);
}

template <typename T, int V>
__device__ __forceinline__ void load_elems(const T* p, float (&v)[V]) {
  if constexpr (V == 1) {
    v[0] = ElemTraits<T>::to_float(*p);
  } else {
    uint4 raw[V * sizeof(T) / 16];
#pragma unroll
    for (int q = 0; q < static_cast<int>(V * sizeof(T) / 16); ++q) raw[q] = reinterpret_cast<const uint4*>(p)[q];
    const T* e = reinterpret_cast<const T*>(raw);
#pragma unroll
    for (int q = 0; q < V; ++q) v[q] = ElemTraits<T>::to_float(e[q]);
  }
}

template <typename T, int V>
__global__ void __launch_bounds__(256) amax_kernel(const T* in, int64_t ld, int64_t rows, int64_t cols,
                                                   uint32_t* parts) {
  grid_dep_wait();
  grid_dep_launch();
  const int64_t per_row = (cols + V - 1) / V, total = rows * per_row;
  uint32_t m = 0;
#pragma unroll 4
  for (int64_t t = static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x; t < total;
       t += static_cast<int64_t>(gridDim.x) * 256) {
    const int64_t r = rows == 1 ? 0 : (total <= 0x7fffffffLL ? static_cast<uint32_t>(t) / static_cast<uint32_t>(per_row) : t / per_row);
    const int64_t c0 = (t - r * per_row) * V;
    const T* p = in + r * ld + c0;
    if (V == 1 || c0 + V <= cols) {
      float v[V];
      load_elems<T, V>(p, v);
#pragma unroll
      for (int q = 0; q < V; ++q) m = max(m, abs_bits(v[q]));
    } else {
      for (int64_t q = 0; q < cols - c0; ++q) m = max(m, abs_bits(ElemTraits<T>::to_float(p[q])));
    }
  }
  m = block_max(m);
  if (threadIdx.x == 0) parts[blockIdx.x] = m;
}

// the scale of the tensor, in every thread; stored by the first block
__device__ __forceinline__ float tensor_scale(const uint32_t* parts, int nparts, float* scale) {
  uint32_t m = 0;
  for (int t = threadIdx.x; t < nparts; t += 256) m = max(m, parts[t]);
  m = block_max(m);
  const float amax = __uint_as_float(m);
  const float s = amax > 0.f ? amax * (1.f / 448.f) : 1.f;  // (torch divides by a constant this way)
  if (blockIdx.x == 0 && threadIdx.x == 0) *scale = s;
  return s;
}

// v / s rounded as a division rounds it.  With inv = 1 / s rounded, one residual step on v * inv gives that
// quotient (Markstein, "Computation of elementary functions on the IBM RISC System/6000 processor",
// theorem on division) as long as the residual of a value that matters is no denormal number.  Values
// below 2^-11 s quantise to zero either way; the residual of a larger one is a multiple of 2^-48 times it,
// at least 2^-119 for scales from 2^-60 on.  Other scales divide.  So does a scale of 1, the one that a
// tensor with a NaN gets: its infinities are 448, and would be NaN by the residual step.  Three instructions
// instead of a division's dozen, which bound the quantising kernels (16.6 -> 12.6 us for 12544 x 768 bf16,
// 20.4 -> 18.4 us transposing; both include the wait for the first launch).
struct Scale {
  float s, inv;
  bool plain;  // divide
  __device__ explicit Scale(float v) : s(v), inv(1.f / v), plain(!(v > 0x1p-60f && v < 0x1p60f) || v == 1.f) {}
  __device__ __forceinline__ float quotient(float v) const {
    if (plain) return v / s;
    const float q = v * inv;
    return fmaf(fmaf(-q, s, v), inv, q);
  }
};
// two neighbouring values; the conversion saturates at 448, which is the clamp, and keeps a NaN
__device__ __forceinline__ uint32_t quantise2(float v0, float v1, const Scale& s) {
  return __nv_cvt_float2_to_fp8x2(make_float2(s.quotient(v0), s.quotient(v1)), __NV_SATFINITE, __NV_E4M3);
}
__device__ __forceinline__ uint8_t quantise1(float v, const Scale& s) {
  return __nv_cvt_float_to_fp8(s.quotient(v), __NV_SATFINITE, __NV_E4M3);
}

template <typename T, int V>
__global__ void __launch_bounds__(256)
    quantize_kernel(const T* in, int64_t in_ld, uint8_t* out, int64_t out_ld, int64_t rows,
                    int64_t cols, const uint32_t* parts, int nparts, float* scale) {
  grid_dep_wait();
  grid_dep_launch();
  const Scale s(tensor_scale(parts, nparts, scale));
  constexpr int C = V == 1 ? 2 : V;
  const int64_t per_row = (cols + 15) / 16, total = rows * per_row;  // 16 results per thread and step
  for (int64_t t = static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x; t < total;
       t += static_cast<int64_t>(gridDim.x) * 256) {
    const int64_t r = rows == 1 ? 0 : (total <= 0x7fffffffLL ? static_cast<uint32_t>(t) / static_cast<uint32_t>(per_row) : t / per_row);
    const int64_t c0 = (t - r * per_row) * 16;
    const T* src = in + r * in_ld + c0;
    uint8_t* dst = out + r * out_ld + c0;
    if (c0 + 16 <= cols) {
      uint32_t w[4] = {0, 0, 0, 0};
#pragma unroll
      for (int q = 0; q < 16 / C; ++q) {
        float v[C];
        if constexpr (V == 1) {
          load_elems<T, 1>(src + q * 2, reinterpret_cast<float(&)[1]>(v[0]));
          load_elems<T, 1>(src + q * 2 + 1, reinterpret_cast<float(&)[1]>(v[1]));
        } else {
          load_elems<T, V>(src + q * V, v);
        }
#pragma unroll
        for (int e = 0; e < C; e += 2) w[(q * C + e) >> 2] |= quantise2(v[e], v[e + 1], s) << (((q * C + e) & 2) * 8);
      }
      *reinterpret_cast<uint4*>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
    } else {
      for (int64_t q = 0; q < cols - c0; ++q) dst[q] = quantise1(ElemTraits<T>::to_float(src[q]), s);
    }
  }
}

// in: (rows, cols) contiguous, out: (cols, rows) with row stride out_ld.  A tile of 128 rows x 64 columns
// goes through shared memory as bytes; a padded pitch keeps the column reads on distinct banks.
template <typename T, int V>
__global__ void __launch_bounds__(256)
    quantize_transpose_kernel(const T* in, uint8_t* out, int64_t out_ld, int64_t rows,
                              int64_t cols, uint32_t tiles_x, const uint32_t* parts, int nparts, float* scale) {
  constexpr int TR = 128, TC = 64, PITCH = TC + 4;
  __shared__ __align__(16) uint8_t tile[TR * PITCH];
  grid_dep_wait();
  grid_dep_launch();
  const Scale s(tensor_scale(parts, nparts, scale));
  const int64_t r0 = static_cast<int64_t>(blockIdx.x / tiles_x) * TR, c0 = static_cast<int64_t>(blockIdx.x % tiles_x) * TC;
  for (int t = threadIdx.x; t < TR * TC / V; t += 256) {
    const int r = t / (TC / V), c = t % (TC / V) * V;
    if (r0 + r >= rows) break;
    if (V > 1 && c0 + c + V <= cols) {
      float v[V];
      load_elems<T, V>(in + (r0 + r) * cols + c0 + c, v);
#pragma unroll
      for (int e = 0; e < V; e += 4) {
        *reinterpret_cast<uint32_t*>(tile + r * PITCH + c + e) =
            quantise2(v[e % V], v[(e + 1) % V], s) | quantise2(v[(e + 2) % V], v[(e + 3) % V], s) << 16;
      }
    } else {
      for (int e = 0; e < V; ++e)
        if (c0 + c + e < cols) tile[r * PITCH + c + e] = quantise1(ElemTraits<T>::to_float(in[(r0 + r) * cols + c0 + c + e]), s);
    }
  }
  __syncthreads();
  for (int t = threadIdx.x; t < TC * TR / 16; t += 256) {
    const int c = t / (TR / 16), r = t % (TR / 16) * 16;
    if (c0 + c >= cols) break;
    uint8_t* dst = out + (c0 + c) * out_ld + r0 + r;
    if (r0 + r + 16 <= rows) {
      uint32_t w[4] = {0, 0, 0, 0};
#pragma unroll
      for (int e = 0; e < 16; ++e) w[e >> 2] |= static_cast<uint32_t>(tile[(r + e) * PITCH + c]) << ((e & 3) * 8);
      *reinterpret_cast<uint4*>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
    } else {
      for (int e = 0; e < 16; ++e)
        if (r0 + r + e < rows) dst[e] = tile[(r + e) * PITCH + c];
    }
  }
}

constexpr int kParts = 148 * 4;

template <typename T>
int quantize_typed(const T* in, int64_t in_ld, uint8_t* out, int64_t out_ld, int64_t rows, int64_t cols, bool transpose,
                   uint32_t* parts, float* scale, cudaStream_t stream) {
  constexpr int V = 16 / sizeof(T);
  const bool vec = reinterpret_cast<uintptr_t>(in) % 16 == 0 && (in_ld * sizeof(T)) % 16 == 0;
  const int64_t r1 = in_ld == cols ? 1 : rows, c1 = in_ld == cols ? rows * cols : cols;  // one run where rows touch
  const bool vec1 = vec || (r1 == 1 && reinterpret_cast<uintptr_t>(in) % 16 == 0);
  auto blocks = [](int64_t threads, int64_t most) {
    const int64_t b = (threads + 255) / 256;
    return static_cast<unsigned>(b < most ? b : most);
  };
  const int64_t work = r1 * ((c1 + (vec1 ? V : 1) - 1) / (vec1 ? V : 1));
  const int nparts = static_cast<int>(blocks((work + 3) / 4, kParts));
  cudaError_t err = vec1 ? tc::launch_pdl(amax_kernel<T, V>, nparts, 256, 0, stream, in, in_ld, r1, c1, parts)
                         : tc::launch_pdl(amax_kernel<T, 1>, nparts, 256, 0, stream, in, in_ld, r1, c1, parts);
  count_launch();
  if (err == cudaSuccess && !transpose) {
    const bool flat = in_ld == cols && out_ld == cols;
    const int64_t rr = flat ? 1 : rows, cc = flat ? rows * cols : cols;
    const unsigned grid = blocks(rr * ((cc + 15) / 16), 148 * 8);
    // (rows of the destination are 16-byte multiples, or all of them one run)
    err = (flat ? vec1 : vec) ? tc::launch_pdl(quantize_kernel<T, V>, grid, 256, 0, stream, in, in_ld, out, out_ld, rr, cc,
                              static_cast<const uint32_t*>(parts), nparts, scale)
                              : tc::launch_pdl(quantize_kernel<T, 1>, grid, 256, 0, stream, in, in_ld, out, out_ld, rr, cc,
                              static_cast<const uint32_t*>(parts), nparts, scale);
    count_launch();
  } else if (err == cudaSuccess) {
    const int64_t tx = (cols + 63) / 64, ty = (rows + 127) / 128;
    if (tx * ty > 0x7fffffffLL) return set_error(KSMM_ERR_UNSUPPORTED, "quantisation: the grid limit is exceeded");
    err = vec ? tc::launch_pdl(quantize_transpose_kernel<T, V>, static_cast<unsigned>(tx * ty), 256, 0, stream, in, out,
                               out_ld, rows, cols, static_cast<uint32_t>(tx), static_cast<const uint32_t*>(parts), nparts, scale)
              : tc::launch_pdl(quantize_transpose_kernel<T, 1>, static_cast<unsigned>(tx * ty), 256, 0, stream, in, out,
                               out_ld, rows, cols, static_cast<uint32_t>(tx), static_cast<const uint32_t*>(parts), nparts, scale);
    count_launch();
  }
  if (err == cudaSuccess) err = cudaGetLastError();
  if (err != cudaSuccess) return set_error(KSMM_ERR_CUDA, "quantisation launch failed: %s", cudaGetErrorString(err));
  return KSMM_OK;
}

}  // namespace

size_t quantize_parts_bytes() { return kParts * sizeof(uint32_t); }

int launch_quantize(const void* in, int dtype, int64_t in_ld, void* out, int64_t out_ld, int64_t rows, int64_t cols,
                    bool transpose, void* parts, float* scale, cudaStream_t stream) {
  if (rows <= 0 || cols <= 0) return KSMM_OK;
  uint8_t* o = static_cast<uint8_t*>(out);
  uint32_t* pt = static_cast<uint32_t*>(parts);
  if (dtype == KSMM_F32)
    return quantize_typed(static_cast<const float*>(in), in_ld, o, out_ld, rows, cols, transpose, pt, scale, stream);
  if (dtype == KSMM_F16)
    return quantize_typed(static_cast<const __half*>(in), in_ld, o, out_ld, rows, cols, transpose, pt, scale, stream);
  if (dtype == KSMM_BF16)
    return quantize_typed(static_cast<const __nv_bfloat16*>(in), in_ld, o, out_ld, rows, cols, transpose, pt, scale, stream);
  return set_error(KSMM_ERR_UNSUPPORTED, "quantisation takes fp32, fp16 and bf16");
}

}  // namespace ksmm
