// Out-of-place 2-D transpose (1-, 2- and 4-byte elements) used by the
// layout-conversion path: a batch-first factor that no direct kernel covers is
// run as transpose -> batch-last kernel -> transpose.
//
// One CTA moves a 64 x 64 tile through shared memory: 16-byte global loads
// along the input rows, element-wise shared stores into a padded tile, strided
// shared reads along the tile columns, 16-byte global stores in which the lanes
// of a warp follow the output rows (whole 128-byte lines per warp).  Edges and
// unaligned shapes fall back to element accesses.
#include "backward.h"
#include "common.cuh"

namespace ksmm {

template <typename T>
__global__ void __launch_bounds__(256)
    transpose_kernel(const T* __restrict__ in, T* __restrict__ out, int64_t rows, int64_t cols,
                     int64_t in_ld, int64_t out_ld, int vec_in, int vec_out, unsigned tiles_x) {
  constexpr int TILE = 64;
  constexpr int V = 16 / sizeof(T);            // elements per 16-byte vector
  constexpr int VPR = TILE / V;                // vectors per tile row
  // one extra 4-byte word per tile row keeps the column reads of a warp on distinct banks
  constexpr int PITCH = TILE + 4 / static_cast<int>(sizeof(T));
  __shared__ T tile[TILE][PITCH];
  // tiles are numbered row-major in one grid dimension (either extent may exceed 65535 tiles)
  const int64_t r0 = static_cast<int64_t>(blockIdx.x / tiles_x) * TILE;
  const int64_t c0 = static_cast<int64_t>(blockIdx.x % tiles_x) * TILE;
  const int tid = threadIdx.x;

  // ---- load: rows r0.., columns c0.. --------------------------------------------
  if (vec_in && c0 + TILE <= cols) {
    for (int v = tid; v < TILE * VPR; v += 256) {
      const int r = v / VPR, cv = v % VPR;
      if (r0 + r >= rows) break;
      const uint4 raw = *reinterpret_cast<const uint4*>(in + (r0 + r) * in_ld + c0 + cv * V);
      const T* e = reinterpret_cast<const T*>(&raw);
#pragma unroll
      for (int q = 0; q < V; ++q) tile[r][cv * V + q] = e[q];
    }
  } else {
    for (int v = tid; v < TILE * TILE; v += 256) {
      const int r = v / TILE, c = v % TILE;
      if (r0 + r < rows && c0 + c < cols) tile[r][c] = in[(r0 + r) * in_ld + c0 + c];
    }
  }
  __syncthreads();
  // ---- store: output rows c0.., output columns r0.. ----------------------------------
  if (vec_out && r0 + TILE <= rows) {
    for (int v = tid; v < TILE * VPR; v += 256) {
      // lanes walk along an output row, so that a warp writes whole 128-byte lines
      const int c = v / VPR, rv = v % VPR;
      if (c0 + c >= cols) break;
      uint4 raw;
      T* e = reinterpret_cast<T*>(&raw);
#pragma unroll
      for (int q = 0; q < V; ++q) e[q] = tile[rv * V + q][c];
      *reinterpret_cast<uint4*>(out + (c0 + c) * out_ld + r0 + rv * V) = raw;
    }
  } else {
    for (int v = tid; v < TILE * TILE; v += 256) {
      const int c = v / TILE, r = v % TILE;
      if (r0 + r < rows && c0 + c < cols) out[(c0 + c) * out_ld + r0 + r] = tile[r][c];
    }
  }
}

// in: rows x cols with row stride in_ld (0 = cols), out: cols x rows with row stride out_ld (0 = rows);
// `es` = element size in bytes
int launch_transpose(const void* in, void* out, int64_t rows, int64_t cols, int es,
                     cudaStream_t stream, int64_t out_ld, int64_t in_ld) {
  if (rows <= 0 || cols <= 0) return KSMM_OK;
  if (in_ld == 0) in_ld = cols;
  if (out_ld == 0) out_ld = rows;
  const int64_t gx = (cols + 63) / 64, gy = (rows + 63) / 64;
  if (gx * gy > 0x7fffffffLL)
    return set_error(KSMM_ERR_UNSUPPORTED, "transpose of %lld x %lld exceeds the grid limits",
                     static_cast<long long>(rows), static_cast<long long>(cols));
  const int V = 16 / es;
  const int vec_in = in_ld % V == 0 && reinterpret_cast<uintptr_t>(in) % 16 == 0;
  const int vec_out = out_ld % V == 0 && reinterpret_cast<uintptr_t>(out) % 16 == 0;
  const unsigned grid = static_cast<unsigned>(gx * gy), tx = static_cast<unsigned>(gx);
  if (es == 4)
    transpose_kernel<uint32_t><<<grid, 256, 0, stream>>>(static_cast<const uint32_t*>(in), static_cast<uint32_t*>(out),
                                                         rows, cols, in_ld, out_ld, vec_in, vec_out, tx);
  else if (es == 2)
    transpose_kernel<uint16_t><<<grid, 256, 0, stream>>>(static_cast<const uint16_t*>(in), static_cast<uint16_t*>(out),
                                                         rows, cols, in_ld, out_ld, vec_in, vec_out, tx);
  else
    transpose_kernel<uint8_t><<<grid, 256, 0, stream>>>(static_cast<const uint8_t*>(in), static_cast<uint8_t*>(out),
                                                        rows, cols, in_ld, out_ld, vec_in, vec_out, tx);
  count_launch();
  cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess)
    return set_error(KSMM_ERR_CUDA, "transpose launch failed: %s", cudaGetErrorString(err));
  return KSMM_OK;
}

// Copy of a matrix between two row strides: the way in for batch-last tensors whose rows are not
// 16-byte multiples, which no tensor map can address.  Rows of the destination are aligned, rows of
// the source start anywhere.  A thread makes 16-byte pieces of the destination out of the two aligned
// 16-byte words that hold them in the source (byte shifts in registers), so that every access of a warp
// is a run of whole lines; the last piece of a row, and pieces whose words would reach outside the
// source tensor, go element by element.  Bound by memory: 384 x 6501 fp16 (10 MB moved) 3 us, 9 us with
// one element per thread and access.
struct PitchArgs {
  const uint8_t* in;
  uint8_t* out;
  int64_t in_ld, out_ld;  // bytes
  int64_t rows;
  int64_t bytes;          // of a row
  uint32_t pieces;        // 16-byte pieces per row, the last one possibly partial
};

template <int ES>
__global__ void __launch_bounds__(256) copy_rows_kernel(const PitchArgs A) {
  const uint8_t* in_end = A.in + (A.rows - 1) * A.in_ld + A.bytes;
  const int64_t total = A.rows * A.pieces;
  for (int64_t t = static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x; t < total;
       t += static_cast<int64_t>(gridDim.x) * 256) {
    const int64_t r = total <= 0xffffffffLL ? static_cast<uint32_t>(t) / A.pieces : t / A.pieces;
    const int64_t x = (t - r * A.pieces) * 16;
    const uint8_t* src = A.in + r * A.in_ld + x;
    uint8_t* dst = A.out + r * A.out_ld + x;
    const uint32_t sh = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(src) & 15);
    const uint8_t* w0 = src - sh;
    if (x + 16 <= A.bytes && w0 >= A.in && w0 + (sh ? 32 : 16) <= in_end) {
      const uint4 lo = *reinterpret_cast<const uint4*>(w0);
      uint4 hi = make_uint4(0, 0, 0, 0);
      if (sh) hi = *reinterpret_cast<const uint4*>(w0 + 16);
      // bytes sh .. sh + 15 of the 32: by 8, by 4, then within a word
      uint32_t v0 = lo.x, v1 = lo.y, v2 = lo.z, v3 = lo.w, v4 = hi.x, v5 = hi.y, v6 = hi.z;
      const uint32_t v7 = hi.w;
      if (sh & 8) { v0 = v2; v1 = v3; v2 = v4; v3 = v5; v4 = v6; v5 = v7; }
      if (sh & 4) { v0 = v1; v1 = v2; v2 = v3; v3 = v4; v4 = v5; }
      const uint32_t b = (sh & 3) * 8;
      uint4 o;
      o.x = __funnelshift_r(v0, v1, b);
      o.y = __funnelshift_r(v1, v2, b);
      o.z = __funnelshift_r(v2, v3, b);
      o.w = __funnelshift_r(v3, v4, b);
      *reinterpret_cast<uint4*>(dst) = o;
    } else {
      const int n = static_cast<int>(min(A.bytes - x, static_cast<int64_t>(16)));
      for (int e = 0; e < n; e += ES) {
        if constexpr (ES == 4) *reinterpret_cast<uint32_t*>(dst + e) = *reinterpret_cast<const uint32_t*>(src + e);
        else if constexpr (ES == 2) *reinterpret_cast<uint16_t*>(dst + e) = *reinterpret_cast<const uint16_t*>(src + e);
        else dst[e] = src[e];
      }
    }
  }
}

// out and out_ld * es are multiples of 16 bytes
int launch_copy_rows(const void* in, int64_t in_ld, void* out, int64_t out_ld, int64_t rows, int64_t cols, int es,
                     cudaStream_t stream) {
  if (rows <= 0 || cols <= 0) return KSMM_OK;
  PitchArgs A;
  A.in = static_cast<const uint8_t*>(in);
  A.out = static_cast<uint8_t*>(out);
  A.in_ld = in_ld * es;
  A.out_ld = out_ld * es;
  A.rows = rows;
  A.bytes = cols * es;
  const int64_t pieces = (A.bytes + 15) / 16;
  if (pieces > 0x7fffffffLL) return set_error(KSMM_ERR_UNSUPPORTED, "row copy: too many columns");
  A.pieces = static_cast<uint32_t>(pieces);
  const int64_t blocks = (rows * pieces + 255) / 256;
  const unsigned grid = static_cast<unsigned>(blocks < 148 * 32 ? blocks : 148 * 32);
  if (es == 4) copy_rows_kernel<4><<<grid, 256, 0, stream>>>(A);
  else if (es == 2) copy_rows_kernel<2><<<grid, 256, 0, stream>>>(A);
  else copy_rows_kernel<1><<<grid, 256, 0, stream>>>(A);
  count_launch();
  cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess)
    return set_error(KSMM_ERR_CUDA, "row copy launch failed: %s", cudaGetErrorString(err));
  return KSMM_OK;
}

}  // namespace ksmm
