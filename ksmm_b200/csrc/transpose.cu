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
                     int64_t out_ld, int vec_in, int vec_out, unsigned tiles_x) {
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
      const uint4 raw = *reinterpret_cast<const uint4*>(in + (r0 + r) * cols + c0 + cv * V);
      const T* e = reinterpret_cast<const T*>(&raw);
#pragma unroll
      for (int q = 0; q < V; ++q) tile[r][cv * V + q] = e[q];
    }
  } else {
    for (int v = tid; v < TILE * TILE; v += 256) {
      const int r = v / TILE, c = v % TILE;
      if (r0 + r < rows && c0 + c < cols) tile[r][c] = in[(r0 + r) * cols + c0 + c];
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

// in: rows x cols row-major, out: cols x rows with row stride out_ld (0 = rows); `es` = element size in bytes
int launch_transpose(const void* in, void* out, int64_t rows, int64_t cols, int es,
                     cudaStream_t stream, int64_t out_ld) {
  if (rows <= 0 || cols <= 0) return KSMM_OK;
  if (out_ld == 0) out_ld = rows;
  const int64_t gx = (cols + 63) / 64, gy = (rows + 63) / 64;
  if (gx * gy > 0x7fffffffLL)
    return set_error(KSMM_ERR_UNSUPPORTED, "transpose of %lld x %lld exceeds the grid limits",
                     static_cast<long long>(rows), static_cast<long long>(cols));
  const int V = 16 / es;
  const int vec_in = cols % V == 0 && reinterpret_cast<uintptr_t>(in) % 16 == 0;
  const int vec_out = out_ld % V == 0 && reinterpret_cast<uintptr_t>(out) % 16 == 0;
  const unsigned grid = static_cast<unsigned>(gx * gy), tx = static_cast<unsigned>(gx);
  if (es == 4)
    transpose_kernel<uint32_t><<<grid, 256, 0, stream>>>(static_cast<const uint32_t*>(in), static_cast<uint32_t*>(out),
                                                         rows, cols, out_ld, vec_in, vec_out, tx);
  else if (es == 2)
    transpose_kernel<uint16_t><<<grid, 256, 0, stream>>>(static_cast<const uint16_t*>(in), static_cast<uint16_t*>(out),
                                                         rows, cols, out_ld, vec_in, vec_out, tx);
  else
    transpose_kernel<uint8_t><<<grid, 256, 0, stream>>>(static_cast<const uint8_t*>(in), static_cast<uint8_t*>(out),
                                                        rows, cols, out_ld, vec_in, vec_out, tx);
  count_launch();
  cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess)
    return set_error(KSMM_ERR_CUDA, "transpose launch failed: %s", cudaGetErrorString(err));
  return KSMM_OK;
}

// Copy of a matrix between two row strides: the way in for batch-last tensors whose rows are not
// 16-byte multiples, which no tensor map can address.  One CTA moves 256 x VO elements of one row
// after another; the side with 16-byte rows uses 16-byte accesses, the other one element
// accesses in which neighbouring lanes take neighbouring elements (through shared memory).
template <typename T>
__global__ void __launch_bounds__(256)
    copy_rows_kernel(const T* __restrict__ in, int64_t in_ld, T* __restrict__ out, int64_t out_ld, int64_t rows,
                     int64_t cols) {
  constexpr int SPAN = 1024;  // elements of a row per CTA and step
  const int64_t c0 = static_cast<int64_t>(blockIdx.x) * SPAN;
  const int n = static_cast<int>(min(cols - c0, static_cast<int64_t>(SPAN)));
  for (int64_t r = blockIdx.y; r < rows; r += gridDim.y) {
    const T* src = in + r * in_ld + c0;
    T* dst = out + r * out_ld + c0;
    T v[SPAN / 256];
#pragma unroll
    for (int q = 0; q < SPAN / 256; ++q)
      if (q * 256 + static_cast<int>(threadIdx.x) < n) v[q] = src[q * 256 + threadIdx.x];
#pragma unroll
    for (int q = 0; q < SPAN / 256; ++q)
      if (q * 256 + static_cast<int>(threadIdx.x) < n) dst[q * 256 + threadIdx.x] = v[q];
  }
}

int launch_copy_rows(const void* in, int64_t in_ld, void* out, int64_t out_ld, int64_t rows, int64_t cols, int es,
                     cudaStream_t stream) {
  if (rows <= 0 || cols <= 0) return KSMM_OK;
  const int64_t gx = (cols + 1023) / 1024;
  if (gx > 0x7fffffffLL) return set_error(KSMM_ERR_UNSUPPORTED, "row copy: too many columns");
  const dim3 grid(static_cast<unsigned>(gx), static_cast<unsigned>(rows < 32768 ? rows : 32768));
  if (es == 4)
    copy_rows_kernel<uint32_t><<<grid, 256, 0, stream>>>(static_cast<const uint32_t*>(in), in_ld,
                                                         static_cast<uint32_t*>(out), out_ld, rows, cols);
  else if (es == 2)
    copy_rows_kernel<uint16_t><<<grid, 256, 0, stream>>>(static_cast<const uint16_t*>(in), in_ld,
                                                         static_cast<uint16_t*>(out), out_ld, rows, cols);
  else
    copy_rows_kernel<uint8_t><<<grid, 256, 0, stream>>>(static_cast<const uint8_t*>(in), in_ld,
                                                        static_cast<uint8_t*>(out), out_ld, rows, cols);
  count_launch();
  cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess)
    return set_error(KSMM_ERR_CUDA, "row copy launch failed: %s", cudaGetErrorString(err));
  return KSMM_OK;
}

}  // namespace ksmm
