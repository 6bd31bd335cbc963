// Out-of-place 2-D transpose (1-, 2- and 4-byte elements): the ends of a chain that runs in the other
// layout, batch-first factors that no direct kernel covers, operands of weight gradients; and the copy of
// rows into padded rows.
//
// One CTA moves a tile of 16 KB through shared memory in 32-bit words.  A word holds R = 4 / size
// neighbouring input rows of one column: a thread loads 16 bytes of each of R rows, pairs them up in
// registers (byte permutes) and stores 16 / size words; an output row then is a run of words, read and
// written in 16-byte pieces.  The words of a column are swizzled in groups of four by the column's
// 16-byte piece, which makes both sides free of bank conflicts.  Four 16-byte loads per thread are in
// flight.  What bounds it is memory: 12544 x 3072 fp16 (154 MB moved) 31 -> 22 us, fp32 54 -> 47 us,
// against one shared access per element and side before.
#include "backward.h"
#include "common.cuh"

namespace ksmm {

template <int ES>
struct Tr {
  static constexpr int R = 4 / ES;               // input rows per word
  static constexpr int V = 16 / ES;              // elements per 16-byte piece
  static constexpr int TR = ES == 4 ? 64 : 128;  // tile rows
  static constexpr int TC = ES == 1 ? 128 : 64;  // tile columns
  static constexpr int WPC = TR / R;             // words per column
  static constexpr int LANES = TR * ES / 16;     // threads that write one output row of the tile
  // warp units: 8 pieces of a row x 4 words' rows
  static constexpr int UNITS = (WPC / 4) * (TC / (8 * V));
  static_assert(TC * WPC * 4 == 16384 && UNITS % 8 == 0, "tile");
  // word w of column c
  static __device__ __forceinline__ int at(int c, int w) { return c * WPC + (w ^ (((c / V) & 7) << 2)); }
};

// the R rows' pieces v[r] -> the words of the piece's columns
template <int ES>
__device__ __forceinline__ void pair_up(const uint4 (&v)[4 / ES], uint32_t (&w)[16 / ES]) {
  if constexpr (ES == 4) {
    w[0] = v[0].x; w[1] = v[0].y; w[2] = v[0].z; w[3] = v[0].w;
  } else if constexpr (ES == 2) {
    const uint32_t a[4] = {v[0].x, v[0].y, v[0].z, v[0].w}, b[4] = {v[1].x, v[1].y, v[1].z, v[1].w};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      w[2 * q] = __byte_perm(a[q], b[q], 0x5410);
      w[2 * q + 1] = __byte_perm(a[q], b[q], 0x7632);
    }
  } else {
    const uint32_t a[4] = {v[0].x, v[0].y, v[0].z, v[0].w}, b[4] = {v[1].x, v[1].y, v[1].z, v[1].w};
    const uint32_t c[4] = {v[2].x, v[2].y, v[2].z, v[2].w}, d[4] = {v[3].x, v[3].y, v[3].z, v[3].w};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const uint32_t ab0 = __byte_perm(a[q], b[q], 0x5140), ab1 = __byte_perm(a[q], b[q], 0x7362);
      const uint32_t cd0 = __byte_perm(c[q], d[q], 0x5140), cd1 = __byte_perm(c[q], d[q], 0x7362);
      w[4 * q] = __byte_perm(ab0, cd0, 0x5410);
      w[4 * q + 1] = __byte_perm(ab0, cd0, 0x7632);
      w[4 * q + 2] = __byte_perm(ab1, cd1, 0x5410);
      w[4 * q + 3] = __byte_perm(ab1, cd1, 0x7632);
    }
  }
}

// DT: element type of the sums (a ksmm_dtype_t), or -1.  With sums, sums[row tile][column] is the fp32 sum of
// the column over the tile's rows: a bias gradient's first stage, from the gradient that passes by.
template <int ES, int DT>
__global__ void __launch_bounds__(256)
    transpose_kernel(const uint8_t* __restrict__ in, uint8_t* __restrict__ out, int64_t rows, int64_t cols,
                     int64_t in_ld, int64_t out_ld, int vec_in, int vec_out, unsigned tiles_x,
                     float* __restrict__ sums) {
  using C = Tr<ES>;
  constexpr int R = C::R, V = C::V;
  __shared__ __align__(16) uint32_t tile[C::TC * C::WPC];
  uint8_t* const tile_b = reinterpret_cast<uint8_t*>(tile);
  // tiles are numbered row-major in one grid dimension (either extent may exceed 65535 tiles)
  const int64_t r0 = static_cast<int64_t>(blockIdx.x / tiles_x) * C::TR;
  const int64_t c0 = static_cast<int64_t>(blockIdx.x % tiles_x) * C::TC;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  // ---- load: 8 pieces x 4 words' rows per warp and unit --------------------------------
  constexpr int PER = C::UNITS / 8;
  uint4 v[PER][R];
  const bool inside = vec_in && r0 + C::TR <= rows && c0 + C::TC <= cols;
  if (inside) {
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      const int unit = warp + u * 8;
      const int c = (unit / (C::WPC / 4) * 8 + (lane & 7)) * V, w = unit % (C::WPC / 4) * 4 + (lane >> 3);
      const uint8_t* src = in + ((r0 + w * R) * in_ld + c0 + c) * ES;
#pragma unroll
      for (int r = 0; r < R; ++r) v[u][r] = *reinterpret_cast<const uint4*>(src + r * in_ld * ES);
    }
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      const int unit = warp + u * 8;
      const int c = (unit / (C::WPC / 4) * 8 + (lane & 7)) * V, w = unit % (C::WPC / 4) * 4 + (lane >> 3);
      uint32_t word[V];
      pair_up<ES>(v[u], word);
#pragma unroll
      for (int j = 0; j < V; ++j) tile[C::at(c + j, w)] = word[j];
    }
  } else {
    // edges and unaligned rows: element by element, neighbouring threads on neighbouring columns
    for (int e = threadIdx.x; e < C::TR * C::TC; e += 256) {
      const int r = e / C::TC, c = e % C::TC;
      uint8_t* dst = tile_b + C::at(c, r / R) * 4 + (r % R) * ES;
      const bool ok = r0 + r < rows && c0 + c < cols;
      const uint8_t* src = in + ((r0 + r) * in_ld + c0 + c) * ES;
      if constexpr (ES == 4) *reinterpret_cast<uint32_t*>(dst) = ok ? *reinterpret_cast<const uint32_t*>(src) : 0u;
      else if constexpr (ES == 2) *reinterpret_cast<uint16_t*>(dst) = ok ? *reinterpret_cast<const uint16_t*>(src) : uint16_t{0};
      else *dst = ok ? *src : uint8_t{0};
    }
  }
  __syncthreads();
  // ---- store: output rows c0.., 16-byte pieces of output columns r0.. ------------------------
#pragma unroll 4
  for (int t = threadIdx.x; t < C::TC * C::LANES; t += 256) {
    const int c = t / C::LANES, q = t % C::LANES;
    const uint4 o = *reinterpret_cast<const uint4*>(tile + C::at(c, 4 * q));
    if constexpr (DT >= 0) {
      // (rows and columns that do not exist hold zeros)
      float s = 0.f;
      const uint32_t w4[4] = {o.x, o.y, o.z, o.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        if constexpr (DT == KSMM_F32) {
          s += __uint_as_float(w4[e]);
        } else if constexpr (DT == KSMM_F16) {
          const __half2 h = *reinterpret_cast<const __half2*>(&w4[e]);
          s += __low2float(h) + __high2float(h);
        } else {
          s += __uint_as_float(w4[e] << 16) + __uint_as_float(w4[e] & 0xffff0000u);
        }
      }
#pragma unroll
      for (int d = C::LANES / 2; d > 0; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
      if (q == 0 && c0 + c < cols) sums[static_cast<int64_t>(blockIdx.x / tiles_x) * cols + c0 + c] = s;
    }
    if (c0 + c >= cols) continue;
    uint8_t* dst = out + ((c0 + c) * out_ld + r0 + q * V) * ES;
    if (vec_out && r0 + (q + 1) * V <= rows) {
      *reinterpret_cast<uint4*>(dst) = o;
    } else {
      const uint32_t w4[4] = {o.x, o.y, o.z, o.w};
#pragma unroll
      for (int e = 0; e < V; ++e) {
        if (r0 + q * V + e >= rows) break;
        const uint32_t x = w4[e / R] >> (8 * ES * (e % R));
        if constexpr (ES == 4) reinterpret_cast<uint32_t*>(dst)[e] = x;
        else if constexpr (ES == 2) reinterpret_cast<uint16_t*>(dst)[e] = static_cast<uint16_t>(x);
        else dst[e] = static_cast<uint8_t>(x);
      }
    }
  }
}

int transpose_row_tiles(int64_t rows, int es) {
  const int64_t tr = es == 4 ? Tr<4>::TR : Tr<2>::TR;
  return static_cast<int>((rows + tr - 1) / tr);
}

// in: rows x cols with row stride in_ld (0 = cols), out: cols x rows with row stride out_ld (0 = rows);
// `es` = element size in bytes
int launch_transpose(const void* in, void* out, int64_t rows, int64_t cols, int es,
                     cudaStream_t stream, int64_t out_ld, int64_t in_ld, float* sums, int sum_dtype) {
  if (rows <= 0 || cols <= 0) return KSMM_OK;
  if (in_ld == 0) in_ld = cols;
  if (out_ld == 0) out_ld = rows;
  const int tr = es == 4 ? Tr<4>::TR : Tr<2>::TR, tc = es == 1 ? Tr<1>::TC : Tr<2>::TC;
  const int64_t gx = (cols + tc - 1) / tc, gy = (rows + tr - 1) / tr;
  if (gx * gy > 0x7fffffffLL)
    return set_error(KSMM_ERR_UNSUPPORTED, "transpose of %lld x %lld exceeds the grid limits",
                     static_cast<long long>(rows), static_cast<long long>(cols));
  const int V = 16 / es;
  const int vec_in = in_ld % V == 0 && reinterpret_cast<uintptr_t>(in) % 16 == 0;
  const int vec_out = out_ld % V == 0 && reinterpret_cast<uintptr_t>(out) % 16 == 0;
  const unsigned grid = static_cast<unsigned>(gx * gy), tx = static_cast<unsigned>(gx);
  const uint8_t* src = static_cast<const uint8_t*>(in);
  uint8_t* dst = static_cast<uint8_t*>(out);
  auto go = [&](auto kern) { kern<<<grid, 256, 0, stream>>>(src, dst, rows, cols, in_ld, out_ld, vec_in, vec_out, tx, sums); };
  if (sums) {
    if (sum_dtype == KSMM_F32) go(transpose_kernel<4, KSMM_F32>);
    else if (sum_dtype == KSMM_F16) go(transpose_kernel<2, KSMM_F16>);
    else go(transpose_kernel<2, KSMM_BF16>);
  } else if (es == 4) {
    go(transpose_kernel<4, -1>);
  } else if (es == 2) {
    go(transpose_kernel<2, -1>);
  } else {
    go(transpose_kernel<1, -1>);
  }
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
// source tensor, go element by element.  384 x 6501 fp16, 5 MB read from DRAM and 5 MB
// written: 6.7 us, a launch and the loads' latency.
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
