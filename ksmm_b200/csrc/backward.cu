// Backward of one Kronecker-sparse factor.
//
//   forward    Y4[i,j,l,n] = sum_k W[i,j,k,l] X4[i,k,l,n]
//   dX         dX4[i,k,l,n] = sum_j W[i,j,k,l] dY4[i,j,l,n]: the same multiplication with pattern
//              (a,c,b,d) and every b x c block transposed, so it runs on the forward kernels once
//              the blocks have been transposed (transpose_blocks_kernel below);
//   dW         dW[i,j,k,l] = sum_n dY4[i,j,l,n] X4[i,k,l,n]: a*d independent (c x B) @ (B x b)
//              products whose contraction runs over the batch.  In kernel format the result of block
//              (i,l) is the row-major (c, b) matrix dWk[(i*d + l)*c + k, j].
//
// dW on the tensor cores (16-bit inputs, fp32 accumulation in TMEM): accumulator rows are k, columns
// are j, the K dimension of the MMAs is the batch, 64 entries per stage.  The two operands are
// independent: a batch-last one has rows of consecutive batch entries (K-major, fetched by the 4-D
// map over (batch, d, features, a) that the forward kernel uses for its input), a batch-first one
// with d = 1 has rows of consecutive features (MN-major).  A batch-first operand with d > 1, or one
// whose rows are not 16-byte multiples, is first copied into a batch-last tensor with padded rows in
// the workspace.  fp32 runs on tc_wgrad_f32.cu the same way.
//
// What bounds it: the wait for operands from L2, 52 GB/s per SM with three stages in flight (no unit is
// saturated: (1,768,192,4) fp16 at 25088 entries has the tensor pipe at 56 %, DRAM at 59 %, L2 at 41 %).
// A CTA that owns 128 x 256 outputs reads 48 KB per 64 batch entries, so a (1,768,192,4) factor reads its
// input three times and its output gradient twice; with two accumulators one above the other (MB = 2,
// 256 x 256 outputs, all 512 columns of TMEM) the gradient, four times the larger operand, is read once.
// Blocks have few tiles, so the batch is split over CTAs; every CTA writes an fp32 partial tile (staged through the idle ring, TMA
// store) and a second kernel sums the partials in a fixed order (bitwise repeatable) and converts.
// The number of splits minimises a time model (wgrad_splits), because whole waves of CTAs, the
// chunks per CTA and the bytes of the partials all depend on it.
//
// Roles of the tensor kernel (320 threads): warp 0 TMA producer, warp 1 TMEM owner and MMA issuer,
// warps 2..9 epilogue.  Waits are bounded and report through the device status word.
//
// The reference has no backward: Kernel.backward is a stub
// (src/ksmm_py/layer/kronecker_sparse/kernel.py:323-329).
#include <cuda.h>

#include <algorithm>
#include <atomic>
#include <cfloat>
#include <cstdint>

#include "backward.h"
#include "tc_host.h"
#include "tc_kernel.h"
#include "tc_ptx.cuh"

namespace ksmm {

// ---------------------------------------------------------------------------
// block transposes of kernel-format weights: (nblk, c, b) -> (nblk, b, c)
// ---------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256)
    transpose_blocks_kernel(const T* __restrict__ in, T* __restrict__ out, int c, int b) {
  __shared__ T tile[32][33];
  const int64_t base = static_cast<int64_t>(blockIdx.z) * c * b;
  const int k0 = blockIdx.y * 32, j0 = blockIdx.x * 32;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  for (int r = ty; r < 32; r += 8)
    if (k0 + r < c && j0 + tx < b) tile[r][tx] = in[base + static_cast<int64_t>(k0 + r) * b + j0 + tx];
  __syncthreads();
  for (int r = ty; r < 32; r += 8)
    if (j0 + r < b && k0 + tx < c) out[base + static_cast<int64_t>(j0 + r) * c + k0 + tx] = tile[tx][r];
}

int launch_transpose_blocks(const void* in, void* out, int64_t nblk, int c, int b, int es,
                            cudaStream_t stream) {
  if (nblk <= 0) return KSMM_OK;
  if (nblk > 65535)
    return set_error(KSMM_ERR_UNSUPPORTED, "weight transpose: %lld blocks exceed the grid limit",
                     static_cast<long long>(nblk));
  dim3 grid((b + 31) / 32, (c + 31) / 32, static_cast<unsigned>(nblk));
  if (grid.y > 65535) return set_error(KSMM_ERR_UNSUPPORTED, "weight transpose: c too large");
  if (es == 4)
    transpose_blocks_kernel<uint32_t><<<grid, 256, 0, stream>>>(static_cast<const uint32_t*>(in),
                                                                static_cast<uint32_t*>(out), c, b);
  else if (es == 2)
    transpose_blocks_kernel<uint16_t><<<grid, 256, 0, stream>>>(static_cast<const uint16_t*>(in),
                                                                static_cast<uint16_t*>(out), c, b);
  else
    transpose_blocks_kernel<uint8_t><<<grid, 256, 0, stream>>>(static_cast<const uint8_t*>(in),
                                                               static_cast<uint8_t*>(out), c, b);
  count_launch();
  cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess)
    return set_error(KSMM_ERR_CUDA, "weight transpose launch failed: %s", cudaGetErrorString(err));
  return KSMM_OK;
}

// ---------------------------------------------------------------------------
// dW, FFMA fallback: one thread per (k, j) of a 16 x 16 tile, the batch in steps of 32 through
// shared memory; any type, layout and alignment
// ---------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256)
    wgrad_simt_kernel(const T* __restrict__ x, const T* __restrict__ g, T* __restrict__ dw, int64_t batch,
                      int a, int b, int c, int d, int bs_last) {
  __shared__ float xs[16][33], gs[16][33];
  const int blk = blockIdx.z, i = blk / d, l = blk % d;
  const int k0 = blockIdx.y * 16, j0 = blockIdx.x * 16;
  const int tk = threadIdx.x >> 4, tj = threadIdx.x & 15;
  const int64_t n_in = static_cast<int64_t>(a) * c * d, n_out = static_cast<int64_t>(a) * b * d;
  float acc = 0.f;
  for (int64_t n0 = 0; n0 < batch; n0 += 32) {
    for (int e = threadIdx.x; e < 16 * 32; e += 256) {
      // batch-last: lanes walk the batch; batch-first: lanes walk the features
      const int r = bs_last ? e >> 5 : e & 15, nn = bs_last ? e & 31 : e >> 4;
      const int64_t n = n0 + nn;
      float xv = 0.f, gv = 0.f;
      if (n < batch) {
        if (k0 + r < c) {
          const int64_t f = (static_cast<int64_t>(i) * c + k0 + r) * d + l;
          xv = ElemTraits<T>::to_float(x[bs_last ? f * batch + n : n * n_in + f]);
        }
        if (j0 + r < b) {
          const int64_t f = (static_cast<int64_t>(i) * b + j0 + r) * d + l;
          gv = ElemTraits<T>::to_float(g[bs_last ? f * batch + n : n * n_out + f]);
        }
      }
      xs[r][nn] = xv;
      gs[r][nn] = gv;
    }
    __syncthreads();
#pragma unroll
    for (int nn = 0; nn < 32; ++nn) acc = fmaf(xs[tk][nn], gs[tj][nn], acc);
    __syncthreads();
  }
  if (k0 + tk < c && j0 + tj < b)
    dw[(static_cast<int64_t>(blk) * c + k0 + tk) * b + j0 + tj] = ElemTraits<T>::from_float(acc);
}

namespace tc {

struct ParamsW {
  int a, b, c, d;
  int tiles_k, tiles_j, splits;
  int nchunks;  // ceil(batch / 64)
  uint32_t idesc;
  float* part;  // (splits, a*d, c, b) fp32
  int tma_part;  // b % 4 == 0: partial tiles leave through TMA
  int* status;
};

constexpr int kThreadsW = 10 * 32;

template <int MB, int NT, int SX>
struct CfgW {
  static constexpr int A_BYTES = MB * 128 * 128;  // MB x 128 k x 64 batch entries (either order)
  static constexpr int B_BYTES = NT * 128;        // NT j x 64 batch entries
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int NBAR = 2 * SX + 1;
  static constexpr int BAR_BYTES = 256;
  static constexpr int SMEM_BYTES = SX * STAGE_BYTES + BAR_BYTES + 1024;
  static constexpr int TMEM_COLS = MB * NT;
  static_assert(MB == 1 || MB == 2, "accumulators above one another");
  static_assert(NT == 64 || NT == 128 || NT == 256, "j tile");
  static_assert(SMEM_BYTES <= 232448, "shared memory budget");
  static_assert(SMEM_BYTES > 116 * 1024, "one CTA per SM, so that the TMEM allocation never waits");
  static_assert(8 * NBAR + 16 <= BAR_BYTES, "barrier area");
};

// X_LAST / G_LAST: layout of the input / of the output gradient
template <bool X_LAST, bool G_LAST, int MB, int NT, int SX>
__global__ void __launch_bounds__(kThreadsW, 1)
    ksmm_tc_wgrad_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmG,
                         const __grid_constant__ CUtensorMap tmP, const ParamsW P) {
  using C = CfgW<MB, NT, SX>;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t sm0 = (raw + 1023u) & ~1023u;
  uint8_t* sm_gen = smem_raw + (sm0 - raw);
  const uint32_t ring0 = sm0;
  const uint32_t bar0 = ring0 + SX * C::STAGE_BYTES;
  uint8_t* bar_gen = sm_gen + SX * C::STAGE_BYTES;
  auto full_bar = [&](int s) { return bar0 + 8u * s; };
  auto empty_bar = [&](int s) { return bar0 + 8u * (SX + s); };
  const uint32_t tfull_bar = bar0 + 8u * (2 * SX);
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(bar_gen + 8 * C::NBAR);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bar_gen + 8 * C::NBAR + 4);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < SX; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    mbar_init(tfull_bar, 1);
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 0 && lane == 0) {
    prefetch_tensormap(&tmX);
    prefetch_tensormap(&tmG);
    prefetch_tensormap(&tmP);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_slot)), C::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // everything above overlaps the tail of the previous kernel in the stream; memory comes after this
  grid_dep_wait();
  grid_dep_launch();

  // CTA -> (split, block, k tile, j tile); the split owns a contiguous range of 64-entry chunks.  The
  // tiles of one (split, block) are neighbours: they share their operands in L2 at the same time.
  uint32_t t = blockIdx.x;
  const int tj = static_cast<int>(t % P.tiles_j); t /= P.tiles_j;
  const int tk = static_cast<int>(t % P.tiles_k); t /= P.tiles_k;
  const int sp = static_cast<int>(t % P.splits);
  const int blk = static_cast<int>(t / P.splits);
  const int i = blk / P.d, l = blk % P.d;
  const int k0 = tk * (MB * 128), j0 = tj * NT;
  const int ch_begin = static_cast<int>(static_cast<int64_t>(sp) * P.nchunks / P.splits);
  const int ch_end = static_cast<int>(static_cast<int64_t>(sp + 1) * P.nchunks / P.splits);

  if (warp == 0) {
    if (lane == 0) {
      uint32_t si = 0, sph = 0;
      for (int ch = ch_begin; ch < ch_end; ++ch) {
        if (!mbar_wait<64>(empty_bar(si), sph ^ 1u, abort_flag, P.status, 51)) break;
        const uint32_t dst = ring0 + si * C::STAGE_BYTES;
        const uint32_t bar = full_bar(si);
        mbar_expect_tx(bar, C::STAGE_BYTES);
        const int n0 = ch * 64;
        if constexpr (X_LAST) {
#pragma unroll
          for (int mb = 0; mb < MB; ++mb) tma_load_4d(dst + mb * 128 * 128, &tmX, bar, n0, l, k0 + mb * 128, i);
        } else {
          // 64 batch rows x 64 features per box; M groups of 64 follow one another
#pragma unroll
          for (int kb = 0; kb < 2 * MB; ++kb) tma_load_3d(dst + kb * 64 * 128, &tmX, bar, k0 + kb * 64, blk, n0);
        }
        if constexpr (G_LAST) {
          tma_load_4d(dst + C::A_BYTES, &tmG, bar, n0, l, j0, i);
        } else {
#pragma unroll
          for (int jb = 0; jb < NT / 64; ++jb)
            tma_load_3d(dst + C::A_BYTES + jb * 64 * 128, &tmG, bar, j0 + jb * 64, blk, n0);
        }
        if (++si == SX) { si = 0; sph ^= 1u; }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (lane == 0) {
      // descriptor words that never change: SBO = 1024 bytes, version 1, 128-byte swizzle
      constexpr uint32_t kDescHi = (1024u >> 4) | (1u << 14) | (2u << 29);
      // K-major (batch-last): 32 bytes per k step inside the swizzle row, LBO unused;
      // MN-major (batch-first): LBO = one 64-wide group (64 rows x 128 bytes), 16 rows per k step
      constexpr uint32_t kLboK = 1u << 16, kLboMN = static_cast<uint32_t>((64 * 128) >> 4) << 16;
      constexpr uint32_t kStepK = 32u >> 4, kStepMN = (16u * 128u) >> 4;
      uint32_t si = 0, sph = 0;
      bool ok = true;
      for (int ch = ch_begin; ch < ch_end; ++ch) {
        if (!mbar_wait<0>(full_bar(si), sph, abort_flag, P.status, 52)) { ok = false; break; }
        tc_fence_after();
        const uint32_t asrc = ring0 + si * C::STAGE_BYTES, bsrc = asrc + C::A_BYTES;
        const uint32_t alo = (asrc >> 4) | (X_LAST ? kLboK : kLboMN), blo = (bsrc >> 4) | (G_LAST ? kLboK : kLboMN);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const uint64_t bdesc = (static_cast<uint64_t>(kDescHi) << 32) | (blo + k * (G_LAST ? kStepK : kStepMN));
#pragma unroll
          for (int mb = 0; mb < MB; ++mb) {
            const uint64_t adesc = (static_cast<uint64_t>(kDescHi) << 32) |
                                   (alo + mb * ((128 * 128) >> 4) + k * (X_LAST ? kStepK : kStepMN));
            umma<2>(tmem_base + mb * NT, adesc, bdesc, P.idesc, (ch != ch_begin || k != 0) ? 1u : 0u);
          }
        }
        umma_commit(empty_bar(si));
        if (++si == SX) { si = 0; sph ^= 1u; }
      }
      if (ok) umma_commit(tfull_bar);
    }
    __syncwarp();
  } else {
    // epilogue: lane = accumulator row k; 32 columns (j) per TMEM load.  MB = 2: four warps per
    // accumulator; MB = 1: the two groups of four warps take alternate column groups.
    const int q = warp & 3, h = (warp - 2) >> 2;
    const int mb = MB == 2 ? h : 0;
    int got = 1;
    if (lane == 0) got = mbar_wait<128>(tfull_bar, 0u, abort_flag, P.status, 53) ? 1 : 0;
    got = __shfl_sync(0xffffffffu, got, 0);
    const int krow0 = k0 + mb * 128 + q * 32;
    if (got && krow0 < P.c) {
      tc_fence_after();
      const int k = krow0 + lane;
      const int pz = sp * P.a * P.d + blk;
      // every load has been consumed by the MMAs: the ring is free for staging tiles
      const uint32_t stg0 = ring0 + (warp - 2) * 2 * 4096;
      uint32_t sti = 0;
#pragma unroll 1
      for (int cg = MB == 2 ? 0 : h; cg < NT / 32; cg += MB == 2 ? 1 : 2) {
        if (j0 + cg * 32 >= P.b) break;
        uint32_t r[32];
        if (ch_end > ch_begin) {
          tmem_ld32(tmem_base + (static_cast<uint32_t>(q * 32) << 16) + mb * NT + cg * 32, r);
          tmem_ld_wait();
        } else {  // a split without chunks: its partial tile is zero
#pragma unroll
          for (int e = 0; e < 32; ++e) r[e] = 0u;
        }
        if (P.tma_part) {
          const uint32_t stg = stg0 + sti * 4096u;
          sti ^= 1u;
          if (lane == 0) bulk_wait_read<1>();  // the store before the last has read this staging tile
          __syncwarp();
#pragma unroll
          for (int ch = 0; ch < 8; ++ch)
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(stg + lane * 128 + ((ch ^ (lane & 7)) << 4)),
                         "r"(r[ch * 4]), "r"(r[ch * 4 + 1]), "r"(r[ch * 4 + 2]), "r"(r[ch * 4 + 3])
                         : "memory");
          fence_proxy_async();
          __syncwarp();
          if (lane == 0) {
            tma_store_3d(&tmP, stg, j0 + cg * 32, krow0, pz);
            bulk_commit();
          }
        } else if (k < P.c) {
          float* row = P.part + (static_cast<int64_t>(pz) * P.c + k) * P.b + j0 + cg * 32;
#pragma unroll
          for (int e = 0; e < 32; ++e)
            if (j0 + cg * 32 + e < P.b) row[e] = __uint_as_float(r[e]);
        }
      }
      if (lane == 0) bulk_wait<0>();
    }
    __syncwarp();
  }

  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    __nanosleep(20000);
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, C::TMEM_COLS);
  }
}

// What an fp32 sum that is not finite is computed again from.  The split of the operands (tc_wgrad_f32.cu) turns
// an infinite one into NaN, its rest being inf - inf, and may overflow a little below the largest float.
struct Again {
  const float *x, *g;
  int64_t batch;
  int b, c, d;
  // address of (feature r of block (i, l), entry n): i * i + r * r + l * l + n * n
  struct Strides { int64_t i, r, l, n; } xs, gs;
};

// the sum of products of element e in the order and precision of wgrad_simt_kernel
__device__ __noinline__ float sum_again(const Again& A, int64_t e) {
  const int j = static_cast<int>(e % A.b), k = static_cast<int>(e / A.b % A.c);
  const int64_t blk = e / A.b / A.c, i = blk / A.d, l = blk % A.d;
  const float* x = A.x + i * A.xs.i + k * A.xs.r + l * A.xs.l;
  const float* g = A.g + i * A.gs.i + j * A.gs.r + l * A.gs.l;
  float acc = 0.f;
  for (int64_t n0 = 0; n0 < A.batch && acc == acc; n0 += 32) {  // (a NaN stays one)
    const int64_t end = min(n0 + 32, A.batch);
#pragma unroll 8
    for (int64_t n = n0; n < end; ++n) acc = fmaf(x[n * A.xs.n], g[n * A.gs.n], acc);
  }
  return acc;
}

// Sums the partial tiles of the splits in a fixed order and converts to the weights' type.  Four
// elements per thread (elems is a multiple of 4 in the vector form), four splits in flight.
template <typename T, int V>
__global__ void __launch_bounds__(256)
    wgrad_reduce_kernel(const float* part, T* dw, int64_t elems, int splits, const Again A) {
  // (no read-only loads in this kernel: the compiler may move those above the wait)
  grid_dep_wait();
  grid_dep_launch();
  const int64_t n = elems / V;
  for (int64_t e = static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x; e < n;
       e += static_cast<int64_t>(gridDim.x) * 256) {
    float s[V] = {};
#pragma unroll 4
    for (int q = 0; q < splits; ++q) {
      float v[V];
      if constexpr (V == 4) {
        const float4 f = *reinterpret_cast<const float4*>(part + q * elems + e * V);
        v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
      } else {
        v[0] = part[q * elems + e];
      }
#pragma unroll
      for (int u = 0; u < V; ++u) s[u] += v[u];
    }
    if constexpr (sizeof(T) == 4) {
#pragma unroll
      for (int u = 0; u < V; ++u)
        if (!(fabsf(s[u]) <= FLT_MAX)) s[u] = sum_again(A, e * V + u);
    }
    store_vec<T, V>(dw + e * V, s);
  }
}

template <typename T>
static cudaError_t launch_reduce(const Problem& p, const WgradOperand& x, const WgradOperand& g, const float* part,
                                 int splits, cudaStream_t stream) {
  void* dw = p.out;
  const int64_t elems = static_cast<int64_t>(p.a) * p.b * p.c * p.d, d = p.d;
  auto strides = [&](const WgradOperand& o, int64_t f) {
    if (o.last) return Again::Strides{f * d * o.ld, d * o.ld, o.ld, 1};
    if (o.regrouped) return Again::Strides{f * d, 1, f, p.a * f * d};
    return Again::Strides{f * d, d, 1, p.a * f * d};
  };
  const Again A{static_cast<const float*>(x.ptr), static_cast<const float*>(g.ptr), p.batch, p.b, p.c, p.d,
                strides(x, p.c), strides(g, p.b)};
  const bool vec = elems % 4 == 0 && reinterpret_cast<uintptr_t>(dw) % 16 == 0;
  const int64_t items = vec ? elems / 4 : elems;
  const unsigned grid = static_cast<unsigned>(std::min<int64_t>((items + 255) / 256, 148 * 8));
  if (vec)
    return launch_pdl(wgrad_reduce_kernel<T, 4>, grid, 256, 0, stream, part, static_cast<T*>(dw), elems, splits, A);
  return launch_pdl(wgrad_reduce_kernel<T, 1>, grid, 256, 0, stream, part, static_cast<T*>(dw), elems, splits, A);
}

template <bool X_LAST, bool G_LAST, int MB, int NT, int SX>
static int launch_w(const Problem& p, const WgradOperand& x, const WgradOperand& g, float* part, int splits,
                    cudaStream_t stream) {
  using C = CfgW<MB, NT, SX>;
  auto kern = ksmm_tc_wgrad_kernel<X_LAST, G_LAST, MB, NT, SX>;
  static std::atomic<bool> attr_set[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !attr_set[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES);
    if (e != cudaSuccess)
      return set_error(KSMM_ERR_CUDA, "cannot reserve %d bytes of shared memory: %s", C::SMEM_BYTES,
                       cudaGetErrorString(e));
    attr_set[dev] = true;
  }
  const uint64_t a = p.a, b = p.b, c = p.c, d = p.d, B = p.batch;
  CUtensorMap tmX, tmG, tmP;
  int st;
  // batch-last: (batch, d, features, a), 64 batch entries x 128 (NT) features per box;
  // batch-first (d = 1): (features, a, batch), 64 features x 64 batch entries per box
  auto operand_map = [&](CUtensorMap* tm, bool last, const WgradOperand& o, uint64_t f, uint32_t rows) {
    if (last) {
      const uint64_t L = o.ld;
      const uint64_t dims[4] = {B, d, f, a}, str[4] = {1, L, d * L, f * d * L};
      const uint32_t box[4] = {64, 1, rows, 1};
      return encode_map(tm, p.in_dtype, 4, o.ptr, dims, str, box);
    }
    // (regrouped rows have a * d blocks one after the other)
    const uint64_t dims[3] = {f, a * d, B}, str[3] = {1, f, a * d * f};
    const uint32_t box[3] = {64, 1, 64};
    return encode_map(tm, p.in_dtype, 3, o.ptr, dims, str, box);
  };
  if ((st = operand_map(&tmX, X_LAST, x, c, 128)) != KSMM_OK) return st;
  if ((st = operand_map(&tmG, G_LAST, g, b, NT)) != KSMM_OK) return st;
  ParamsW P;
  P.a = p.a; P.b = p.b; P.c = p.c; P.d = p.d;
  P.tiles_k = (p.c + MB * 128 - 1) / (MB * 128);
  P.tiles_j = (p.b + NT - 1) / NT;
  P.splits = splits;
  P.nchunks = static_cast<int>((p.batch + 63) / 64);
  P.part = part;
  P.tma_part = p.b % 4 == 0 ? 1 : 0;
  tmP = tmX;  // unused otherwise
  if (P.tma_part) {
    const uint64_t dims[3] = {b, c, static_cast<uint64_t>(splits) * a * d}, str[3] = {1, b, b * c};
    const uint32_t box[3] = {32, 32, 1};
    if ((st = encode_map(&tmP, KSMM_F32, 3, part, dims, str, box)) != KSMM_OK) return st;
  }
  P.status = status_word();
  if (!P.status) return set_error(KSMM_ERR_CUDA, "cannot resolve the device status word");
  const uint32_t fmt = p.in_dtype == KSMM_BF16 ? 1u : 0u;
  // fp32 accumulate, M = 128, N = NT; batch-last operands are K-major, batch-first ones MN-major
  P.idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | (X_LAST ? 0u : 1u << 15) | (G_LAST ? 0u : 1u << 16) |
            (static_cast<uint32_t>(NT >> 3) << 17) | (static_cast<uint32_t>(128 >> 4) << 24);
  const int64_t grid = static_cast<int64_t>(p.a) * p.d * splits * P.tiles_k * P.tiles_j;
  if (grid <= 0 || grid > 0x7fffffffLL)
    return set_error(KSMM_ERR_UNSUPPORTED, "weight gradient: %lld tiles exceed the grid limit",
                     static_cast<long long>(grid));
  cudaError_t err = launch_pdl(kern, static_cast<unsigned>(grid), kThreadsW, C::SMEM_BYTES, stream, tmX, tmG, tmP, P);
  count_launch();
  if (err == cudaSuccess) err = cudaGetLastError();
  if (err != cudaSuccess)
    return set_error(KSMM_ERR_CUDA, "weight-gradient kernel launch failed: %s", cudaGetErrorString(err));
  return KSMM_OK;
}

template <bool X_LAST, bool G_LAST>
static int launch_w_tile(const Problem& p, const WgradOperand& x, const WgradOperand& g, float* part, int mb, int nt,
                         int splits, cudaStream_t stream) {
  if (mb == 2) {
    if (nt == 64) return launch_w<X_LAST, G_LAST, 2, 64, 5>(p, x, g, part, splits, stream);
    if (nt == 128) return launch_w<X_LAST, G_LAST, 2, 128, 4>(p, x, g, part, splits, stream);
    return launch_w<X_LAST, G_LAST, 2, 256, 3>(p, x, g, part, splits, stream);
  }
  if (nt == 64) return launch_w<X_LAST, G_LAST, 1, 64, 8>(p, x, g, part, splits, stream);
  if (nt == 128) return launch_w<X_LAST, G_LAST, 1, 128, 6>(p, x, g, part, splits, stream);
  return launch_w<X_LAST, G_LAST, 1, 256, 4>(p, x, g, part, splits, stream);
}

}  // namespace tc

// ---------------------------------------------------------------------------
// plan of one weight gradient
// ---------------------------------------------------------------------------
namespace {

constexpr size_t align256(size_t v) { return (v + 255) / 256 * 256; }

struct WgradPlan {
  bool tc = false;                 // tensor cores; else the FFMA kernel
  bool copy_x = false, copy_g = false;
  int64_t ld_copy = 0;             // row stride of the copies
  int mb = 1, nt = 256, splits = 1;
  size_t x_bytes = 0, g_bytes = 0, part_bytes = 0;
  size_t total() const { return x_bytes + g_bytes + part_bytes; }
};

// Splits of the batch.  A CTA's time is its chunks plus its partial tile, both as bytes that cross
// L2 (45 to 52 GB/s per SM in the 16-bit kernel: 308 MB in 41 us on 144 CTAs), plus a fixed 2 us; CTAs run in waves of one per SM; the
// reduction then reads all partials.
int wgrad_splits(int64_t tiles, int64_t nchunks, double chunk_bytes, double tile_bytes, double elems) {
  int sms = tc::num_sms();
  if (sms <= 0) sms = 148;
  const int64_t most = std::min<int64_t>(64, std::max<int64_t>(1, nchunks / 2));
  double best = 1e30;
  int pick = 1;
  for (int64_t s = 1; s <= most; ++s) {
    const double waves = static_cast<double>((tiles * s + sms - 1) / sms);
    const double chunks = static_cast<double>((nchunks + s - 1) / s);
    const double us = waves * ((chunks * chunk_bytes + tile_bytes) / 45e3 + 2.0) + s * elems * 4.0 / 5e6;
    if (us < best * 0.995) { best = us; pick = static_cast<int>(s); }
  }
  return pick;
}

bool wgrad_operand_direct(const Problem& p, const WgradOperand& o, int feat, bool check_pointers) {
  const int es = dtype_size(p.in_dtype);
  if (check_pointers && reinterpret_cast<uintptr_t>(o.ptr) % 16) return false;
  if (o.last) return (o.ld * es) % 16 == 0;
  // fp32 batch-first operands are addressed in atoms of 32 features
  return (p.d == 1 || o.regrouped) && (p.in_dtype == KSMM_F32 ? feat % 32 == 0 : (feat * es) % 16 == 0);
}

WgradPlan plan_wgrad(const Problem& p, const WgradOperand& x, const WgradOperand& g, bool check_pointers) {
  WgradPlan w;
  if (p.batch <= 0 || p.batch > 0x7fffffffLL) return w;
  const bool f32 = p.in_dtype == KSMM_F32;
  if (!f32 && p.in_dtype != KSMM_F16 && p.in_dtype != KSMM_BF16) return w;
  if (f32 && p.batch < 128) return w;  // the FFMA kernel is the faster one there (tc_wgrad_f32.cu)
  w.copy_x = !wgrad_operand_direct(p, x, p.c, check_pointers);
  w.copy_g = !wgrad_operand_direct(p, g, p.b, check_pointers);
  // The padding of a tile is all the work there is for blocks of a few rows; the FFMA kernel, one CTA
  // per 16 x 16 outputs, takes those unless the 16-bit operands can be used as they stand.
  if ((p.b < 16 || p.c < 16) && (f32 || w.copy_x || w.copy_g)) return w;
  w.tc = true;
  w.ld_copy = (p.batch + 63) / 64 * 64;
  const size_t es = dtype_size(p.in_dtype), ad = static_cast<size_t>(p.a) * p.d;
  if (w.copy_x) w.x_bytes = align256(ad * p.c * w.ld_copy * es);
  if (w.copy_g) w.g_bytes = align256(ad * p.b * w.ld_copy * es);
  const double elems = static_cast<double>(ad) * p.b * p.c;
  const int64_t blocks = static_cast<int64_t>(ad);
  if (f32) {
    w.mb = 1;
    w.nt = p.b <= 64 ? 64 : 128;
    // (a chunk of 32 entries takes 1.5 us whatever its bytes; 63e3 for it gave the same times)
    w.splits = wgrad_splits(blocks * ((p.c + 127) / 128) * ((p.b + w.nt - 1) / w.nt), (p.batch + 31) / 32,
                            w.nt == 64 ? 22e3 : 30e3, 128.0 * w.nt * 4, elems);
  } else {
    w.mb = p.c > 128 ? 2 : 1;
    w.nt = p.b <= 64 ? 64 : (p.b <= 128 ? 128 : 256);
    const int cr = std::min(p.c, w.mb * 128), br = std::min(p.b, w.nt);  // rows that exist
    w.splits = wgrad_splits(blocks * ((p.c + w.mb * 128 - 1) / (w.mb * 128)) * ((p.b + w.nt - 1) / w.nt),
                            (p.batch + 63) / 64, 128.0 * (cr + br), 4.0 * cr * br, elems);
  }
  w.part_bytes = static_cast<size_t>(w.splits) * static_cast<size_t>(elems) * sizeof(float);
  return w;
}

// batch-last copy with padded rows of an operand that the tensor kernels cannot address
int wgrad_copy(const Problem& p, WgradOperand* o, int feat, void* dst, int64_t ld, cudaStream_t stream) {
  const int64_t rows = static_cast<int64_t>(p.a) * feat * p.d;
  const int es = dtype_size(p.in_dtype);
  const int st = o->last ? launch_copy_rows(o->ptr, o->ld, dst, ld, rows, p.batch, es, stream)
                         : launch_transpose(o->ptr, dst, p.batch, rows, es, stream, ld);
  *o = WgradOperand{dst, 1, ld};
  return st;
}

}  // namespace

bool wgrad_any_layout(const Problem& p) {
  return p.b >= 16 && p.c >= 16 && p.batch > 0 && p.batch <= 0x7fffffffLL && !(p.in_dtype == KSMM_F32 && p.batch < 128);
}

// ---------------------------------------------------------------------------
// gradient of the bias: sums over the batch in a fixed order.  16-bit gradients are summed in fp32.  Of fp32
// gradients a few neighbours at a time are summed in fp32 and these sums in fp64: a chain of fp32 additions
// as long as a thread's share of the batch would be the result's error (1.5e-7 to 3.6e-7 relative at 6272 to
// 50176 entries, against 1e-7 by a tree).
// ---------------------------------------------------------------------------
namespace {

template <typename T>
struct LongSum { using type = float; };
template <>
struct LongSum<float> { using type = double; };

// V neighbouring elements as floats (V * sizeof(T) = 16, or V = 1)
template <typename T, int V>
__device__ __forceinline__ void load16(const T* p, float (&v)[V]) {
  if constexpr (V == 1) {
    v[0] = ElemTraits<T>::to_float(*p);
  } else {
    const uint4 raw = *reinterpret_cast<const uint4*>(p);
    const T* e = reinterpret_cast<const T*>(&raw);
#pragma unroll
    for (int q = 0; q < V; ++q) v[q] = ElemTraits<T>::to_float(e[q]);
  }
}

// batch-last: one CTA per feature.  Bound by memory: 1536 x 6272 fp32 in 10 us (30 us by the framework's
// reduction)
template <typename T, int V>
__global__ void __launch_bounds__(128) bias_grad_rows_kernel(const T* __restrict__ g, int64_t ld, T* __restrict__ out, int64_t batch) {
  using Sum = typename LongSum<T>::type;
  const T* row = g + static_cast<int64_t>(blockIdx.x) * ld;
  Sum s = 0;
  const int64_t whole = batch / V * V;
#pragma unroll 4
  for (int64_t n = threadIdx.x * V; n < whole; n += 128 * V) {
    float v[V];
    load16<T, V>(row + n, v);
    if constexpr (V == 4) {
      s += (v[0] + v[1]) + (v[2] + v[3]);
    } else {
#pragma unroll
      for (int q = 0; q < V; ++q) s += v[q];
    }
  }
  for (int64_t n = whole + threadIdx.x; n < batch; n += 128) s += ElemTraits<T>::to_float(row[n]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  __shared__ Sum part[4];
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0)
    out[blockIdx.x] = ElemTraits<T>::from_float(static_cast<float>((part[0] + part[1]) + (part[2] + part[3])));
}

constexpr int kBiasSlices = 64;

// batch-first: a CTA sums 32 V features over a slice of the batch, its eight warps every eighth row; a
// second launch adds the slices.  12544 x 3072 fp16 (77 MB) in 15 us (36 us by the framework's reduction)
template <typename T, int V>
__global__ void __launch_bounds__(256)
    bias_grad_cols_kernel(const T* __restrict__ g, float* __restrict__ part, int64_t batch, int64_t feats) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t f0 = (static_cast<int64_t>(blockIdx.x) * 32 + lane) * V;
  const int64_t n_begin = blockIdx.y * batch / kBiasSlices, n_end = (blockIdx.y + 1) * batch / kBiasSlices;
  using Sum = typename LongSum<T>::type;
  Sum s[V] = {};
  if (f0 < feats) {
#pragma unroll 4
    for (int64_t n = n_begin + warp; n < n_end; n += 8) {
      float v[V];
      load16<T, V>(g + n * feats + f0, v);
#pragma unroll
      for (int q = 0; q < V; ++q) s[q] += v[q];
    }
  }
  __shared__ Sum sum[8][32 * V + 1];
#pragma unroll
  for (int q = 0; q < V; ++q) sum[warp][q * 32 + lane] = s[q];
  __syncthreads();
  for (int e = threadIdx.x; e < 32 * V; e += 256) {
    Sum t = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) t += sum[w][e];
    const int64_t f = (static_cast<int64_t>(blockIdx.x) * 32 + (e & 31)) * V + (e >> 5);
    if (f < feats) part[blockIdx.y * feats + f] = static_cast<float>(t);
  }
}
template <typename T>
__global__ void __launch_bounds__(256) bias_grad_sum_kernel(const float* __restrict__ part, int slices, T* __restrict__ out, int64_t feats) {
  const int64_t f = static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x;
  if (f >= feats) return;
  typename LongSum<T>::type s = 0;
#pragma unroll 8
  for (int q = 0; q < slices; ++q) s += part[q * feats + f];
  out[f] = ElemTraits<T>::from_float(static_cast<float>(s));
}

template <typename T>
int bias_grad_typed(const T* g, int last, int64_t ld, T* out, float* part, int64_t batch, int64_t feats, cudaStream_t stream) {
  constexpr int V = 16 / sizeof(T);
  const bool al = reinterpret_cast<uintptr_t>(g) % 16 == 0;
  if (feats > 0x7fffffffLL) return set_error(KSMM_ERR_UNSUPPORTED, "bias gradient: too many features");
  if (last) {
    if (al && ld % V == 0)
      bias_grad_rows_kernel<T, V><<<static_cast<unsigned>(feats), 128, 0, stream>>>(g, ld, out, batch);
    else
      bias_grad_rows_kernel<T, 1><<<static_cast<unsigned>(feats), 128, 0, stream>>>(g, ld, out, batch);
  } else {
    const bool vec = al && feats % V == 0;
    const int64_t span = vec ? 32 * V : 32;
    const dim3 grid(static_cast<unsigned>((feats + span - 1) / span), kBiasSlices);
    if (vec) bias_grad_cols_kernel<T, V><<<grid, 256, 0, stream>>>(g, part, batch, feats);
    else bias_grad_cols_kernel<T, 1><<<grid, 256, 0, stream>>>(g, part, batch, feats);
    count_launch();
    bias_grad_sum_kernel<T><<<static_cast<unsigned>((feats + 255) / 256), 256, 0, stream>>>(part, kBiasSlices, out, feats);
  }
  count_launch();
  cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess) return set_error(KSMM_ERR_CUDA, "bias-gradient launch failed: %s", cudaGetErrorString(err));
  return KSMM_OK;
}

}  // namespace

size_t bias_grad_workspace_bytes(int64_t feats) { return static_cast<size_t>(feats) * kBiasSlices * sizeof(float); }

int launch_bias_grad(const void* g, int last, int64_t ld, void* out, void* workspace, int64_t batch, int64_t feats,
                     int dtype, cudaStream_t stream) {
  float* part = static_cast<float*>(workspace);
  if (dtype == KSMM_F32)
    return bias_grad_typed(static_cast<const float*>(g), last, ld, static_cast<float*>(out), part, batch, feats, stream);
  if (dtype == KSMM_F16)
    return bias_grad_typed(static_cast<const __half*>(g), last, ld, static_cast<__half*>(out), part, batch, feats, stream);
  return bias_grad_typed(static_cast<const __nv_bfloat16*>(g), last, ld, static_cast<__nv_bfloat16*>(out), part, batch,
                         feats, stream);
}

int launch_bias_sum(const float* part, int slices, void* out, int64_t feats, int dtype, cudaStream_t stream) {
  const unsigned grid = static_cast<unsigned>((feats + 255) / 256);
  if (dtype == KSMM_F32) bias_grad_sum_kernel<<<grid, 256, 0, stream>>>(part, slices, static_cast<float*>(out), feats);
  else if (dtype == KSMM_F16) bias_grad_sum_kernel<<<grid, 256, 0, stream>>>(part, slices, static_cast<__half*>(out), feats);
  else bias_grad_sum_kernel<<<grid, 256, 0, stream>>>(part, slices, static_cast<__nv_bfloat16*>(out), feats);
  count_launch();
  cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess) return set_error(KSMM_ERR_CUDA, "bias-gradient launch failed: %s", cudaGetErrorString(err));
  return KSMM_OK;
}

size_t wgrad_workspace_bytes(const Problem& p, const WgradOperand& x, const WgradOperand& g) {
  return plan_wgrad(p, x, g, false).total();
}

// p.out = dW (kernel format, input dtype); x = X, g = dY
int wgrad_launch(const Problem& p, WgradOperand x, WgradOperand g, void* workspace, size_t workspace_bytes,
                 cudaStream_t stream) {
  const int64_t elems = static_cast<int64_t>(p.a) * p.b * p.c * p.d;
  if (p.batch == 0) {
    cudaError_t e = cudaMemsetAsync(p.out, 0, elems * dtype_size(p.in_dtype), stream);
    return e == cudaSuccess ? KSMM_OK : set_error(KSMM_ERR_CUDA, "memset failed: %s", cudaGetErrorString(e));
  }
  const WgradPlan w = plan_wgrad(p, x, g, true);
  if (w.tc && workspace && reinterpret_cast<uintptr_t>(workspace) % 16 == 0 && workspace_bytes >= w.total()) {
    char* ws = static_cast<char*>(workspace);
    float* part = reinterpret_cast<float*>(ws + w.x_bytes + w.g_bytes);
    int st = KSMM_OK;
    if (w.copy_x && (st = wgrad_copy(p, &x, p.c, ws, w.ld_copy, stream)) != KSMM_OK) return st;
    if (w.copy_g && (st = wgrad_copy(p, &g, p.b, ws + w.x_bytes, w.ld_copy, stream)) != KSMM_OK) return st;
    if (p.in_dtype == KSMM_F32) {
      st = wgrad_f32_launch(p, x, g, part, w.nt, w.splits, stream);
    } else if (x.last) {
      st = g.last ? tc::launch_w_tile<true, true>(p, x, g, part, w.mb, w.nt, w.splits, stream)
                  : tc::launch_w_tile<true, false>(p, x, g, part, w.mb, w.nt, w.splits, stream);
    } else {
      st = g.last ? tc::launch_w_tile<false, true>(p, x, g, part, w.mb, w.nt, w.splits, stream)
                  : tc::launch_w_tile<false, false>(p, x, g, part, w.mb, w.nt, w.splits, stream);
    }
    if (st != KSMM_OK) return st;
    cudaError_t err = p.in_dtype == KSMM_F32   ? tc::launch_reduce<float>(p, x, g, part, w.splits, stream)
                      : p.in_dtype == KSMM_F16 ? tc::launch_reduce<__half>(p, x, g, part, w.splits, stream)
                                               : tc::launch_reduce<__nv_bfloat16>(p, x, g, part, w.splits, stream);
    count_launch();
    if (err == cudaSuccess) err = cudaGetLastError();
    if (err != cudaSuccess)
      return set_error(KSMM_ERR_CUDA, "weight-gradient reduction launch failed: %s", cudaGetErrorString(err));
    return KSMM_OK;
  }
  if (x.last != g.last || (x.last && (x.ld != p.batch || g.ld != p.batch)))
    return set_error(KSMM_ERR_WORKSPACE, "weight gradient: operands in two layouts need a workspace of %zu bytes",
                     w.total());
  const int64_t nblk = static_cast<int64_t>(p.a) * p.d;
  if (nblk > 65535 || (p.c + 15) / 16 > 65535)
    return set_error(KSMM_ERR_UNSUPPORTED, "weight gradient: too many blocks for the fallback kernel");
  dim3 grid((p.b + 15) / 16, (p.c + 15) / 16, static_cast<unsigned>(nblk));
  if (p.in_dtype == KSMM_F32)
    wgrad_simt_kernel<float><<<grid, 256, 0, stream>>>(static_cast<const float*>(x.ptr),
                                                       static_cast<const float*>(g.ptr),
                                                       static_cast<float*>(p.out), p.batch, p.a, p.b, p.c, p.d,
                                                       x.last);
  else if (p.in_dtype == KSMM_F16)
    wgrad_simt_kernel<__half><<<grid, 256, 0, stream>>>(static_cast<const __half*>(x.ptr),
                                                        static_cast<const __half*>(g.ptr),
                                                        static_cast<__half*>(p.out), p.batch, p.a, p.b, p.c, p.d,
                                                        x.last);
  else if (p.in_dtype == KSMM_BF16)
    wgrad_simt_kernel<__nv_bfloat16><<<grid, 256, 0, stream>>>(
        static_cast<const __nv_bfloat16*>(x.ptr), static_cast<const __nv_bfloat16*>(g.ptr),
        static_cast<__nv_bfloat16*>(p.out), p.batch, p.a, p.b, p.c, p.d, x.last);
  else
    return set_error(KSMM_ERR_UNSUPPORTED, "weight gradients exist for fp32, fp16 and bf16");
  count_launch();
  cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess)
    return set_error(KSMM_ERR_CUDA, "weight-gradient kernel launch failed: %s", cudaGetErrorString(err));
  return KSMM_OK;
}

}  // namespace ksmm
