// fp32 weight gradients on the tensor cores:
//   dW[i,j,k,l] = sum_n dY4[i,j,l,n] X4[i,k,l,n],
// a*d independent (c x B) @ (B x b) products.  Every operand is cut into three bf16 values, each the rounded
// rest of the ones before it: v = v1 + v2 + v3 exactly (8 + 8 + 8 bits, the signs of the rests included; below
// 2^-110 the last one may fall under the smallest bf16).  A term is the six products x1 g1, x1 g2, x2 g1,
// x2 g2, x1 g3, x3 g1, each exact in fp32; x2 g3 and x3 g2, at most 2^-25 of it, are left out (2^-28 on average,
// next to the 2^-25.3 of one rounding), so that a term is as exact as an fp32 FMA's.  (Two tf32 parts cannot
// hold 24 bits: one bit was dropped from a quarter of the operands, and gradients of a few entries were two to
// three times as far from 64 bits as by FFMAs.)  The six bf16 products take the tensor time of three tf32
// ones.  Infinite operands give NaN, their rest being inf - inf; the reduction in backward.cu computes sums
// that are not finite once more.
//
// Accumulator rows are k (128 per tile), columns j (NT = 64 or 128), the K dimension of the MMAs is
// the batch, 32 entries per chunk.  TMA delivers raw tiles into one ring; eight splitter warps write their pieces
// [x1 | x2 | x3 | g1 | g2 | g3] into a second one, whose stages the MMAs read.  g2 follows g1 directly, so
// the two are one operand of 2 NT rows.  A batch-last operand has rows of consecutive batch entries: K-major
// pieces with rows of 64 bytes and the 64-byte swizzle.  A batch-first one (d = 1) has rows of consecutive
// features: MN-major pieces, groups of 64 features x 32 batch rows with the 128-byte swizzle.  The split is
// element-wise, so any combination of the two works.
//
// The contraction is long (a training batch), and the tensor core truncates when it adds into its
// accumulator, once per step of 16 entries.  So the accumulator only ever sums kFlush chunks (128
// entries, 8 additions); the epilogue warps then add it, rounded to nearest, to sums in registers,
// while the MMAs fill the other accumulator buffer.  Relative error against 64 bits for N(0,1) operands
// (the FFMA kernel's in brackets): 7.6e-8 (1.8e-7) at 128 entries, 8.3e-8 (3.2e-7) at 320, 1.4e-7 to 1.8e-7
// (1.4e-6) at 6272, 2.6e-8 (2.5e-8) where a single entry is not zero.  With two tf32 parts it was 2.0e-7, 2.0e-7,
// 3.5e-7 and 8.1e-8.  Below 128 entries the FFMA kernel runs: its launch is the shorter one there, (6,64,64,1) at
// 128 entries 20 us against 26, (1,768,192,2) 34 against 33 and at 256 46 against 33.
//
// What bounds it: the chain of a chunk, about 1.5 us for NT = 128 (TMA, split, ten MMAs), at the number of stages
// that fit; tensor pipe 31 %, issue slots 48 %, shared memory 27 % by loads and stores and 23 % by the MMAs.  (1,768,192,2) at 6272 batch entries: 58 us with the reduction, as with two tf32 parts (485 us on the
// FFMA kernel); (1,64,64,16) at 12544 52 us (56 with the tf32 parts), (1,768,192,4) 184 (177), batch-first
// (1,768,768,1) 148 (134).  For (1,768,192,2) six splitter warps take 62 us, four 64, ten 60; two raw stages and three
// of pieces 67.
//
// Roles (576 threads): warp 0 TMA producer, warp 1 TMEM owner and MMA issuer, warps 2..9 splitters,
// warps 10..17 epilogue.  Waits are bounded and report through the device status word.
#include <cuda.h>

#include <atomic>

#include "backward.h"
#include "tc_host.h"
#include "tc_kernel.h"
#include "tc_ptx.cuh"

namespace ksmm {
namespace tc {

struct ParamsWF {
  int a, b, c, d;
  int tiles_k, tiles_j, splits;
  int nchunks;      // ceil(batch / 32)
  uint32_t idesc;   // N = NT
  uint32_t idesc2;  // N = 2 NT
  float* part;      // (splits, a*d, c, b)
  int tma_part;     // b % 4 == 0: partial tiles leave through TMA
  int* status;
};

constexpr int kSplitWarpsWF = 8;
constexpr int kThreadsWF = (2 + kSplitWarpsWF + 8) * 32;
constexpr int kFlush = 4;  // chunks per accumulator buffer

// the three pieces of two neighbouring values; v becomes the rest of the first two
__device__ __forceinline__ uint32_t next_piece(float& v0, float& v1) {
  const __nv_bfloat162 p = __floats2bfloat162_rn(v0, v1);
  const uint32_t w = *reinterpret_cast<const uint32_t*>(&p);
  v0 -= __uint_as_float(w << 16);
  v1 -= __uint_as_float(w & 0xffff0000u);
  return w;
}

// Cuts one unit of a tile, eight values that lie next to each other in 16-byte pieces of a 128-byte swizzled raw row,
// into 16 bytes of each piece tile.  K-major (LAST): row = feature, q = octet of batch entries; MN-major: row =
// batch entry, q = octet of features.  Eight neighbouring lanes take eight rows: no bank conflicts on either side.
template <bool LAST>
__device__ __forceinline__ void split_unit(uint32_t raw, uint32_t pieces, uint32_t piece_bytes, int u, int rows) {
  const int row = LAST ? u & (rows - 1) : u & 31, q = LAST ? u / rows : u >> 5;
  const uint32_t src = raw + (LAST ? row * 128 : (q >> 2) * 4096 + row * 128);
  const int p = (LAST ? q : q & 3) * 2;
  const uint32_t dst = pieces + (LAST ? row * 64 + ((q ^ ((row >> 1) & 3)) << 4)
                                      : (q >> 3) * 4096 + row * 128 + (((q & 7) ^ (row & 7)) << 4));
  float v[8];
#pragma unroll
  for (int h = 0; h < 2; ++h)
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v[4 * h]), "=f"(v[4 * h + 1]), "=f"(v[4 * h + 2]), "=f"(v[4 * h + 3])
                 : "r"(src + (((p + h) ^ (row & 7)) << 4))
                 : "memory");
#pragma unroll
  for (int t = 0; t < 3; ++t) {
    uint32_t w[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) w[e] = next_piece(v[2 * e], v[2 * e + 1]);
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst + t * piece_bytes), "r"(w[0]), "r"(w[1]), "r"(w[2]),
                 "r"(w[3])
                 : "memory");
  }
}

// RT raw stages, ST stages of pieces
template <int NT, int RT, int ST>
struct CfgWF {
  static constexpr int X_RAW = 128 * 128, RAW_BYTES = X_RAW + NT * 128;  // 32 batch entries of 128 k and NT j (either order)
  static constexpr int X_PIECE = 128 * 64, G_PIECE = NT * 64;
  static constexpr int G_OFF = 3 * X_PIECE;
  static constexpr int STAGE_BYTES = 3 * X_PIECE + 3 * G_PIECE;
  static constexpr int NBAR = 2 * RT + 2 * ST + 4;
  static constexpr int BAR_BYTES = 256;
  static constexpr int SMEM_BYTES = RT * RAW_BYTES + ST * STAGE_BYTES + BAR_BYTES + 1024;
  static constexpr int BUF_COLS = 2 * NT;  // leading accumulator | small-terms accumulator
  static constexpr int TMEM_COLS = 2 * BUF_COLS;
  static_assert(NT == 64 || NT == 128, "j tile");
  static_assert(RT * RAW_BYTES >= 8 * (NT / 64) * 4096, "staging of the partial tile");
  static_assert(SMEM_BYTES <= 232448, "shared memory budget");
  static_assert(SMEM_BYTES > 116 * 1024, "one CTA per SM, so that the TMEM allocation never waits");
  static_assert(8 * NBAR + 16 <= BAR_BYTES, "barrier area");
};

template <bool X_LAST, bool G_LAST, int NT, int RT, int ST>
__global__ void __launch_bounds__(kThreadsWF, 1)
    ksmm_tc_wgrad_f32_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmG,
                             const __grid_constant__ CUtensorMap tmP, const ParamsWF P) {
  using C = CfgWF<NT, RT, ST>;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t sm0 = (raw + 1023u) & ~1023u;
  uint8_t* sm_gen = smem_raw + (sm0 - raw);
  const uint32_t raw0 = sm0, stage0 = raw0 + RT * C::RAW_BYTES;
  const uint32_t bar0 = stage0 + ST * C::STAGE_BYTES;
  uint8_t* bar_gen = sm_gen + RT * C::RAW_BYTES + ST * C::STAGE_BYTES;
  auto full_bar = [&](int s) { return bar0 + 8u * s; };                    // TMA: raw tiles landed
  auto read_bar = [&](int s) { return bar0 + 8u * (RT + s); };             // splitters: raw tiles read
  auto split_bar = [&](int s) { return bar0 + 8u * (2 * RT + s); };        // splitters: pieces written
  auto free_bar = [&](int s) { return bar0 + 8u * (2 * RT + ST + s); };    // MMA commit: pieces consumed
  auto tfull_bar = [&](int q) { return bar0 + 8u * (2 * RT + 2 * ST + q); };
  auto tempty_bar = [&](int q) { return bar0 + 8u * (2 * RT + 2 * ST + 2 + q); };
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(bar_gen + 8 * C::NBAR);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bar_gen + 8 * C::NBAR + 4);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < RT; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(read_bar(s), kSplitWarpsWF);
    }
    for (int s = 0; s < ST; ++s) {
      mbar_init(split_bar(s), kSplitWarpsWF);
      mbar_init(free_bar(s), 1);
    }
    for (int q = 0; q < 2; ++q) {
      mbar_init(tfull_bar(q), 1);
      mbar_init(tempty_bar(q), 8);
    }
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

  uint32_t t = blockIdx.x;
  const int tj = static_cast<int>(t % P.tiles_j); t /= P.tiles_j;
  const int tk = static_cast<int>(t % P.tiles_k); t /= P.tiles_k;
  const int sp = static_cast<int>(t % P.splits);
  const int blk = static_cast<int>(t / P.splits);
  const int i = blk / P.d, l = blk % P.d;
  const int k0 = tk * 128, j0 = tj * NT;
  const int ch_begin = static_cast<int>(static_cast<int64_t>(sp) * P.nchunks / P.splits);
  const int ch_end = static_cast<int>(static_cast<int64_t>(sp + 1) * P.nchunks / P.splits);

  if (warp == 0) {
    // ===================== TMA producer =====================
    if (lane == 0) {
      uint32_t si = 0, sph = 0;
      for (int ch = ch_begin; ch < ch_end; ++ch) {
        if (!mbar_wait<64>(read_bar(si), sph ^ 1u, abort_flag, P.status, 81)) break;
        const uint32_t dst = raw0 + si * C::RAW_BYTES;
        const uint32_t bar = full_bar(si);
        mbar_expect_tx(bar, C::RAW_BYTES);
        const int n0 = ch * 32;
        if constexpr (X_LAST) tma_load_4d(dst, &tmX, bar, n0, l, k0, i);
        else tma_load_4d(dst, &tmX, bar, 0, n0, k0 / 32, blk);
        if constexpr (G_LAST) tma_load_4d(dst + C::X_RAW, &tmG, bar, n0, l, j0, i);
        else tma_load_4d(dst + C::X_RAW, &tmG, bar, 0, n0, j0 / 32, blk);
        if (++si == RT) { si = 0; sph ^= 1u; }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ===================== MMA issuer =====================
    if (lane == 0) {
      uint32_t si = 0, sph = 0, ut = 0;
      bool ok = true;
      for (int ch = ch_begin; ch < ch_end && ok; ++ut) {
        const uint32_t buf = ut & 1u, bph = (ut >> 1) & 1u;
        if (!mbar_wait<0>(tempty_bar(buf), bph ^ 1u, abort_flag, P.status, 82)) { ok = false; break; }
        tc_fence_after();
        const uint32_t dcol = tmem_base + buf * C::BUF_COLS, dsmall = dcol + NT;
        const int stop = min(ch + kFlush, ch_end);
        for (bool first = true; ch < stop; ++ch, first = false) {
          if (!mbar_wait<0>(split_bar(si), sph, abort_flag, P.status, 83)) { ok = false; break; }
          tc_fence_after();
          const uint32_t xb = stage0 + si * C::STAGE_BYTES, gb = xb + C::G_OFF;
          // K-major: 8 rows of 64 bytes are 512 bytes apart, a k step of 16 entries is 32 bytes inside the row;
          // MN-major: 4 KB between groups of 64 features, 1 KB between groups of 8 batch rows
          auto xd = [&](int t, int ks) {
            const uint32_t at = xb + t * C::X_PIECE;
            return X_LAST ? make_desc(at + ks * 32, 16, 512, 4) : make_desc(at + ks * 2048, 4096, 1024, 2);
          };
          auto gd = [&](int t, int ks) {
            const uint32_t at = gb + t * C::G_PIECE;
            return G_LAST ? make_desc(at + ks * 32, 16, 512, 4) : make_desc(at + ks * 2048, 4096, 1024, 2);
          };
#pragma unroll
          for (int ks = 0; ks < 2; ++ks) {
            // x1 * [g1 | g2]: the leading accumulator and, next to it, the small one
            umma<2>(dcol, xd(0, ks), gd(0, ks), P.idesc2, (first && ks == 0) ? 0u : 1u);
            umma<2>(dsmall, xd(0, ks), gd(2, ks), P.idesc, 1u);
            umma<2>(dsmall, xd(1, ks), gd(0, ks), P.idesc, 1u);
            umma<2>(dsmall, xd(1, ks), gd(1, ks), P.idesc, 1u);
            umma<2>(dsmall, xd(2, ks), gd(0, ks), P.idesc, 1u);
          }
          umma_commit(free_bar(si));
          if (++si == ST) { si = 0; sph ^= 1u; }
        }
        if (ok) umma_commit(tfull_bar(buf));
      }
    }
    __syncwarp();
  } else if (warp < 2 + kSplitWarpsWF) {
    // ===================== splitters =====================
    const int tt = (warp - 2) * 32 + lane;
    constexpr int kXU = 128 * 4, kU = kXU + NT * 4;  // units of 8 values
    uint32_t ri = 0, rph = 0, si = 0, sph = 0;
    for (int ch = ch_begin; ch < ch_end; ++ch) {
      int got = 1;
      if (lane == 0)
        got = mbar_wait<32>(full_bar(ri), rph, abort_flag, P.status, 84) &&
              mbar_wait<32>(free_bar(si), sph ^ 1u, abort_flag, P.status, 86) ? 1 : 0;
      got = __shfl_sync(0xffffffffu, got, 0);
      if (!got) break;
      const uint32_t rb = raw0 + ri * C::RAW_BYTES, sb = stage0 + si * C::STAGE_BYTES;
#pragma unroll 2
      for (int u = tt; u < kU; u += kSplitWarpsWF * 32) {
        if (u < kXU) split_unit<X_LAST>(rb, sb, C::X_PIECE, u, 128);
        else split_unit<G_LAST>(rb + C::X_RAW, sb + C::G_OFF, C::G_PIECE, u - kXU, NT);
      }
      fence_proxy_async();  // the pieces are read by the tensor core through the async proxy
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(split_bar(si));
        mbar_arrive(read_bar(ri));
      }
      if (++ri == RT) { ri = 0; rph ^= 1u; }
      if (++si == ST) { si = 0; sph ^= 1u; }
    }
    __syncwarp();
  } else {
    // ===================== epilogue =====================
    // lane = accumulator row k, NT / 2 columns per warp, summed in registers over the buffers
    const int q = warp & 3, h = (warp - 2 - kSplitWarpsWF) >> 2;
    const uint32_t tm = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + h * (NT / 2);
    float acc[NT / 2];
#pragma unroll
    for (int e = 0; e < NT / 2; ++e) acc[e] = 0.f;
    bool ok = true;
    uint32_t ut = 0;
    for (int ch = ch_begin; ch < ch_end; ch += kFlush, ++ut) {
      const uint32_t buf = ut & 1u, bph = (ut >> 1) & 1u;
      int got = 1;
      if (lane == 0) got = mbar_wait<128>(tfull_bar(buf), bph, abort_flag, P.status, 85) ? 1 : 0;
      got = __shfl_sync(0xffffffffu, got, 0);
      if (!got) { ok = false; break; }
      tc_fence_after();
#pragma unroll
      for (int cg = 0; cg < NT / 2; cg += 16) {
        uint32_t r[16], rs[16];
        tmem_ld16(tm + buf * C::BUF_COLS + cg, r);
        tmem_ld16(tm + buf * C::BUF_COLS + NT + cg, rs);
        tmem_ld_wait();
#pragma unroll
        for (int e = 0; e < 16; ++e) acc[cg + e] += __uint_as_float(r[e]) + __uint_as_float(rs[e]);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(tempty_bar(buf));
    }
    const int krow0 = k0 + q * 32;
    if (ok && krow0 < P.c) {
      // the last buffer is complete, so every raw tile has been read: that ring is free for staging
      const int pz = sp * P.a * P.d + blk;
#pragma unroll
      for (int cg = 0; cg < NT / 64; ++cg) {
        const int jc = j0 + h * (NT / 2) + cg * 32;
        if (jc >= P.b) break;
        if (P.tma_part) {
          const uint32_t stg = raw0 + ((warp - 2 - kSplitWarpsWF) * 2 + cg) * 4096;
#pragma unroll
          for (int c4 = 0; c4 < 8; ++c4)
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(stg + lane * 128 + ((c4 ^ (lane & 7)) << 4)),
                         "r"(__float_as_uint(acc[cg * 32 + c4 * 4])), "r"(__float_as_uint(acc[cg * 32 + c4 * 4 + 1])),
                         "r"(__float_as_uint(acc[cg * 32 + c4 * 4 + 2])), "r"(__float_as_uint(acc[cg * 32 + c4 * 4 + 3]))
                         : "memory");
          fence_proxy_async();
          __syncwarp();
          if (lane == 0) {
            tma_store_3d(&tmP, stg, jc, krow0, pz);
            bulk_commit();
          }
        } else if (krow0 + lane < P.c) {
          float* row = P.part + (static_cast<int64_t>(pz) * P.c + krow0 + lane) * P.b + jc;
#pragma unroll
          for (int e = 0; e < 32; ++e)
            if (jc + e < P.b) row[e] = acc[cg * 32 + e];
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

template <bool X_LAST, bool G_LAST, int NT, int RT, int ST>
static int launch_wf(const Problem& p, const WgradOperand& x, const WgradOperand& g, float* part, int splits,
                     cudaStream_t stream) {
  using C = CfgWF<NT, RT, ST>;
  auto kern = ksmm_tc_wgrad_f32_kernel<X_LAST, G_LAST, NT, RT, ST>;
  static std::atomic<bool> attr_set[64];  // zero-initialised; set once per device (a repeated set is harmless)
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
  auto operand_map = [&](CUtensorMap* tm, bool last, const WgradOperand& o, uint64_t f, uint32_t rows) {
    if (last) {
      // (batch, d, features, a): 32 batch entries x `rows` features per box
      const uint64_t L = o.ld;
      const uint64_t dims[4] = {B, d, f, a}, str[4] = {1, L, d * L, f * d * L};
      const uint32_t box[4] = {32, 1, rows, 1};
      return encode_map(tm, KSMM_F32, 4, o.ptr, dims, str, box);
    }
    // (feature % 32, batch, feature / 32, block): rows / 32 atoms of 32 features x 32 batch rows.  The a blocks of
    // d = 1 and the a * d of block-ordered rows follow one another.
    const uint64_t dims[4] = {32, B, f / 32, a * d}, str[4] = {1, a * d * f, 32, f};
    const uint32_t box[4] = {32, 32, rows / 32, 1};
    return encode_map(tm, KSMM_F32, 4, o.ptr, dims, str, box);
  };
  if ((st = operand_map(&tmX, X_LAST, x, c, 128)) != KSMM_OK) return st;
  if ((st = operand_map(&tmG, G_LAST, g, b, NT)) != KSMM_OK) return st;
  ParamsWF P;
  P.a = p.a; P.b = p.b; P.c = p.c; P.d = p.d;
  P.tiles_k = (p.c + 127) / 128;
  P.tiles_j = (p.b + NT - 1) / NT;
  P.splits = splits;
  P.nchunks = static_cast<int>((p.batch + 31) / 32);
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
  // fp32 accumulate, bf16 operands, M = 128; batch-last operands are K-major, batch-first ones MN-major
  const uint32_t common = (1u << 4) | (1u << 7) | (1u << 10) | (X_LAST ? 0u : 1u << 15) | (G_LAST ? 0u : 1u << 16) |
                          (static_cast<uint32_t>(128 >> 4) << 24);
  P.idesc = common | (static_cast<uint32_t>(NT >> 3) << 17);
  P.idesc2 = common | (static_cast<uint32_t>(2 * NT >> 3) << 17);
  const int64_t grid = static_cast<int64_t>(p.a) * p.d * splits * P.tiles_k * P.tiles_j;
  if (grid <= 0 || grid > 0x7fffffffLL)
    return set_error(KSMM_ERR_UNSUPPORTED, "weight gradient: %lld tiles exceed the grid limit",
                     static_cast<long long>(grid));
  cudaError_t err = launch_pdl(kern, static_cast<unsigned>(grid), kThreadsWF, C::SMEM_BYTES, stream, tmX, tmG, tmP, P);
  count_launch();
  if (err == cudaSuccess) err = cudaGetLastError();
  if (err != cudaSuccess)
    return set_error(KSMM_ERR_CUDA, "weight-gradient kernel launch failed: %s", cudaGetErrorString(err));
  return KSMM_OK;
}

template <bool X_LAST, bool G_LAST>
static int launch_wf_tile(const Problem& p, const WgradOperand& x, const WgradOperand& g, float* part, int nt,
                          int splits, cudaStream_t stream) {
  return nt == 64 ? launch_wf<X_LAST, G_LAST, 64, 4, 3>(p, x, g, part, splits, stream)
                  : launch_wf<X_LAST, G_LAST, 128, 4, 2>(p, x, g, part, splits, stream);
}

}  // namespace tc

int wgrad_f32_launch(const Problem& p, const WgradOperand& x, const WgradOperand& g, float* part, int nt, int splits,
                     cudaStream_t stream) {
  if (x.last)
    return g.last ? tc::launch_wf_tile<true, true>(p, x, g, part, nt, splits, stream)
                  : tc::launch_wf_tile<true, false>(p, x, g, part, nt, splits, stream);
  return g.last ? tc::launch_wf_tile<false, true>(p, x, g, part, nt, splits, stream)
                : tc::launch_wf_tile<false, false>(p, x, g, part, nt, splits, stream);
}

}  // namespace ksmm
