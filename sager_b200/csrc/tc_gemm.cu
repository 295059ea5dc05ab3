// tc_gemm.cu - the fp16 tensor-core family of the reference's prefill path
// (include/sager/kernels/cuda_ops.hpp:104-152; src/kernels/cuda/tc_gemm.cu): Q4_K
// weights dequantised to fp16, then  y[t][row] = sum_k x[t][k] * w[row][k]  with
// fp32 accumulation. The reference hands the GEMM to a library; here it is one
// tcgen05 kernel:
//
//   * warp 0 moves operand tiles (128 rows x 64 halfs) global -> shared with TMA
//     through two tensor maps encoded by the launcher and passed as kernel
//     parameters, a four-stage ring of (weights, activations) tile pairs;
//   * warp 1 owns tensor memory and issues tcgen05.mma kind::f16 (M 128, N up to
//     128, K 16 per instruction, fp32 accumulators in 128 TMEM columns);
//   * warps 2-5 read the accumulators back (tcgen05.ld) and store fp16 or fp32
//     rows, 32 consecutive weight rows of one token per warp store.
//
// Two operand layouts are built: 128-byte swizzled tiles (one 2-D box per tile) and
// unswizzled 8x16-byte core matrices (a 3-D box whose innermost extent is one core
// matrix row). Every wait is bounded; an expired wait raises the status word and the
// CTA still releases its tensor memory.
#include <cuda.h>

#include <atomic>
#include <cstring>

#include <algorithm>

#include "api_util.cuh"
#include "q4k_common.cuh"
#include "umma.cuh"

namespace sgr {
namespace {

constexpr int kBM = 128;            // weight rows per CTA (MMA M)
constexpr int kBN = 128;            // token rows per CTA (max MMA N)
constexpr int kBK = 64;             // halfs per stage and operand row: 128 bytes
constexpr int kTcStages = 4;
constexpr int kTileBytes = kBM * kBK * 2;                 // 16 KB, both operands
constexpr int kTcThreads = 192;
constexpr int kTcSmem = 1024 /*alignment slack*/ + 1024 /*barriers*/ + kTcStages * 2 * kTileBytes;
constexpr int kTcCols = 128;

enum { kLayoutSwizzled = 0, kLayoutCore = 1 };

// Shared-memory operand descriptors (K-major).
//   swizzled: rows of 128 bytes, eight-row groups 1024 bytes apart, 128-byte swizzle
//   core:     8x16-byte core matrices; K-adjacent ones a whole column of the tile apart
//             (tile rows x 16 bytes), eight-row groups 128 bytes apart
__device__ __forceinline__ uint64_t tc_desc(uint32_t saddr, int layout, int tile_rows) {
  const uint64_t start = (saddr & 0x3FFFFu) >> 4;
  if (layout == kLayoutSwizzled)
    return start | (static_cast<uint64_t>(1) << 16) | (static_cast<uint64_t>(1024 >> 4) << 32) |
           (static_cast<uint64_t>(1) << 46) | (static_cast<uint64_t>(2) << 61);
  return start | (static_cast<uint64_t>(tile_rows) << 16) /* tile_rows * 16 bytes >> 4 */ |
         (static_cast<uint64_t>(128 >> 4) << 32) | (static_cast<uint64_t>(1) << 46);
}
// D fp32, A and B fp16, both K-major, M = 128, N = n
__device__ __forceinline__ uint32_t tc_idesc(int n) {
  return (1u << 4) | (static_cast<uint32_t>(n >> 3) << 17) | (static_cast<uint32_t>(kBM >> 4) << 24);
}
__device__ __forceinline__ void tc_mma(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc,
                                       uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}"
      ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate), "r"(0u)
      : "memory");
}
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void tc_ld16(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
        "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tc_tma_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
               ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar)) : "memory");
}
// into this CTA's shared memory, the bytes counted at a barrier of the CTA pair (an address in the cluster's shared memory)
__device__ __forceinline__ void tc_tma_2d_pair(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
               ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}
__device__ __forceinline__ void tc_tma_3d(uint32_t dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar) {
  asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
               ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar)) : "memory");
}

struct TcArgs {
  void* y;
  int n_rows, k, n_tokens;
  int layout;
  int bn;                 // token rows per CTA: 128, or 64 when that is what fills the machine
  int* status;
};

template <bool F32OUT>
__global__ void __launch_bounds__(kTcThreads) tc_gemm_kernel(const __grid_constant__ CUtensorMap map_w,
                                                             const __grid_constant__ CUtensorMap map_x,
                                                             const TcArgs a) {
  extern __shared__ unsigned char tc_smem_raw[];
  const uint32_t base = (smem_u32(tc_smem_raw) + 1023u) & ~1023u;
  unsigned char* smem = tc_smem_raw + (base - smem_u32(tc_smem_raw));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem);          // full[S], empty[S], acc
  uint64_t* full = bars;
  uint64_t* empty = bars + kTcStages;
  uint64_t* acc_full = bars + 2 * kTcStages;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * kTcStages + 1);
  int* fail = reinterpret_cast<int*>(tmem_slot + 1);
  const uint32_t tiles = base + 1024;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row0 = blockIdx.x * kBM, tok0 = blockIdx.y * a.bn;
  const int ntok = min(a.bn, a.n_tokens - tok0);
  const uint32_t b_bytes = static_cast<uint32_t>(a.bn) * kBK * 2;
  const int n_mma = max(16, (ntok + 15) & ~15);
  const int nkb = a.k / kBK;

  if (threadIdx.x == 0) {
    for (int i = 0; i < kTcStages; ++i) {
      mbar_init(full + i, 1);
      mbar_init(empty + i, 1);
    }
    mbar_init(acc_full, 1);
    *fail = 0;
    fence_barrier_init();
    fence_proxy_async();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(kTcCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    if (lane == 0) {
      for (int kb = 0; kb < nkb; ++kb) {
        const int s = kb % kTcStages;
        if (kb >= kTcStages && !mbar_wait(empty + s, ((kb / kTcStages) - 1) & 1)) {
          atomicExch(fail, 1);
          break;
        }
        mbar_expect_tx(full + s, kTileBytes + b_bytes);
        const uint32_t ta = tiles + s * 2 * kTileBytes, tb = ta + kTileBytes;
        if (a.layout == kLayoutSwizzled) {
          tc_tma_2d(ta, &map_w, kb * kBK, row0, full + s);
          tc_tma_2d(tb, &map_x, kb * kBK, tok0, full + s);
        } else {
          tc_tma_3d(ta, &map_w, 0, row0, kb * (kBK / 8), full + s);
          tc_tma_3d(tb, &map_x, 0, tok0, kb * (kBK / 8), full + s);
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      const uint32_t idesc = tc_idesc(n_mma);
      // bytes between K = 16 slices of a tile
      const int kstep_a = a.layout == kLayoutSwizzled ? 32 : 2 * kBM * 16;
      const int kstep_b = a.layout == kLayoutSwizzled ? 32 : 2 * a.bn * 16;
      bool ok = true;
      for (int kb = 0; kb < nkb && ok; ++kb) {
        const int s = kb % kTcStages;
        ok = mbar_wait(full + s, (kb / kTcStages) & 1);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t ta = tiles + s * 2 * kTileBytes, tb = ta + kTileBytes;
#pragma unroll
        for (int j = 0; j < kBK / 16; ++j)
          tc_mma(tmem, tc_desc(ta + j * kstep_a, a.layout, kBM), tc_desc(tb + j * kstep_b, a.layout, a.bn), idesc,
                 (kb | j) != 0);
        tc_commit(empty + s);
      }
      if (!ok) atomicExch(fail, 1);
      tc_commit(acc_full);             // arrives when everything issued so far has finished
    }
  } else {
    const int quarter = warp & 3;      // the TMEM lanes this warp may read
    const bool ok = mbar_wait(acc_full, 0);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (!ok && lane == 0) atomicExch(fail, 1);
    const int row = row0 + quarter * 32 + lane;
    if (__all_sync(0xFFFFFFFFu, ok && *reinterpret_cast<volatile int*>(fail) == 0)) {
      for (int c = 0; c < ntok; c += 16) {
        uint32_t v[16];
        tc_ld16(tmem + (static_cast<uint32_t>(quarter * 32) << 16) + c, v);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (row < a.n_rows) {
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            if (c + i < ntok) {
              const size_t o = static_cast<size_t>(tok0 + c + i) * a.n_rows + row;
              if constexpr (F32OUT) reinterpret_cast<float*>(a.y)[o] = __uint_as_float(v[i]);
              else reinterpret_cast<uint16_t*>(a.y)[o] = f2h(__uint_as_float(v[i]));
            }
          }
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTcCols) : "memory");
  }
  if (threadIdx.x == 0 && *fail != 0 && a.status != nullptr) atomicExch(a.status, 1);
}

// ---- dequantisation ----------------------------------------------------------------------
// Lane l of a warp owns weights 8l .. 8l+7 of one super-block: sub-block l/4, its
// (l%4)-th octet. The warp's 32 stores are one contiguous 512-byte run.
// value = fp16( fma(d*sc, q, -(dmin*m)) ): one rounding to fp32, one to fp16
// (src/kernels/cuda/tc_gemm.cu:58-95 of the reference).
__device__ __forceinline__ uint4 dequant_octet(const unsigned char* blk, int lane) {
  const uint32_t dm = __ldg(reinterpret_cast<const uint32_t*>(blk));
  const Scales6 s6 = unpack_scales6(__ldg(reinterpret_cast<const uint32_t*>(blk + 4)),
                                    __ldg(reinterpret_cast<const uint32_t*>(blk + 8)),
                                    __ldg(reinterpret_cast<const uint32_t*>(blk + 12)));
  const int sb = lane >> 2, q = lane & 3;
  const float sd = h2f(static_cast<uint16_t>(dm & 0xFFFFu)) *
                   static_cast<float>(((sb < 4 ? s6.sc[0] : s6.sc[1]) >> (8 * (sb & 3))) & 0xFFu);
  const float sm = h2f(static_cast<uint16_t>(dm >> 16)) *
                   static_cast<float>(((sb < 4 ? s6.mn[0] : s6.mn[1]) >> (8 * (sb & 3))) & 0xFFu);
  const uint32_t* qp = reinterpret_cast<const uint32_t*>(blk + 16 + (sb >> 1) * 32 + q * 8);
  const uint2 w = make_uint2(__ldg(qp), __ldg(qp + 1));
  const int shift = (sb & 1) * 4;
  auto half_of = [&](uint32_t word, int byte) -> uint32_t {
    const uint32_t nib = (word >> (8 * byte + shift)) & 0xFu;
    return f2h(__fmaf_rn(sd, static_cast<float>(nib), -sm));
  };
  uint4 o;
  o.x = half_of(w.x, 0) | (half_of(w.x, 1) << 16);
  o.y = half_of(w.x, 2) | (half_of(w.x, 3) << 16);
  o.z = half_of(w.y, 0) | (half_of(w.y, 1) << 16);
  o.w = half_of(w.y, 2) | (half_of(w.y, 3) << 16);
  return o;
}

// ---- Q4_K weights: the dequantisation inside the GEMM ------------------------------------------
// Persistent: a CTA, or a pair of CTAs (CG = 2, cta_group::2), takes units of 128 weight rows per CTA x up to 256 token rows. The
// rows are the M lanes of tensor memory, so a thread dequantises its row of a block in registers and stores it as the
// tensor-memory operand (tcgen05.st); only the activations go through shared memory, of a pair's each CTA half.
//   * warps 0-7: unpack, four to a block, even and odd blocks, on into the next unit; a block is two of four slots in tensor memory,
//     so neither four waits for the other's
//   * warps 8-15: epilogue, a quarter of the lanes and half of the columns each, sixteen columns at a time (all of them into registers
//     first, so that the accumulators are free earlier, is straight-line code and lost more: 2048 x 512 over 1457 tokens 8.55 us, now 6.5, 4096 x 512
//     over 1000 10.9 and 8.6, 4096 x 2048 over 2048 29.8 and 29.3)
//   * warp 16: activation tiles (TMA, 128-byte swizzle, 64 k a stage)
//   * warp 17: block columns of the weights (a TMA copy of 128 blocks each), four in flight
//   * warp 18: tensor memory and (a pair's first CTA) MMA issue
// 4096 x 2048 over 2048 rows (MMAs 16 us at two units each, 20.8 at the library's rate): 38.5 us with a CTA per unit, whose start and epilogue
// nothing covered, 32.8 persistent and in pairs, 31.8 with the weights by TMA (one warp's cp.async, 36 to a block with a division
// each, took longer than the block: 130 x 4096 over 333 rows 28 -> 21), 31.2 with four slots instead of three (those with pairs of N = 240;
// inputs from HBM 37.9, and 38.4 with the N = 256 that mma_columns asks for). The tensor pipe of an SM with two units is busy for 67 % of its
// cycles, about 2,050 to a block; the rest is the start, the last epilogue, the scratch (by the estimate below 2 us) and hand-overs.
// `scratch` receives the dequantised rows: with few units by CTAs of their own on the SMs left over (a thread's 16-byte pieces of
// its row take longer than its block: 1000 x 4096 over 75 rows 33.8 -> 22.6 us, over 64 rows 54.5 -> 22.5), else each token
// tile writes its share of the blocks. (Written by the epilogue warps out of the weights' ring, 512 bytes a row: 33.8 us for 31.0.)
constexpr int kQ4Unpack = 8, kQ4Epi = 8, kQ4WarpX = kQ4Unpack + kQ4Epi, kQ4WarpW = kQ4WarpX + 1, kQ4WarpMma = kQ4WarpW + 1;
constexpr int kQ4Threads = (kQ4WarpMma + 1) * 32, kQ4WStages = 4, kQ4WBytes = 128 * kW4, kQ4Slots = 4;
constexpr int kQ4BBytes = 128 * 1024;             // activation ring: 4 stages of 256 rows, 8 of 128 or fewer
constexpr int kQ4Smem = 1024 + 1024 + kQ4BBytes + kQ4WStages * kQ4WBytes;
enum { kQ4WFull = 0, kQ4WEmpty = 4, kQ4AFull = 8, kQ4AEmpty = 12, kQ4BFull = 16, kQ4BEmpty = 24, kQ4AccFull = 32, kQ4AccEmpty = 33, kQ4Drain = 34 };

// The four weights of a word under `mask` (its low or its high nibbles), sd * q + sm rounded to fp16: 2^23 + q by byte insertion,
// - 2^23 exactly. (Nibbles as 1024 + q in fp16 and an addition in mixed precision, half the integer instructions: no faster.)
__device__ __forceinline__ void dequant_word(uint32_t raw, uint32_t mask, f32x2 sd, f32x2 sm, uint32_t& v01, uint32_t& v23) {
  const f32x2 magic = splat2(-8388608.f);
  const uint32_t nib = raw & mask;
  const f32x2 q01 = add2(pack2(__byte_perm(nib, 0x4B000000u, 0x7440), __byte_perm(nib, 0x4B000000u, 0x7441)), magic);
  const f32x2 q23 = add2(pack2(__byte_perm(nib, 0x4B000000u, 0x7442), __byte_perm(nib, 0x4B000000u, 0x7443)), magic);
  const f32x2 f01 = fma2(sd, q01, sm), f23 = fma2(sd, q23, sm);
  v01 = h2_bits(__floats2half2_rn(part2(f01, 0), part2(f01, 1)));
  v23 = h2_bits(__floats2half2_rn(part2(f23, 0), part2(f23, 1)));
}

// Columns of an MMA over n tokens: M = 128 of one CTA takes any multiple of 16, a pair's M = 256 with A in tensor memory multiples of 32 (what
// CUTLASS's SM100_MMA_F16BF16_2x1SM_TS asserts). The tokens past a tile's end are the next tile's or, past the matrix, zeros; their sums are
// not stored.
template <int CG>
__host__ __device__ constexpr int mma_columns(int n) { return (n + 16 * CG - 1) / (16 * CG) * (16 * CG); }

struct Q4Args {
  const unsigned char* w;
  uint16_t *y, *scratch;
  int n_rows, k, n_tokens;
  int bn, stages, tiles;                          // token rows per unit, activation stages, token tiles
  int row_units, units, workers;                  // groups of CG row tiles, units, CTAs that work on them (the others: scratch)
  int tiles_write;                                // the token tiles write the scratch
  int* status;
};

template <int CG>
__global__ void __launch_bounds__(kQ4Threads, 1) tc_gemm_q4_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, const Q4Args a) {
  extern __shared__ unsigned char tc_smem_raw[];
  const uint32_t base = (smem_u32(tc_smem_raw) + 1023u) & ~1023u;
  unsigned char* smem = tc_smem_raw + (base - smem_u32(tc_smem_raw));
  uint64_t* bar = reinterpret_cast<uint64_t*>(smem);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + 512);
  volatile int* fail = reinterpret_cast<volatile int*>(smem + 516);
  unsigned char* w_sm = smem + 1024 + kQ4BBytes;
  const uint32_t b_sm = base + 1024;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nb = a.k / kQK;
  if (static_cast<int>(blockIdx.x) >= a.workers) {        // writes a row tile's dequantised blocks, a warp per block
    pdl_wait();
    pdl_launch_dependents();
    const int row_tiles = (a.n_rows + 127) / 128, i = blockIdx.x - a.workers, row0 = i % row_tiles * 128;
    const int blocks = min(128, a.n_rows - row0) * nb, part = i / row_tiles, parts = (gridDim.x - a.workers) / row_tiles;
    if (part >= parts) return;
    const unsigned char* w = a.w + static_cast<size_t>(row0) * nb * kW4;
    uint4* out = reinterpret_cast<uint4*>(a.scratch + static_cast<size_t>(row0) * a.k);
    const int stride = parts * (kQ4Threads / 32);
    for (int b = part * (kQ4Threads / 32) + warp; b < blocks; b += 4 * stride) {
      uint4 v[4];                                 // four blocks' loads in flight
#pragma unroll
      for (int u = 0; u < 4; ++u) v[u] = dequant_octet(w + static_cast<size_t>(min(b + u * stride, blocks - 1)) * kW4, lane);
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (b + u * stride < blocks) out[static_cast<size_t>(b + u * stride) * 32 + lane] = v[u];
    }
    return;
  }
  const uint32_t rank = CG == 2 ? blockIdx.x & 1u : 0u, b_bytes = static_cast<uint32_t>(a.bn / CG) * 128;

  if (threadIdx.x == 0) {
    for (int i = 0; i < kQ4WStages; ++i) { mbar_init(&bar[kQ4WFull + i], 1); mbar_init(&bar[kQ4WEmpty + i], 4); }
    for (int i = 0; i < kQ4Slots; ++i) { mbar_init(&bar[kQ4AFull + i], 4 * CG); mbar_init(&bar[kQ4AEmpty + i], 1); }
    for (int i = 0; i < 8; ++i) { mbar_init(&bar[kQ4BFull + i], 1); mbar_init(&bar[kQ4BEmpty + i], 1); }
    mbar_init(&bar[kQ4AccFull], 1);
    mbar_init(&bar[kQ4AccEmpty], kQ4Epi * CG);
    mbar_init(&bar[kQ4Drain], 1);
    *fail = 0;
    fence_barrier_init();
    fence_proxy_async();
  }
  if (warp == kQ4WarpMma) {
    __syncwarp();
    asm volatile("tcgen05.alloc.cta_group::%2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512), "n"(CG) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::%0.sync.aligned;" ::"n"(CG) : "memory");
  }
  tc_fence_before();
  __syncthreads();
  if constexpr (CG == 2) cluster_sync();          // the other CTA's barriers are there
  tc_fence_after();
  const uint32_t tmem = *tmem_slot, tmem_a = tmem + 256;
  auto wait_warp = [&](int b, unsigned parity) {
    if (__all_sync(0xFFFFFFFFu, mbar_wait_tight(&bar[b], parity)) != 0) return true;
    *fail = 1;
    return false;
  };
  // arrives at a barrier of the CTA that issues the MMAs; `first` is that barrier's address there
  auto arrive_first = [&](uint64_t* b, uint32_t first) {
    if constexpr (CG == 1) mbar_arrive_one(b);
    else mbar_arrive_cluster(first);
  };
  // units of this CTA (pair): f(first weight row of this CTA, first token row, token rows, token tile) -> false ends the walk
  auto for_units = [&](auto f) {
    for (int u = blockIdx.x / CG; u < a.units; u += a.workers / CG) {
      const int t = u / a.row_units, tok0 = t * a.bn;
      if (!f(((u - t * a.row_units) * CG + static_cast<int>(rank)) * 128, tok0, min(a.bn, a.n_tokens - tok0), t)) return;
    }
  };

  if (warp < kQ4Unpack) {
    const int grp = warp >> 2, r = (warp & 3) * 32 + lane;
    const uint32_t lanes = static_cast<uint32_t>((warp & 3) * 32) << 16, a_full = cluster_addr(&bar[kQ4AFull], 0);
    pdl_wait();                                   // scratch may still be read by the kernel before
    pdl_launch_dependents();
    const int share = a.tiles;                    // the units of token tile t write blocks t, t + share, ... to scratch
    int job0 = 0;                                 // blocks of the units before this one
    for_units([&](int row0, int, int, int tile) {
      uint16_t* row_out = a.scratch + static_cast<size_t>(min(row0 + r, a.n_rows - 1)) * a.k;
      for (int b = (grp ^ job0) & 1; b < nb; b += 2) {
        const int job = job0 + b, st = job % kQ4WStages;
        if (!wait_warp(kQ4WFull + st, (job / kQ4WStages) & 1)) return false;
        const uint4* blk = reinterpret_cast<const uint4*>(w_sm + st * kQ4WBytes + r * kW4);
        const uint4 hdr = blk[0];
        const float d = h2f(static_cast<uint16_t>(hdr.x & 0xFFFFu)), dmin = h2f(static_cast<uint16_t>(hdr.x >> 16));
        const Scales6 s6 = unpack_scales6(hdr.y, hdr.z, hdr.w);
        const bool keep = a.tiles_write && b % share == tile && row0 + r < a.n_rows;
#pragma unroll 1
        for (int g = 0; g < 4; ++g) {
          const int x = 2 * job + (g >> 1), slot = x % kQ4Slots;
          const uint4 q0 = blk[1 + 2 * g], q1 = blk[2 + 2 * g];
          const uint32_t raw[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
          const uint32_t scw = (g < 2 ? s6.sc[0] : s6.sc[1]) >> (16 * (g & 1)), mnw = (g < 2 ? s6.mn[0] : s6.mn[1]) >> (16 * (g & 1));
          uint32_t v[32];
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            // sub-block 2 g + h: value = fp16(fma(d * sc, q, -(dmin * mn))); the odd one's nibbles come sixteen-fold, its scale as a sixteenth (exact)
            const f32x2 sd = splat2((h ? 0.0625f : 1.f) * (d * static_cast<float>((scw >> (8 * h)) & 0xFFu)));
            const f32x2 sm = splat2(-(dmin * static_cast<float>((mnw >> (8 * h)) & 0xFFu)));
#pragma unroll
            for (int i = 0; i < 8; ++i) dequant_word(raw[i], h ? 0xF0F0F0F0u : 0x0F0F0F0Fu, sd, sm, v[16 * h + 2 * i], v[16 * h + 2 * i + 1]);
          }
          if ((g & 1) == 0) {
            if (!wait_warp(kQ4AEmpty + slot, ((x / kQ4Slots) & 1) ^ 1u)) return false;
            tc_fence_after();
          }
          tmem_st32(tmem_a + lanes + slot * 64 + (g & 1) * 32, v);
          if (keep) {
            uint4* o = reinterpret_cast<uint4*>(row_out + b * kQK + g * 64);
#pragma unroll
            for (int i = 0; i < 8; ++i) o[i] = make_uint4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
          }
          if (g & 1) {
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            tc_fence_before();
            __syncwarp();
            if (lane == 0) arrive_first(&bar[kQ4AFull + slot], a_full + 8 * slot);
          }
        }
        if (lane == 0) mbar_arrive_one(&bar[kQ4WEmpty + st]);
      }
      job0 += nb;
      return true;
    });
  } else if (warp < kQ4Unpack + kQ4Epi) {
    // this thread's weight row, half of the token columns; lane pairs trade halves so that a store is two rows of one token
    const int quarter = warp & 3, half = ((warp - kQ4Unpack) >> 2) * (a.bn >> 1);
    const uint32_t src = tmem + (static_cast<uint32_t>(quarter * 32) << 16) + half, acc_empty = cluster_addr(&bar[kQ4AccEmpty], 0);
    const bool pairs = (a.n_rows & 1) == 0 && (reinterpret_cast<uintptr_t>(a.y) & 3u) == 0;
    const int odd = lane & 1;
    const uint32_t sel = odd ? 0x3276u : 0x5410u;
    unsigned ph = 0;
    pdl_wait();                                   // y may still be read by the kernel before
    for_units([&](int row0, int tok0, int ntok, int) {
      if (!wait_warp(kQ4AccFull, ph)) return false;
      ph ^= 1u;
      tc_fence_after();
      const int cols = min(a.bn >> 1, ntok - half), row = row0 + quarter * 32 + lane, last = row < a.n_rows ? cols : 0;
      uint16_t* y = a.y + static_cast<size_t>(tok0 + half) * a.n_rows + row;
      if (pairs) y += odd ? a.n_rows - 1 : 0;
#pragma unroll 2
      for (int c = 0; c < cols; c += 16) {
        uint32_t v[16];
        tc_ld16(src + c, v);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const uint32_t h = h2_bits(__floats2half2_rn(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1])));      // tokens t, t + 1
          const int t = c + 2 * i;
          if (pairs) {
            const uint32_t w = __byte_perm(h, __shfl_xor_sync(0xFFFFFFFFu, h, 1), sel);
            if (t + odd < last) *reinterpret_cast<uint32_t*>(y) = w;
          } else {
            if (t < last) y[0] = static_cast<uint16_t>(h & 0xFFFFu);
            if (t + 1 < last) y[a.n_rows] = static_cast<uint16_t>(h >> 16);
          }
          y += 2 * static_cast<size_t>(a.n_rows);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) arrive_first(&bar[kQ4AccEmpty], acc_empty);
      return true;
    });
  } else if (warp == kQ4WarpX) {
    const uint32_t b_full = cluster_addr(&bar[kQ4BFull], 0);
    int s = 0;
    unsigned ph = 1;
    pdl_wait();
    if (lane == 0) {
      for_units([&](int, int tok0, int ntok, int) {
        const int from = tok0 + static_cast<int>(rank) * (mma_columns<CG>(ntok) >> 1);
        for (int kb = 0; kb < 4 * nb; ++kb) {
          if (!mbar_wait_tight(&bar[kQ4BEmpty + s], ph)) {
            *fail = 1;
            return false;
          }
          // (of a pair: the first CTA's barrier counts both halves; its phase cannot be over before its own expect)
          if (rank == 0) mbar_expect_tx(&bar[kQ4BFull + s], CG * b_bytes);
          if constexpr (CG == 1) tc_tma_2d(b_sm + s * b_bytes, &map_x, kb * kBK, tok0, &bar[kQ4BFull + s]);
          else tc_tma_2d_pair(b_sm + s * b_bytes, &map_x, kb * kBK, from, b_full + 8 * s);
          if (++s == a.stages) { s = 0; ph ^= 1u; }
        }
        return true;
      });
    }
  } else if (warp == kQ4WarpW) {
    // (the weights do not depend on the kernel before) Rows past the matrix arrive as zeros and are never stored.
    int st = 0;
    unsigned ph = 1;
    if (lane == 0) {
      for_units([&](int row0, int, int, int) {
        for (int b = 0; b < nb; ++b) {
          if (!mbar_wait_tight(&bar[kQ4WEmpty + st], ph)) {
            *fail = 1;
            return false;
          }
          mbar_expect_tx(&bar[kQ4WFull + st], kQ4WBytes);
          tc_tma_2d(smem_u32(w_sm + st * kQ4WBytes), &map_w, b * kW4, row0, &bar[kQ4WFull + st]);
          if (++st == kQ4WStages) { st = 0; ph ^= 1u; }
        }
        return true;
      });
    }
  } else {
    if (rank == 0) {
      const uint32_t lead = elect_one();
      int slot = 0, s = 0;
      unsigned slot_ph = 0, s_ph = 0, acc_ph = 1;
      for_units([&](int, int, int ntok, int) {
        const uint32_t idesc = __shfl_sync(0xFFFFFFFFu, umma_idesc_f16(mma_columns<CG>(ntok), 128 * CG), 0);
        if (!wait_warp(kQ4AccEmpty, acc_ph)) return false;
        acc_ph ^= 1u;
        for (int x = 0; x < 2 * nb; ++x) {        // half-blocks
          if (!wait_warp(kQ4AFull + slot, slot_ph)) return false;
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            if (!wait_warp(kQ4BFull + s, s_ph)) return false;
            tc_fence_after();
            const uint32_t db = umma_desc_swizzled(b_sm + s * b_bytes), ta = tmem_a + slot * 64 + j * 32;
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) umma_ts<CG>(lead, tmem, ta + kk * 8, db + kk * 2, kDescSwizzled, idesc, (x | j | kk) != 0);
            if (lead) umma_commit<CG>(&bar[kQ4BEmpty + s]);
            if (++s == a.stages) { s = 0; s_ph ^= 1u; }
          }
          if (lead) umma_commit<CG>(&bar[kQ4AEmpty + slot]);
          if (++slot == kQ4Slots) { slot = 0; slot_ph ^= 1u; }
        }
        if (lead) umma_commit<CG>(&bar[kQ4AccFull]);
        return true;
      });
      if (lead) umma_commit<CG>(&bar[kQ4Drain]);  // everything issued has finished before tensor memory goes back
    }
    mbar_wait_tight(&bar[kQ4Drain], 0);
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if constexpr (CG == 2) cluster_sync();          // neither CTA goes while the other may still arrive at its barriers
  if (warp == kQ4WarpMma) {
    __syncwarp();
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::%2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512), "n"(CG) : "memory");
  }
  if (threadIdx.x == 0 && *fail != 0 && a.status != nullptr) atomicExch(a.status, 1);
}

__global__ void __launch_bounds__(256) dequant_rows_kernel(const unsigned char* __restrict__ w,
                                                           uint4* __restrict__ out, long long n_blocks) {
  const int lane = threadIdx.x & 31;
  const long long warps = static_cast<long long>(gridDim.x) * (blockDim.x >> 5);
  for (long long b = static_cast<long long>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5); b < n_blocks;
       b += warps)
    out[b * 32 + lane] = dequant_octet(w + b * kW4, lane);
}

// The routed experts of one layer into a ring of fp16 slots
// (src/kernels/cuda/tc_gemm.cu:124-152 of the reference): slot e % ring holds
// rows_per rows of k halfs starting at element dst_row0; with two tables the first
// half of the rows comes from tab_a[e], the second from tab_b[e]. Experts without
// routed rows (off[e+1] <= off[e]) and null table entries are skipped.
__global__ void __launch_bounds__(256) dequant_experts_kernel(const unsigned char* const* __restrict__ tab_a,
                                                              const unsigned char* const* __restrict__ tab_b,
                                                              const int* __restrict__ off, uint16_t* slots,
                                                              long long dst_row0, int rows_per, int nb, int ring,
                                                              long long slot_elems) {
  const int e = blockIdx.y;
  if (off[e + 1] <= off[e]) return;
  const int lane = threadIdx.x & 31;
  const int half_rows = rows_per >> 1;
  const long long blocks = static_cast<long long>(rows_per) * nb;
  const long long warps = static_cast<long long>(gridDim.x) * (blockDim.x >> 5);
  uint16_t* dst = slots + static_cast<long long>(e & (ring - 1)) * slot_elems + dst_row0;
  for (long long b = static_cast<long long>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5); b < blocks;
       b += warps) {
    int r = static_cast<int>(b / nb);
    const int blk = static_cast<int>(b - static_cast<long long>(r) * nb);
    const unsigned char* src = tab_a[e];
    if (tab_b != nullptr && r >= half_rows) {
      src = tab_b[e];
      r -= half_rows;
    }
    if (src == nullptr) continue;
    reinterpret_cast<uint4*>(dst)[b * 32 + lane] =
        dequant_octet(src + (static_cast<long long>(r) * nb + blk) * kW4, lane);
  }
}

__global__ void __launch_bounds__(256) cast_f32_f16_kernel(const float4* __restrict__ src, uint2* __restrict__ dst,
                                                           long long n4) {
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < n4;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const float4 v = __ldg(src + i);
    dst[i] = make_uint2(f2h(v.x) | (static_cast<uint32_t>(f2h(v.y)) << 16),
                        f2h(v.z) | (static_cast<uint32_t>(f2h(v.w)) << 16));
  }
}

// ---- host side ---------------------------------------------------------------------------
typedef CUresult (*EncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                             const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                             CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeFn tc_encoder() {
  static std::atomic<EncodeFn> cached{nullptr};
  EncodeFn f = cached.load(std::memory_order_acquire);
  if (f != nullptr) return f;
  void* fn = nullptr;
  cudaDriverEntryPointQueryResult qres;
  if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres) != cudaSuccess ||
      fn == nullptr || qres != cudaDriverEntryPointSuccess)
    return nullptr;
  f = reinterpret_cast<EncodeFn>(fn);
  cached.store(f, std::memory_order_release);
  return f;
}

std::atomic<int> g_tc_layout{kLayoutSwizzled};

// A [rows][k] fp16 matrix as operand tiles of 128 rows x 64 halfs.
bool operand_map(CUtensorMap* tm, const void* base, int rows, int k, int layout, int tile_rows) {
  EncodeFn enc = tc_encoder();
  if (enc == nullptr) return false;
  if (layout == kLayoutSwizzled) {
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(k), static_cast<cuuint64_t>(rows)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(k) * 2};
    const cuuint32_t box[2] = {kBK, static_cast<cuuint32_t>(tile_rows)};
    const cuuint32_t estr[2] = {1u, 1u};
    return enc(tm, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
  }
  // (8 halfs, rows, k / 8): the box lands as [k-chunk][row][16 bytes]
  const cuuint64_t dims[3] = {8, static_cast<cuuint64_t>(rows), static_cast<cuuint64_t>(k / 8)};
  const cuuint64_t strides[2] = {static_cast<cuuint64_t>(k) * 2, 16};
  const cuuint32_t box[3] = {8, static_cast<cuuint32_t>(tile_rows), kBK / 8};
  const cuuint32_t estr[3] = {1u, 1u, 1u};
  return enc(tm, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// A [rows][k] Q4_K matrix as tiles of one block column of 128 rows.
bool weight_map(CUtensorMap* tm, const void* base, int rows, int k) {
  EncodeFn enc = tc_encoder();
  if (enc == nullptr) return false;
  const cuuint64_t dims[2] = {static_cast<cuuint64_t>(k / kQK) * kW4, static_cast<cuuint64_t>(rows)};
  const cuuint64_t strides[1] = {static_cast<cuuint64_t>(k / kQK) * kW4};
  const cuuint32_t box[2] = {kW4, 128};
  const cuuint32_t estr[2] = {1u, 1u};
  return enc(tm, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <bool F32OUT>
int launch_tc_gemm(const void* w16, const void* x16, void* y, int n_rows, int k, int n_tokens, cudaStream_t s) {
  if (n_rows <= 0 || n_tokens <= 0) return kOk;
  if (!w16 || !x16 || !y || k <= 0) return kErrArg;
  if (k % kBK != 0) return kErrUnsupported;
  if ((reinterpret_cast<uintptr_t>(w16) | reinterpret_cast<uintptr_t>(x16)) & 15u) return kErrAlign;
  if (reinterpret_cast<uintptr_t>(y) & (F32OUT ? 3u : 1u)) return kErrAlign;
  const int layout = g_tc_layout.load(std::memory_order_relaxed);
  // 128 x 128 tiles when they fill the machine, else 128 x 64 for twice the CTAs
  const int row_tiles = (n_rows + kBM - 1) / kBM;
  const int bn = row_tiles * ((n_tokens + kBN - 1) / kBN) >= 148 ? kBN : 64;
  CUtensorMap mw, mx;
  if (!operand_map(&mw, w16, n_rows, k, layout, kBM) || !operand_map(&mx, x16, n_tokens, k, layout, bn))
    return kErrUnsupported;
  auto kern = tc_gemm_kernel<F32OUT>;
  // the opt-in to more than 48 KB of dynamic shared memory is a per-device attribute
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kTcSmem) != cudaSuccess)
    return kErrLaunch;
  TcArgs a{y, n_rows, k, n_tokens, layout, bn, status_word()};
  kern<<<dim3(row_tiles, (n_tokens + bn - 1) / bn), kTcThreads, kTcSmem, s>>>(mw, mx, a);
  return cudaPeekAtLastError() == cudaSuccess ? kOk : kErrLaunch;
}

int grid_for(long long warps_needed, int warps_per_cta) {
  const long long ctas = (warps_needed + warps_per_cta - 1) / warps_per_cta;
  return static_cast<int>(ctas < 1 ? 1 : (ctas > 148 * 16 ? 148 * 16 : ctas));
}

int launch_dequant(const void* w, void* out16, long long n_blocks, cudaStream_t s) {
  if (n_blocks <= 0) return kOk;
  dequant_rows_kernel<<<grid_for(n_blocks, 8), 256, 0, s>>>(static_cast<const unsigned char*>(w),
                                                           static_cast<uint4*>(out16), n_blocks);
  return cudaPeekAtLastError() == cudaSuccess ? kOk : kErrLaunch;
}

struct Q4Plan {
  int cg, bn, tiles, units, workers, spare;      // CTAs to a unit, its token rows, token tiles, units, CTAs that work on them, CTAs per row tile for the scratch
  bool ahead;                                    // the scratch is written by the dequantisation kernel
  double us;
};
// Token rows per unit, CTAs that share a unit, and who writes the scratch: what takes the least by estimates in us, fitted to
// 47 shapes of 512 to 8192 rows, 512 to 4096 columns and 64 to 2048 tokens. us of a pair's units / of a single CTA's, each at their best, inputs
// from HBM: 4096 x 2048 over 2048 tokens 38.5 / 39.5, 4096 x 4096 70.5 / 73.5, 4096 x 4096 over 1000 40.5 / 42.3, 2048 x 2048 20.1 / 20.2, 4096 x 1024 22.5 / 22.5.
// (Back to back, all of them in L2, rows of up to eight blocks are 3 to 5 % faster by single CTAs.)
//   the start, 4, and the last unit's epilogue, 1.5 for 256 tokens
//   a block column of a unit: 1.0 and, with the square of its tokens, up to 0.35 more, a fifth more when every SM works; a pair
//     brings half of the activations per CTA and gains 6 % past 128 tokens, but costs 0.3 to set up
//   the scratch, per block of a row tile: SMs that the units leave idle, in whole columns of row tiles, 3.2 / spare beside
//     the units' 1.3 and epilogue; the units of a row tile themselves, 2 for each block that one
//     of its token tiles writes on top of it; or the dequantisation kernel ahead of the
//     GEMM, 2.5 us and the bytes at 5 TB/s (8192 x 4096 over 64 tokens: 53 us by one spare column, 41 by the kernel ahead).
Q4Plan q4_plan(int sms, int n_rows, int k, int n_tokens) {
  const int row_tiles = (n_rows + 127) / 128, nb = k / kQK;
  Q4Plan p{};
  for (int cg = 1; cg <= (row_tiles > 1 ? 2 : 1); ++cg) {
    for (int most = 256, last = 0; most >= 32; most -= 16) {
      const int t = (n_tokens - 1) / most + 1, each = (n_tokens - 1) / t + 1;            // tiles of nearly equal length
      const int bn = cg == 1 ? mma_columns<1>(each) : mma_columns<2>(each);
      if (bn == last) continue;
      last = bn;
      Q4Plan c{cg, bn, (n_tokens + bn - 1) / bn, 0, 0, 0, false, 0.};
      const long long units = static_cast<long long>((row_tiles + cg - 1) / cg) * c.tiles;
      if (units > 0x3FFFFFFF) continue;
      c.units = static_cast<int>(units);
      c.workers = std::min(c.units, sms / cg) * cg;
      const int waves = (c.units * cg + c.workers - 1) / c.workers;
      const double wide = bn / 256.;
      c.us = 4 + 1.5 * wide + 0.3 * (cg - 1) + waves * nb * (1 + 0.35 * wide * wide) * (1 + 0.2 * c.workers / sms) * (cg == 1 && bn > 128 ? 1.06 : 1.);
      const int spare = std::min(nb, (sms - c.workers) / row_tiles);
      const double by_spare = spare > 0 ? std::max(0., nb * (3.2 / spare - 1.3) - 1.5 * wide) : 1e30, by_tiles = 2. * ((nb + c.tiles - 1) / c.tiles);
      const double by_kernel = 2.5 + static_cast<double>(n_rows) * k * 2.5625 / 5e6;
      c.spare = by_spare < by_tiles ? spare : 0;
      if (by_kernel < std::min(by_spare, by_tiles)) {
        c.spare = 0;
        c.ahead = true;
      }
      c.us += std::min(by_kernel, std::min(by_spare, by_tiles));
      if (p.cg == 0 || c.us < p.us) p = c;
    }
  }
  return p;
}

int launch_tc_q4(const void* w, const uint16_t* x, uint16_t* y, uint16_t* scratch, int n_rows, int k, int n_tokens, cudaStream_t s) {
  if ((reinterpret_cast<uintptr_t>(x) & 15u) || (reinterpret_cast<uintptr_t>(y) & 1u)) return kErrAlign;
  const int sms = device_sms(), row_tiles = (n_rows + 127) / 128, nb = k / kQK;
  if (sms <= 0) return kErrLaunch;
  const Q4Plan p = q4_plan(sms, n_rows, k, n_tokens);
  if (p.cg == 0) return kErrUnsupported;
  CUtensorMap mx, mw;
  if (!weight_map(&mw, w, n_rows, k) || !operand_map(&mx, x, n_tokens, k, kLayoutSwizzled, p.bn / p.cg)) return kErrUnsupported;
  Q4Args a{};
  a.scratch = scratch; a.y = y;
  a.n_rows = n_rows; a.k = k; a.n_tokens = n_tokens; a.w = static_cast<const unsigned char*>(w);
  a.bn = p.bn;
  a.stages = std::min(8, kQ4BBytes * p.cg / (p.bn * 128));
  a.tiles = p.tiles;
  a.row_units = (row_tiles + p.cg - 1) / p.cg;
  a.units = p.units;
  a.workers = p.workers;
  a.tiles_write = p.spare == 0 && !p.ahead;
  a.status = status_word();
  if (p.ahead) {
    const int rc = launch_dequant(w, scratch, static_cast<long long>(n_rows) * nb, s);
    if (rc != kOk) return rc;
  }
  const dim3 grid(p.workers + (p.spare * row_tiles + p.cg - 1) / p.cg * p.cg);
  if (p.cg == 1) {
    if (!opt_in_smem<tc_gemm_q4_kernel<1>>(kQ4Smem)) return kErrLaunch;
    return launch_pdl(tc_gemm_q4_kernel<1>, grid, kQ4Threads, kQ4Smem, s, mx, mw, a);
  }
  if (!opt_in_smem<tc_gemm_q4_kernel<2>>(kQ4Smem)) return kErrLaunch;
  return launch_pdl<2>(tc_gemm_q4_kernel<2>, grid, kQ4Threads, kQ4Smem, s, mx, mw, a);
}

}  // namespace
}  // namespace sgr

using namespace sgr;

SGR_API void* sgr_tc_handle(void) { return reinterpret_cast<void*>(tc_encoder()); }

SGR_API size_t sgr_tc_scratch_elems(int max_rows, int max_k) {
  return static_cast<size_t>(max_rows > 0 ? max_rows : 1) * static_cast<size_t>(max_k > 0 ? max_k : 1);
}

SGR_API int sgr_tc_set_operand_layout(int layout) {
  if (layout != kLayoutSwizzled && layout != kLayoutCore) return kErrArg;
  g_tc_layout.store(layout, std::memory_order_relaxed);
  return kOk;
}

SGR_API int sgr_tc_gemm_f16_raw(const void* w16, const void* x16, void* y16, int n_rows, int k, int n_tokens,
                                void* stream) {
  return launch_tc_gemm<false>(w16, x16, y16, n_rows, k, n_tokens, as_stream(stream));
}

SGR_API int sgr_tc_gemm_f16_f32out_raw(const void* w16, const void* x16, float* y32, int n_rows, int k,
                                       int n_tokens, void* stream) {
  return launch_tc_gemm<true>(w16, x16, y32, n_rows, k, n_tokens, as_stream(stream));
}

SGR_API int sgr_dequant_q4_k_f16(const void* w, uint16_t* out16, int n_rows, int k, void* stream) {
  if (n_rows <= 0) return kOk;
  if (!w || !out16 || k <= 0 || k % kQK != 0) return kErrArg;
  if ((reinterpret_cast<uintptr_t>(w) & 3u) || (reinterpret_cast<uintptr_t>(out16) & 15u)) return kErrAlign;
  return launch_dequant(w, out16, static_cast<long long>(n_rows) * (k / kQK), as_stream(stream));
}

SGR_API int sgr_tc_gemm_q4_k_f16(const void* w, const uint16_t* x, uint16_t* y, uint16_t* scratch, int n_rows,
                                 int k, int n_tokens, void* stream) {
  if (n_rows <= 0 || n_tokens <= 0) return kOk;
  if (!w || !x || !y || !scratch) return kErrArg;
  // the reference's own refusals (callers then take the GEMV path): k a power of two
  // >= 256, weights 16-byte aligned
  if (k < kQK || (k & (k - 1)) != 0) return kErrUnsupported;
  if (reinterpret_cast<uintptr_t>(w) & 15u) return kErrAlign;
  if (reinterpret_cast<uintptr_t>(scratch) & 15u) return kErrAlign;
  return launch_tc_q4(w, x, y, scratch, n_rows, k, n_tokens, as_stream(stream));
}

SGR_API int sgr_tc_gemm_q4_k_plan(int* plan, int sms, int n_rows, int k, int n_tokens) {
  if (!plan || sms <= 0 || n_rows <= 0 || n_tokens <= 0 || k < kQK || k % kQK != 0) return kErrArg;
  const Q4Plan p = q4_plan(sms, n_rows, k, n_tokens);
  if (p.cg == 0) return kErrUnsupported;
  const int v[7] = {p.cg, p.bn, p.tiles, p.units, p.workers, p.spare, p.ahead};
  std::memcpy(plan, v, sizeof(v));
  return kOk;
}

SGR_API int sgr_dequant_experts_q4_k_f16(const void* const* tab_a, const void* const* tab_b, const int* off,
                                         void* slots, long long dst_row0, int rows_sl2, int k, int n_experts,
                                         int ring, long long slot_elems, void* stream) {
  if (n_experts <= 0) return kOk;
  if (!tab_a || !off || !slots || k <= 0 || k % kQK != 0 || rows_sl2 < 1 || rows_sl2 > 24 || ring <= 0 ||
      (ring & (ring - 1)) != 0)
    return kErrArg;
  if ((reinterpret_cast<uintptr_t>(slots) & 15u) || (dst_row0 & 7) || (slot_elems & 7)) return kErrAlign;
  const int rows_per = 1 << rows_sl2;
  const int nb = k / kQK;
  const long long blocks = static_cast<long long>(rows_per) * nb;
  int gx = grid_for(blocks, 8);
  if (gx > 64) gx = 64;                                     // x n_experts CTAs; grid-stride inside
  dequant_experts_kernel<<<dim3(gx, n_experts), 256, 0, as_stream(stream)>>>(
      reinterpret_cast<const unsigned char* const*>(tab_a), reinterpret_cast<const unsigned char* const*>(tab_b),
      off, static_cast<uint16_t*>(slots), dst_row0, rows_per, nb, ring, slot_elems);
  return cudaPeekAtLastError() == cudaSuccess ? kOk : kErrLaunch;
}

SGR_API int sgr_tc_router_f32(const float* w_f32, const uint16_t* x, float* y, uint16_t* scratch, int n_rows,
                              int k, int n_tokens, void* stream) {
  if (n_rows <= 0 || n_tokens <= 0) return kOk;
  if (!w_f32 || !x || !y || !scratch || k <= 0) return kErrArg;
  if (k % kBK != 0) return kErrUnsupported;
  if ((reinterpret_cast<uintptr_t>(w_f32) & 15u) || (reinterpret_cast<uintptr_t>(scratch) & 15u)) return kErrAlign;
  const long long n4 = static_cast<long long>(n_rows) * k / 4;
  cast_f32_f16_kernel<<<grid_for((n4 + 31) / 32, 8), 256, 0, as_stream(stream)>>>(
      reinterpret_cast<const float4*>(w_f32), reinterpret_cast<uint2*>(scratch), n4);
  if (cudaPeekAtLastError() != cudaSuccess) return kErrLaunch;
  return launch_tc_gemm<true>(scratch, x, y, n_rows, k, n_tokens, as_stream(stream));
}
