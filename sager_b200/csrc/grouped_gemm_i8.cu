// grouped_gemm_i8.cu - the prefill MoE grouped GEMM on the 5th-generation tensor cores:
// tcgen05.mma with the weights as the tensor-memory operand and the accumulators in tensor memory.
//
// It replaces the reference's prefill expert math for chunks of many tokens
// (dequant_experts_q4_k_f16 + one cublasGemmEx per expert and matrix,
// src/kernels/cuda/tc_gemm.cu:124-152, 209-240, driven from
// src/core/session.cpp:2643-2760) but keeps the arithmetic of the reference's
// Q4_K x Q8_K path (gemv_grouped_tab_q4_k_q8_f16out_mtok, q4_k.cu:765-836): Q8_K
// activations, integer dots, fp32 scaling - so it is checked against that
// path, not against the fp16 one.
//
// The integers ride in fp16 operands (kind::f16, fp32 accumulators): sc * q <= 945 and an int8 code
// are exact in fp16, their products are exact, and a super-block's sum is an integer that fp32 holds
// exactly while the partial sums stay below 2^24 - sum |code| below 17,754 in a block is enough, N(0, 1) rows
// have about 8,700. A block that goes on to 3 x 10^7 (codes and nibbles all near their largest) loses up to two
// units in each of the at most eight steps past 2^24, where an int32 sum would be rounded once (measured: up to
// six units). One accumulator takes the 256 products of a block; a second one takes the min term in a single
// K = 16 step, mn x (bsum & 63) + (64 mn) x (bsum >> 6). Per output and block the epilogue then reads two fp32
// values and spends three operations, where the int8 form of the same idea (6-bit scales split over
// two u8 operand tiles, four int32 accumulators) spends about twenty, four of them conversions.
//
// The 128 weight rows of a tile are the M lanes of tensor memory, so a thread that owns a row
// unpacks its block in registers and stores it with tcgen05.st: weights never cross shared memory
// as operands (two bytes per weight written and read again there was the int8 form's limit).
//
// Persistent: one CTA per SM takes work units round-robin. A unit is one expert, one or several
// tiles of 128 weight rows, and at most 80 of the expert's token rows; a job is one super-block
// column of a tile. The roles run as a pipeline over mbarriers:
//   * a producer warp brings the [128 rows][144 B] block columns into a ring, one TMA copy each through the expert's
//     descriptor (made by the quantiser's launch); the plain entry, which has no memory for descriptors, uses two warps and
//     cp.async. Plain loads where an expert's base is only 2-byte aligned;
//   * eight unpack warps (thread = weight row; four warps take the even jobs, four the odd ones):
//     nibbles -> sc * q as packed fp16 with one logic and one FMA instruction per two weights, in
//     three half-block slots of tensor memory; the min operand and (d, dmin) go to shared memory;
//   * the activation tiles of one block, two in flight: two warps copy them (cp.async) from rows
//     that already are operands (kOpBlk bytes per block, written by quantize_operand: a prefill
//     chunk), or eight warps make them from Q8_K rows (the plain entry, which has no scratch; they
//     cost more instructions than everything else together). Rows of at most two blocks keep their
//     tiles for all weight tiles of the unit;
//   * one warp issues the 17 MMAs of a job (M = 128, N = tokens rounded up to 16, K = 16);
//   * eight epilogue warps fold xd * (d * D0 - dmin * D1) into fp32 registers, each warp 32 rows of
//     every second tile (gate / up alternate), while the next job's MMAs run into the other of two
//     accumulator sets.
// The gate and up projections run as one pass: their jobs alternate over the same activation tiles.
// What runs per job is kept compact: with the five roles on a scheduler a loop that is unrolled over a
// whole block waits for its instructions (a third of all stall cycles did).
// The shared expert is one more expert whose rows are all the chunk's rows.
//
// Operand tiles in shared memory use the canonical K-major layout without swizzle: 8 rows x 16
// bytes per core matrix, the two K halves 128 bytes apart, 8-row groups 256 bytes apart.
// Every wait is bounded; on expiry the CTA raises the status word, frees its tensor
// memory and returns.
#include <algorithm>

#include "api_util.cuh"
#include "quantize_dev.cuh"
#include "tmap_dev.cuh"
#include "umma.cuh"

namespace sgr {
namespace {

constexpr int kGemmRows = 128;                    // weight rows per tile = MMA M = tensor-memory lanes
constexpr int kGemmTok = 80;                      // token rows per unit = max MMA N
// (Four stages: a fifth to seventh hides nothing more, and what shared memory does not take is L1 cache - 2048 rows, two layers:
// 892 us with seven, 876 with four. With two producers on cp.async and one stager it was 913. The plain entry, 256 experts, 512 rows
// of 2048: 2 / 24 / 64 / 128 token rows per expert 68 / 83 / 123 / 235 us with seven, 66 / 77 / 109 / 205 with four.)
constexpr int kStages = 4, kStageBytes = kGemmRows * kW4;     // 18,432
constexpr int kBTile = kGemmTok * 32;             // one K = 16 step of the activations
constexpr int kBBytes = 17 * kBTile;              // 16 code steps + the split sums
constexpr int kMinBytes = kGemmRows * 32;         // the min operand of a job
constexpr int kTmemCols = 512;                    // two accumulator sets of 2 x 80 columns, three half-block slots of 64
constexpr int kColSet = 2 * kGemmTok, kColA = 2 * kColSet, kASlots = 3;
static_assert(kColA + 64 * kASlots <= kTmemCols, "tensor memory");

// warps: epilogue | MMA, and three that copy: two producers (RAW) or one producer and two stagers | unpack | converting stagers
constexpr int kEpiWarps = 8, kWarpMma = kEpiWarps, kWarpProd0 = kEpiWarps + 1, kCopyStagers = 2, kWarpUnpack0 = kEpiWarps + 4,
              kUnpackGroups = 2, kWarpStage0 = kWarpUnpack0 + 4 * kUnpackGroups, kStageWarps = 8;
// Threads and registers per thread of each role (setmaxnreg). The sum over the warpgroups is at most
// what the launch holds.
template <bool RAW>
struct Cfg {
  static constexpr int kThreads = (kWarpStage0 + (RAW ? kStageWarps : 0)) * 32;
  static constexpr int kRegsLaunch = RAW ? 72 : 96, kRegsEpi = RAW ? 112 : 136, kRegsUnpack = RAW ? 56 : 72, kRegsCtrl = RAW ? 56 : 64,
                       kRegsStage = 56;
  static_assert(256 * (kRegsEpi + kRegsUnpack + (RAW ? kRegsStage : 0)) + 128 * kRegsCtrl <= kThreads * kRegsLaunch, "registers");
};

// shared-memory map (bytes)
constexpr int kOffW = 1024;
constexpr int kOffB = kOffW + kStages * kStageBytes;
constexpr int kOffMin = kOffB + 2 * kBBytes;                      // [2][128 rows][16 halfs] min operand
constexpr int kOffDd = kOffMin + 2 * kMinBytes;                   // [4][128] float2 (d, dmin)
constexpr int kOffXd = kOffDd + 4 * kGemmRows * 8;                // [4][80] fp32 activation scales
constexpr int kGemmSmem = kOffXd + 4 * kGemmTok * 4;
static_assert(kGemmSmem <= 227 * 1024, "shared memory");

enum { kBarWFull = 0, kBarWEmpty = kBarWFull + kStages, kBarAFull = kBarWEmpty + kStages, kBarAEmpty = kBarAFull + kASlots,
       kBarBFull = kBarAEmpty + kASlots, kBarBEmpty = kBarBFull + 2, kBarAccFull = kBarBEmpty + 2,
       kBarAccEmpty = kBarAccFull + 4,   // full: per epilogue group and set
        kBarDrain = kBarAccEmpty + 2, kBarCount };

struct GemmArgs {
  const unsigned char* const* tab0;    // [n_expert] gate (or the only matrix)
  const unsigned char* const* tab1;    // [n_expert] up
  const int* off;                      // [n_expert + 1] grouped slots of each expert
  const int* rows;                     // activation row of a grouped slot; null: the slot itself
  const unsigned char* xq;             // Q8_K rows (RAW) or operand rows
  uint16_t *y, *y1;                    // [slots][n_rows] of tab0 / tab1
  int n_rows, nb, n_expert;
  int tiles, group, groups;            // row tiles per matrix, per unit, units per expert and pass
  const unsigned char *sw0, *sw1, *sxq;   // one more expert over s_rows rows of its own (null: none)
  uint16_t *sy, *sy1;
  int s_rows, s_step, s_items;         // its rows, rows per unit, units
  int n_items;
  const unsigned char* maps;           // (operand rows) [n_expert + 1][3] descriptors, or null; the matrix of tab0 is map0
  int map0;
  int* status;
};

// address of (row, 16-byte K half) inside a canonical tile
__device__ __forceinline__ int tile_at(int row, int khalf) { return (row >> 3) * 256 + khalf * 128 + (row & 7) * 16; }

// One work unit and the walk over a CTA's units; every role walks the same list on its own.
struct Unit {
  const unsigned char *w0, *w1;        // null: the expert is absent
  const unsigned char* xq;
  const int* rows;
  uint16_t *y, *y1;
  int tile0, n_tiles;                  // row tiles
  int expert;
  int slot0, nt, n_mma;                // first slot, token rows, MMA N
};
struct Walk {
  int it, m = 0, t0 = 0, step = 0, slot = 0;
  const unsigned char *w0 = nullptr, *w1 = nullptr;
  __device__ __forceinline__ explicit Walk(int first) : it(first) {}
  template <bool DUAL>
  __device__ __forceinline__ bool next(const GemmArgs& a, Unit& u) {
    for (; it < a.n_items; it += gridDim.x) {
      const bool shared = it < a.s_items;
      const int i = shared ? it : it - a.s_items;
      const int e = i / a.groups;                     // expert, or pass of the shared one
      u.tile0 = (i - e * a.groups) * a.group;
      u.n_tiles = min(a.group, a.tiles - u.tile0);
      if (shared) {
        u.w0 = a.sw0; u.w1 = a.sw1; u.xq = a.sxq; u.rows = nullptr; u.y = a.sy; u.y1 = a.sy1; u.expert = a.n_expert;
        u.slot0 = e * a.s_step;
        u.nt = min(a.s_step, a.s_rows - u.slot0);
        it += gridDim.x;
      } else {
        if (m == 0) {
          slot = __ldg(a.off + e);
          m = __ldg(a.off + e + 1) - slot;
          if (m <= 0) { m = 0; continue; }
          w0 = a.tab0[e];
          w1 = DUAL ? a.tab1[e] : w0;
          if (w1 == nullptr) w0 = nullptr;
          t0 = 0;
          const int passes = (m + kGemmTok - 1) / kGemmTok;
          step = ((m + passes - 1) / passes + 15) & ~15;
        }
        u.w0 = w0; u.w1 = w1; u.xq = a.xq; u.rows = a.rows; u.y = a.y; u.y1 = a.y1; u.expert = e;
        u.slot0 = slot + t0;
        u.nt = min(step, m - t0);
        t0 += step;
        if (t0 >= m) { m = 0; it += gridDim.x; }
      }
      u.n_mma = (u.nt + 15) & ~15;
      return true;
    }
    return false;
  }
};
// The jobs of a unit in order: f(tile, block, matrix, fill) -> false ends the walk. `fill` numbers the
// activation tiles staged for the unit: one per block when they are shared by gate and up or stay for
// all row tiles (at most two blocks), else one per (tile, block).
template <bool DUAL, typename F>
__device__ __forceinline__ bool for_jobs(const GemmArgs& a, const Unit& u, F f) {
  int fill = 0;
#pragma unroll 1
  for (int t = 0; t < u.n_tiles; ++t) {
    if (a.nb <= 2) fill = 0;
#pragma unroll 1
    for (int b = 0; b < a.nb; ++b, ++fill)
#pragma unroll 1
      for (int m = 0; m < (DUAL ? 2 : 1); ++m)
        if (!f(t, b, m, fill)) return false;
  }
  return true;
}
__device__ __forceinline__ int fills_of(const GemmArgs& a, const Unit& u) { return a.nb <= 2 ? a.nb : u.n_tiles * a.nb; }

// STREAM: weights first to leave L2 (streams_weights)
template <bool DUAL, bool RAW, bool STREAM>
__global__ void __launch_bounds__(Cfg<RAW>::kThreads, 1) grouped_gemm_kernel(const GemmArgs a) {
  extern __shared__ __align__(1024) unsigned char smem[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  uint64_t* bar = reinterpret_cast<uint64_t*>(smem);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + 512);
  volatile int* fail = reinterpret_cast<volatile int*>(smem + 516);
  static_assert(kBarCount * 8 <= 512, "barriers");

  if (tid == 0) {
    for (int i = 0; i < kStages; ++i) { mbar_init(&bar[kBarWFull + i], RAW ? 32 : 1); mbar_init(&bar[kBarWEmpty + i], 4); }
    for (int i = 0; i < kASlots; ++i) { mbar_init(&bar[kBarAFull + i], 4); mbar_init(&bar[kBarAEmpty + i], 1); }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bar[kBarBFull + i], RAW ? kStageWarps : 32 * kCopyStagers); mbar_init(&bar[kBarBEmpty + i], 1);
      mbar_init(&bar[kBarAccFull + i], 1); mbar_init(&bar[kBarAccFull + 2 + i], 1);
      mbar_init(&bar[kBarAccEmpty + i], kEpiWarps / 2);
    }
    mbar_init(&bar[kBarDrain], 1);
    *fail = 0;
    fence_barrier_init();
  }
  if (warp == kWarpMma) {
    __syncwarp();
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  // a wait that gives up flags the CTA and ends its role; the others' waits then run out as well
  auto wait_warp = [&](int b, unsigned parity) {
    if (__all_sync(0xFFFFFFFFu, mbar_wait_tight(&bar[b], parity)) != 0) return true;
    *fail = 1;
    return false;
  };
  const int row_bytes = a.nb * kW4;
  pdl_wait();                                        // plan and activations come from the kernels before this one
  pdl_launch_dependents();
  Walk wk(blockIdx.x);
  Unit u;

  if (warp < kEpiWarps) {
    // ---------------- epilogue: this thread's weight row of every second tile ----------------
    // (of the gate or of the up matrix when both run)
    regs_inc<Cfg<RAW>::kRegsEpi>();
    const unsigned grp = warp >> 2;
    const int row = (warp & 3) * 32 + lane;                   // accumulator lane = weight row in the tile
    const uint32_t lane_base = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16);
    const float2* dd_sm = reinterpret_cast<const float2*>(smem + kOffDd) + row;
    const float* xd_sm = reinterpret_cast<const float*>(smem + kOffXd);
    f32x2 acc[kGemmTok / 2];                                  // two token columns each
#pragma unroll
    for (int c = 0; c < kGemmTok / 2; ++c) acc[c] = 0ull;
    unsigned job = 0, fill0 = 0, tile_no = 0, seen = 0;        // seen: phase of each set's barrier
    while (wk.next<DUAL>(a, u)) {
      if (u.w0 == nullptr) {                                   // absent expert: zero rows
        uint16_t* y = DUAL && grp ? u.y1 : u.y;
        for (int t = 0; t < u.n_tiles; ++t) {
          const int r = (u.tile0 + t) * kGemmRows + row;
          if (r < a.n_rows)
            for (int c = DUAL ? 0 : grp; c < u.nt; c += DUAL ? 1 : 2) y[static_cast<size_t>(u.slot0 + c) * a.n_rows + r] = 0;
        }
        continue;
      }
      const bool ok = for_jobs<DUAL>(a, u, [&](int t, int b, int m, int fill) {
        const unsigned j = job++;
        const int set = j & 1;
        if ((DUAL ? m : (tile_no + t) & 1) != grp) return true;
        if (!wait_warp(kBarAccFull + 2 * grp + set, (seen >> set) & 1)) return false;
        seen ^= 1u << set;
        tc_fence_after();
        const float2 dd = dd_sm[(j & 3) * kGemmRows];
        const f32x2 d2 = splat2(dd.x), nm2 = splat2(-dd.y);
        const ulonglong2* xd = reinterpret_cast<const ulonglong2*>(xd_sm + ((fill0 + fill) & 3) * kGemmTok);
        const uint32_t d0 = lane_base + set * kColSet;
#pragma unroll
        for (int c = 0; c < kGemmTok; c += 8) {
          if (c >= u.n_mma) break;
          uint32_t v0[8], v1[8];
          tmem_ld8(d0 + c, v0);
          tmem_ld8(d0 + kGemmTok + c, v1);
          const ulonglong2 xa = xd[c / 4], xb = xd[c / 4 + 1];
          const f32x2 xv[4] = {xa.x, xa.y, xb.x, xb.y};
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int q = 0; q < 4; ++q)           // acc += xd * (d * D0 - dmin * D1)
            acc[c / 2 + q] = fma2(xv[q], fma2(nm2, pack2(v1[2 * q], v1[2 * q + 1]), mul2(d2, pack2(v0[2 * q], v0[2 * q + 1]))), acc[c / 2 + q]);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_one(&bar[kBarAccEmpty + set]);
        if (b + 1 == a.nb) {                                   // the tile is complete
          const int r = (u.tile0 + t) * kGemmRows + row;
          uint16_t* yp = (DUAL && grp ? u.y1 : u.y) + static_cast<size_t>(u.slot0) * a.n_rows + r;
          const int n_left = r < a.n_rows ? u.nt : 0;
#pragma unroll
          for (int c = 0; c < kGemmTok; c += 8) {
            if (c >= u.n_mma) break;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const uint32_t h = h2_bits(__floats2half2_rn(part2(acc[c / 2 + q], 0), part2(acc[c / 2 + q], 1)));
              if (c + 2 * q < n_left) yp[0] = static_cast<uint16_t>(h & 0xFFFFu);
              if (c + 2 * q + 1 < n_left) yp[a.n_rows] = static_cast<uint16_t>(h >> 16);
              yp += 2 * a.n_rows;
              acc[c / 2 + q] = 0ull;
            }
          }
        }
        return true;
      });
      if (!ok) break;
      fill0 += fills_of(a, u);
      tile_no += u.n_tiles;
    }
  } else if (warp >= kWarpUnpack0 && warp < kWarpStage0) {
    // ---------------- unpack: this thread's weight row of a block -> tensor memory ----------------
    // Group g of four warps takes jobs g, g + G, ... The halves of a job (sub-blocks 0-3 / 4-7) go round three
    // slots of tensor memory: half 2j + h into slot (2j + h) mod 3. (Two groups are as far ahead of the
    // tensor core as they can be: a third one's first wait could take a slot's phase for the one before it.)
    regs_dec<Cfg<RAW>::kRegsUnpack>();
    constexpr int G = kUnpackGroups;
    const int grp = (warp - kWarpUnpack0) >> 2;
    const int r = (warp & 3) * 32 + lane;
    const uint32_t a_base = tmem + kColA + (static_cast<uint32_t>((warp & 3) * 32) << 16);
    const __half2 k1024 = __float2half2_rn(1024.f), n1024 = __float2half2_rn(-1024.f), n64 = __float2half2_rn(-64.f);
    const __half2 k16th = __float2half2_rn(0.0625f);
    const uint32_t mlo = 0x000F000Fu, mhi = 0x00F000F0u, magic = 0x64006400u;
    int to_mine = grp;                                           // jobs until this group's next one
    unsigned job = grp;                                          // its number
    int st = grp % kStages, slot = 2 * grp % kASlots;            // its ring stage and first slot
    unsigned st_ph = 0, slot_ph = 1u ^ ((2 * grp / kASlots) & 1);
    bool ok = true;
    while (ok && wk.next<DUAL>(a, u)) {
      if (u.w0 == nullptr) continue;
      const int n_jobs = u.n_tiles * a.nb * (DUAL ? 2 : 1);
#pragma unroll 1
      for (; to_mine < n_jobs; to_mine += G) {
        if (!(ok = wait_warp(kBarWFull + st, st_ph))) break;
        const uint4* blk = reinterpret_cast<const uint4*>(smem + kOffW + st * kStageBytes + r * kW4);
        const uint4 hdr = blk[0];
        const Scales6 s6 = unpack_scales6(hdr.y, hdr.z, hdr.w);
        uint32_t scw = s6.sc[0];
#pragma unroll 1
        for (int g = 0; g < 4; ++g) {
          const uint4 q0 = blk[1], q1 = blk[2];
          blk += 2;
          const uint32_t raw[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
          // scales of the two sub-blocks of a 32-byte group, splat; nibbles enter as 1024 + q and 1024 + 16 q
          const __half2 se = __hsub2(bits_h2(__byte_perm(scw, 0x64646464u, 0x4040)), k1024);
          const __half2 so = __hsub2(bits_h2(__byte_perm(scw, 0x64646464u, 0x4141)), k1024);
          const __half2 ce = __hmul2(se, n1024), so16 = __hmul2(so, k16th), co = __hmul2(so, n64);
          scw = g == 1 ? s6.sc[1] : scw >> 16;
          if ((g & 1) == 0) {
            if (!(ok = wait_warp(kBarAEmpty + slot, slot_ph))) break;
            tc_fence_after();
          }
          const uint32_t dst = a_base + slot * 64 + (g & 1) * 32;
#pragma unroll
          for (int i = 0; i < 8; i += 4) {
            uint32_t v[8], w[8];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const uint32_t odd = raw[i + q] >> 8;
              v[2 * q] = h2_bits(__hfma2(bits_h2(and_or(raw[i + q], mlo, magic)), se, ce));
              v[2 * q + 1] = h2_bits(__hfma2(bits_h2(and_or(odd, mlo, magic)), se, ce));
              w[2 * q] = h2_bits(__hfma2(bits_h2(and_or(raw[i + q], mhi, magic)), so16, co));
              w[2 * q + 1] = h2_bits(__hfma2(bits_h2(and_or(odd, mhi, magic)), so16, co));
            }
            tmem_st8(dst + 2 * i, v);
            tmem_st8(dst + 16 + 2 * i, w);
          }
          if (g == 0) {                                          // min operand and block scales of this job
            uint32_t mn[4], mn64[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const __half2 p = __hsub2(bits_h2(__byte_perm(s6.mn[i >> 1], 0x64646464u, (i & 1) ? 0x4342 : 0x4140)), k1024);
              mn[i] = h2_bits(p);
              mn64[i] = h2_bits(__hmul2(p, __float2half2_rn(64.f)));
            }
            unsigned char* min_sm = smem + kOffMin + (job & 1) * kMinBytes;
            *reinterpret_cast<uint4*>(min_sm + tile_at(r, 0)) = make_uint4(mn[0], mn[1], mn[2], mn[3]);
            *reinterpret_cast<uint4*>(min_sm + tile_at(r, 1)) = make_uint4(mn64[0], mn64[1], mn64[2], mn64[3]);
            reinterpret_cast<float2*>(smem + kOffDd)[(job & 3) * kGemmRows + r] =
                make_float2(h2f(static_cast<uint16_t>(hdr.x & 0xFFFFu)), h2f(static_cast<uint16_t>(hdr.x >> 16)));
            fence_proxy_async();                                 // min operand -> visible to the tensor core
          }
          if (g & 1) {
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_one(&bar[kBarAFull + slot]);
            if (g == 1 && ++slot == kASlots) { slot = 0; slot_ph ^= 1u; }
          }
        }
        if (!ok) break;
        if (lane == 0) mbar_arrive_one(&bar[kBarWEmpty + st]);         // the stage has been read
        job += G;
        st += G;
        if (st >= kStages) { st -= kStages; st_ph ^= 1u; }
        slot += 2 * G - 1;                                       // from the second half to the next job's first
        while (slot >= kASlots) { slot -= kASlots; slot_ph ^= 1u; }
      }
      to_mine -= n_jobs;
    }
  } else if (warp < kWarpUnpack0) {
    regs_dec<Cfg<RAW>::kRegsCtrl>();
    if (warp == kWarpMma) {
      // ---------------- MMA issue: the whole warp walks, one elected lane issues ----------------
      // (the instructions carry the elected lane's predicate: for 16 MMAs of N = 16 with two waits and two commits
      // 329 cycles, in a branch of the elected lane 446, as a loop 944, from a lone thread 720)
      unsigned job = 0, fill0 = 0, tile_no = 0;
      int slot = 0;
      unsigned slot_ph = 0;
      const uint32_t d_min = umma_desc_core(smem_u32(smem + kOffMin)), d_b = umma_desc_core(smem_u32(smem + kOffB));
      const uint32_t lead = elect_one();
      bool ok = true;
      while (ok && wk.next<DUAL>(a, u)) {
        if (u.w0 == nullptr) continue;
        const uint32_t idesc = __shfl_sync(0xFFFFFFFFu, umma_idesc_f16(u.n_mma), 0);
        ok = for_jobs<DUAL>(a, u, [&](int t, int, int m, int fill) {
          const unsigned set = job & 1, f = fill0 + fill, buf = f & 1;
          if (!DUAL || m == 0) {
            if (!wait_warp(kBarBFull + buf, (f >> 1) & 1)) return false;
            if (!RAW) fence_proxy_async();                       // copied tiles (cp.async is generic) -> the tensor core
          }
          if (!wait_warp(kBarAccEmpty + set, ((job >> 1) & 1) ^ 1u)) return false;
          const uint32_t db = d_b + buf * (kBBytes >> 4), dm = d_min + set * (kMinBytes >> 4);
          const uint32_t d0 = tmem + set * kColSet, d1 = d0 + kGemmTok;
          // the activation tiles are free after their last job
          const bool last_use = DUAL ? m == 1 : (a.nb > 2 || t + 1 == u.n_tiles);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            if (!wait_warp(kBarAFull + slot, slot_ph)) return false;
            tc_fence_after();
            const uint32_t ta = tmem + kColA + slot * 64;
#pragma unroll
            for (int k = 0; k < 8; ++k) umma_ts(lead, d0, ta + k * 8, db + (h * 8 + k) * (kBTile >> 4), kDescCore, idesc, (h | k) != 0);
            if (h == 1) umma_ss(lead, d1, dm, db + 16 * (kBTile >> 4), kDescCore, idesc, 0u);
            if (lead) {
              umma_commit(&bar[kBarAEmpty + slot]);
              if (h == 1) {
                umma_commit(&bar[kBarAccFull + 2 * (DUAL ? m : (tile_no + t) & 1) + set]);
                if (last_use) umma_commit(&bar[kBarBEmpty + buf]);
              }
            }
            __syncwarp();
            if (++slot == kASlots) { slot = 0; slot_ph ^= 1u; }
          }
          ++job;
          return true;
        });
        fill0 += fills_of(a, u);
        tile_no += u.n_tiles;
      }
      if (elect_one()) umma_commit(&bar[kBarDrain]);             // everything issued has finished before tensor memory goes back
      mbar_wait_tight(&bar[kBarDrain], 0);
    } else if (!RAW && warp == kWarpProd0) {
      // ---------------- producer: a block column of 128 rows is one TMA copy ----------------
      unsigned st = 0, st_ph = 1;
      while (wk.next<DUAL>(a, u)) {
        if (u.w0 == nullptr) continue;
        const uintptr_t align = (reinterpret_cast<uintptr_t>(u.w0) | reinterpret_cast<uintptr_t>(u.w1)) & 15u;
        const unsigned char* map = a.maps + (static_cast<size_t>(u.expert) * 3 + a.map0) * 128;
        if (a.maps != nullptr && align == 0 && lane == 0) {
          tmap_acquire(map);
          if (DUAL) tmap_acquire(map + 128);
        }
        const bool ok = for_jobs<DUAL>(a, u, [&](int t, int b, int m, int) {
          const unsigned s = st;
          if (!wait_warp(kBarWEmpty + s, st_ph)) return false;
          if (++st == kStages) { st = 0; st_ph ^= 1u; }
          unsigned char* stage = smem + kOffW + s * kStageBytes;
          const int row0 = (u.tile0 + t) * kGemmRows;
          const unsigned char* src = (m == 0 ? u.w0 : u.w1) + static_cast<size_t>(row0) * row_bytes + b * kW4;
          if (align == 0) {
            if (a.maps == nullptr) {
              cp_load_box(stage, src, kGemmRows, row_bytes, &bar[kBarWFull + s], lane);
              __syncwarp();
              if (lane == 0) mbar_arrive_one(&bar[kBarWFull + s]);
            } else if (lane == 0) {
              mbar_expect_tx(&bar[kBarWFull + s], kStageBytes);
              tma_load_box<STREAM>(stage, map + 128 * m, b * kW4, row0, &bar[kBarWFull + s]);
            }
          } else {                                               // a base off a 16-byte boundary
            warp_copy_unaligned(stage, kStageBytes / 16, lane, reinterpret_cast<uintptr_t>(src), false, [&](int p) { return src + p / 9 * row_bytes + p % 9 * 16; });
            asm volatile("cp.async.wait_all;" ::: "memory");
            fence_proxy_async();                                 // the next fill of the stage may be a TMA copy
            __syncwarp();
            if (lane == 0) mbar_arrive_one(&bar[kBarWFull + s]);
          }
          __syncwarp();
          return true;
        });
        if (!ok) break;
      }
    } else if (RAW && warp < kWarpProd0 + 2) {
      // ---------------- producers: block columns of 128 rows into the ring, alternate jobs ----------------
      // 16-byte piece p = 9 * row + c of a stage goes to lane p % 32; nine steps of 32 pieces are 32 rows, so a lane
      // keeps the source offsets of nine steps.
      const unsigned p = warp - kWarpProd0;
      uint32_t offs[9];
#pragma unroll
      for (int q = 0; q < 9; ++q) offs[q] = (q * 32 + lane) / 9 * row_bytes + (q * 32 + lane) % 9 * 16;
      unsigned job = 0, st = 0, st_ph = 1;
      while (wk.next<DUAL>(a, u)) {
        if (u.w0 == nullptr) continue;
        const bool ok = for_jobs<DUAL>(a, u, [&](int t, int b, int m, int) {
          const unsigned s = st, ph = st_ph;
          if (++st == kStages) { st = 0; st_ph ^= 1u; }
          if ((job++ & 1) != p) return true;
          if (!wait_warp(kBarWEmpty + s, ph)) return false;
          const unsigned char* base = m == 0 ? u.w0 : u.w1;
          const int row0 = (u.tile0 + t) * kGemmRows;
          const unsigned char* src = base + static_cast<size_t>(row0) * row_bytes + b * kW4;
          unsigned char* stage = smem + kOffW + s * kStageBytes;
          const uintptr_t align = reinterpret_cast<uintptr_t>(base) & 15u;
          if (align == 0 && row0 + kGemmRows <= a.n_rows) {
            const uint32_t dst = smem_u32(stage) + lane * 16;
#pragma unroll 1
            for (int g = 0; g < 4; ++g) {
#pragma unroll
              for (int q = 0; q < 9; ++q) cp_async16(dst + (g * 9 + q) * 512, src + offs[q]);
              src += 32 * row_bytes;
            }
            cp_async_arrive(&bar[kBarWFull + s]);
          } else {                                               // ragged last tile, or a base off a 16-byte boundary
            const int last = a.n_rows - 1 - row0;                // rows past the matrix (never stored): zero, or its last one
            auto piece = [&](int p) { return src + min(p / 9, last) * row_bytes + p % 9 * 16; };
            if (align == 0) {
#pragma unroll 4
              for (int q = lane; q < kStageBytes / 16; q += 32) cp_async16_or_zero(smem_u32(stage) + q * 16, piece(q), q / 9 <= last);
              cp_async_arrive(&bar[kBarWFull + s]);
            } else if (warp_copy_unaligned(stage, kStageBytes / 16, lane, align, false, piece)) {
              mbar_arrive_one(&bar[kBarWFull + s]);
            } else {
              cp_async_arrive(&bar[kBarWFull + s]);
            }
          }
          return true;
        });
        if (!ok) break;
      }
      asm volatile("cp.async.wait_all;" ::: "memory");
    } else if constexpr (!RAW) {
      // ---------------- copying stagers: operand rows of one block, 16 bytes per lane and step ----------------
      // lane = (row of eight, one of four 16-byte pieces); each warp takes half of a row's codes, the first one the split sums
      // too and the second one the scales
      const int half = warp - kWarpProd0 - 1, r8 = lane & 7, pc = lane >> 3;
      constexpr int kGroups = kGemmTok / 8, kGroups32 = (kGemmTok + 31) / 32;
      const size_t xrow_bytes = static_cast<size_t>(a.nb) * kOpBlk;
      const uint32_t lane_dst = smem_u32(smem + kOffB) + (pc >> 1) * kBTile + tile_at(r8, pc & 1);      // (of the first half)
      const uint32_t xd_dst = smem_u32(smem + kOffXd) + lane * 4;
      unsigned fill = 0;
      while (wk.next<DUAL>(a, u)) {
        if (u.w0 == nullptr) continue;
        auto row_of = [&](int t) {
          const int s = u.slot0 + min(t, u.nt - 1);             // columns past the last row repeat it; never stored
          return u.rows != nullptr ? __ldg(u.rows + s) : s;
        };
          int row[kGroups32];                                     // of tokens lane, lane + 32, ...
#pragma unroll
        for (int g = 0; g < kGroups32; ++g) row[g] = row_of(g * 32 + lane);
        const int n_fills = fills_of(a, u);
        bool ok = true;
        int blk = 0;
#pragma unroll 1
        for (int f = 0; f < n_fills; ++f, ++fill) {
          const int buf = fill & 1;
          ok = wait_warp(kBarBEmpty + buf, ((fill >> 1) & 1) ^ 1u);
          if (!ok) break;
          const unsigned char* src = u.xq + static_cast<size_t>(blk) * kOpBlk;
          if (++blk == a.nb) blk = 0;
          const uint32_t dst = lane_dst + buf * kBBytes;
#pragma unroll
          for (int g = 0; g < kGroups; ++g)
            if (g * 8 < u.n_mma) {
              const unsigned char* xb = src + __shfl_sync(0xFFFFFFFFu, row[g / 4], (g & 3) * 8 + r8) * xrow_bytes + pc * 16;
#pragma unroll
              for (int q = 0; q < 4; ++q) cp_async16(dst + half * 8 * kBTile + g * 256 + q * 2 * kBTile, xb + half * 256 + q * 64);
              if (half == 0 && pc < 2) cp_async16(dst + g * 256 + 16 * kBTile, xb + 512);
            }
#pragma unroll
          for (int g = 0; g < kGroups32; ++g)
            if (half == 1 && g * 32 + lane < u.n_mma)
              asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(xd_dst + ((fill & 3) * kGemmTok + g * 32) * 4),
                           "l"(src + row[g] * xrow_bytes + 544)
                           : "memory");
          cp_async_arrive(&bar[kBarBFull + buf]);
        }
        if (!ok) break;
      }
      asm volatile("cp.async.wait_all;" ::: "memory");
    }
  } else if constexpr (RAW) {
    // ---------------- converting stagers: one block of the unit's Q8_K rows -> operand tiles ----------------
    // Warp w takes 64 codes of every second group of eight rows, a lane 16 codes of one row of a group (blocks of
    // 276 bytes start on 4-byte boundaries: word loads), and thread i the sums and the scale of row i. A fill's
    // loads are issued before its buffer is awaited.
    regs_dec<Cfg<RAW>::kRegsStage>();
    const int w = (warp - kWarpStage0) & 3, gh = (warp - kWarpStage0) >> 2, i = tid - kWarpStage0 * 32;
    const int r8 = lane & 7, pc = lane >> 3;
    constexpr int kGroups = kGemmTok / 16;                      // row groups per warp
    const size_t xrow_bytes = static_cast<size_t>(a.nb) * kX8;
    float* xd_sm = reinterpret_cast<float*>(smem + kOffXd);
    const __half2 m1152 = __float2half2_rn(-1152.f), m1024 = __float2half2_rn(-1024.f);
    unsigned fill = 0;
    while (wk.next<DUAL>(a, u)) {
      if (u.w0 == nullptr) continue;
      auto row_of = [&](int t) {
        const int s = u.slot0 + min(t, u.nt - 1);               // columns past the last row repeat it; never stored
        return u.rows != nullptr ? __ldg(u.rows + s) : s;
      };
      const int n_fills = fills_of(a, u);
      int row[kGroups];
#pragma unroll
      for (int g = 0; g < kGroups; ++g) row[g] = row_of((2 * g + gh) * 8 + r8);
      const int row_i = row_of(i);
      bool ok = true;
      int blk = 0;
#pragma unroll 1
      for (int f = 0; f < n_fills; ++f, ++fill) {
        const int buf = fill & 1;
        unsigned char* tiles = smem + kOffB + buf * kBBytes;
        const unsigned char* xblk = u.xq + static_cast<size_t>(blk) * kX8;
        if (++blk == a.nb) blk = 0;
        uint32_t cw[kGroups][4];
#pragma unroll
        for (int g = 0; g < kGroups; ++g)
          if ((2 * g + gh) * 8 < u.n_mma) {
            const uint32_t* xb = reinterpret_cast<const uint32_t*>(xblk + row[g] * xrow_bytes) + 1 + w * 16 + pc * 4;
#pragma unroll
            for (int q = 0; q < 4; ++q) cw[g][q] = __ldg(xb + q);
          }
        uint32_t sums[5] = {0u, 0u, 0u, 0u, 0u};                // scale, four words of sub-block sums
        if (i < u.n_mma) {
          const uint32_t* xb = reinterpret_cast<const uint32_t*>(xblk + row_i * xrow_bytes);
          sums[0] = __ldg(xb);
#pragma unroll
          for (int q = 0; q < 4; ++q) sums[1 + q] = __ldg(xb + 65 + q);
        }
        ok = wait_warp(kBarBEmpty + buf, ((fill >> 1) & 1) ^ 1u);
        if (!ok) break;
#pragma unroll
        for (int g = 0; g < kGroups; ++g)
          if ((2 * g + gh) * 8 < u.n_mma) {
            uint32_t h[8];                                       // codes (0, 2), (1, 3) of every word, as the weights' nibbles
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const uint32_t x = cw[g][q] ^ 0x80808080u;
              h[2 * q] = h2_bits(__hadd2(bits_h2(and_or(x, 0x00FF00FFu, 0x64006400u)), m1152));
              h[2 * q + 1] = h2_bits(__hadd2(bits_h2(__byte_perm(x, 0x64646464u, 0x4341)), m1152));
            }
            unsigned char* t = tiles + (w * 4 + pc) * kBTile;
            *reinterpret_cast<uint4*>(t + tile_at((2 * g + gh) * 8 + r8, 0)) = make_uint4(h[0], h[1], h[2], h[3]);
            *reinterpret_cast<uint4*>(t + tile_at((2 * g + gh) * 8 + r8, 1)) = make_uint4(h[4], h[5], h[6], h[7]);
          }
        if (i < u.n_mma) {
          uint32_t lo[4], hi[4];                                 // bsum = 64 * hi + lo
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            lo[q] = h2_bits(__hadd2(bits_h2(and_or(sums[1 + q], 0x003F003Fu, 0x64006400u)), m1024));
            const int s0 = static_cast<int16_t>(sums[1 + q] & 0xFFFFu) >> 6, s1 = static_cast<int16_t>(sums[1 + q] >> 16) >> 6;
            hi[q] = h2_bits(__hadd2(bits_h2(static_cast<uint32_t>(s0 + 128) | (static_cast<uint32_t>(s1 + 128) << 16) | 0x64006400u), m1152));
          }
          unsigned char* t = tiles + 16 * kBTile;
          *reinterpret_cast<uint4*>(t + tile_at(i, 0)) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
          *reinterpret_cast<uint4*>(t + tile_at(i, 1)) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
          xd_sm[(fill & 3) * kGemmTok + i] = __uint_as_float(sums[0]);
        }
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) mbar_arrive_one(&bar[kBarBFull + buf]);
      }
      if (!ok) break;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (tid == 0 && *fail && a.status != nullptr) atomicExch(a.status, 6);
  if (warp == kWarpMma) {
    __syncwarp();
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
  }
}

template <bool DUAL, bool RAW, bool STREAM>
int launch_gemm(GemmArgs a, cudaStream_t stream) {
  a.status = status_word();
  const int sms = device_sms();
  if (a.status == nullptr || sms <= 0) return kErrLaunch;      // the kernel reports an expired wait through the word
  a.tiles = (a.n_rows + kGemmRows - 1) / kGemmRows;
  // Rows of at most two blocks keep their activation tiles for a unit's row tiles: four tiles per unit
  // make the staging an eighth of the jobs' time and still leave about seven units per SM for 256 experts.
  // With fewer units than SMs the other SMs would have nothing to do: then smaller units (8 experts of 2048 x 512 over 64 /
  // 300 rows each: 10.8 / 26.7 us, with units of four tiles 17.8 / 62.5).
  a.group = !DUAL && a.nb <= 2 ? std::min(4, a.tiles) : 1;
  while (a.group > 1 && static_cast<long long>((a.tiles + a.group - 1) / a.group) * a.n_expert < sms) a.group /= 2;
  a.groups = (a.tiles + a.group - 1) / a.group;
  if (a.sw0 != nullptr && a.s_rows > 0) {
    const int passes = (a.s_rows + kGemmTok - 1) / kGemmTok;
    a.s_step = ((a.s_rows + passes - 1) / passes + 15) & ~15;
    a.s_items = a.groups * ((a.s_rows + a.s_step - 1) / a.s_step);
  } else {
    a.s_items = 0;
  }
  const long long n_items = static_cast<long long>(a.groups) * a.n_expert + a.s_items;
  if (n_items > 0x7FFFFFFF - 1024) return kErrUnsupported;
  a.n_items = static_cast<int>(n_items);
  if (!opt_in_smem<grouped_gemm_kernel<DUAL, RAW, STREAM>>(kGemmSmem)) return kErrLaunch;
  return launch_pdl(grouped_gemm_kernel<DUAL, RAW, STREAM>, dim3(std::min(a.n_items, sms)), Cfg<RAW>::kThreads, kGemmSmem, stream, a);
}

// Rows of fp16 values - or SwiGLU of two rows, rounded to fp16 as silu_mul_f16 does - -> operand rows
// (api_util.cuh): the Q8_K quantiser of quantize_block_f16 with the codes, the split sums and the scale in
// the form the GEMM copies. Two slabs in one launch, the first bounded by *d_rows on the device; and, in map_ctas CTAs of
// their own, the experts' descriptors. One warp per block or expert.
constexpr int kQuantWarps = 4;
__global__ void __launch_bounds__(kQuantWarps * 32)
quantize_operand_kernel(const uint16_t* __restrict__ x0, const uint16_t* __restrict__ u0,
                        unsigned char* __restrict__ out0, long long n0, const int* __restrict__ d_rows,
                        const uint16_t* __restrict__ x1, const uint16_t* __restrict__ u1,
                        unsigned char* __restrict__ out1, long long n1, int nb, unsigned map_ctas,
                        const __grid_constant__ MapArgs m) {
  __shared__ __align__(128) unsigned char patch[kQuantWarps][384];
  pdl_wait();
  pdl_launch_dependents();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (blockIdx.x < map_ctas) {
    const int e = blockIdx.x * kQuantWarps + warp;
    if (e <= m.n_expert) make_maps(m, e, patch[warp], lane);
    return;
  }
  long long b = static_cast<long long>(blockIdx.x - map_ctas) * kQuantWarps + warp;
  const uint16_t *x = x0, *u = u0;
  unsigned char* out = out0;
  if (b >= n0) {
    b -= n0;
    if (b >= n1) return;
    x = x1;
    u = u1;
    out = out1;
  } else if (d_rows != nullptr && b >= static_cast<long long>(*d_rows) * nb) {
    return;
  }
  float v[8];
  load_lane8(x + b * kQK, lane, v);
  if (u != nullptr) {
    float uv[8];
    load_lane8(u + b * kQK, lane, uv);
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = h2f(f2h(silu_mul(v[i], uv[i])));
  }
  int q[8], sum;
  const float d = quantize_lane8(v, q, sum);
  out += b * kOpBlk;
  uint32_t h[4];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    h[2 * i] = h2_bits(__floats2half2_rn(static_cast<float>(q[4 * i]), static_cast<float>(q[4 * i + 2])));
    h[2 * i + 1] = h2_bits(__floats2half2_rn(static_cast<float>(q[4 * i + 1]), static_cast<float>(q[4 * i + 3])));
  }
  reinterpret_cast<uint4*>(out)[lane] = make_uint4(h[0], h[1], h[2], h[3]);
  if ((lane & 3) == 0) {                                        // four lanes hold one sub-block: bsum = 64 * hi + lo
    uint16_t* s = reinterpret_cast<uint16_t*>(out + 512) + (lane >> 2);
    s[0] = f2h(static_cast<float>(sum & 63));
    s[8] = f2h(static_cast<float>(sum >> 6));
  }
  if (lane == 0) *reinterpret_cast<float*>(out + 544) = d;
}

GemmArgs args_of(const ExpertGemm& g) {
  GemmArgs a{};
  a.tab0 = g.tab; a.off = g.off; a.rows = g.rows; a.xq = g.xq; a.y = g.y;
  a.n_rows = g.n_rows; a.nb = g.k / kQK; a.n_expert = g.n_expert;
  a.sw0 = a.sw1 = static_cast<const unsigned char*>(g.shared_w);
  a.sxq = g.shared_xq; a.sy = g.shared_y; a.s_rows = g.shared_rows;
  a.maps = static_cast<const unsigned char*>(g.maps);
  return a;
}

}  // namespace

int gemm_gate_up(const ExpertGemm& g, const unsigned char* const* tab_up, uint16_t* y_up, const void* shared_up,
                 uint16_t* shared_y_up, cudaStream_t stream) {
  GemmArgs a = args_of(g);
  a.tab1 = tab_up; a.y1 = y_up;
  a.sw1 = static_cast<const unsigned char*>(shared_up); a.sy1 = shared_y_up;
  if (!g.operand_rows) return launch_gemm<true, true, false>(a, stream);
  return g.stream ? launch_gemm<true, false, true>(a, stream) : launch_gemm<true, false, false>(a, stream);
}
int gemm_grouped(const ExpertGemm& g, cudaStream_t stream) {
  GemmArgs a = args_of(g);
  a.map0 = 2;
  if (!g.operand_rows) return launch_gemm<false, true, false>(a, stream);
  return g.stream ? launch_gemm<false, false, true>(a, stream) : launch_gemm<false, false, false>(a, stream);
}
int quantize_operand(const uint16_t* x0, const uint16_t* u0, void* out0, long long rows0, const int* d_rows,
                     const uint16_t* x1, const uint16_t* u1, void* out1, long long rows1, int k, const ExpertMaps& em, bool make_maps,
                     cudaStream_t stream) {
  const int nb = k / kQK;
  const long long ctas = ((rows0 + rows1) * nb + kQuantWarps - 1) / kQuantWarps;
  MapArgs m{};
  if (!map_args(em, make_maps, &m)) return kErrUnsupported;
  const unsigned map_ctas = make_maps && em.maps != nullptr ? static_cast<unsigned>(em.n_expert / kQuantWarps + 1) : 0;
  if (ctas + map_ctas > 0x7FFFFFFF) return kErrUnsupported;
  if (ctas + map_ctas == 0) return kOk;
  return launch_pdl(quantize_operand_kernel, dim3(static_cast<unsigned>(ctas + map_ctas)), kQuantWarps * 32, 0, stream, x0, u0,
                    static_cast<unsigned char*>(out0), rows0 * nb, d_rows, x1, u1, static_cast<unsigned char*>(out1), rows1 * nb, nb,
                    map_ctas, m);
}

}  // namespace sgr

using namespace sgr;

// y[off[e] + t][r] = W_e[r][:] . xq[off[e] + t][:] for every expert e and its rows
// t < off[e+1] - off[e]; fp16 out, row length n_rows. w_tab[e] == null: zero rows.
SGR_API int sgr_moe_grouped_gemm_i8(const void* const* w_tab, const int* off, const void* xq,
                                    uint16_t* y, int n_rows, int k, int n_expert, void* stream) {
  if (n_expert <= 0 || n_rows <= 0) return kOk;
  if (!w_tab || !off || !xq || !y || k <= 0 || k % kQK != 0) return kErrArg;
  if (reinterpret_cast<uintptr_t>(xq) & 15u) return kErrAlign;
  if (n_expert > 65535) return kErrUnsupported;
  ExpertGemm g{};
  g.tab = reinterpret_cast<const unsigned char* const*>(w_tab);
  g.off = off;
  g.xq = static_cast<const unsigned char*>(xq);
  g.y = y;
  g.n_rows = n_rows;
  g.k = k;
  g.n_expert = n_expert;
  return gemm_grouped(g, as_stream(stream));
}
