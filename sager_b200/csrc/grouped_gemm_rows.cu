// grouped_gemm_rows.cu - the prefill MoE grouped GEMM for chunks that leave an expert few token rows.
//
// Same contract and same values as the tcgen05 form (grouped_gemm_i8.cu; both replace the reference's prefill expert math,
// src/kernels/cuda/tc_gemm.cu:124-152, 209-240): Q8_K activations, exact integer sums per super-block, and per block
//     acc = fma(xd, fma(-dmin, M, d * S), acc)
// in block order, so the two agree to the bit (while S stays below 2^24, which the tensor-memory accumulator holds
// exactly). That form unpacks every weight to fp16 and passes a block column through five roles whatever the number of
// token rows: 1,800 cycles per 128 rows x 256 weights at 16 rows, 2,500 at 64, where HBM needs 800. Here a consumer warp
// keeps sixteen weight rows and their sums from the first block column to the last (as the decode layer's row-streaming
// kernel, expert_rows.cuh): nibbles go into mma.sync m16n8k32 with one logic instruction per four, the sub-block scales
// are applied to the int32 results.
//
// Persistent, one CTA per SM. A unit is 128 (gate, up) row pairs, or 256 rows, of one expert and at most 32 of its
// token rows, and is handed out by itself, so that the passes of a hot expert spread over the SMs; its block columns stream through a ring of four stages (256 blocks of 144 bytes by two TMA copies, and
// that block of the token rows by one bulk copy each). Sixteen consumer warps, one weight warp, two activation warps; a
// consumer returns its share of the weight bytes as soon as they are in registers. Gate and up rows of the same index meet
// in a warp, so SwiGLU happens on the accumulators (rounded to fp16 first, as the reference's staged rows are). Waits are
// bounded; an expiry raises the status word.
#include <algorithm>

#include "api_util.cuh"
#include "quantize_dev.cuh"
#include "tile.cuh"
#include "tmap_dev.cuh"

namespace sgr {
namespace {

constexpr int kTok = 32;                                     // token rows per unit
constexpr int kConsumerWarps = 16, kWeightWarp = kConsumerWarps, kFirstXWarp = kWeightWarp + 1, kXWarps = 2;
constexpr int kThreads = (kFirstXWarp + kXWarps) * 32;
constexpr int kStages = 4;
constexpr int kHalfBytes = 128 * kW4, kWBytes = 2 * kHalfBytes;
// activation part of a stage: a 288-byte block (kRowBlk, api_util.cuh) per token row; rows 76 words apart, so
// that eight rows' 16 bytes lie in different banks
constexpr int kXRow = 304, kXCodes = 16, kXSums = 272, kXBytes = kTok * kXRow;
static_assert(kRowBlk <= kXRow && kXSums + 16 == kRowBlk, "block layout");
constexpr int kStageBytes = (kWBytes + kXBytes + 127) & ~127;
constexpr int kHdr = 1024;                                    // the last 256 bytes are zeros
constexpr int kSmem = kHdr + kStages * kStageBytes;
static_assert(kSmem <= 227 * 1024, "shared memory");

struct RowsArgs {
  const unsigned char* const* tab0;    // [E] gate (or the only matrix)
  const unsigned char* const* tab1;    // [E] up
  const unsigned char* maps;           // [E + 1][3] descriptors (null: none); the matrix of tab0 is map0
  int map0;
  const int* off;                      // [E + 1] grouped slots of each expert
  const int* rows;                     // source row of a grouped slot; null: the slot itself
  const unsigned char *xq, *sxq;       // activation rows in 288-byte blocks; the shared expert's
  uint16_t *y, *sy;                    // [slots][n_rows]
  const unsigned char *sw0, *sw1;      // the shared expert (null: none)
  int n_rows, nb, n_expert, groups;    // row groups per matrix
  int s_rows, s_step, s_items;
  unsigned* next;                      // items handed out beyond the first of every CTA
  int* status;
};

// One unit, as the weight warp publishes it in shared memory for the activation warps.
struct alignas(16) Unit {
  int slot0, nt, flags;                // first slot, token rows (0: end of the list), 1 shared / 2 absent
  int pad;
};
constexpr int kListSlots = 8;          // units published ahead: at most one per stage, and the one being read
static_assert(kListSlots >= kStages + 3, "a reader could be overtaken");

struct Desc {      // one 16-byte load per stage and warp
  int flags;       // bits 0-7 token rows, 8 first column, 9 last, 10 absent, 11 shared, 12 end of the list
  int slot0, group;
  int pad;
};

// (as one instruction: sums of products are otherwise regrouped into a multiplication, a multiply-add and an addition)
__device__ __forceinline__ int imad(int a, int b, int c) {
  int d;
  asm("mad.lo.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}
// One super-block of a warp's sixteen rows against NT groups of eight token rows; as warp_mma_block (tile.cuh) with the
// fp32 steps spelled out, and with the even sub-blocks' scales taken sixteen-fold instead of their sums.
template <int NT, typename Loaded>
__device__ __forceinline__ void rows_block(const unsigned char* a_ptr, const unsigned char* h_lo, const unsigned char* h_hi,
                                           const unsigned char* xs, float (&acc)[4][4], int lane, Loaded loaded) {
  const int gid = lane >> 2, tig = lane & 3;
  const uint4 h0 = *reinterpret_cast<const uint4*>(h_lo);
  const uint4 h1 = *reinterpret_cast<const uint4*>(h_hi);
  uint32_t raw[4][4];
#pragma unroll
  for (int g = 0; g < 4; ++g) ldmatrix_x4(raw[g], a_ptr + g * 32);
  loaded();
  const float d_lo = 0.0625f * h2f(static_cast<uint16_t>(h0.x & 0xFFFFu)), m_lo = -h2f(static_cast<uint16_t>(h0.x >> 16));
  const float d_hi = 0.0625f * h2f(static_cast<uint16_t>(h1.x & 0xFFFFu)), m_hi = -h2f(static_cast<uint16_t>(h1.x >> 16));
  const Scales6 s_lo = unpack_scales6(h0.y, h0.z, h0.w), s_hi = unpack_scales6(h1.y, h1.z, h1.w);
  int isum[NT][4];
#pragma unroll
  for (int n = 0; n < NT; ++n)
#pragma unroll
    for (int j = 0; j < 4; ++j) isum[n][j] = 0;
  const int zero[4] = {0, 0, 0, 0};
  // matrices of an activation load: (tokens, k 0-15 / 16-31) of sub-block 2g, then of 2g + 1
  const unsigned char* b_ptr = xs + (lane & 7) * kXRow + kXCodes + (lane >> 3) * 16;
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    uint32_t lo[4], hi[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      lo[j] = raw[g][j] & 0x0F0F0F0Fu;
      hi[j] = raw[g][j] & 0xF0F0F0F0u;            // sixteen-fold
    }
    const int sh = 2 * (g & 1);
    const int sc0_lo = __byte_perm(s_lo.sc[g >> 1], 0, 0x4440 + sh) << 4, sc1_lo = __byte_perm(s_lo.sc[g >> 1], 0, 0x4441 + sh);
    const int sc0_hi = __byte_perm(s_hi.sc[g >> 1], 0, 0x4440 + sh) << 4, sc1_hi = __byte_perm(s_hi.sc[g >> 1], 0, 0x4441 + sh);
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      uint32_t b[4];
      ldmatrix_x4(b, b_ptr + n * 8 * kXRow + g * 64);
      int c0[4], c1[4];
      mma_u8s8(c0, lo, b[0], b[1], zero);
      mma_u8s8(c1, hi, b[2], b[3], zero);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        isum[n][j] = imad(j < 2 ? sc0_lo : sc0_hi, c0[j], isum[n][j]);
        isum[n][j] = imad(j < 2 ? sc1_lo : sc1_hi, c1[j], isum[n][j]);
      }
    }
  }
  const uint32_t ma[4] = {tig == 0 ? s_lo.mn[0] : (tig == 1 ? s_lo.mn[1] : 0u), tig == 0 ? s_hi.mn[0] : (tig == 1 ? s_hi.mn[1] : 0u), 0u, 0u};
#pragma unroll
  for (int n = 0; n < NT; ++n) {
    // parts of the sub-block sums 4 tig .. 4 tig + 3 of token 8 n + gid (lanes whose mins are zero read another's)
    const uint2 sv = *reinterpret_cast<const uint2*>(xs + (8 * n + gid) * kXRow + kXSums + 8 * (tig & 1));
    int dl[4], dh[4];
    mma_u8s8(dl, ma, sv.x, 0u, zero);
    mma_u8s8(dh, ma, sv.y, 0u, zero);
    const float* xd = reinterpret_cast<const float*>(xs + (8 * n + 2 * tig) * kXRow);
    const float xd0 = xd[0], xd1 = xd[kXRow / 4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float s = __fmul_rn(j < 2 ? d_lo : d_hi, static_cast<float>(isum[n][j]));
      acc[n][j] = __fmaf_rn(j & 1 ? xd1 : xd0, __fmaf_rn(j < 2 ? m_lo : m_hi, static_cast<float>(imad(dh[j], 128, dl[j])), s), acc[n][j]);
    }
  }
}

// Weight warp: a stage's two halves of 128 blocks where the TMA unit cannot bring them - no descriptors, or a base off a 16-byte
// boundary - and the barrier's arrival.
__device__ __forceinline__ void copy_blocks(unsigned char* st, const unsigned char* b0, const unsigned char* b1, int row_bytes, bool aligned,
                                                uint64_t* bar, int lane) {
  if (aligned) {
#pragma unroll 1
    for (int h = 0; h < 2; ++h) cp_load_box(st + h * kHalfBytes, h ? b1 : b0, 128, row_bytes, bar, lane);
  } else {
    const uintptr_t a0 = reinterpret_cast<uintptr_t>(b0), a1 = reinterpret_cast<uintptr_t>(b1);
    warp_copy_unaligned(st, kWBytes / 16, lane, a0 | a1, ((a0 ^ a1) & 2u) != 0, [&](int p) {
      const int r = p / 9, h = r >> 7;
      return (h ? b1 : b0) + static_cast<size_t>(r & 127) * row_bytes + (p - r * 9) * 16;
    });
    asm volatile("cp.async.wait_all;" ::: "memory");
    fence_proxy_async();                             // the next fill of this stage may come from the TMA unit
  }
  __syncwarp();
  if (lane == 0) mbar_arrive_one(bar);
}

// STREAM: weights first to leave L2 (streams_weights)
template <bool DUAL, bool STREAM>
__global__ void __launch_bounds__(kThreads, 1) grouped_gemm_rows_kernel(const RowsArgs a) {
  extern __shared__ __align__(128) unsigned char smem[];
  uint64_t* full = reinterpret_cast<uint64_t*>(smem);            // [kStages] copies landed
  uint64_t* wempty = full + kStages;                             // weight part may be refilled
  uint64_t* xempty = wempty + kStages;                           // activation part may be refilled
  volatile unsigned* published = reinterpret_cast<volatile unsigned*>(smem + 132);
  Desc* desc = reinterpret_cast<Desc*>(smem + 256);
  Unit* list = reinterpret_cast<Unit*>(smem + 512);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  unsigned char* const zeros = smem + kHdr - 256;
  if (tid < 64) reinterpret_cast<uint32_t*>(zeros)[tid] = 0u;
  if (tid == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full[s], 1 + kXWarps);
      mbar_init(&wempty[s], kConsumerWarps);
      mbar_init(&xempty[s], kConsumerWarps);
    }
    *published = 0;
    fence_barrier_init();
  }
  __syncthreads();
  pdl_wait();                                        // plan, descriptors and activations come from the kernels before this one
  pdl_launch_dependents();
  auto wait = [&](uint64_t* b, unsigned parity) {
    if (__all_sync(0xFFFFFFFFu, mbar_wait(b, parity)) != 0) return true;
    if (lane == 0) atomicExch(a.status, 6);
    return false;
  };
  int s = 0;
  unsigned ph = 0;
  auto advance = [&] { if (++s == kStages) { s = 0; ph ^= 1u; } };

  if (warp == kWeightWarp) {
    // ---------------- weights ----------------
    // Items are units: one pass of an expert's token rows over one row group, handed out as CTAs come to want them. (With rounds of
    // fixed length the slowest CTA had 293,000 cycles of 241,000 on average, 777 rows over 256 experts. With all passes of an
    // expert in one item a chunk waited for its hot experts: two layers, 832 rows over 256 experts, 439 us evenly spread, 804
    // with a fifth of the experts in 70 % of the routes, 1409 with one in almost all of them; 439 / 469 / 421 by passes.)
    // The passes of a row group follow one another, so that the CTAs that read the same weights do so together. Where an item
    // lies is looked up in a window of 32 experts that only moves on, a lane per expert, while the item before it streams; the
    // next window's loads are under way before it is needed. (96 rows, two layers: 228 us with loads and look-up
    // between two items, 220 with the loads ahead, 214 like this.)
    const int row_bytes = a.nb * kW4;
    unsigned k = 0;                                  // units published
    auto publish = [&](int slot0, int nt, int flags) {
      if (lane == 0) {
        Unit* e = list + k % kListSlots;
        e->slot0 = slot0; e->nt = nt; e->flags = flags;
        __threadfence_block();
        *published = k + 1;
      }
      ++k;
    };
    int e0 = 0, w_slot, w_rows, w_end = 0;           // the window: this lane's expert's first slot and rows, items up to and with it
    const unsigned char *w_0, *w_1;                  // ... and its matrices
    int n_slot = 0, n_to = 0;                        // the same of the window after it, on its way
    const unsigned char *n_0 = nullptr, *n_1 = nullptr;
    auto passes_of = [](int rows) { return (rows + kTok - 1) / kTok; };
    auto request = [&](int e) {
      const int c = min(e, a.n_expert - 1);
      n_slot = __ldg(a.off + c);
      n_to = __ldg(a.off + c + (e < a.n_expert ? 1 : 0));      // (past the end: no rows)
      n_0 = a.tab0[c];
      n_1 = DUAL ? a.tab1[c] : n_0;
    };
    auto window = [&](int before) {                  // the window at e0 becomes the present one
      const int to = n_to;
      w_slot = n_slot;
      w_0 = n_0;
      w_1 = n_1;
      request(e0 + 32 + lane);
      w_rows = to - w_slot;
      if (!__any_sync(0xFFFFFFFFu, w_rows > kTok)) {           // (a scan costs a launch of short items 0.6 us at its start)
        w_end = __popc(__ballot_sync(0xFFFFFFFFu, w_rows > 0) & ((2u << lane) - 1)) * a.groups;
      } else {
        w_end = passes_of(w_rows) * a.groups;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
          const int v = __shfl_up_sync(0xFFFFFFFFu, w_end, off);
          if (lane >= off) w_end += v;
        }
      }
      w_end += before;
    };
    auto lane_ptr = [](const unsigned char* p, int from) {
      return reinterpret_cast<const unsigned char*>(__shfl_sync(0xFFFFFFFFu, reinterpret_cast<unsigned long long>(p), from));
    };
    request(lane);
    window(0);
    struct Item { int e, group, slot, nt; const unsigned char *w0, *w1; };
    auto find = [&](unsigned item) {
      Item f;
      if (item < static_cast<unsigned>(a.s_items)) {
        const int pass = static_cast<int>(item) / a.groups;
        f.e = a.n_expert;
        f.group = static_cast<int>(item) - pass * a.groups;
        f.slot = pass * a.s_step;
        f.nt = min(a.s_step, a.s_rows - f.slot);
        f.w0 = a.sw0;
        f.w1 = a.sw1;
        return f;
      }
      const int i = static_cast<int>(item) - a.s_items;
      for (int before; i >= (before = __shfl_sync(0xFFFFFFFFu, w_end, 31)) && e0 < a.n_expert;) {
        e0 += 32;
        window(before);
      }
      f.e = f.group = f.slot = f.nt = 0;             // no rows: the list is at its end
      f.w0 = f.w1 = nullptr;
      if (e0 >= a.n_expert) return f;
      const int at = __popc(__ballot_sync(0xFFFFFFFFu, w_end <= i)), rows = __shfl_sync(0xFFFFFFFFu, w_rows, at);
      const int passes = passes_of(rows), r = i - (__shfl_sync(0xFFFFFFFFu, w_end, at) - passes * a.groups);
      f.slot = __shfl_sync(0xFFFFFFFFu, w_slot, at);
      f.group = r;
      f.nt = rows;
      if (passes > 1) {
        const int step = ((rows + passes - 1) / passes + 7) & ~7;
        f.group = r / passes;
        const int t0 = (r - f.group * passes) * step;
        f.slot += t0;
        f.nt = min(step, rows - t0);
      }
      f.e = e0 + at;
      f.w0 = lane_ptr(w_0, at);
      f.w1 = DUAL ? lane_ptr(w_1, at) : f.w0;
      return f;
    };
    const int look = (a.nb - 1) / 2;                 // the column under which the next item is looked up
    for (Item it = find(blockIdx.x), after; it.nt > 0; it = after) {
      unsigned later = 0;
      if (lane == 0) later = atomicAdd(a.next, 1u);
      const int e = it.e, group = it.group, slot = it.slot, nt = it.nt;
      const unsigned char *w0 = it.w0, *w1 = it.w1;
      const bool shared = e == a.n_expert;
      const uintptr_t align = (reinterpret_cast<uintptr_t>(w0) | reinterpret_cast<uintptr_t>(w1)) & 15u;
      const bool absent = w0 == nullptr || w1 == nullptr;
      const unsigned char* map0 = a.maps + (static_cast<size_t>(e) * 3 + a.map0) * 128;
      const int row0 = group * (DUAL ? 128 : 256);
      if (a.maps != nullptr && !absent && align == 0 && lane == 0) {
        tmap_acquire(map0);
        if (DUAL) tmap_acquire(map0 + 128);
      }
      publish(slot, nt, (shared ? 1 : 0) | (absent ? 2 : 0));
#pragma unroll 1
      for (int b = 0; b < a.nb; ++b) {
        if (!wait(&wempty[s], ph ^ 1u)) return;
        unsigned char* st = smem + kHdr + s * kStageBytes;
        if (lane == 0) {
          Desc d;
          d.flags = nt | (b == 0 ? 1 << 8 : 0) | (b + 1 == a.nb ? 1 << 9 : 0) | (absent ? 1 << 10 : 0) | (shared ? 1 << 11 : 0);
          d.slot0 = slot; d.group = group; d.pad = 0;
          desc[s] = d;
        }
        if (absent) {
          if (lane == 0) mbar_arrive_one(&full[s]);
        } else if (align == 0 && a.maps != nullptr) {
          if (lane == 0) {
            mbar_expect_tx(&full[s], kWBytes);
            tma_load_box<STREAM>(st, map0, b * kW4, row0, &full[s]);
            tma_load_box<STREAM>(st + kHalfBytes, DUAL ? map0 + 128 : map0, b * kW4, DUAL ? row0 : row0 + 128, &full[s]);
          }
        } else {
          const unsigned char* b0 = w0 + static_cast<size_t>(row0) * row_bytes + b * kW4;
          copy_blocks(st, b0, DUAL ? w1 + static_cast<size_t>(row0) * row_bytes + b * kW4 : b0 + static_cast<size_t>(128) * row_bytes,
                      row_bytes, align == 0, &full[s], lane);
        }
        __syncwarp();
        if (b == look) after = find(__shfl_sync(0xFFFFFFFFu, later, 0) + gridDim.x);
        advance();
      }
    }
    publish(0, 0, 0);
    if (!wait(&wempty[s], ph ^ 1u)) return;
    if (lane == 0) {                                 // one last stage that only says that the list is at its end
      Desc d;
      d.flags = 1 << 12; d.slot0 = d.group = d.pad = 0;
      desc[s] = d;
      mbar_arrive_one(&full[s]);
    }
  } else if (warp >= kFirstXWarp) {
    // ---------------- activations: one bulk copy of 288 bytes per token row and block ----------------
    const int x = warp - kFirstXWarp, t = kXWarps * lane + x;      // this lane's token row
    const size_t xrow = static_cast<size_t>(a.nb) * kRowBlk;
    for (unsigned k = 0;; ++k) {
      unsigned it = 0;
      if (lane == 0)
        while (*published <= k && ++it < (1u << 24)) __nanosleep(20);
      if (__shfl_sync(0xFFFFFFFFu, it, 0) >= (1u << 24)) {
        if (lane == 0) atomicExch(a.status, 6);
        return;
      }
      __threadfence_block();
      const Unit u = list[k % kListSlots];
      if (u.nt == 0) break;
      const bool shared = u.flags & 1, copies = !(u.flags & 2) && t < u.nt;
      int row = u.slot0 + t;
      if (copies && !shared && a.rows != nullptr) row = __ldg(a.rows + row);
      const unsigned char* src = (shared ? a.sxq : a.xq) + static_cast<size_t>(row) * xrow;
      const int mine = u.flags & 2 ? 0 : (u.nt - x + kXWarps - 1) / kXWarps;     // rows of this warp
#pragma unroll 1
      for (int b = 0; b < a.nb; ++b, src += kRowBlk) {
        if (!wait(&xempty[s], ph ^ 1u)) return;
        if (lane == 0) {
          if (mine > 0) mbar_expect_tx(&full[s], mine * kRowBlk);
          else mbar_arrive_one(&full[s]);
        }
        __syncwarp();
        if (copies) bulk_g2s(smem + kHdr + s * kStageBytes + kWBytes + t * kXRow, src, kRowBlk, &full[s]);
        advance();
      }
    }
    if (!wait(&xempty[s], ph ^ 1u)) return;
    if (lane == 0) mbar_arrive_one(&full[s]);
  } else {
    // ---------------- consumers: sixteen rows each ----------------
    float acc[4][4];
    const int gid = lane >> 2, tig = lane & 3;
    // unit u of the sixteen: gate rows 0 .. 7 and the up rows of the same indices, or sixteen adjacent rows
    auto row_at = [&](int u) { return DUAL ? ((u & 7) + 8 * warp) * kW4 + (u >> 3) * kHalfBytes : (16 * warp + u) * kW4; };
    const int w_off = row_at((lane & 7) + ((lane >> 3) & 1) * 8) + 16 + (lane >> 4) * 16, own_lo = row_at(gid), own_hi = row_at(gid + 8);
    for (;; advance()) {
      if (!wait(&full[s], ph)) return;
      const Desc d = desc[s];
      if (d.flags >> 12 & 1) break;
      const int nt = d.flags & 255;
      unsigned char* st = smem + kHdr + s * kStageBytes;
      if (d.flags >> 8 & 1) {
#pragma unroll
        for (int n = 0; n < 4; ++n)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[n][j] = 0.f;
      }
      auto loaded = [&] {
        __syncwarp();
        if (lane == 0) mbar_arrive_one(&wempty[s]);
      };
      if (d.flags >> 10 & 1) {
        loaded();
      } else if (nt <= 4) {
        const unsigned char* xs = st + kWBytes;
        const uint4 h0 = *reinterpret_cast<const uint4*>(st + own_lo), h1 = *reinterpret_cast<const uint4*>(st + own_hi);
        const unsigned char* b_row = b_row4(xs + kXCodes, kXRow, zeros, lane);
        warp_mma_block4(st + w_off, h0, h1, [&](int g) { return b_row + g * 64; }, lane, loaded,
                        [&] { return *reinterpret_cast<const uint32_t*>(xs + (gid >> 1) * kXRow + kXSums + (tig & 1) * 8 + (gid & 1) * 4); },
                        [&](int r, int isum, int msum) {
                          const uint32_t dm = r ? h1.x : h0.x;
                          const float s = __fmul_rn(0.0625f * h2f(static_cast<uint16_t>(dm & 0xFFFFu)), static_cast<float>(isum));
                          const float v = __fmaf_rn(-h2f(static_cast<uint16_t>(dm >> 16)), static_cast<float>(msum), s);
                          acc[0][r] = __fmaf_rn(*reinterpret_cast<const float*>(xs + tig * kXRow), v, acc[0][r]);
                        });
      } else if (nt <= 8) rows_block<1>(st + w_off, st + own_lo, st + own_hi, st + kWBytes, acc, lane, loaded);
      else if (nt <= 16) rows_block<2>(st + w_off, st + own_lo, st + own_hi, st + kWBytes, acc, lane, loaded);
      else if (nt <= 24) rows_block<3>(st + w_off, st + own_lo, st + own_hi, st + kWBytes, acc, lane, loaded);
      else rows_block<4>(st + w_off, st + own_lo, st + own_hi, st + kWBytes, acc, lane, loaded);
      __syncwarp();
      if (lane == 0) mbar_arrive_one(&xempty[s]);
      if (!(d.flags >> 9 & 1)) continue;
      // ---- the unit is complete for this warp's rows: the lanes of two neighbouring rows trade halves, so that a
      // store is two rows of one token ----
      uint16_t* y = (d.flags >> 11 & 1) ? a.sy : a.y;
      if (nt <= 4) {                                 // token tig; row pairs by the even lanes
        const __half2 v = __floats2half2_rn(acc[0][0], acc[0][1]);
        uint32_t mine = *reinterpret_cast<const uint32_t*>(&v);
        if (DUAL) {
          const __half h = __float2half(silu_mul(__low2float(v), __high2float(v)));
          mine = *reinterpret_cast<const uint16_t*>(&h);
        }
        const uint32_t other = __shfl_xor_sync(0xFFFFFFFFu, mine, 4);
        if (tig < nt && (gid & 1) == 0) {
          uint16_t* o = y + static_cast<size_t>(d.slot0 + tig) * a.n_rows + d.group * (DUAL ? 128 : 256) + (DUAL ? 8 : 16) * warp + gid;
          *reinterpret_cast<uint32_t*>(o) = __byte_perm(mine, other, 0x5410);
          if (!DUAL) *reinterpret_cast<uint32_t*>(o + 8) = __byte_perm(mine, other, 0x7632);
        }
        continue;
      }
      const int odd = gid & 1;
      const uint32_t sel = odd ? 0x3276u : 0x5410u;
      const int row = d.group * (DUAL ? 128 : 256) + (DUAL ? 8 : 16) * warp + gid - odd;
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        if (8 * n >= nt) break;
        const int t = 8 * n + 2 * tig + odd;
        uint16_t* o = y + static_cast<size_t>(d.slot0 + t) * a.n_rows + row;
        const __half2 lo = __floats2half2_rn(acc[n][0], acc[n][1]), hi = __floats2half2_rn(acc[n][2], acc[n][3]);
        auto trade = [&](__half2 v) {
          const uint32_t mine = *reinterpret_cast<const uint32_t*>(&v);
          return __byte_perm(mine, __shfl_xor_sync(0xFFFFFFFFu, mine, 4), sel);
        };
        if (DUAL) {
          const uint32_t h = trade(__floats2half2_rn(silu_mul(__low2float(lo), __low2float(hi)), silu_mul(__high2float(lo), __high2float(hi))));
          if (t < nt) *reinterpret_cast<uint32_t*>(o) = h;
        } else {
          const uint32_t v0 = trade(lo), v1 = trade(hi);
          if (t < nt) {
            *reinterpret_cast<uint32_t*>(o) = v0;
            *reinterpret_cast<uint32_t*>(o + 8) = v1;
          }
        }
      }
    }
  }
}

template <bool DUAL, bool STREAM>
int launch_rows(RowsArgs a, long long routes, cudaStream_t stream) {
  a.status = status_word();
  const int sms = device_sms();
  if (a.status == nullptr || sms <= 0) return kErrLaunch;
  a.groups = a.n_rows / (DUAL ? 128 : 256);
  a.s_items = 0;
  if (a.sw0 != nullptr && a.s_rows > 0) {
    const int passes = (a.s_rows + kTok - 1) / kTok;
    a.s_step = ((a.s_rows + passes - 1) / passes + 7) & ~7;
    a.s_items = a.groups * ((a.s_rows + a.s_step - 1) / a.s_step);
  }
  // (the routed items' number is known on the device alone: passes of kTok rows are at most one more per expert than the rows make)
  const long long n_items = static_cast<long long>(a.groups) * (a.n_expert + routes / kTok) + a.s_items;
  if (n_items > 0x7FFFFFFF - 1024) return kErrUnsupported;
  if (!opt_in_smem<grouped_gemm_rows_kernel<DUAL, STREAM>>(kSmem)) return kErrLaunch;
  return launch_pdl(grouped_gemm_rows_kernel<DUAL, STREAM>, dim3(static_cast<unsigned>(std::min<long long>(n_items, sms))), kThreads, kSmem, stream, a);
}

// Rows of fp16 values -> Q8_K rows in blocks of kRowBlk bytes, two slabs
// in one launch, the first bounded by *d_rows on the device; and, in CTAs of their own (map_ctas of them), the descriptors of every
// expert's three matrices. One warp per block or expert.
constexpr int kQuantWarps = 4;
__global__ void __launch_bounds__(kQuantWarps * 32)
quantize_rows_kernel(const uint16_t* __restrict__ x0, unsigned char* __restrict__ out0, long long n0, const int* __restrict__ d_rows,
                     const uint16_t* __restrict__ x1, unsigned char* __restrict__ out1, long long n1, int nb, unsigned map_ctas,
                     const __grid_constant__ MapArgs m) {
  __shared__ __align__(128) unsigned char patch[kQuantWarps][384];
  pdl_wait();
  pdl_launch_dependents();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (blockIdx.x == 0 && threadIdx.x < 4) m.counters[threadIdx.x] = 0u;
  if (blockIdx.x < map_ctas) {
    const int e = blockIdx.x * kQuantWarps + warp;
    if (e <= m.n_expert) make_maps(m, e, patch[warp], lane);
    return;
  }
  long long b = static_cast<long long>(blockIdx.x - map_ctas) * kQuantWarps + warp;
  const uint16_t* x = x0;
  unsigned char* out = out0;
  if (b >= n0) {
    b -= n0;
    if (b >= n1) return;
    x = x1;
    out = out1;
  } else if (d_rows != nullptr && b >= static_cast<long long>(*d_rows) * nb) {
    return;
  }
  float v[8];
  load_lane8(x + b * kQK, lane, v);
  int q[8], sum;
  const float d = quantize_lane8(v, q, sum);
  uint32_t* o32 = reinterpret_cast<uint32_t*>(out + b * kRowBlk);
  auto pack = [&](int i) {
    return (q[i] & 0xFF) | ((q[i + 1] & 0xFF) << 8) | ((q[i + 2] & 0xFF) << 16) | (static_cast<uint32_t>(q[i + 3] & 0xFF) << 24);
  };
  if (lane == 0) o32[0] = __float_as_uint(d);
  *reinterpret_cast<uint2*>(o32 + 4 + 2 * lane) = make_uint2(pack(0), pack(4));
  if ((lane & 3) == 0) {                           // sub-block lane / 4
    unsigned char* parts = reinterpret_cast<unsigned char*>(o32 + 68) + (lane >> 4) * 8 + ((lane >> 2) & 3);
    parts[0] = static_cast<unsigned char>(sum & 127);
    parts[4] = static_cast<unsigned char>((sum >> 7) & 0xFF);
  }
}

RowsArgs args_of(const ExpertGemm& g, int map0) {
  RowsArgs a{};
  a.maps = static_cast<const unsigned char*>(g.maps);
  a.next = g.counters + map0;
  a.tab0 = g.tab; a.map0 = map0; a.off = g.off; a.rows = g.rows; a.xq = g.xq; a.y = g.y;
  a.n_rows = g.n_rows; a.nb = g.k / kQK; a.n_expert = g.n_expert;
  a.sw0 = a.sw1 = static_cast<const unsigned char*>(g.shared_w);
  a.sxq = g.shared_xq; a.sy = g.shared_y; a.s_rows = g.shared_rows;
  return a;
}

}  // namespace

int gemm_rows_gate_up(const ExpertGemm& g, const unsigned char* const* tab_up, const void* shared_up, cudaStream_t stream) {
  RowsArgs a = args_of(g, 0);
  a.tab1 = tab_up;
  a.sw1 = static_cast<const unsigned char*>(shared_up);
  return g.stream ? launch_rows<true, true>(a, g.routes, stream) : launch_rows<true, false>(a, g.routes, stream);
}
int gemm_rows_down(const ExpertGemm& g, cudaStream_t stream) {
  const RowsArgs a = args_of(g, 2);
  return g.stream ? launch_rows<false, true>(a, g.routes, stream) : launch_rows<false, false>(a, g.routes, stream);
}

int quantize_rows(const uint16_t* x0, void* out0, long long rows0, const int* d_rows, const uint16_t* x1, void* out1, long long rows1,
                  int k, const ExpertMaps& em, bool make_maps, cudaStream_t stream) {
  const int nb = k / kQK;
  const long long ctas = ((rows0 + rows1) * nb + kQuantWarps - 1) / kQuantWarps;
  MapArgs m{};
  if (!map_args(em, make_maps, &m)) return kErrUnsupported;
  const unsigned map_ctas = make_maps && em.maps != nullptr ? static_cast<unsigned>(em.n_expert / kQuantWarps + 1) : 0;
  if (ctas + map_ctas > 0x7FFFFFFF) return kErrUnsupported;
  if (ctas + map_ctas == 0) return kOk;
  return launch_pdl(quantize_rows_kernel, dim3(static_cast<unsigned>(ctas + map_ctas)), kQuantWarps * 32, 0, stream, x0,
                    static_cast<unsigned char*>(out0), rows0 * nb, d_rows, x1, static_cast<unsigned char*>(out1), rows1 * nb, nb, map_ctas, m);
}

}  // namespace sgr
