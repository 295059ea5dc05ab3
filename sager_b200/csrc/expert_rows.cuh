// expert_rows.cuh - the expert kernel for layers with many token rows (part of
// moe_layer.cu, which defines LayerDev and the plan before including this file).
//
// A persistent kernel, one CTA per SM: 16 consumer warps, a preparing warp, a weight warp,
// two activation warps and two finisher warps.
// Work is cut into groups: the 256 (gate, up) row pairs of one block of h of one tile (up to 16
// token rows of one expert) - or half of them where groups are few -, or 256 rows of its down
// matrix. A group is streamed through a ring of three shared-memory stages one super-block column
// at a time: a stage holds the 144-byte blocks of 256 weight rows for one block index, plus
// that block of the tile's activation rows, re-laid for the dot engine. Every
// consumer warp owns sixteen of the rows - eight gate rows
// and the eight up rows of the same indices, so SwiGLU needs no exchange - and
// keeps its sums in registers from the first column to the last: no partial sums
// in shared memory, no barrier between the warps; they synchronise by the stages' mbarriers
// (full; weight part free; activation part free) and, once per block of h, by those of its buffer.
//
// The weight part of a stage arrives by TMA: two tiled copies per stage (boxes of
// 144 bytes x 128 rows) through 2-D tensor maps over [rows][row bytes]. The maps
// are made on the host for a placeholder address; the preparing warp patches a group's
// descriptors some stages ahead of its copies: the expert's base addresses go into shared-memory
// copies (tensormap.replace), are published to a per-CTA ring of descriptors in global
// memory (tensormap.cp_fenceproxy) and acquired by the weight warp before use. (16-byte cp.async
// copies reach the same HBM rate on their own, but every one of them passes through
// the load/store pipe that the consumers' shared-memory loads need; bulk copies of
// 144 bytes are issue-bound at roughly one per 60 cycles and warp.) The activation
// warps copy the stage's block of the tile's activation rows with
// cp.async. The two roles walk the same list of stages independently, so the
// weight stream never waits for an activation row that is not ready yet. Experts
// whose pointers are not 16-byte aligned cannot go through TMA: the weight warp
// copies them with plain loads.
//
// Gate/up groups leave h in shared memory, where the finisher warps quantise it to Q8_K (padded
// 288-byte blocks, 16-byte copyable) and publish the block; half groups exchange their halves through
// global memory first. A down group's activations are copied once its tile's blocks are all
// published; the preparing warp watches for that (bounded) and draws no further group meanwhile.
// Down groups write fp32 y; after a grid-wide barrier the CTAs add
// residual + sum_k w_k * y_k + shared expert (combine_flat).
//
// What bounds it at 64 rows over 256 experts (hidden 2048, n_ff 512, 160 distinct experts under the
// benchmark's skew: 284 MB, 44 us of HBM): 90 us per layer with the route kernel, of which 28 until the
// first stage is there, 65 of streaming - 49 without the arithmetic, whose integer instructions hold the
// stages back -, 7 of barrier and blend (101 with five stages, one finisher and blocks of h shared by two CTAs).
#pragma once

namespace rs {

constexpr int kTok = 16;                        // token rows per tile
constexpr int kConsumerWarps = 16;
constexpr int kConsumers = kConsumerWarps * 32;
constexpr int kXWarps = 2;                      // activation-row producers
constexpr int kXThreads = kXWarps * 32;
constexpr int kPrepWarp = kConsumerWarps, kWeightWarp = kPrepWarp + 1, kFirstXWarp = kWeightWarp + 1, kFinishWarp = kFirstXWarp + kXWarps;
constexpr int kFinishWarps = 2;
constexpr int kThreads = (kFinishWarp + kFinishWarps) * 32;
constexpr int kStageCount = 3;
constexpr int kHalfRows = 128;                  // a stage is two halves of 128 rows
constexpr int kHalfBytes = kHalfRows * kW4;     // 18432
constexpr int kWBytes = 2 * kHalfBytes;
// activation part of a stage: codes [16][272] | int16 sums [16][8] | scales [16] at 16-byte steps
constexpr int kXCodes = kTok * kXqStride;
constexpr int kXBytes = kXCodes + kTok * 16 + kTok * 16;
constexpr int kStageBytes = (kWBytes + kXBytes + 127) & ~127;
constexpr int kHq = 288;                        // padded Q8_K block of h: d | 12 bytes | 256 codes | 8 sums
constexpr int kHdr = 4096;
// The plan of a layer, built by every CTA for itself when the routing was made by this call's own
// route kernel: row masks [E] | offsets [E + 1] | scan scratch | tile records | rows of the slots | slot
// of every route. One round trip for the routing and a few barriers per CTA, all CTAs at once, instead
// of one CTA planning in global memory while 147 wait (8 us per layer at 64 rows).
constexpr int kPlanExperts = 256, kPlanRoutes = 512;
constexpr int kPlanTiles = kPlanExperts + kPlanRoutes / kTok + 8;     // a tile per expert, per further 16 rows, shared expert's
constexpr int kPlanOffMask = 0, kPlanOffOff = kPlanExperts * 8, kPlanOffScan = kPlanOffOff + 1152;
constexpr int kPlanOffRec = kPlanOffScan + 512, kPlanOffRows = kPlanOffRec + kPlanTiles * 16;
constexpr int kPlanOffSlot = kPlanOffRows + kPlanRoutes;               // (a source row is below 64: one byte)
constexpr int kPlanOffTab = kPlanOffSlot + kPlanRoutes * 4;             // the layer's pointer table [3][E]
constexpr int kPlanBytes = (kPlanOffTab + 3 * kPlanExperts * 8 + 127) & ~127;
// h of a gate/up group, [16][256] fp32, two groups in turn (the padded row keeps the consumers' stores off one bank)
constexpr int kHRow = 260;
constexpr int kHBytes = kTok * kHRow * 4;
constexpr size_t kSmem = kHdr + kPlanBytes + static_cast<size_t>(kStageCount) * kStageBytes + 2 * kHBytes;
constexpr int kGateUpPairs = 256;               // pairs per gate/up group: one block of h, streamed as two halves of 128 pairs,
                                                // or one of the halves where groups are few (Sched::split)
constexpr int kDownRows = 256;                  // rows per down group
constexpr int kFullArrivals = 1 + kXThreads;      // weight warp: one arrival; activation warps: a thread's copies landed
constexpr int kAhead = kAheadStages;
constexpr int kMapRing = kAhead + kStageCount + 2;   // descriptor slots per CTA: groups (of one stage at least) that are
                                                 // published and not issued, in flight, and the one being patched

static_assert(kSmem <= 227 * 1024, "ring exceeds shared memory");
static_assert(kMapRing <= kTmapSlots, "the workspace holds kTmapSlots descriptor pairs per CTA");

struct Desc {     // one 16-byte shared-memory load per stage and warp
  int flags;     // bit 0 kind (0 gate/up, 1 down), bit 1 expert absent, bits 2-7 token rows,
                 // bits 8-15 block column, bit 16 last column, bit 17 end of this CTA's list,
                 // bit 18 second half of a gate/up group, bits 20-31 group number in this CTA
  int tile;
  int hrow0;     // first h / y row of the tile
  int row0;      // first pair (gate/up) or first row (down) of the group
  __device__ __forceinline__ int kind() const { return flags & 1; }
  __device__ __forceinline__ int absent() const { return (flags >> 1) & 1; }
  __device__ __forceinline__ int ntok() const { return (flags >> 2) & 63; }
  __device__ __forceinline__ int blk() const { return (flags >> 8) & 255; }
  __device__ __forceinline__ int last() const { return (flags >> 16) & 1; }
  __device__ __forceinline__ int end() const { return (flags >> 17) & 1; }     // no more stages for this CTA
  __device__ __forceinline__ int half() const { return (flags >> 18) & 1; }
  __device__ __forceinline__ int seq() const { return (flags >> 20) & 4095; }
};

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
// arrive on `bar` once every cp.async this thread has issued so far has landed
__device__ __forceinline__ void cp_async_arrive(uint64_t* bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// The service warps' wait: they wait most of the time, and their polls took a fifth of the issue slots that the consumers need.
__device__ __forceinline__ bool mbar_wait_idle(uint64_t* bar, uint32_t parity) {
  for (int it = 0; it < (1 << 20); ++it) {
    if (mbar_try_wait(bar, parity)) return true;
    __nanosleep(40);
  }
  return false;
}
__device__ __forceinline__ void rs_consumers_sync() {
  asm volatile("bar.sync 5, %0;" ::"n"(kConsumers) : "memory");
}

// Groups are handed out dynamically, in one global order: every gate/up group of the
// layer (tile-major), then every down group. A CTA starts with group blockIdx.x and takes
// further ones from a global counter; its weight warp draws the next number while it
// streams the current group and publishes the CTA's list in shared memory for the other
// roles. Equal finishing times need no cost model this way, and a tile's down groups are
// drawn long after its gate/up groups were (the whole gate/up list lies between).
struct Group {
  int kind, tile, gi, nb;        // 0 gate/up / 1 down, tile, group inside the tile, stages
  bool valid;
};
struct Sched {
  int n_gu, total, nbh, nbf, gpt_gu, gpt_dn;
  int split;                     // 1: a gate/up group is half a block of h (bit 0 of gi tells which)
  __device__ __forceinline__ Group decode(int g) const {
    Group r;
    r.valid = g >= 0 && g < total;
    r.kind = g >= n_gu ? 1 : 0;
    const int local = r.kind ? g - n_gu : g;
    const int gpt = r.kind ? gpt_dn : gpt_gu;
    r.tile = r.valid ? local / gpt : 0;
    r.gi = local - r.tile * gpt;
    r.nb = r.kind ? nbf : (2 - split) * nbh;
    return r;
  }
};
constexpr int kListSlots = 16;

// One entry of a CTA's group list, published by the preparing warp some stages ahead of the copies,
// with everything the other roles would otherwise fetch from global memory again. A reader lags by at
// most kAhead + kStageCount + 1 groups and the two whose h waits for the finisher warp.
struct alignas(16) GEntry {
  int id;          // global group number, -1 = end of this CTA's list
  int bits;        // bit 0: the expert's pointers are null; bit 1: they are 16-byte aligned
  const unsigned char* maps;    // the group's descriptors
  int4 rc;         // the tile's record: expert, token rows, first h / y row, first entry of grows
  const unsigned char* w[3];    // the expert's matrices
  unsigned char rows[kTok];     // gate/up groups: source row of the tile's token slot t in the quantised inputs
  volatile int there;           // down groups: the tile's h has been seen complete
};
static_assert(kListSlots > kAhead + kStageCount + 1 + 2, "a reader could be overtaken");
static_assert(sizeof(GEntry) * kListSlots + 2048 <= kHdr, "group list exceeds the header");

// One warp: Q8_K-quantise block `hb` of h, rows `src` in shared memory, into the padded rows
// [hrow0, hrow0 + ntok) of L.hq (arithmetic of src/kernels/cpu/q4_avx2.cpp:77-94 in the reference,
// the same as stage_quantized_f32). The down groups of the tile wait for it, and beside sixteen
// consumer warps a chain of instructions takes ten cycles each: R rows go through it side by side
// (one after the other, a row took 0.85 us).
template <int R>
__device__ __forceinline__ void quantize_h_rows(const LayerDev& L, const float* src, int hrow0, int ntok, int hb, int lane) {
  const size_t hq_stride = static_cast<size_t>(L.nbf) * kHq;
  float4 a[R], b[R];
#pragma unroll
  for (int u = 0; u < R; ++u) {
    const float4* p = reinterpret_cast<const float4*>(src + min(u, ntok - 1) * kHRow) + lane * 2;
    a[u] = p[0];
    b[u] = p[1];
  }
  uint32_t lo[R], hi[R], sums[R];
  float d[R];
#pragma unroll
  for (int u = 0; u < R; ++u) {
    const float v[8] = {a[u].x, a[u].y, a[u].z, a[u].w, b[u].x, b[u].y, b[u].z, b[u].w};
    int q[8], sum;
    d[u] = quantize_lane8(v, q, sum);
    lo[u] = (q[0] & 0xFF) | ((q[1] & 0xFF) << 8) | ((q[2] & 0xFF) << 16) | (static_cast<uint32_t>(q[3] & 0xFF) << 24);
    hi[u] = (q[4] & 0xFF) | ((q[5] & 0xFF) << 8) | ((q[6] & 0xFF) << 16) | (static_cast<uint32_t>(q[7] & 0xFF) << 24);
    sums[u] = (static_cast<uint32_t>(sum) & 0xFFFFu) | (static_cast<uint32_t>(__shfl_down_sync(0xFFFFFFFFu, sum, 4)) << 16);
  }
#pragma unroll
  for (int u = 0; u < R; ++u) {
    if (u >= ntok) break;                        // warp-uniform
    uint32_t* o32 = reinterpret_cast<uint32_t*>(L.hq + static_cast<size_t>(hrow0 + u) * hq_stride + hb * kHq);
    if (lane == 0) o32[0] = __float_as_uint(d[u]);
    *reinterpret_cast<uint2*>(o32 + 4 + 2 * lane) = make_uint2(lo[u], hi[u]);
    if ((lane & 7) == 0) o32[68 + (lane >> 3)] = sums[u];
  }
}
// (batches of four rows in turn between the finisher warps, `f` is this one's number)
__device__ __forceinline__ void quantize_h_block(const LayerDev& L, const float* src, int hrow0, int ntok, int hb, int f, int lane) {
#pragma unroll 1
  for (int t0 = 4 * f; t0 < ntok; t0 += 4 * kFinishWarps) {
    if (ntok - t0 > 2) quantize_h_rows<4>(L, src + t0 * kHRow, hrow0 + t0, ntok - t0, hb, lane);
    else quantize_h_rows<2>(L, src + t0 * kHRow, hrow0 + t0, ntok - t0, hb, lane);
  }
}

// Half a super-block (sub-blocks 4 * half .. 4 * half + 3) of one weight row against a tile's only token row, for a
// pair of adjacent lanes that share the weight row: the integer sums of the two halves are added across the pair before
// the one fp32 rounding, so the result equals block_dot's. `x` is the activation part of the stage. The consumers'
// integer pipe bounds the stage: odd sub-blocks stay sixteen-fold. (From two rows on the MMA below costs less: 64 rows
// over 256 experts 90.4 -> 88.8 us per layer, 8 rows 50.8 -> 49.6; at one row it loses, 93.6 and 55.2.)
__device__ __forceinline__ float half_dot(const uint4& hdr, const uint4 (&wq)[4], int half, const unsigned char* x) {
  const Scales6 s6 = unpack_scales6(hdr.y, hdr.z, hdr.w);
  const uint32_t scw = half ? s6.sc[1] : s6.sc[0], mnw = half ? s6.mn[1] : s6.mn[0];
  const unsigned char* codes = x + half * 144;                 // (the second half of a block lies 16 bytes further on)
  int isum = 0, hsum = 0;                                      // hsum: sixteen-fold, below 2^29
#pragma unroll
  for (int gg = 0; gg < 2; ++gg) {
    const uint4 q0 = wq[2 * gg], q1 = wq[2 * gg + 1];
    const uint32_t raw[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
    uint32_t lo[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) lo[i] = raw[i] & 0x0F0F0F0Fu;
    const uint4* xa = reinterpret_cast<const uint4*>(codes + 64 * gg);
    const uint4 x0 = xa[0], x1 = xa[1], x2 = xa[2], x3 = xa[3];
    isum += static_cast<int>(__byte_perm(scw, 0, 0x4440 + 2 * gg)) * dot8(lo, x0, x1);
    hsum += static_cast<int>(__byte_perm(scw, 0, 0x4441 + 2 * gg)) * dot8_high(raw, x2, x3);
  }
  const uint2 bs = *reinterpret_cast<const uint2*>(x + kXCodes + half * 8);
  const int min_sum = __dp2a_hi(static_cast<int>(bs.y), static_cast<int>(mnw), __dp2a_lo(static_cast<int>(bs.x), static_cast<int>(mnw), 0));
  const int mine = isum + (hsum >> 4);
  const int is = mine + __shfl_xor_sync(0xFFFFFFFFu, mine, 1);
  const int ms = min_sum + __shfl_xor_sync(0xFFFFFFFFu, min_sum, 1);
  const float d = h2f(static_cast<uint16_t>(hdr.x & 0xFFFFu)), dmin = h2f(static_cast<uint16_t>(hdr.x >> 16));
  return *reinterpret_cast<const float*>(x + kXCodes + kTok * 16) * (d * static_cast<float>(is) - dmin * static_cast<float>(ms));
}

// Every thread of the CTA: the plan of build_plan (moe_layer.cu) in shared memory - same masks, same
// tile order (shared expert's tiles, tiles of more than half a tile's rows, the rest, each in expert
// order), same slots. CTA 0 also silences rows with ids outside [0, E) as moe_dispatch_scan does
// (moe.cu:385-398 of the reference) and leaves the counts in meta. Returns the number of tiles.
__device__ __forceinline__ int build_plan_shared(const LayerDev& L, unsigned char* ps, int tid) {
  unsigned long long* mask = reinterpret_cast<unsigned long long*>(ps + kPlanOffMask);
  int* off_s = reinterpret_cast<int*>(ps + kPlanOffOff);
  int* scan = reinterpret_cast<int*>(ps + kPlanOffScan);          // [3][40]: warp totals of rows, tiles, heavy tiles; [120]: bad ids
  int4* rec_s = reinterpret_cast<int4*>(ps + kPlanOffRec);
  unsigned char* rows_s = ps + kPlanOffRows;
  int* slot_s = reinterpret_cast<int*>(ps + kPlanOffSlot);
  const int lane = tid & 31, wp = tid >> 5;
  const int total = L.n * L.K;
  // (the masks and the count of bad ids were cleared before the wait for the route kernel)
  for (int i = tid; i < 3 * L.E; i += kThreads) {                 // the layer's pointer table, beside everything else
    const int m = i >= 2 * L.E ? 2 : (i >= L.E ? 1 : 0);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(ps + kPlanOffTab + i * 8)),
                 "l"(L.tab + static_cast<size_t>(m) * L.tab_stride + (i - m * L.E)) : "memory");
  }
  int my_e = -1, my_r = 0;
  if (tid < total) {                            // kPlanRoutes <= kThreads: a route per thread
    my_r = tid / L.K;
    const int kk = tid - my_r * L.K;
    my_e = __ldcg(L.idx + static_cast<size_t>(my_r) * L.rstride + kk);
    if (my_e < 0 || my_e >= L.E) {
      if (blockIdx.x == 0) {
        for (int q = 0; q <= L.K; ++q) L.w[static_cast<size_t>(my_r) * L.rstride + q] = 0.f;
        atomicAdd(&scan[120], 1);
      }
      my_e = -1;
    } else if (my_e >= L.e_lo && my_e < L.e_hi) {
      atomicOr(&mask[my_e], 1ull << my_r);
    } else {
      my_e = -1;
    }
  }
  __syncthreads();
  auto is_heavy = [](int rows_in_tile) { return 2 * rows_in_tile > kTok; };
  int c = 0, t = 0, h = 0;
  if (tid < L.E) {
    c = __popcll(mask[tid]);
    t = (c + kTok - 1) / kTok;
    h = c / kTok + (is_heavy(c % kTok) ? 1 : 0);
  }
  int ic = c, it = t, ih = h;                   // inclusive scans inside the warps that hold experts
  if (tid < kPlanExperts) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int uc = __shfl_up_sync(0xFFFFFFFFu, ic, o), ut = __shfl_up_sync(0xFFFFFFFFu, it, o);
      const int uh = __shfl_up_sync(0xFFFFFFFFu, ih, o);
      if (lane >= o) { ic += uc; it += ut; ih += uh; }
    }
    if (lane == 31) { scan[wp] = ic; scan[40 + wp] = it; scan[80 + wp] = ih; }
  }
  __syncthreads();
  int rows_total = 0, tiles_total = 0, heavy_total = 0, pc = 0, pt = 0, phv = 0;
#pragma unroll
  for (int w = 0; w < kPlanExperts / 32; ++w) {
    if (w < wp) { pc += scan[w]; pt += scan[40 + w]; phv += scan[80 + w]; }
    rows_total += scan[w]; tiles_total += scan[40 + w]; heavy_total += scan[80 + w];
  }
  const int sh_tiles = (L.sh[0] != nullptr && L.sh_hi > L.sh_lo) ? (L.sh_hi - L.sh_lo + kTok - 1) / kTok : 0;
  if (tid < L.E) {
    const int ar = pc + ic - c;                 // exclusive prefixes of this expert
    int at_heavy = sh_tiles + (phv + ih - h), at_light = sh_tiles + heavy_total + ((pt + it - t) - (phv + ih - h));
    off_s[tid] = ar;
    for (int t0 = 0; t0 < c; t0 += kTok) {
      const int ct = min(kTok, c - t0);
      const int at = is_heavy(ct) ? at_heavy++ : at_light++;
      rec_s[at] = make_int4(tid, ct, ar + t0, ar + t0);
    }
  }
  if (tid == 0) off_s[L.E] = rows_total;
  if (tid < sh_tiles) {
    const int t0 = tid * kTok;
    rec_s[tid] = make_int4(L.E, min(kTok, L.sh_hi - L.sh_lo - t0), L.n_max * L.K + L.sh_lo + t0, L.sh_lo + t0);
  }
  __syncthreads();
  if (tid < total) {
    int pos = -1;
    if (my_e >= 0) {
      pos = off_s[my_e] + __popcll(mask[my_e] & ((1ull << my_r) - 1ull));
      rows_s[pos] = static_cast<unsigned char>(my_r);
    }
    slot_s[tid] = pos;
  }
  if (blockIdx.x == 0 && tid == 0) {
    L.meta[0] = rows_total;
    L.meta[1] = tiles_total + sh_tiles;
    L.meta[2] = scan[120];
    L.meta[3] = sh_tiles;
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  return tiles_total + sh_tiles;
}

// STREAM: weights first to leave L2 (streams_weights)
template <bool STREAM>
__global__ void __launch_bounds__(kThreads, 1) expert_rows_kernel(const LayerDev L) {
  extern __shared__ __align__(128) unsigned char smem[];
  uint64_t* full = reinterpret_cast<uint64_t*>(smem);
  uint64_t* empty = reinterpret_cast<uint64_t*>(smem + 64);      // a stage's activation part may be refilled
  uint64_t* wempty = reinterpret_cast<uint64_t*>(smem + 192);    // a stage's weight part may be refilled
  int* flag = reinterpret_cast<int*>(smem + 128);
  uint64_t* hfull = reinterpret_cast<uint64_t*>(smem + 160);     // [2] h of a gate/up group is in shared memory
  uint64_t* hempty = reinterpret_cast<uint64_t*>(smem + 176);    // [2] ... and has been quantised
  Desc* desc = reinterpret_cast<Desc*>(smem + 384);
  unsigned char* plan_s = smem + kHdr;
  unsigned char* stages = smem + kHdr + kPlanBytes;
  float* hs = reinterpret_cast<float*>(stages + static_cast<size_t>(kStageCount) * kStageBytes);   // [2][16][kHRow]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  if (tid == 0) {
    for (int s = 0; s < kStageCount; ++s) {
      mbar_init(&full[s], kFullArrivals);
      mbar_init(&empty[s], kConsumerWarps);
      mbar_init(&wempty[s], kConsumerWarps);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&hfull[s], kConsumerWarps);
      mbar_init(&hempty[s], kFinishWarps);
    }
    *reinterpret_cast<volatile unsigned*>(smem + 144) = 0u;
    *reinterpret_cast<volatile unsigned*>(smem + 148) = 0u;
    fence_barrier_init();
  }
  if (L.plan_in_kernel) {           // shared memory of the plan that must start out clear
    for (int e = tid; e < kPlanExperts; e += kThreads) reinterpret_cast<unsigned long long*>(plan_s + kPlanOffMask)[e] = 0ull;
    if (tid == 0) reinterpret_cast<int*>(plan_s + kPlanOffScan)[120] = 0;
  }
  unsigned char* smaps = smem + 1024;                                 // three 128-byte descriptors being patched
  uint32_t* tmpl = reinterpret_cast<uint32_t*>(smem + 1408);          // the two host-made descriptors
  if (tid == kPrepWarp * 32) {
#pragma unroll
    for (int i = 0; i < 32; ++i) {               // constant indices only (see LayerDev)
      tmpl[i] = L.tmap_gu[i];
      tmpl[32 + i] = L.tmap_dn[i];
    }
  }
  __syncthreads();
  pdl_wait();                       // routing and quantised rows (and, without a plan of its own, the plan) come from the route kernel
  pdl_launch_dependents();

  Sched sc;
  sc.gpt_dn = L.H / kDownRows;      // groups per tile
  sc.nbh = L.nbh; sc.nbf = L.nbf;
  // the plan: this CTA's own copy in shared memory, or the one a plan kernel left in the workspace
  const bool plan_own = L.plan_in_kernel != 0;
  if (plan_own && L.wait_flags != nullptr) {
    // owner side of an expert-parallel layer: the routing is in the records the home ranks store into
    // this rank's memory; every CTA waits (bounded) for their arrival words. A word that never comes
    // raises the status; the CTA then goes on with the records of an earlier step (valid memory).
    if (tid < L.wait_count) {
      const unsigned want = *L.wait_step * L.wait_mul + L.wait_add;
      unsigned it = 0, v;
      do {
        asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(L.wait_flags + tid) : "memory");
      } while (static_cast<int>(v - want) < 0 && ++it < L.wait_limit && (__nanosleep(64), true));
      if (static_cast<int>(v - want) < 0) atomicExch(L.status, 8);
    }
    __syncthreads();
  }
  const int n_tiles = plan_own ? build_plan_shared(L, plan_s, tid) : L.meta[1];
  const int4* rec_p = plan_own ? reinterpret_cast<const int4*>(plan_s + kPlanOffRec) : L.rec;
  const int* slot_p = plan_own ? reinterpret_cast<const int*>(plan_s + kPlanOffSlot) : L.gslot;
  auto tile_rec = [&](int tile) { return plan_own ? rec_p[tile] : __ldcg(rec_p + tile); };
  // Groups of whole blocks quantise their h in the CTA; with fewer of them than two thirds of the CTAs, halves of a block
  // and an exchange through global memory are faster (us per layer: hidden 2048, n_ff 512, 5 rows, 82 blocks: 44.6
  // against 47.2, 8 rows, 118 blocks: 52.4 against 51.4).
  sc.split = 3 * n_tiles * L.nbf < 2 * static_cast<int>(gridDim.x) ? 1 : 0;
  sc.gpt_gu = L.nbf << sc.split;
  sc.n_gu = n_tiles * sc.gpt_gu;
  sc.total = sc.n_gu + n_tiles * sc.gpt_dn;
  const int rb_h = L.nbh * kW4, rb_f = L.nbf * kW4;
  GEntry* glist = reinterpret_cast<GEntry*>(smem + 2048);                       // [kListSlots] this CTA's groups
  volatile unsigned* g_pub = reinterpret_cast<volatile unsigned*>(smem + 144);  // entries of glist published
  volatile unsigned* issued = reinterpret_cast<volatile unsigned*>(smem + 148); // stages the weight warp has issued
  // a follower role's k-th group (bounded wait for the preparing warp to publish it)
  auto follow = [&](int k, bool& ok) -> const GEntry* {
    unsigned it = 0;
    if (lane == 0)
      while (*g_pub <= static_cast<unsigned>(k) && ++it < kSpinLimit) __nanosleep(20);
    it = __shfl_sync(0xFFFFFFFFu, it, 0);
    ok = it < kSpinLimit;
    __threadfence_block();
    return glist + k % kListSlots;
  };

  if (warp == kPrepWarp) {
    // ---------------- preparing warp ----------------
    // Draws the CTA's groups and publishes each with its record, pointers and patched descriptors: three
    // dependent round trips and the descriptor proxies' fences per group (2.5 us together), which the
    // weight warp, when it did them between its copies, could not hide behind a down group's two stages.
    // A number drawn is a group that no other CTA can take, and a gate/up group that waits long for its
    // CTA delays its tile's h, on which the down groups elsewhere depend: so a number is drawn only when
    // the weight warp has kAhead published stages or fewer left.
    unsigned char* gmaps = L.tmaps + static_cast<size_t>(blockIdx.x) * kMapRing * 2 * 128;
    const unsigned char* const* ptab = reinterpret_cast<const unsigned char* const*>(plan_s + kPlanOffTab);
    unsigned planned = 0;                        // stages of the groups published so far
    int drawn = blockIdx.x;                      // the first group is this CTA's own number
    bool have = true;
    int map_seq = 0;
    for (int k = 0;; ++k) {
      unsigned it = 0;
      if (lane == 0) {
        while (planned - *issued > static_cast<unsigned>(kAhead) && ++it < kSpinLimit) __nanosleep(20);
        if (!have) drawn = static_cast<int>(atomicAdd(&L.cnt[10], 1u));
      }
      it = __shfl_sync(0xFFFFFFFFu, it, 0);
      if (it >= kSpinLimit) {
        if (lane == 0) atomicExch(L.status, 2);
        return;
      }
      const int id = __shfl_sync(0xFFFFFFFFu, drawn, 0);
      const Group g = sc.decode(id);
      int4 rc = make_int4(0, 0, 0, 0);
      const unsigned char *w0 = nullptr, *w1 = nullptr, *w2 = nullptr, *maps = nullptr;
      int row = 0;
      unsigned ready = 0u;
      bool absent = false, aligned = true;
      have = false;
      if (g.valid) {
        rc = tile_rec(g.tile);
        const bool shared = rc.x == L.E;
        // a down group's activation rows are the tile's quantised h: seen complete here (acquire)
        if (g.kind == 1) {
          ready = ld_acquire(L.ready + g.tile);
          have = ready >= static_cast<unsigned>(kFinishWarps * L.nbf);     // a short group: its successor's number at hand when it starts
          if (have && lane == 0) drawn = static_cast<int>(atomicAdd(&L.cnt[10], 1u));
          have = __any_sync(0xFFFFFFFFu, have && lane == 0);
        }
        w0 = shared ? L.sh[0] : (plan_own ? ptab[rc.x] : L.tab[rc.x]);
        w1 = shared ? L.sh[1] : (plan_own ? ptab[L.E + rc.x] : L.tab[L.tab_stride + rc.x]);
        w2 = shared ? L.sh[2] : (plan_own ? ptab[2 * L.E + rc.x] : L.tab[2 * L.tab_stride + rc.x]);
        if (g.kind == 0 && lane < rc.y)
          row = shared ? rc.w + lane : (plan_own ? plan_s[kPlanOffRows + rc.w + lane] : __ldcg(L.grows + rc.w + lane));
        absent = w0 == nullptr || w1 == nullptr || w2 == nullptr;
        aligned = ((reinterpret_cast<uintptr_t>(w0) | reinterpret_cast<uintptr_t>(w1) | reinterpret_cast<uintptr_t>(w2)) & 15u) == 0;
        if (!absent && aligned) {
          // descriptors of the matrices this group reads (gate and up, or down), in the next slot of the
          // CTA's ring: the ring keeps the descriptors of earlier groups intact while their copies fly
          unsigned char* slot = gmaps + static_cast<size_t>(map_seq % kMapRing) * 2 * 128;
          ++map_seq;
          uint32_t* m = reinterpret_cast<uint32_t*>(smaps);
          if (g.kind == 0) {
            m[lane] = tmpl[lane];
            m[32 + lane] = tmpl[lane];
            __syncwarp();
            if (lane == 0) {
              tmap_replace_addr(smaps, w0);
              tmap_replace_addr(smaps + 128, w1);
            }
            __syncwarp();
            tmap_publish(slot, smaps);
            tmap_publish(slot + 128, smaps + 128);
          } else {
            m[64 + lane] = tmpl[32 + lane];
            __syncwarp();
            if (lane == 0) tmap_replace_addr(smaps + 256, w2);
            __syncwarp();
            tmap_publish(slot, smaps + 256);
          }
          __syncwarp();
          maps = slot;
        }
      }
      GEntry* e = glist + k % kListSlots;
      if (lane < kTok) e->rows[lane] = static_cast<unsigned char>(row);
      if (lane == 0) {
        e->id = g.valid ? id : -1;
        e->bits = (absent ? 1 : 0) | (aligned ? 2 : 0);
        e->there = have ? 1 : 0;
        e->maps = maps;
        e->rc = rc;
        e->w[0] = w0; e->w[1] = w1; e->w[2] = w2;
      }
      __syncwarp();
      if (lane == 0) {
        __threadfence_block();
        *g_pub = static_cast<unsigned>(k) + 1u;
      }
      if (!g.valid) return;
      planned += static_cast<unsigned>(g.nb);
      if (g.kind == 1 && !have && !absent) {
        // its h is not there yet: no further groups until it is. (A CTA early to the down groups would otherwise
        // fill its ring with them and keep them to itself, while the CTAs that make the h end up with none.)
        it = 0;
        // (one poller per CTA, which tells the activation warps: more of them slowed the counters they wait for)
        if (lane == 0) {
          while (ld_acquire(L.ready + g.tile) < static_cast<unsigned>(kFinishWarps * L.nbf) && ++it < kSpinLimit) __nanosleep(50);
          __threadfence_block();
          if (it < kSpinLimit) e->there = 1;
        }
        it = __shfl_sync(0xFFFFFFFFu, it, 0);
        if (it >= kSpinLimit) {
          if (lane == 0) atomicExch(L.status, 4);
          return;
        }
      }
    }
  }

  if (warp == kWeightWarp) {
    // ---------------- weight warp: the copies of the published groups, stage by stage ----------------
    int q = 0, s = 0;
    unsigned ph = 0;
    for (int k = 0;; ++k) {
      bool got;
      const GEntry* ge = follow(k, got);
      if (!got) {
        if (lane == 0) atomicExch(L.status, 7);
        return;
      }
      const Group wk = sc.decode(ge->id);
      if (!wk.valid) {                           // end of the list: one last stage that only says so
        if (!mbar_wait_idle(&wempty[s], ph ^ 1u)) {
          if (lane == 0) atomicExch(L.status, 2);
          return;
        }
        if (lane == 0) {
          Desc d;
          d.flags = 1 << 17; d.tile = 0; d.hrow0 = 0; d.row0 = 0;
          desc[s] = d;
          mbar_arrive(&full[s]);
        }
        return;
      }
      const int4 rc = ge->rc;
      const bool absent = (ge->bits & 1) != 0, aligned = (ge->bits & 2) != 0;
      const unsigned char* maps = ge->maps;
      if (!absent && aligned && lane == 0) {
        if (wk.kind == 0) {
          tmap_acquire(maps);
          tmap_acquire(maps + 128);
        } else {
          tmap_acquire(maps);
        }
      }
      const int cols = wk.kind == 0 ? L.nbh : L.nbf;
      for (int i = 0; i < wk.nb; ++i) {
        int half = 0, row0 = wk.gi * kDownRows, blk = i;
        if (wk.kind == 0) {
          half = sc.split ? wk.gi & 1 : (i >= cols ? 1 : 0);
          row0 = (wk.gi >> sc.split) * kGateUpPairs + half * kHalfRows;
          if (i >= cols) blk -= cols;
        }
        if (!mbar_wait_idle(&wempty[s], ph ^ 1u)) {
          if (lane == 0) atomicExch(L.status, 2);
          return;
        }
        unsigned char* st = stages + static_cast<size_t>(s) * kStageBytes;
        if (lane == 0) {
          Desc d;
          d.flags = wk.kind | (absent ? 2 : 0) | (rc.y << 2) | (blk << 8) | (blk == cols - 1 ? 1 << 16 : 0) |
                    (half << 18) | ((k & 4095) << 20);
          d.tile = wk.tile; d.hrow0 = rc.z; d.row0 = row0;
          desc[s] = d;
        }
        if (!absent && aligned) {
          if (lane == 0) {
            mbar_expect_tx(&full[s], kWBytes);      // this lane's arrival, with the bytes to come
            if (wk.kind == 0) {
              tma_load_box<STREAM>(st, maps, blk * kW4, row0, &full[s]);
              tma_load_box<STREAM>(st + kHalfBytes, maps + 128, blk * kW4, row0, &full[s]);
            } else {
              tma_load_box<STREAM>(st, maps, blk * kW4, row0, &full[s]);
              tma_load_box<STREAM>(st + kHalfBytes, maps, blk * kW4, row0 + kHalfRows, &full[s]);
            }
          }
        } else {
          if (!absent) {                           // sources without 16-byte alignment: plain loads
            const unsigned char *b0, *b1;
            int rb;
            if (wk.kind == 0) {
              rb = rb_h;
              b0 = ge->w[0] + static_cast<size_t>(row0) * rb_h + blk * kW4;
              b1 = ge->w[1] + static_cast<size_t>(row0) * rb_h + blk * kW4;
            } else {
              rb = rb_f;
              b0 = ge->w[2] + static_cast<size_t>(row0) * rb_f + blk * kW4;
              b1 = b0 + static_cast<size_t>(kHalfRows) * rb_f;
            }
            const uintptr_t a0 = reinterpret_cast<uintptr_t>(b0), a1 = reinterpret_cast<uintptr_t>(b1);
            warp_copy_unaligned(st, 2 * kHalfBytes / 16, lane, a0 | a1, ((a0 ^ a1) & 2u) != 0, [&](int p) {
              const int r = p / 9, h = r / kHalfRows;
              return (h ? b1 : b0) + static_cast<size_t>(r - h * kHalfRows) * rb + (p - r * 9) * 16;
            });
            asm volatile("cp.async.wait_all;" ::: "memory");
            fence_proxy_async();                   // the next fill of this stage may come from the TMA unit
          }
          __syncwarp();                            // every lane's part of the stage (and of its descriptor) is written
          if (lane == 0) mbar_arrive(&full[s]);
        }
        __syncwarp();
        ++q;
        if (lane == 0) *issued = static_cast<unsigned>(q);
        if (++s == kStageCount) { s = 0; ph ^= 1u; }
      }
    }
  }

  if (warp >= kFirstXWarp && warp < kFirstXWarp + kXWarps) {
    // ---------------- activation warps ----------------
    const int xtid = tid - kFirstXWarp * 32;
    int myoff = 0;                              // lane t < 16: byte offset of token slot t's row
    int s = 0;                                  // ring position and its phase
    unsigned ph = 0;
    for (int k = 0;; ++k) {
      bool got;
      const GEntry* ge = follow(k, got);
      if (!got) {
        if (lane == 0) atomicExch(L.status, 7);
        return;
      }
      const Group wk = sc.decode(ge->id);
      const int4 rc = ge->rc;
      const bool absent = (ge->bits & 1) != 0;
      if (!wk.valid) {                           // end of the list: count in at the last stage and leave
        if (!mbar_wait_idle(&empty[s], ph ^ 1u)) {
          if (lane == 0) atomicExch(L.status, 2);
          return;
        }
        cp_async_arrive(&full[s]);
        return;
      }
      myoff = 0;
      if (wk.kind == 0) {
        if (lane < rc.y) myoff = ge->rows[lane] * L.xq16_stride;
      } else {
        if (lane < rc.y) myoff = (rc.z + lane) * L.nbf * kHq;
        if (!absent) {                        // the tile's h must be quantised and published
          unsigned it = 0;
          if (lane == 0)
            while (ge->there == 0 && ++it < kSpinLimit) __nanosleep(20);
          it = __shfl_sync(0xFFFFFFFFu, it, 0);
          __threadfence_block();
          if (it >= kSpinLimit) {
            if (lane == 0) atomicExch(L.status, 4);
            return;
          }
        }
      }
      for (int i = 0; i < wk.nb; ++i) {
      const int blk = wk.kind == 0 && i >= L.nbh ? i - L.nbh : i;
      if (!mbar_wait_idle(&empty[s], ph ^ 1u)) {
        if (lane == 0) atomicExch(L.status, 2);
        return;
      }
      unsigned char* xs = stages + static_cast<size_t>(s) * kStageBytes + kWBytes;
      if (!absent) {
        // 288-byte blocks (quantised inputs for gate/up, quantised h for down): 16-byte copies
        const unsigned char* xsrc = (wk.kind == 0 ? L.xq16 : L.hq) + blk * kHq;
        const int total = rc.y * (kHq / 16);
        for (int base = 0; base < total; base += kXThreads) {      // warp-uniform trip count
          const int p = base + xtid;
          const bool valid = p < total;
          const int t = valid ? p / (kHq / 16) : 0;
          const int c = p - t * (kHq / 16);
          const int off = __shfl_sync(0xFFFFFFFFu, myoff, t);
          if (valid) {
            // scale | codes (second half of the block 16 bytes further on: see XTile::mid_pad) | sums
            unsigned char* dst = c == 0 ? xs + kXCodes + kTok * 16 + t * 16
                                        : (c <= 16 ? xs + t * kXqStride + (c - 1) * 16 + (c > 8 ? 16 : 0)
                                                   : xs + kXCodes + t * 16);
            cp_async16(dst, xsrc + off + c * 16);
          }
        }
      }
      cp_async_arrive(&full[s]);
      if (++s == kStageCount) { s = 0; ph ^= 1u; }
      }   // block columns of the group
    }
  }

  if (warp >= kFinishWarp) {
    // ---------------- finisher warps ----------------
    // Take the finished gate/up groups of this CTA in order: quantise the group's block of h for the
    // tile's rows from shared memory and publish it, each its own rows. A group of half a block leaves its
    // half in global memory first; the CTA that comes second takes the other half from there and
    // quantises. The consumers never wait for any of this, except for a buffer to be free again two
    // groups later.
    const int f = warp - kFinishWarp;
    for (int g = 0;; ++g) {
      bool got;
      const GEntry* ge = follow(g, got);
      if (!got) {
        if (lane == 0) atomicExch(L.status, 7);
        return;
      }
      const Group wk = sc.decode(ge->id);
      if (!wk.valid || wk.kind == 1) return;     // a CTA's gate/up groups all come before its down groups
      const int4 rc = ge->rc;
      const bool absent = (ge->bits & 1) != 0;
      const int buf = g & 1;
      if (!__all_sync(0xFFFFFFFFu, mbar_wait_idle(&hfull[buf], (g >> 1) & 1))) {
        if (lane == 0) atomicExch(L.status, 6);
        return;
      }
      float* hb = hs + buf * kTok * kHRow;
      const int blk = wk.gi >> sc.split;
      bool mine = !absent;
      if (sc.split && !absent) {
        const int half = wk.gi & 1;
        float* own = L.hbuf + static_cast<size_t>(rc.z) * L.FF + blk * kQK + half * kHalfRows + lane * 4;
        for (int t = 4 * f; t < rc.y; t = (t & 3) == 3 ? t + 1 + 4 * (kFinishWarps - 1) : t + 1)
          *reinterpret_cast<float4*>(own + static_cast<size_t>(t) * L.FF) = *reinterpret_cast<const float4*>(hb + t * kHRow + half * kHalfRows + lane * 4);
        __syncwarp();
        unsigned old = 0;
        if (lane == 0)
          asm volatile("atom.acq_rel.gpu.global.or.b32 %0, [%1], %2;" : "=r"(old) : "l"(L.tile_cnt + 2 * wk.tile + f), "r"(1u << blk) : "memory");
        mine = (__shfl_sync(0xFFFFFFFFu, old, 0) >> blk & 1u) != 0;
        __syncwarp();
        if (mine) {
          const float* other = L.hbuf + static_cast<size_t>(rc.z) * L.FF + blk * kQK + (half ^ 1) * kHalfRows + lane * 4;
          for (int t0 = 4 * f; t0 < rc.y; t0 += 4 * kFinishWarps) {
            float4 v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u)
              v[u] = __ldcg(reinterpret_cast<const float4*>(other + static_cast<size_t>(min(t0 + u, rc.y - 1)) * L.FF));
#pragma unroll
            for (int u = 0; u < 4; ++u)
              if (t0 + u < rc.y) *reinterpret_cast<float4*>(hb + (t0 + u) * kHRow + (half ^ 1) * kHalfRows + lane * 4) = v[u];
          }
          __syncwarp();
        }
      }
      if (mine) quantize_h_block(L, hb, rc.z, rc.y, blk, f, lane);
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&hempty[buf]);
        // (the release is cumulative: it covers the other lanes' stores, ordered before it by the warp barrier)
        if (mine) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(L.ready + wk.tile) : "memory");
      }
    }
    return;
  }

  // ---------------- consumers ----------------
  float acc[2][4];                               // (one token row: acc[0][0])
  bool ok = true;
  // offsets in a stage, set when a group's half or a down group starts: this lane's half-block row, or its ldmatrix row and
  // the rows gid and gid + 8 that it owns results of
  int w_off = 0, own_lo = 0, own_hi = 0;
  int s = 0;
  unsigned ph = 0;
  for (;; ph ^= s == kStageCount - 1 ? 1u : 0u, s = s == kStageCount - 1 ? 0 : s + 1) {
    if (!mbar_wait(&full[s], ph)) {
      if (lane == 0) atomicExch(L.status, 3);
      ok = false;
      break;
    }
    const Desc d = desc[s];
    if (d.end()) break;
    const int d_kind = d.kind(), d_mode = d.absent(), d_ntok = d.ntok(), d_blk = d.blk(), d_last = d.last(), d_seq = d.seq();
    unsigned char* st = stages + static_cast<size_t>(s) * kStageBytes;
    if (d_blk == 0) {
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[0][j] = acc[1][j] = 0.f;
      // unit u of the warp's sixteen: gate rows 0 .. 7 and the up rows of the same pairs, or sixteen down rows
      auto row_at = [&](int u) {
        return d_kind == 0 ? ((u & 7) + 8 * warp) * kW4 + (u >> 3) * kHalfBytes : (16 * warp + u) * kW4;
      };
      if (d_ntok == 1) {
        w_off = row_at(lane >> 1);
      } else {
        w_off = row_at((lane & 7) + ((lane >> 3) & 1) * 8) + 16 + (lane >> 4) * 16;
        own_lo = row_at(lane >> 2);
        own_hi = row_at((lane >> 2) + 8);
      }
    }
    bool w_released = false;
    if (d_mode == 0 && d_ntok == 1) {
      // the lane's half block goes to registers and the weight part of the stage back to the
      // weight warp before the arithmetic: its refill is the long round trip of the ring
      const uint4* wrow = reinterpret_cast<const uint4*>(st + w_off);
      const int half = lane & 1;
      const uint4 hdr = wrow[0];
      uint4 wq[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) wq[i] = wrow[1 + 4 * half + i];
      __syncwarp();
      if (lane == 0) mbar_arrive(&wempty[s]);
      w_released = true;
      acc[0][0] += half_dot(hdr, wq, half, st + kWBytes);
    } else if (d_mode == 0) {
      XTile xt;
      xt.qs = reinterpret_cast<int8_t*>(st + kWBytes);
      xt.bs = reinterpret_cast<int16_t*>(st + kWBytes + kXCodes);
      xt.bl = nullptr;
      xt.d = reinterpret_cast<float*>(st + kWBytes + kXCodes + kTok * 16);
      xt.nb = 1;
      xt.tok_stride = kXqStride;
      xt.d_step = 4;
      xt.mid_pad = 16;
      auto loaded = [&]() {
        __syncwarp();
        if (lane == 0) mbar_arrive(&wempty[s]);
      };
      w_released = true;
      if (d_ntok <= 8) warp_mma_block<1>(st + w_off, st + own_lo, st + own_hi, xt, acc, loaded);
      else warp_mma_block<2>(st + w_off, st + own_lo, st + own_hi, xt, acc, loaded);
    }
    __syncwarp();
    if (lane == 0) {                             // this warp no longer reads the stage
      if (!w_released) mbar_arrive(&wempty[s]);
      mbar_arrive(&empty[s]);
    }
    if (!d_last) continue;

    // ---- the group is complete for this warp's rows ----
    const int gid = lane >> 2, tig = lane & 3;
    if (d_kind == 0) {
      if ((sc.split || d.half() == 0) && !mbar_wait(&hempty[d_seq & 1], ((d_seq >> 1) & 1) ^ 1u)) {
        if (lane == 0) atomicExch(L.status, 6);
        ok = false;
        break;
      }
      if (d_mode == 1) {
        if (d.row0 == 0 && d.half() == 0 && warp == 0 && lane == 0 && L.mail != nullptr) {
          const int e = tile_rec(d.tile).x;
          if (e != L.E) {
            const int mi = atomicAdd(L.mail_n, 1);
            if (mi < L.E) L.mail[mi] = e;
          }
        }
      } else {
        float* hb = hs + (d_seq & 1) * kTok * kHRow + d.half() * kHalfRows + 8 * warp;
        if (d_ntok == 1) {
          const float g = acc[0][0], u = __shfl_down_sync(0xFFFFFFFFu, g, 16);
          if (lane < 16 && (lane & 1) == 0) hb[lane >> 1] = g / (1.f + expf(-g)) * u;
        } else {
#pragma unroll
          for (int n = 0; n < 2; ++n) {
            const int t0 = 8 * n + 2 * tig;
            if (t0 < d_ntok) {
              const float g = acc[n][0], u = acc[n][2];
              hb[t0 * kHRow + gid] = g / (1.f + expf(-g)) * u;
            }
            if (t0 + 1 < d_ntok) {
              const float g = acc[n][1], u = acc[n][3];
              hb[(t0 + 1) * kHRow + gid] = g / (1.f + expf(-g)) * u;
            }
          }
        }
      }
      __syncwarp();
      if ((sc.split || d.half() == 1) && lane == 0) mbar_arrive(&hfull[d_seq & 1]);
    } else {
      if (d_mode == 1) {
        for (int j = lane; j < 16 * d_ntok; j += 32)
          L.ybuf[static_cast<size_t>(d.hrow0 + j / 16) * L.H + d.row0 + 16 * warp + (j & 15)] = 0.f;
        continue;
      }
      if (d_ntok == 1) {
        if ((lane & 1) == 0) L.ybuf[static_cast<size_t>(d.hrow0) * L.H + d.row0 + 16 * warp + (lane >> 1)] = acc[0][0];
      } else {
        const int col = d.row0 + 16 * warp + gid;
#pragma unroll
        for (int n = 0; n < 2; ++n) {
          const int t0 = 8 * n + 2 * tig;
          if (t0 < d_ntok) {
            L.ybuf[static_cast<size_t>(d.hrow0 + t0) * L.H + col] = acc[n][0];
            L.ybuf[static_cast<size_t>(d.hrow0 + t0) * L.H + col + 8] = acc[n][2];
          }
          if (t0 + 1 < d_ntok) {
            L.ybuf[static_cast<size_t>(d.hrow0 + t0 + 1) * L.H + col] = acc[n][1];
            L.ybuf[static_cast<size_t>(d.hrow0 + t0 + 1) * L.H + col + 8] = acc[n][3];
          }
        }
      }
    }
  }

  // ---- all y rows written everywhere: blend ------------------------------------------------
  // (the barrier orders the other threads' stores before thread 0's release, which is cumulative)
  rs_consumers_sync();
  if (tid == 0) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&L.cnt[9]) : "memory");
    unsigned it = 0;
    while (ld_acquire(&L.cnt[9]) < gridDim.x && ++it < kSpinLimit) {
    }
    flag[0] = (it < kSpinLimit && ok) ? 1 : 0;
  }
  rs_consumers_sync();
  if (!flag[0]) {
    if (tid == 0) atomicExch(L.status, 5);
    return;
  }
  combine_flat(L, blockIdx.x * kConsumers + tid, gridDim.x * kConsumers, slot_p, plan_own);
  if (L.ep_out != nullptr) {
    // Owner side of an expert-parallel layer: the rows went straight into the home ranks' buffers;
    // the last CTA to finish tells the home ranks.
    // (CTA barrier, then one thread's acquire-release count; its system-scope fence is cumulative)
    rs_consumers_sync();
    if (tid == 0) {
      if (atom_add_acq_rel(&L.cnt[11], 1u) == gridDim.x - 1) {
        L.cnt[11] = 0u;
        const unsigned v = *L.ep_step * L.ep_mul + L.ep_add;
        set_arrival_words(L.ep_flags, L.ep_world, v);
      }
    }
  }
}

}  // namespace rs
