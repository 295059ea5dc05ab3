// token_layer.cuh - one MoE layer for one to four token rows in ONE persistent launch
// (part of moe_layer.cu, which defines LayerDev, the workspace and the helpers used here).
//
// The single-token layer is latency-bound: 18 MB of weights are 3 us of HBM time, and
// every dependent step around them - a launch, a global round trip, a grid-wide
// barrier - costs about as much again. This kernel keeps the chain as short as the data
// dependencies allow. One CTA per SM, sixteen consumer warps and a producer warp:
//
//   before the previous kernel's results are needed (programmatic dependent launch):
//     the CTA's router rows and its share of the shared expert's gate / up / down rows
//     are already on their way into shared memory - none of them depends on routing
//   phase 1  Q8_K-quantise the rows (every CTA, redundantly: 4 KB per row), logits of the
//            CTA's experts (a warp per expert row and token, the reference kernel's FMA order,
//            so logits are bit-identical), published for the other CTAs; the shared expert's
//            gate / up share while theirs arrive
//   phase 2  every CTA selects redundantly from the n x E logits: for each row one warp picks
//            and one adds up the softmax; from the picks warp 0 builds the list of tiles
//            (distinct experts, each with the set of rows routed to it). The producer warp
//            then issues the weight copies (TMA): the CTA's pairs of the routed gate / up
//            rows through a ring AND its rows of the down matrices, so the down weights
//            arrive while gate / up computes
//   phase 3  gate / up dots (dp4a or the int8 MMA, integer sub-block dots exact), SwiGLU, fp32 h rows to
//            global memory, grid barrier; with dp4a the first down weights go into registers meanwhile
//   phase 4  every CTA quantises the h rows it needs (all of them: a few KB from L2),
//            runs the down dots for its H / grid output rows of EVERY tile, and - since
//            all of a row's expert contributions are then in this CTA - adds
//            residual + sum_k w_k * y_k + shared in place. No second barrier.
//
// What it is bound by: at one row the chain (hidden 2048, n_ff 512, 256 experts, 8 used: 13.2 us per
// layer, 2.3 to the logits, 1 until a CTA has all of them, 2 for picks and tables, 1.5 for the first bytes, 2 for
// gate / up, 2 for the barrier, 1 + 1 for h and the down rows; 13.8 with a barrier between logits and selection, 15.1 with the loops over rows
// of larger layers, whose live values were spilled, 26.6 with eight warps on whole blocks and the selection in sequence). A further
// row costs 3 to 7 us - 20.7 / 23.9 / 27.1 us at 2 / 3 / 4 rows, by dp4a 21.7 / 28.3 / 32.7 -, where its bytes cost 2.2: at four rows, without
// the terms of gate / up 2.3 us less, without those of the down rows 2.9, with four of the 36 h rows in every CTA 1.6 (at two rows 1.7, 2.2 and 0.7).
//
// Work split: gate / up by pairs (a flat range of (tile, pair) per CTA, of equal cost), down by output
// rows. Contracts are those of the two-launch path: null table entry = absent expert
// (zero contribution, id mailed), weight pointers may be only 2-byte aligned (then the
// producer copies with plain loads), routing written to route_idx / route_w.
#pragma once

namespace tk {

constexpr int kMaxTok = 4;                 // token rows per call
constexpr int kWarps = 16;                 // consumer warps: four to a scheduler, the dots are chains of latencies
constexpr int kConsumers = kWarps * 32;
constexpr int kGroupWarps = 8;             // ring stages alternate between two groups of consumer warps
constexpr int kGroupThreads = kGroupWarps * 32;
constexpr int kThreads = kConsumers + 32;  // + producer warp
constexpr int kPairsStage = 16;            // (gate, up) row pairs per ring stage, at least
constexpr int kRing = 2;
constexpr int kDownTiles = 16;             // tiles whose down rows are resident in their own region; as many again in the ring
constexpr int kMaxTiles = 33;              // n * K + 1 <= 33
constexpr int kHdr = 1024;
constexpr int kTables = 4096;

// Quantised rows laid out for lanes that each take half a block: a half is 128 codes, four int16 sums and the block's
// scale in 192 bytes, a block 400, so that the eight lanes of a shared-memory access - four blocks x two halves of a
// row, or two rows of two blocks - read sixteen bytes each from different banks.
constexpr int kHalf = 192, kHBlk = 2 * kHalf + 16;
struct HTile {
  unsigned char* p;
  int nb;
  __device__ __forceinline__ unsigned char* blk(int row, int b) const { return p + static_cast<size_t>(row * nb + b) * kHBlk; }
};

// One super-block of sixteen weight rows against up to four of the rows above (warp_mma_block4): term(r, v) with the block term of
// fragment row gid (r = 0) and gid + 8 and of token tig, before the token's scale. `row` and `row_m` are the blocks of tokens
// (lane & 7) / 2 and gid / 2 (any where there is no such token).
template <typename Loaded, typename Term>
__device__ __forceinline__ void mma_terms(const unsigned char* a_ptr, const unsigned char* own0, const unsigned char* own1, const unsigned char* row,
                                          const unsigned char* row_m, const unsigned char* zeros, int lane, Loaded loaded, Term term) {
  const uint4 h0 = *reinterpret_cast<const uint4*>(own0), h1 = *reinterpret_cast<const uint4*>(own1);
  const bool codes = (lane & 1) == (lane >> 4);
  const unsigned char* b0 = codes ? row + (lane >> 3) * 16 : zeros;
  const int step = codes ? 64 : 0, half = codes ? kHalf : 0;
  warp_mma_block4(a_ptr, h0, h1, [&](int g) { return b0 + (g >> 1) * half + (g & 1) * step; }, lane, loaded,
                  [&] {
                    const uint2 sv = *reinterpret_cast<const uint2*>(row_m + (lane & 1) * kHalf + 128);
                    const int high = (lane >> 2) & 1;                 // bsum = 128 * high + low
                    const uint32_t mask = high ? 0x00FF00FFu : 0x007F007Fu;
                    return __byte_perm((sv.x >> (7 * high)) & mask, (sv.y >> (7 * high)) & mask, 0x6420);
                  },
                  [&](int r, int isum, int msum) {
                    const uint32_t dm = r ? h1.x : h0.x;
                    const float d = 0.0625f * h2f(static_cast<uint16_t>(dm & 0xFFFFu)), dmin = h2f(static_cast<uint16_t>(dm >> 16));
                    term(r, d * static_cast<float>(isum) - dmin * static_cast<float>(msum));
                  });
}

struct Tables {                            // built after the selection, the same in every CTA
  int n_tiles;
  int n_hrows;
  int tile_e[kMaxTiles];                   // expert id (E = shared)
  int tile_mask[kMaxTiles];                // rows routed to it
  int tile_hrow0[kMaxTiles];               // first h / y row
  int tile_mode[kMaxTiles];                // 0 TMA, 1 absent, 2 plain loads (unaligned pointers)
  const unsigned char* w[3][kMaxTiles];
  int sel_idx[kMaxTok][kMaxTiles];         // [t][0..K]
  float sel_w[kMaxTok][kMaxTiles];
  int route_hrow[kMaxTok][kMaxTiles];      // [t][kk] -> h / y row of that route, -1 = absent; [t][K] = shared
  float pick_e[kMaxTok][32];               // the K + 1 largest exponentials
};
static_assert(sizeof(Tables) <= kTables, "tables region");

struct StageDesc {
  int tile, pair0, np, mode;
};

// Kernels on the MMA stage each matrix of a stage of `np` pairs as eight chunks of whole rows, 16 bytes apart, so that ldmatrix
// finds its eight rows - one of every chunk - in different banks. (Each row by itself, 16 bytes apart: 32 to 128 copies a stage, which
// cost the narrow rows of hidden 1024 3 us a layer.)
constexpr int kChunkPad = 8 * 16;
struct Chunks {
  int rows, step;        // rows to a chunk; bytes from one to the next
  __device__ __forceinline__ Chunks(int np, int rb) : rows((np + 7) >> 3), step(rows * rb + 16) {}
  __device__ __forceinline__ int matrix() const { return 8 * step; }                                        // bytes from gate to up
  __device__ __forceinline__ int rows_of(int chunk, int np) const { return max(0, min(rows, np - chunk * rows)); }
};

struct Geom {
  int rows_per_cta;      // router rows per CTA
  int nr_max;            // output rows per CTA (down split)
  int sp_max;            // shared-expert pairs per CTA
  int rb_h, rb_f;        // bytes per gate/up row, per down row
  size_t off_prob, off_ptab, off_xh, off_rw, off_xt, off_sh, off_ring, off_dn, off_y, total;
  int stage_pairs, stage_bytes, slot_bytes, down_tiles;
  int part_bytes;        // a stage's block terms: [block][pair][token][gate, up] floats
};
// Whether the MMA kernel keeps the terms of a down row's blocks until all are there: two and three rows add them as reduce_pairs does, which
// for up to two blocks is one after the other.
__host__ __device__ constexpr bool terms_apart(int n, int nbf) { return n < kMaxTok && nbf > 2; }
__host__ __device__ inline Geom geom(int n, int K, int H, int FF, int E, int grid, bool mma) {
  Geom g;
  g.rows_per_cta = (E + grid - 1) / grid;
  g.nr_max = (H + grid - 1) / grid;
  g.sp_max = (FF + grid - 1) / grid;
  g.rb_h = (H / kQK) * kW4;
  g.rb_f = (FF / kQK) * kW4;
  const int hrows = n * (K + 1);                            // (tile, row) pairs at most
  // as many pairs as a group of warps takes at once (narrow rows take few lanes each)
  const int nbh = H / kQK;
  const int lanes = nbh <= 1 ? 2 : (nbh <= 2 ? 4 : (nbh <= 4 ? 8 : (nbh <= 8 ? 16 : 32)));
  g.stage_pairs = kGroupThreads / lanes > kPairsStage ? kGroupThreads / lanes : kPairsStage;
  g.part_bytes = mma ? nbh * g.stage_pairs * 2 * kMaxTok * 4 : 0;
  size_t p = kHdr + kTables;
  auto take = [&](size_t bytes) { const size_t at = p; p = (p + bytes + 127) & ~static_cast<size_t>(127); return at; };
  g.off_prob = take(static_cast<size_t>(n) * ((E + 3) & ~3) * 4);                // rows at 16-byte steps
  g.off_ptab = take(static_cast<size_t>(3) * E * 8);        // the layer's pointer table, read once per CTA
  // x rows as fp16 and the router rows; later the same bytes hold the quantised h rows
  const size_t a = static_cast<size_t>(n) * H * 2 + 128 + static_cast<size_t>(g.rows_per_cta) * H * 4;
  // (on the MMA: and in between the block terms of gate / up, of two stages of each group)
  const size_t b = static_cast<size_t>(hrows) * (FF / kQK) * kHBlk, c = static_cast<size_t>(4) * g.part_bytes;
  g.off_xh = take(a > b ? (a > c ? a : c) : (b > c ? b : c));
  g.off_rw = g.off_xh + ((static_cast<size_t>(n) * H * 2 + 127) & ~static_cast<size_t>(127));
  g.off_xt = take(static_cast<size_t>(n) * (H / kQK) * kHBlk);
  g.off_sh = take(static_cast<size_t>(2) * g.sp_max * g.rb_h);
  g.stage_bytes = 2 * (g.stage_pairs * g.rb_h + (mma ? kChunkPad : 0));
  g.off_ring = take(static_cast<size_t>(kRing) * g.stage_bytes);
  g.slot_bytes = g.nr_max * g.rb_f;
  const int in_ring = kRing * g.stage_bytes / (g.slot_bytes > 0 ? g.slot_bytes : 1);
  g.down_tiles = in_ring < kDownTiles ? in_ring : kDownTiles;      // (none: the caller takes another path)
  g.off_dn = take(static_cast<size_t>(hrows < g.down_tiles ? hrows : g.down_tiles) * g.slot_bytes);
  g.off_y = take(static_cast<size_t>(hrows) * g.nr_max * 4 * (mma && terms_apart(n, FF / kQK) ? FF / kQK : 1));
  g.total = p;
  return g;
}

// Whether a layer of several rows runs its routed tiles on the int8 MMA. It costs a barrier and a sum per stage, which pay when a CTA's
// pairs take more than one pass of both groups, and a row of few blocks leaves little to gain: us per layer, dp4a / MMA,
//   2048 / 512 / 256 experts / top-8 at 2 / 3 / 4 rows (1.7 / 2.6 / 3.5 passes) 21.8 / 28.3 / 32.7, 20.8 / 24.4 / 27.2
//   2048 / 256 / 64 / 8 (0.9 / 1.3 / 1.7) 16.5 / 18.9 / 21.0, 17.2 / 18.7 / 19.8
//   2048 / 768 / 128 / 8 (2.6 / 3.9 / 5.2) 26.1 / 37.7 / 44.4, 25.2 / 32.3 / 35.0
//   1024 / 512 / 128 / 8 (0.9 / 1.3 / 1.7) 17.8 / 20.0 / 22.1, 19.0 / 21.1 / 22.7
//   512 / 256 / 16 / 4 (0.1 / 0.2 / 0.2) 13.2 / 14.0 / 15.1, 13.6 / 14.0 / 14.7.
inline bool use_mma(int n, int K, int H, int FF, int grid) {
  return n > 1 && H / kQK > 4 && static_cast<long long>(n) * K * FF > 2LL * grid * kPairsStage;
}

// Named barriers of the consumers: 6 all of them, 5 the warps that quantise, 1 .. 4 and 8 .. 11 the
// two warps that select for a token row (the logits are there; the picks are: the picking warp only arrives at both, so they cannot be
// one barrier, at which its second arrival could stand for the other warp's), 12 the warps that pick,
// 13 the warp that picks the only row and the second group, 14 and 15 each group.
__device__ __forceinline__ void named_sync(int id, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }
__device__ __forceinline__ void consumers_sync() {
  asm volatile("bar.sync 6, %0;" ::"n"(kConsumers) : "memory");
}
// CTA barrier of the consumers that also tells whether `ok` held in every one of them.
__device__ __forceinline__ bool consumers_all(bool ok) {
  int r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 q, %1, 0;\n\t"
      "bar.red.and.pred p, 6, %2, q;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(r)
      : "r"(ok ? 1 : 0), "n"(kConsumers)
      : "memory");
  return r != 0;
}
__device__ __forceinline__ unsigned long long ld_acquire_u64(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
// Grid-wide barrier on a 64-bit arrival counter that only ever grows: that of the k-th launch on this
// workspace completes when the counter reaches k * G. Waits are bounded: false when the others did not arrive in time. A CTA that
// gives up before the barrier arrives all the same, and counts itself in the word's top byte: the others learn of it when the barrier
// completes and give up too, and the next launch finds a multiple of the grid, a number of its own and so no logits that it could take for its own.
// The counter is read by the producer warp when the kernels before this one have finished - some multiple of
// the grid size plus the arrivals of this launch's CTAs that are already further on, of which one at least is missing, this
// CTA's own -, so the barrier completes at the next multiple. (Read at kernel start, it could lie among the arrivals of a launch before on the
// same workspace, wherever two CTAs fit on one SM.) An arrival is a fire-and-forget releasing add by the thread whose warp
// finishes the work; the producer warp polls and passes the word on through an mbarrier, so no consumer waits for a round trip
// that it could work through.
//
// The logits go from CTA to CTA without a barrier. A word holds a logit and, above it, the launch's number, which no launch before on the
// workspace had (in 32 bits: a word would have to be 2^32 launches old); a warp of each CTA reads a row's words until all have it. Behind
// a barrier they took two more trips: an arrival waits for the stores before it, and the reads begin when the poll returns. There are kXchgCopies of the words, written by
// as many lanes, and a CTA reads one: 148 readers of the same lines are in the writers' way. us per layer at one row, behind the
// barrier, then with 1 / 2 / 4 / 8 / 16 copies: hidden 2048, 256 experts 13.8, 14.3 / 13.6 / 13.4 / 13.2 / 13.2; 1024, 128 12.3, 13.8 / 12.7 / 12.7 /
// 12.3 / 12.0; 2048, 64 12.0, 12.7 / 12.4 / 12.2 / 12.1 / 11.9; 512, 16 10.8, 11.1 / 11.2 / 11.0 / 10.9 / 10.8; two to four rows of the first 21.0 / 24.5 /
// 27.2 and 20.7 / 23.9 / 27.1 with 16. Two warps per CTA that read, or words that are there read again: 16.5. (Copies of the
// barrier's counter as well: no gain.)
__device__ __forceinline__ void put_logit(unsigned long long* p, unsigned tag, float v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(static_cast<unsigned long long>(tag) << 32 | __float_as_uint(v)) : "memory");
}
__device__ __forceinline__ unsigned long long poll_word(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
// Logits first + lane, + 32, ... (at most N) of the row; false when they did not all arrive. Only what is missing is read again.
template <int N>
__device__ __forceinline__ bool get_logits(const unsigned long long* row, unsigned tag, int first, int E, int lane, float (&v)[N]) {
  unsigned missing = 0;
#pragma unroll
  for (int j = 0; j < N; ++j) {
    v[j] = 0.f;
    if (first + lane + 32 * j < E) missing |= 1u << j;
  }
  for (unsigned it = 0; it < kSpinLimit; ++it) {
    unsigned long long w[N];
#pragma unroll
    for (int j = 0; j < N; ++j)
      if (missing >> j & 1) w[j] = poll_word(row + first + lane + 32 * j);
#pragma unroll
    for (int j = 0; j < N; ++j)
      if ((missing >> j & 1) && static_cast<unsigned>(w[j] >> 32) == tag) {
        v[j] = __uint_as_float(static_cast<unsigned>(w[j]));
        missing &= ~(1u << j);
      }
    if (__all_sync(0xFFFFFFFFu, missing == 0)) return true;
    __nanosleep(40);
  }
  return false;
}
constexpr unsigned long long kGaveUp = 1ull << 56, kArrivals = kGaveUp - 1;       // (a grid has fewer than 256 CTAs)
static_assert(kMaxGrid < 256, "the top byte counts the CTAs of a launch that gave up");
__device__ __forceinline__ void grid_arrive(unsigned long long* ctr, bool ok) {
  asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(ctr), "l"(ok ? 1ull : kGaveUp + 1) : "memory");
}
// Launch k + 1's barrier; `gave_up` is the top byte as it was at the launch's start.
__device__ __forceinline__ bool grid_wait(const unsigned long long* ctr, unsigned long long k, unsigned grid, unsigned gave_up) {
  const unsigned long long target = (k + 1) * grid;
  unsigned it = 0;
  unsigned long long v;
  while (((v = ld_acquire_u64(ctr)) & kArrivals) < target && ++it < kSpinLimit) {
  }
  return it < kSpinLimit && static_cast<unsigned>(v >> 56) == gave_up;
}

// One warp: eight values per lane of a 256-value block -> Q8_K codes, sums and scale in a tile
// (arithmetic of src/kernels/cuda/q4_k.cu:94-130 in the reference).
__device__ __forceinline__ void quantize_to_tile(unsigned char* blk, const float (&v)[8], int lane) {
  int q[8], sum;
  const float d = quantize_lane8(v, q, sum);
  unsigned char* half = blk + (lane >> 4) * kHalf;
  *reinterpret_cast<uint2*>(half + (lane & 15) * 8) =
      make_uint2((q[0] & 0xFF) | ((q[1] & 0xFF) << 8) | ((q[2] & 0xFF) << 16) | (static_cast<uint32_t>(q[3] & 0xFF) << 24),
                 (q[4] & 0xFF) | ((q[5] & 0xFF) << 8) | ((q[6] & 0xFF) << 16) | (static_cast<uint32_t>(q[7] & 0xFF) << 24));
  const int sum_next = __shfl_down_sync(0xFFFFFFFFu, sum, 4);
  if ((lane & 7) == 0)
    *reinterpret_cast<uint32_t*>(half + 128 + ((lane >> 3) & 1) * 4) =
        (static_cast<uint32_t>(sum) & 0xFFFFu) | (static_cast<uint32_t>(sum_next) << 16);
  if ((lane & 15) == 0) *reinterpret_cast<float*>(half + 136) = d;
}

// `rows` fp32 rows of h (global memory, FF values each) into a tile, a warp per 256-value block, D blocks' loads
// in flight per warp: every round of them is a trip to L2 (four rows have 72 blocks, 4.5 a warp: two at a time took 3.2 us, all at
// once 2.3).
// (every CTA reads the same few KB: a load too many is 148 more requests to the same L2 lines)
template <int D>
__device__ __forceinline__ void quantize_h_rows(const HTile& xt, int rows, const float* src, int warp, int lane) {
  const int jobs = rows * xt.nb;                   // blocks lie one after another in both places
  for (int j0 = warp; j0 < jobs; j0 += D * kWarps) {
    const float4* p = reinterpret_cast<const float4*>(src + static_cast<size_t>(j0) * kQK) + lane * 2;
    float4 x[D][2];
    x[0][0] = __ldcg(p);
    x[0][1] = __ldcg(p + 1);
#pragma unroll
    for (int d = 1; d < D; ++d)
      if (j0 + d * kWarps < jobs) {                // warp-uniform
        x[d][0] = __ldcg(p + d * kWarps * (kQK / 4));
        x[d][1] = __ldcg(p + d * kWarps * (kQK / 4) + 1);
      }
#pragma unroll
    for (int d = 0; d < D; ++d)
      if (d == 0 || j0 + d * kWarps < jobs) {
        const float v[8] = {x[d][0].x, x[d][0].y, x[d][0].z, x[d][0].w, x[d][1].x, x[d][1].y, x[d][1].z, x[d][1].w};
        quantize_to_tile(xt.blk(0, j0 + d * kWarps), v, lane);
      }
  }
}

// The staged rows of a tile: row `base + (position of the t-th set bit of mask)` when by_bit
// (activation rows are indexed by token), `base + t` otherwise (h rows are stored per tile).
struct RowSet {
  int r0, r1, r2, r3, n;
  __device__ __forceinline__ int at(int t) const { return t == 0 ? r0 : (t == 1 ? r1 : (t == 2 ? r2 : r3)); }
};
__device__ __forceinline__ RowSet rows_of(int mask, int base, bool by_bit) {
  RowSet r;
  r.n = __popc(mask);
  r.r0 = base + (by_bit ? max(__ffs(mask) - 1, 0) : 0);
  const int m1 = mask & (mask - 1), m2 = m1 & (m1 - 1), m3 = m2 & (m2 - 1);
  r.r1 = base + (by_bit ? max(__ffs(m1) - 1, 0) : 1);
  r.r2 = base + (by_bit ? max(__ffs(m2) - 1, 0) : 2);
  r.r3 = base + (by_bit ? max(__ffs(m3) - 1, 0) : 3);
  return r;
}

// Half a super-block of NMAT weight rows in registers: nibbles, the half's four scales and mins, and the block scales of
// the matrix whose value this lane will hold (with two matrices the even lane of a pair ends with the first one's).
template <int NMAT>
struct HalfW {
  uint4 q[NMAT][4];
  uint32_t sc[NMAT], mn[NMAT];
  float d, dmin;
};
template <int NMAT>
__device__ __forceinline__ void load_half(HalfW<NMAT>& W, const unsigned char* const (&w)[NMAT], int half) {
  uint32_t dd = 0;
#pragma unroll
  for (int m = 0; m < NMAT; ++m) {
    const uint4* p = reinterpret_cast<const uint4*>(w[m]);
    const uint4 hdr = p[0];
#pragma unroll
    for (int i = 0; i < 4; ++i) W.q[m][i] = p[1 + 4 * half + i];
    const Scales6 s6 = unpack_scales6(hdr.y, hdr.z, hdr.w);
    W.sc[m] = half ? s6.sc[1] : s6.sc[0];
    W.mn[m] = half ? s6.mn[1] : s6.mn[0];
    if (m == 0 || half) dd = hdr.x;
  }
  W.d = h2f(static_cast<uint16_t>(dd & 0xFFFFu));
  W.dmin = h2f(static_cast<uint16_t>(dd >> 16));
}
// The half blocks W against the rows of `rs` (a lane pair holds a block; the integer sums of the halves meet before the
// one rounding, so the terms are block_dot's). Mostly integer instructions: with two matrices each lane of the pair sends
// the sum it does not keep and both finish one matrix, which halves the shuffles and the arithmetic after them. Whole
// warps call it: `rows` is the warp's largest row count. Not unrolled over rows: every phase of this kernel runs once
// per CTA, so straight-line code is paid for in instruction fetch.
// `out`: this lane's block terms. CHAIN: the sums over the row's `nb` blocks instead, valid in the lanes of the last
// block (lr == nb - 1, `lr` this lane's position in the row), added block after block - the order of the row-streaming
// kernel's consumers, so that layers of four rows and more have the same bits whichever kernel runs them.
template <int NMAT, bool CHAIN>
__device__ __forceinline__ void half_dots(const HalfW<NMAT>& W, int half, const HTile& xt, int blk, int lr, int nb, const RowSet& rs,
                                          int rows, float (&out)[kMaxTok]) {
#pragma unroll
  for (int t = 0; t < kMaxTok; ++t) out[t] = 0.f;
#pragma unroll 1
  for (int t = 0; t < rows; ++t) {
    const unsigned char* xb = xt.blk(rs.at(t < rs.n ? t : 0), blk) + half * kHalf;
    int lo_sum[NMAT], hi_sum[NMAT], is[NMAT], ms[NMAT];              // hi_sum: sixteen-fold, below 2^29
#pragma unroll
    for (int m = 0; m < NMAT; ++m) lo_sum[m] = hi_sum[m] = 0;
#pragma unroll
    for (int gg = 0; gg < 2; ++gg) {
      const uint4* xa = reinterpret_cast<const uint4*>(xb + 64 * gg);
      const uint4 x0 = xa[0], x1 = xa[1], x2 = xa[2], x3 = xa[3];
#pragma unroll
      for (int m = 0; m < NMAT; ++m) {
        const uint4 q0 = W.q[m][2 * gg], q1 = W.q[m][2 * gg + 1];
        const uint32_t raw[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
        uint32_t lo[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) lo[i] = raw[i] & 0x0F0F0F0Fu;
        const uint32_t scw = W.sc[m] >> (16 * gg);
        lo_sum[m] += static_cast<int>(scw & 0xFF) * dot8(lo, x0, x1);
        hi_sum[m] += static_cast<int>((scw >> 8) & 0xFF) * dot8_high(raw, x2, x3);
      }
    }
    const uint4 sd = *reinterpret_cast<const uint4*>(xb + 128);
#pragma unroll
    for (int m = 0; m < NMAT; ++m) {
      is[m] = lo_sum[m] + (hi_sum[m] >> 4);
      ms[m] = __dp2a_hi(static_cast<int>(sd.y), static_cast<int>(W.mn[m]), __dp2a_lo(static_cast<int>(sd.x), static_cast<int>(W.mn[m]), 0));
    }
    const int other_is = NMAT == 1 || !half ? is[NMAT - 1] : is[0], other_ms = NMAT == 1 || !half ? ms[NMAT - 1] : ms[0];
    const int my_is = (half ? is[NMAT - 1] : is[0]) + __shfl_xor_sync(0xFFFFFFFFu, other_is, 1);
    const int my_ms = (half ? ms[NMAT - 1] : ms[0]) + __shfl_xor_sync(0xFFFFFFFFu, other_ms, 1);
    float v = W.d * static_cast<float>(my_is) - W.dmin * static_cast<float>(my_ms);
    if constexpr (CHAIN) {
      const float term = v;
      v = fmaf(__uint_as_float(sd.z), term, 0.f);
#pragma unroll 1
      for (int b = 1; b < nb; ++b) {
        const float before = __shfl_up_sync(0xFFFFFFFFu, v, 2);
        if (lr == b) v = fmaf(__uint_as_float(sd.z), term, before);
      }
    } else {
      v = __uint_as_float(sd.z) * v;
    }
    if (t == 0) out[0] = v;
    else if (t == 1) out[1] = v;
    else if (t == 2) out[2] = v;
    else out[3] = v;
  }
}
// Sum over the blocks of a row, held by lane pairs `2 * lpr` lanes wide, in the order of reduce_lanes, at block 0's lanes.
__device__ __forceinline__ float reduce_pairs(float v, int lpr) {
  for (int off = lpr >> 1; off > 0; off >>= 1) v += __shfl_down_sync(0xFFFFFFFFu, v, 2 * off);
  return v;
}

// Gate / up of `np` pairs staged at st (gate rows, then up rows) for the rows `mask` of one tile by a group of eight
// warps: thread = (pair, block, half), both matrices. SwiGLU, fp32 h rows [hrow0 + slot][FF] to global memory.
// (Inlined at both of its uses: as a function it saved and restored 2,400 warp registers per CTA through local memory.)
// A warp arrives at `empty` (if given) as soon as its weight bytes are in registers: the stage's refill, a DRAM round
// trip, then runs under the arithmetic. Warps without a pair only arrive.
template <bool CHAIN, bool ONE>
__device__ __forceinline__ void gate_up_stage(const unsigned char* st, int np, int mask, int hrow0, int pair0,
                                           const HTile& xt, float* hbuf, int FF, int nbh, int rb_h, int row_lanes, uint64_t* empty,
                                           int threads = kGroupThreads) {
  const int tid = threadIdx.x & (threads - 1), lane = tid & 31;
  const int lpr = 1 << (row_lanes - 1);
  const RowSet rs = ONE ? RowSet{0, 0, 0, 0, 1} : rows_of(mask, 0, true);
  const int tasks = np << row_lanes;
  if ((tid & ~31) >= tasks) {
    if (empty != nullptr && lane == 0) mbar_arrive_one(empty);
    return;
  }
  const int half = tid & 1, lr = (tid >> 1) & (lpr - 1), blk = min(lr, nbh - 1);
#pragma unroll 1
  for (int q = tid; (q & ~31) < tasks; q += threads) {        // warp-uniform
    const int pair = min(q >> row_lanes, np - 1);
    const unsigned char* row = st + pair * rb_h + blk * kW4;
    const unsigned char* const w[2] = {row, row + np * rb_h};
    HalfW<2> W;
    load_half<2>(W, w, half);
    if (empty != nullptr && ((q + threads) & ~31) >= tasks) {
      __syncwarp();
      if (lane == 0) mbar_arrive_one(empty);
    }
    float v[kMaxTok];
    half_dots<2, CHAIN>(W, half, xt, blk, lr, nbh, rs, rs.n, v);
    const int at = CHAIN ? nbh - 1 : 0;
#pragma unroll
    for (int t = 0; t < kMaxTok; ++t) {
      if (t >= rs.n) break;                        // uniform
      const float g = CHAIN ? v[t] : reduce_pairs(lr < nbh ? v[t] : 0.f, lpr), u = __shfl_down_sync(0xFFFFFFFFu, g, 1);          // the odd lanes hold the up row
      if (q < tasks && half == 0 && lr == at) hbuf[static_cast<size_t>(hrow0 + t) * FF + pair0 + pair] = silu_mul(g, u);
    }
  }
}

// The sum of p(0), .. p(L - 1) in the order of reduce_pairs: i and i + L / 2 first.
template <int L, int STEP = 1, typename Term>
__device__ __forceinline__ float tree_sum(Term p, int i = 0) {
  if constexpr (STEP == L) return p(i);
  else return __fadd_rn(tree_sum<L, 2 * STEP>(p, i), tree_sum<L, 2 * STEP>(p, i + STEP));
}

// The same for layers of several rows, on the int8 MMA: a warp takes eight pairs and one block column at a time - gate rows and the
// up rows of the same indices are the sixteen rows of a fragment -, the terms of a row's blocks meet in `part` and are added in
// gate_up_stage's order, so that a row's bits do not depend on which of the two took it. A tile of four rows costs what a tile of one does; by dp4a 16 pairs took 0.25 us and 1.2 more per row of
// the tile, and the CTAs whose tile four rows share finished 8 us after the median one, or took fewer pairs.
// `st` holds chunks of rows of `rb` bytes; a barrier of the group lies between the two functions.
__device__ __forceinline__ void gate_up_terms(const unsigned char* st, int np, const RowSet& rs, const HTile& xt, int nbh, int rb, float* part,
                                              int part_pairs, const unsigned char* zeros, uint64_t* empty) {
  const int tid = threadIdx.x & (kGroupThreads - 1), lane = tid & 31, gid = lane >> 2, tig = lane & 3;
  const int row = rs.at(min((lane & 7) >> 1, rs.n - 1)), row_m = rs.at(min(gid >> 1, rs.n - 1));
  const Chunks ch(np, rb);
  const int tasks = ch.rows * nbh;
  int task = tid >> 5;
  if (task >= tasks && lane == 0) mbar_arrive_one(empty);
#pragma unroll 1
  for (; task < tasks; task += kGroupWarps) {
    const int q = task / nbh, b = task - q * nbh;          // row q of every chunk, block column b
    const unsigned char* col = st + b * kW4 + q * rb;
    auto chunk = [&](int i) { return (i * ch.rows + q < np ? i : 0) * ch.step; };
    // matrices of a weight load: gate rows, up rows of k 0-15, then of k 16-31 of a sub-block
    const unsigned char* a_ptr = col + chunk(lane & 7) + ((lane >> 3) & 1) * ch.matrix() + 16 + (lane >> 4) * 16;
    const unsigned char* own = col + chunk(gid);
    float v[2];
    mma_terms(a_ptr, own, own + ch.matrix(), xt.blk(row, b), xt.blk(row_m, b), zeros, lane,
              [&] {
                if (task + kGroupWarps >= tasks) {                     // this warp's last weight bytes are in registers
                  __syncwarp();
                  if (lane == 0) mbar_arrive_one(empty);
                }
              },
              [&](int r, float t) { v[r] = t; });
    *reinterpret_cast<float2*>(part + ((b * part_pairs + gid * ch.rows + q) * kMaxTok + tig) * 2) = make_float2(v[0], v[1]);
  }
}
template <bool CHAIN>
__device__ __forceinline__ void gate_up_sums(const float* part, int part_pairs, int np, const RowSet& rs, int hrow0, int pair0, const HTile& xt,
                                             float* hbuf, int FF, int nbh) {
  const int tid = threadIdx.x & (kGroupThreads - 1);
#pragma unroll 1
  for (int i = tid; (i & ~31) < np * 2 * kMaxTok; i += kGroupThreads) {        // (pair, token, matrix)
    const int t = (i >> 1) & (kMaxTok - 1), pair = i >> 3;
    const unsigned char* x = xt.blk(rs.at(min(t, rs.n - 1)), 0) + 136;
    float v = 0.f;
    if constexpr (CHAIN) {
#pragma unroll 4
      for (int b = 0; b < nbh; ++b) v = fmaf(*reinterpret_cast<const float*>(x + b * kHBlk), part[(b * part_pairs) * 2 * kMaxTok + i], v);
    } else {                                     // (five to sixteen blocks: use_mma)
      auto term = [&](int b) {
        return b < nbh ? __fmul_rn(*reinterpret_cast<const float*>(x + b * kHBlk), part[(b * part_pairs) * 2 * kMaxTok + i]) : 0.f;
      };
      v = nbh <= 8 ? tree_sum<8>(term) : tree_sum<16>(term);
    }
    const float u = __shfl_down_sync(0xFFFFFFFFu, v, 1);
    if ((i & 1) == 0 && pair < np && t < rs.n) hbuf[static_cast<size_t>(hrow0 + t) * FF + pair0 + pair] = silu_mul(v, u);
  }
}

// The sum of the terms of `nb` blocks, `step` apart from p on and this thread's own, in the order of reduce_pairs.
__device__ __forceinline__ float blocks_tree(float* p, int step, int nb) {
#pragma unroll 1
  for (int off = next_pow2_cap32(nb) >> 1; off > 0; off >>= 1)
#pragma unroll 1
    for (int i = 0; i < min(off, nb); ++i) p[i * step] = __fadd_rn(p[i * step], i + off < nb ? p[(i + off) * step] : 0.f);
  return p[0];
}

// Producer: `bytes` (a multiple of 16) from a source that may be only 2-byte aligned; plain_done() ends a row of them. (Not
// inlined at its six rarely taken uses: straight-line code beside them is paid for in instruction fetch, 0.4 us a layer.)
static __device__ __noinline__ void copy_plain(unsigned char* dst, const unsigned char* src, int bytes, int lane) {
  warp_copy_unaligned(dst, bytes / 16, lane, reinterpret_cast<uintptr_t>(src), false, [&](int p) { return src + static_cast<size_t>(p) * 16; });
}
__device__ __forceinline__ void plain_done() {
  asm volatile("cp.async.wait_all;" ::: "memory");
  fence_proxy_async();
}

// CHAIN: layers of four token rows (see half_dots); one to three have the bits of each row by itself. ONE: layers of one, which are a chain of short steps: what only more rows
// need is neither executed nor fetched. BY_COST: layers whose CTAs take more pairs than a pass of both groups (see routed_share).
// MMA: routed tiles on the int8 MMA (see use_mma). STREAM: weights first to leave L2 (streams_weights).
// APART: with terms_apart (a kernel of its own: its code in the other one cost layers of two blocks to a down row 0.8 us).
template <bool CHAIN, bool ONE, bool BY_COST, bool MMA, bool APART, bool STREAM>
__global__ void __launch_bounds__(kThreads, 1) token_layer_kernel(const LayerDev L) {
  extern __shared__ __align__(128) unsigned char smem[];
  static_assert(!MMA || (!ONE && !BY_COST), "tiles on the MMA cost the same whatever their rows");
  static_assert(!APART || (MMA && !CHAIN), "only a tree needs the terms apart");
  const Geom G = geom(ONE ? 1 : L.n, L.K, L.H, L.FF, L.E, gridDim.x, MMA);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem);              // [kRing]
  uint64_t* empty = full + kRing;                                  // [kRing]
  uint64_t* sh_full = empty + kRing;                               // shared expert's gate / up pairs
  uint64_t* shdn_full = sh_full + 1;                               // shared expert's down rows (slot 0)
  uint64_t* dn_full = shdn_full + 1;                               // [2] routed tiles' down rows, rounds in turn
  uint64_t* dn_empty = dn_full + 2;                                // [2]
  uint64_t* ready = dn_empty + 2;                                  // tables built
  uint64_t* based = ready + 1;                                     // the grid counter has been read: flag[0] is the launch's number
  uint64_t* passed = based + 1;                                    // grid barrier passed (or given up), one phase each
  StageDesc* desc = reinterpret_cast<StageDesc*>(smem + 128);      // [kRing]
  int* flag = reinterpret_cast<int*>(smem + 256);
  unsigned char* zeros = smem + 512;                               // (MMA) sixteen bytes
  Tables& tb = *reinterpret_cast<Tables*>(smem + kHdr);
  float* prob = reinterpret_cast<float*>(smem + G.off_prob);
  const unsigned char** ptab = reinterpret_cast<const unsigned char**>(smem + G.off_ptab);   // [3][E]
  uint16_t* xh = reinterpret_cast<uint16_t*>(smem + G.off_xh);     // [n][H] fp16
  float* rw = reinterpret_cast<float*>(smem + G.off_rw);           // [rows_per_cta][H]
  unsigned char* sh_stage = smem + G.off_sh;
  unsigned char* ring = smem + G.off_ring;
  unsigned char* dn = smem + G.off_dn;
  float* ysm = reinterpret_cast<float*>(smem + G.off_y);           // [hrow][nr_max], terms apart: [block of h][hrow][nr_max]
  const int y_plane = L.n * (L.K + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int cta = blockIdx.x, grid = gridDim.x;
  const int n = ONE ? 1 : L.n, H = L.H, FF = L.FF, E = L.E, K = L.K;
  const bool has_shared = L.sh[0] != nullptr;
  unsigned long long* gctr = reinterpret_cast<unsigned long long*>(L.cnt + 12);

  // this CTA's shares: shared-expert pairs [sp0, sp1), output rows [r0, r1)
  // (products stay below 2^31: at most 33 tiles x 8192 pairs x a cost of 21 x 192 CTAs)
  const unsigned grid_inv = 0xFFFFFFFFu / static_cast<unsigned>(grid);
  auto share = [&](int total, int part) {        // total * part / grid: the estimate is at most one short
    const unsigned x = static_cast<unsigned>(total) * static_cast<unsigned>(part), q = __umulhi(x, grid_inv);
    return static_cast<int>(q + (x - q * static_cast<unsigned>(grid) >= static_cast<unsigned>(grid) ? 1u : 0u));
  };
  const int sp0 = share(FF, cta), sp1 = share(FF, cta + 1), r0 = share(H, cta), r1 = share(H, cta + 1);
  // This CTA's share [pos, end) of the flat (tile, pair) range of the routed tiles; whole warps, after the tables. A pair costs
  // about 0.25 + 1.2 per row of its tile (us per 16 pairs): in equal numbers of pairs the CTAs whose tile four rows share
  // finished gate / up 8 us after the median one. Us per layer at 4 rows skewed / uniform and 3 rows: 39.0 / 37.0 and 31.1 with
  // equal numbers, 33.6 / 34.4 and 29.2 by cost. As long as the two groups take a CTA's pairs in one pass each the
  // numbers do not matter (and the code alone costs layers of hidden 512 a hundredth: they have a kernel without it).
  auto routed_share = [&](int t_first, int tiles, int& pos, int& end) {
    if (!BY_COST || tiles * FF <= grid * 2 * G.stage_pairs) {
      pos = share(tiles * FF, cta);
      end = share(tiles * FF, cta + 1);
      return;
    }
    const int rows = lane < tiles ? __popc(tb.tile_mask[t_first + lane]) : 0, cost = lane < tiles ? 1 + 5 * rows : 0;
    int sum = cost;                              // a pair of every tile up to this one
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int v = __shfl_up_sync(0xFFFFFFFFu, sum, off);
      if (lane >= off) sum += v;
    }
    auto reciprocal = [](unsigned c) { return 0xFFFFFFFFu / c + 1; };      // (quotients below are exact: dividends stay below 2^27)
    const unsigned inv = rows <= 1 ? reciprocal(6) : (rows == 2 ? reciprocal(11) : (rows == 3 ? reciprocal(16) : reciprocal(21)));
    const int all = __shfl_sync(0xFFFFFFFFu, sum, 31) * FF, before = lane < tiles ? (sum - cost) * FF : 0x7FFFFFFF;
    auto from = [&](int x) {
      const int j = __popc(__ballot_sync(0xFFFFFFFFu, before <= x)) - 1;
      return j * FF + static_cast<int>(__umulhi(static_cast<unsigned>(x - __shfl_sync(0xFFFFFFFFu, before, j)), __shfl_sync(0xFFFFFFFFu, inv, j)));
    };
    pos = from(share(all, cta));
    end = from(share(all, cta + 1));
  };
  const int nr = r1 - r0;

  const bool by_pairs = E <= 256 && K < 32;      // warps t and t + 4 select for row t, otherwise warp t
  if (MMA && tid >= 32 && tid < 36) reinterpret_cast<uint32_t*>(zeros)[tid - 32] = 0u;
  if (tid == 0) {
    for (int s = 0; s < kRing; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], kGroupWarps);
    }
    mbar_init(sh_full, 1);
    mbar_init(shdn_full, 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(&dn_full[s], 1);
      mbar_init(&dn_empty[s], kWarps);
    }
    mbar_init(ready, by_pairs ? n + 1 : 1);      // tables built, and every row's picks found to stand (or not: flag[2])
    mbar_init(based, 1);
    mbar_init(passed, 1);
    flag[2] = 0;                                 // a row's picks did not stand
    fence_barrier_init();
    fence_proxy_async();
  }
  __syncthreads();

  if (warp == kWarps) {
    // ---------------- producer warp ----------------
    const bool sh_aligned = ((reinterpret_cast<uintptr_t>(L.sh[0]) | reinterpret_cast<uintptr_t>(L.sh[1]) |
                              reinterpret_cast<uintptr_t>(L.sh[2])) & 15u) == 0;
    if (has_shared) {
      // the shared expert's weights are fixed: fetch this CTA's share before anything else
      const int np = sp1 - sp0;
      if (sh_aligned) {
        if (lane == 0) {
          if (np > 0) {
            mbar_expect_tx(sh_full, static_cast<uint32_t>(2 * np * G.rb_h));
            bulk_g2s_weights<STREAM>(sh_stage, L.sh[0] + static_cast<size_t>(sp0) * G.rb_h, static_cast<uint32_t>(np * G.rb_h), sh_full);
            bulk_g2s_weights<STREAM>(sh_stage + static_cast<size_t>(np) * G.rb_h, L.sh[1] + static_cast<size_t>(sp0) * G.rb_h,
                     static_cast<uint32_t>(np * G.rb_h), sh_full);
          } else {
            mbar_arrive_one(sh_full);
          }
          if (nr > 0) {
            mbar_expect_tx(shdn_full, static_cast<uint32_t>(nr * G.rb_f));
            bulk_g2s_weights<STREAM>(dn, L.sh[2] + static_cast<size_t>(r0) * G.rb_f, static_cast<uint32_t>(nr * G.rb_f), shdn_full);
          } else {
            mbar_arrive_one(shdn_full);
          }
        }
      } else {
        copy_plain(sh_stage, L.sh[0] + static_cast<size_t>(sp0) * G.rb_h, np * G.rb_h, lane);
        copy_plain(sh_stage + static_cast<size_t>(np) * G.rb_h, L.sh[1] + static_cast<size_t>(sp0) * G.rb_h, np * G.rb_h, lane);
        copy_plain(dn, L.sh[2] + static_cast<size_t>(r0) * G.rb_f, nr * G.rb_f, lane);
        plain_done();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive_one(sh_full);
          mbar_arrive_one(shdn_full);
        }
      }
    }
    // (an earlier launch on this workspace may still be at its barrier until now)
    pdl_wait();
    unsigned long long k = 0;                    // launches before this one
    unsigned gave_up = 0;
    if (lane == 0) {
      const unsigned long long word = ld_acquire_u64(gctr);
      k = (word & kArrivals) / grid;
      gave_up = static_cast<unsigned>(word >> 56);
      flag[0] = static_cast<int>(static_cast<unsigned>(k) + 1u);
      __threadfence_block();
      mbar_arrive_one(based);
    }
    bool built = mbar_wait(ready, 0);
    if (built && by_pairs && *reinterpret_cast<volatile int*>(flag + 2) != 0) built = mbar_wait(ready, 1);
    if (!built) {
      if (lane == 0) atomicExch(L.status, 7);
      return;
    }
    const int T = tb.n_tiles;
    const int t_first = has_shared ? 1 : 0;
    // routed gate / up pairs: a flat range of (tile, pair) per CTA
    int pos, pb;
    routed_share(t_first, T - t_first, pos, pb);
    const int cut = min(G.stage_pairs, (pb - pos + 1) / 2);          // both groups get work
    int tile = t_first + pos / FF, pair0 = pos - (tile - t_first) * FF;
    int issued = 0;
    bool down_issued = false;
    int round = 0;
    const int dt = G.down_tiles, rounds = (T + dt - 1) / dt;
    // down rows of the tiles of one round (tile 0 of round 0 is the shared expert's, fetched above)
    auto issue_down_round = [&](int rd) {
      const int j0 = rd * dt, j1 = min(T, j0 + dt);
      unsigned char* to = (rd & 1) ? ring : dn;
      uint64_t* full_bar = &dn_full[rd & 1];
      const int md = j0 + lane < j1 && !(j0 + lane == 0 && has_shared) ? tb.tile_mode[j0 + lane] : 1;
      const uint32_t bytes = static_cast<uint32_t>(__popc(__ballot_sync(0xFFFFFFFFu, md == 0)) * nr * G.rb_f);
      const bool plain = __any_sync(0xFFFFFFFFu, md == 2);
      if (plain) {
        for (int j = j0; j < j1; ++j)
          if (!(j == 0 && has_shared) && tb.tile_mode[j] == 2)
            copy_plain(to + static_cast<size_t>(j - j0) * G.slot_bytes, tb.w[2][j] + static_cast<size_t>(r0) * G.rb_f,
                       nr * G.rb_f, lane);
        plain_done();
        __syncwarp();
      }
      if (lane == 0) {
        if (bytes > 0) mbar_expect_tx(full_bar, bytes);
        else mbar_arrive_one(full_bar);
      }
      __syncwarp();
      const int jl = j0 + lane;                     // a lane per tile
      if (bytes > 0 && md == 0)
        bulk_g2s_weights<STREAM>(to + static_cast<size_t>(lane) * G.slot_bytes, tb.w[2][jl] + static_cast<size_t>(r0) * G.rb_f,
                 static_cast<uint32_t>(nr * G.rb_f), full_bar);
      __syncwarp();
    };
    while (pos < pb) {
      const int s = issued % kRing;
      const unsigned ph = (issued / kRing) & 1;
      if (issued == kRing && !down_issued) {        // the whole ring is in flight: now the down rows
        issue_down_round(0);
        down_issued = true;
        round = 1;
      }
      if (!mbar_wait(&empty[s], ph ^ 1u)) {
        if (lane == 0) atomicExch(L.status, 2);
        return;
      }
      const int np = min(cut, min(FF - pair0, pb - pos));
      const int mode = tb.tile_mode[tile];
      unsigned char* st = ring + static_cast<size_t>(s) * G.stage_bytes;
      if (lane == 0) {
        StageDesc d;
        d.tile = tile; d.pair0 = pair0; d.np = np; d.mode = mode;
        desc[s] = d;
      }
      if (mode == 2) {
        if (!MMA) {
          copy_plain(st, tb.w[0][tile] + static_cast<size_t>(pair0) * G.rb_h, np * G.rb_h, lane);
          copy_plain(st + static_cast<size_t>(np) * G.rb_h, tb.w[1][tile] + static_cast<size_t>(pair0) * G.rb_h, np * G.rb_h, lane);
        } else {
          const Chunks ch(np, G.rb_h);
          for (int i = 0; i < 16; ++i)
            copy_plain(st + i * ch.step, tb.w[i >> 3][tile] + static_cast<size_t>(pair0 + (i & 7) * ch.rows) * G.rb_h, ch.rows_of(i & 7, np) * G.rb_h, lane);
        }
        plain_done();
      }
      __syncwarp();
      if (MMA) {                                    // a lane per chunk
        if (lane == 0) {
          if (mode == 0) mbar_expect_tx(&full[s], static_cast<uint32_t>(2 * np * G.rb_h));
          else mbar_arrive_one(&full[s]);
        }
        __syncwarp();
        const Chunks ch(np, G.rb_h);
        const int rows = ch.rows_of(lane & 7, np);
        if (mode == 0 && lane < 16 && rows > 0)
          bulk_g2s_weights<STREAM>(st + lane * ch.step, tb.w[lane >> 3][tile] + static_cast<size_t>(pair0 + (lane & 7) * ch.rows) * G.rb_h,
                                   static_cast<uint32_t>(rows * G.rb_h), &full[s]);
      } else if (lane == 0) {
        if (mode == 0) {
          mbar_expect_tx(&full[s], static_cast<uint32_t>(2 * np * G.rb_h));
          bulk_g2s_weights<STREAM>(st, tb.w[0][tile] + static_cast<size_t>(pair0) * G.rb_h, static_cast<uint32_t>(np * G.rb_h), &full[s]);
          bulk_g2s_weights<STREAM>(st + static_cast<size_t>(np) * G.rb_h, tb.w[1][tile] + static_cast<size_t>(pair0) * G.rb_h,
                   static_cast<uint32_t>(np * G.rb_h), &full[s]);
        } else {
          mbar_arrive_one(&full[s]);
        }
      }
      __syncwarp();
      pos += np;
      pair0 += np;
      if (pair0 == FF) { pair0 = 0; ++tile; }
      ++issued;
    }
    if (!down_issued) {
      issue_down_round(0);
      round = 1;
    }
    if (round < rounds) {                           // the second round into the ring, once its last stages are in registers
      for (int s = 0; s < kRing; ++s) {
        const int used = (issued - s + kRing - 1) / kRing;
        if (used > 0 && !mbar_wait(&empty[s], (used - 1) & 1)) {
          if (lane == 0) atomicExch(L.status, 2);
          return;
        }
      }
      issue_down_round(round++);
    }
    if (lane == 0) {                                // the barrier's outcome goes to flag[1]
      flag[1] = grid_wait(gctr, k, grid, gave_up) ? 1 : 0;
      __threadfence_block();
      mbar_arrive_one(passed);
    }
    __syncwarp();
    for (; round < rounds; ++round) {               // later rounds reuse the regions
      if (!mbar_wait(&dn_empty[round & 1], (round / 2 - 1) & 1)) {
        if (lane == 0) atomicExch(L.status, 2);
        return;
      }
      issue_down_round(round);
    }
    return;
  }

  // ---------------- consumers ----------------
  const int row_lanes = __ffs(2 * next_pow2_cap32(L.nbh)) - 1;
  // warps 0 .. nlw - 1 take the logits, one (router row, token) at a time; the others quantise x
  const int nl = G.rows_per_cta, nlw = min(nl * n, kGroupWarps);
  // router rows of this CTA's experts: fixed weights, on their way before the previous kernel is awaited
  for (int i = 0; i < nl; ++i) {
    const int e = cta + i * grid;
    if (e >= E) break;
    const float* src = L.router_w + static_cast<size_t>(e) * H;
    float* dst = rw + static_cast<size_t>(i) * H;
    if ((reinterpret_cast<uintptr_t>(L.router_w) & 15u) == 0) {
      for (int c = tid * 4; c < H; c += kConsumers * 4)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst + c)), "l"(src + c) : "memory");
    } else {
      for (int c = tid; c < H; c += kConsumers) dst[c] = __ldg(src + c);
    }
  }
  pdl_wait();
  pdl_launch_dependents();
  if (cta == 0 && tid == 0 && L.mail_n != nullptr) *L.mail_n = 0;

  // The layer's pointer table (3 x E pointers: after the selection the experts' addresses are then one shared-memory
  // read away) and the x rows as fp16, copied by all threads.
  for (int i = tid; i < 3 * E; i += kConsumers) {
    const int m = i >= 2 * E ? 2 : (i >= E ? 1 : 0);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(ptab + i)), "l"(L.tab + static_cast<size_t>(m) * L.tab_stride + (i - m * E))
                 : "memory");
  }
  const int jobs = n * L.nbh, xw = warp - nlw, n_xw = kWarps - nlw;
  for (int i = tid; i < jobs * 32; i += kConsumers)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(xh + i * 8)), "l"(L.xn + static_cast<size_t>(i) * 8) : "memory");
  const HTile xt = {smem + G.off_xt, L.nbh};
  asm volatile("cp.async.wait_all;" ::: "memory");
  consumers_sync();                              // fp16 x rows, router rows and the pointer table are in place
  bool ok = true;
  if (warp < nlw) {
    // logits: lane l adds k = l, l + 32, ... in ascending order with FMA and the lanes meet in a shuffle tree - the
    // order of the reference's kernel (src/kernels/cuda/q4_k.cu:133-149). Eight steps of loads are issued ahead of
    // their FMAs.
#pragma unroll 1
    for (int item = warp; item < nl * n; item += nlw) {
      const int t = (item >= nl) + (item >= 2 * nl) + (item >= 3 * nl), i = item - t * nl;
      const int e = cta + i * grid;
      if (e >= E) continue;
      const float* wr = rw + static_cast<size_t>(i) * H;
      const uint16_t* xr = xh + static_cast<size_t>(t) * H;
      const float b = L.bias != nullptr ? __ldg(L.bias + e) : 0.f;
      float acc = 0.f;
      int k = lane;
#pragma unroll 2
      for (; k + 7 * 32 < H; k += 8 * 32) {
        float wv[8];
        uint16_t xv[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) { wv[j] = wr[k + 32 * j]; xv[j] = xr[k + 32 * j]; }
#pragma unroll
        for (int j = 0; j < 8; ++j) acc = fmaf(wv[j], h2f(xv[j]), acc);
      }
#pragma unroll 1
      for (; k < H; k += 32) acc = fmaf(wr[k], h2f(xr[k]), acc);
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) acc += __shfl_down_sync(0xFFFFFFFFu, acc, off);
      acc = __shfl_sync(0xFFFFFFFFu, acc, 0);
      if (lane < kXchgCopies && mbar_wait(based, 0))         // (set when the kernels before this one have finished)
        put_logit(L.xchg + (lane * n + t) * E + e, static_cast<unsigned>(*reinterpret_cast<volatile int*>(flag)), acc + b);
    }
  } else {
#pragma unroll 1
    for (int job = xw; job < jobs; job += n_xw) {
      float v[8];
      load_lane8(xh + static_cast<size_t>(job) * kQK, lane, v);
      quantize_to_tile(xt.blk(0, job), v, lane);
    }
    named_sync(5, n_xw * 32);
    // the shared expert does not depend on the routing: its gate / up share runs in the second group while the CTAs
    // meet at the barrier (tile 0: every row, h rows 0 .. n-1)
    if (warp >= kGroupWarps && has_shared && sp1 > sp0) {
      if (!mbar_wait(sh_full, 0)) ok = false;
      if (__all_sync(0xFFFFFFFFu, ok))
      {
        // (several rows: two warps to a row, whose threads its few pairs fill as a rule; one row after the other the second group was the
        // last to come to the selection's end. us per layer, 2048 / 256 / 64 experts at 3 rows 18.55 -> 18.2, 1024 / 512 / 128 at 2 / 3 / 4
        // rows 17.4 / 19.75 / 22.05 -> 17.25 / 19.7 / 21.8)
        const int t = ONE ? 0 : (warp - kGroupWarps) >> 1;
        if (t < n)
          gate_up_stage<CHAIN, ONE>(sh_stage, sp1 - sp0, 1 << t, t, sp0, xt, L.hbuf, FF, L.nbh, G.rb_h, row_lanes, nullptr, ONE ? kGroupThreads : 64);
      }
    }
  }

  // ---- selection (every CTA, the same result) and the tile tables ----
  // The picks need no sum, so the tables and the fetch of the picked experts into L2 run while the other warps add. The
  // rare row whose picks do not stand after the division has the tables built once more.
  const int t_first = has_shared ? 1 : 0;
  auto build = [&] {
    // one lane per pick (n * K <= 32): picks of the same expert find each other with a match,
    // the lowest lane of a group founds the tile; tiles are numbered in pick order
    const bool live = lane < n * K;
    const int pt = live ? (lane >= K) + (lane >= 2 * K) + (lane >= 3 * K) : 0, pk = live ? lane - pt * K : 0;
    const int e = live ? tb.sel_idx[pt][pk] : -1 - lane;             // dead lanes match nobody
    const unsigned char *w0 = nullptr, *w1 = nullptr, *w2 = nullptr;
    if (live) { w0 = ptab[e]; w1 = ptab[E + e]; w2 = ptab[2 * E + e]; }
    const bool absent = w0 == nullptr || w1 == nullptr || w2 == nullptr;
    const unsigned same = n == 1 ? 1u << lane : __match_any_sync(0xFFFFFFFFu, e);   // a row's picks are distinct
    const int first = __ffs(same) - 1;
    const bool leader = live && first == lane;
    const unsigned leaders = __ballot_sync(0xFFFFFFFFu, leader);
    const int my_tile = t_first + __popc(leaders & ((1u << first) - 1u));
    int mask = 0;                                                    // rows of the tile: the token of every lane in the group
    const unsigned row = K < 32 ? (1u << K) - 1u : 0xFFFFFFFFu;
#pragma unroll
    for (int t = 0; t < kMaxTok; ++t)
      if (t < n && (same >> (t * K) & row) != 0) mask |= 1 << t;
    // first h / y row of every tile: prefix sum of the founders' row counts
    const int cnt = leader ? __popc(mask) : 0;
    int inc = cnt;
    const int base = has_shared ? n : 0;
    int hrow0;
    if (n == 1) {                                                    // a tile per pick
      hrow0 = base + lane;
      inc = K;
    } else {
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const int v = __shfl_up_sync(0xFFFFFFFFu, inc, off);
        if (lane >= off) inc += v;
      }
      hrow0 = base + __shfl_sync(0xFFFFFFFFu, inc - cnt, first);
    }
    if (leader) {
      const bool aligned = ((reinterpret_cast<uintptr_t>(w0) | reinterpret_cast<uintptr_t>(w1) |
                             reinterpret_cast<uintptr_t>(w2)) & 15u) == 0;
      tb.tile_e[my_tile] = e;
      tb.tile_mask[my_tile] = mask;
      tb.tile_hrow0[my_tile] = hrow0;
      tb.w[0][my_tile] = w0; tb.w[1][my_tile] = w1; tb.w[2][my_tile] = w2;
      tb.tile_mode[my_tile] = absent ? 1 : (aligned ? 0 : 2);
    }
    if (live) tb.route_hrow[pt][pk] = absent ? -1 : hrow0 + __popc(mask & ((1 << pt) - 1));
    if (lane < n) tb.route_hrow[lane][K] = has_shared ? lane : -1;
    if (lane == 31) tb.n_hrows = base + inc;
    if (lane == 0) {
      tb.n_tiles = t_first + __popc(leaders);
      if (has_shared) {
        tb.tile_e[0] = E;
        tb.tile_mask[0] = (1 << n) - 1;
        tb.tile_hrow0[0] = 0;
        tb.w[0][0] = L.sh[0]; tb.w[1][0] = L.sh[1]; tb.w[2][0] = L.sh[2];
        tb.tile_mode[0] = ((reinterpret_cast<uintptr_t>(L.sh[0]) | reinterpret_cast<uintptr_t>(L.sh[1]) |
                            reinterpret_cast<uintptr_t>(L.sh[2])) & 15u) == 0 ? 0 : 2;
      }
    }
    __syncwarp();
  };
  if (warp < 2 * kMaxTok && (warp & (kMaxTok - 1)) < n) {
    const int t = warp & (kMaxTok - 1);
    const unsigned long long* row = L.xchg + ((cta & (kXchgCopies - 1)) * n + t) * E;
    float* pr = prob + static_cast<size_t>(t) * ((E + 3) & ~3);
    float v[8] = {};                             // (one row) this lane's logits
    bool there = true;
    if (warp < kMaxTok) {
      // A CTA without a router row would read from here on, before there can be a logit, and its reads of the lines that a few
      // CTAs are about to write slow those down. us per layer at 1 / 2 / 3 / 4 rows of 512 / 256 / 16, weights in L2: behind a barrier 11.35 / 13.3 /
      // 14.2 / 15.05, words 11.1 / 13.1 / 14.2 / 15.4, with the pause 10.7 / 12.9 / 13.9 / 14.8 (300 to 800 ns within 0.1, launches one by one gain
      // 0.15 more from 600 on; 256 / 256 / 8, one row: 11.3, 10.1, and 10.2 at 500, 10.5 at 800 ns).
      if (cta >= E) __nanosleep(600);
      there = __all_sync(0xFFFFFFFFu, mbar_wait(based, 0)) &&
              get_logits<8>(row, static_cast<unsigned>(*reinterpret_cast<volatile int*>(flag)), 0, min(E, 256), lane, v);
      if (by_pairs) {                            // for the warp that adds
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (lane + 32 * j < E) pr[lane + 32 * j] = v[j];
        __syncwarp();
        asm volatile("bar.arrive %0, 64;" ::"r"(1 + t) : "memory");
      }
    } else if (by_pairs) {
      named_sync(1 + t, 64);
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = lane + 32 * j < E ? pr[lane + 32 * j] : 0.f;
    }
    if (!there) ok = false;                      // (the named barriers below need every warp: it goes on with what is there)
    if (by_pairs) {
      const bool redo = router_select_pair([&](int j) { return v[j]; }, pr, tb.pick_e[t], tb.sel_idx[t], tb.sel_w[t], 8 + t, warp >= kMaxTok, E, K, L.shared_w, lane, [&] {
        if (n == 1) asm volatile("bar.arrive 13, %0;" ::"n"(32 + kGroupThreads) : "memory");   // the second group fetches
        else named_sync(12, n * 32);             // every row's picks are in the tables
        if (warp == 0) build();
      });
      if (redo && lane == 0) *reinterpret_cast<volatile int*>(flag + 2) = 1;
      __syncwarp();
      if (there && lane == 0 && (warp == 0 || warp >= kMaxTok)) mbar_arrive_one(ready);
    } else if (warp < kMaxTok && there) {
      for (int first = 0; first < E; first += 256) {
        if (!get_logits<8>(row, static_cast<unsigned>(*reinterpret_cast<volatile int*>(flag)), first, E, lane, v)) ok = false;
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (first + lane + 32 * j < E) pr[first + lane + 32 * j] = v[j];
      }
      __syncwarp();
      router_select_general(pr, E, K, tb.sel_idx[t], tb.sel_w[t], L.shared_w, lane);
    }
  }
  if (warp >= kGroupWarps && by_pairs && n == 1) {
    // One row: the second group asks for this CTA's slice of the picked experts' matrices (whichever CTA reads it later) to be
    // brought into L2 while warp 0 builds the tables. Line by line: in the copy engine's queue the requests would be
    // ahead of the first stage's copies. (16.3 -> 15.7 us; with more rows the other tiles' bytes only come ahead of the
    // first stages' - 23.5 against 23.1, 31.7 against 30.9, 40.3 against 38.4 us at 2 / 3 / 4 rows.)
    const int g0 = share(FF * (G.rb_h / 16), cta) * 16, g1 = share(FF * (G.rb_h / 16), cta + 1) * 16;
    const int d0 = share(H * (G.rb_f / 16), cta) * 16, d1 = share(H * (G.rb_f / 16), cta + 1) * 16;
    named_sync(13, 32 + kGroupThreads);
    for (int kk = warp - kGroupWarps; kk < K; kk += kGroupWarps) {
      const int e = tb.sel_idx[0][kk];
#pragma unroll
      for (int m = 0; m < 3; ++m) {
        const unsigned char* w = ptab[m * E + e];
        if (w == nullptr) continue;
        for (int o = (m < 2 ? g0 : d0) + lane * 128; o < (m < 2 ? g1 : d1); o += 32 * 128)
          asm volatile("prefetch.global.L2 [%0];" ::"l"(w + o) : "memory");
      }
    }
  }
  if (!consumers_all(ok)) {
    if (tid == 0) {
      atomicExch(L.status, 5);
      grid_arrive(gctr, false);
    }
    return;
  }
  if (!by_pairs || *reinterpret_cast<volatile int*>(flag + 2) != 0) {
    if (warp == 0) {
      build();
      if (lane == 0)
        for (int i = by_pairs ? n + 1 : 1; i > 0; --i) mbar_arrive_one(ready);
    }
    consumers_sync();
  }
  if (cta == 0 && tid < n * (K + 1)) {
    const int t = tid / (K + 1), kk = tid - t * (K + 1);
    if (kk < K) L.idx[static_cast<size_t>(t) * L.rstride + kk] = tb.sel_idx[t][kk];
    L.w[static_cast<size_t>(t) * L.rstride + kk] = tb.sel_w[t][kk];
  }
  if (cta == 0 && L.mail != nullptr && tid >= t_first && tid < tb.n_tiles && tb.tile_mode[tid] == 1) {
    const int mi = atomicAdd(L.mail_n, 1);
    if (mi < E) L.mail[mi] = tb.tile_e[tid];
  }
  const int T = tb.n_tiles;

  // ---- phase 3: gate / up of the routed tiles, SwiGLU; the groups take stages in turn ----
  {
    int pos, pb;
    routed_share(t_first, T - t_first, pos, pb);
    const int group = warp / kGroupWarps;
    int pair0 = pos % FF;
    const int cut = min(G.stage_pairs, (pb - pos + 1) / 2);
    // (where x and the router rows were; two stages' terms per group, so that one barrier a stage is enough)
    float* part = reinterpret_cast<float*>(smem + G.off_xh) + group * (G.part_bytes / 2);
    for (int i = 0; pos < pb && (MMA || ok); ++i) {
      const int s = i % kRing, np = min(cut, min(FF - pair0, pb - pos));    // as the producer cuts the range
      pos += np;
      pair0 = pair0 + np == FF ? 0 : pair0 + np;
      if ((i & 1) != group) continue;
      if constexpr (!MMA) {
        ok = __all_sync(0xFFFFFFFFu, mbar_wait(&full[s], (i / kRing) & 1)) != 0;
        if (!ok) break;
        const StageDesc d = desc[s];
        if (d.mode != 1)
          gate_up_stage<CHAIN, ONE>(ring + static_cast<size_t>(s) * G.stage_bytes, d.np, tb.tile_mask[d.tile], tb.tile_hrow0[d.tile],
                        d.pair0, xt, L.hbuf, FF, L.nbh, G.rb_h, row_lanes, &empty[s]);
        else if (lane == 0) mbar_arrive_one(&empty[s]);
      } else {
        // (whole groups: a warp whose wait ran out goes on to the barriers)
        if (ok) ok = __all_sync(0xFFFFFFFFu, mbar_wait(&full[s], (i / kRing) & 1)) != 0;
        const StageDesc d = desc[s];
        const bool work = ok && d.mode != 1;
        if (ok && !work && lane == 0) mbar_arrive_one(&empty[s]);
        const unsigned char* st = ring + static_cast<size_t>(s) * G.stage_bytes;
        float* terms = part + ((i >> 1) & 1) * (G.part_bytes / 4);
        const RowSet rs = rows_of(work ? tb.tile_mask[d.tile] : 1, 0, true);
        if (work) gate_up_terms(st, d.np, rs, xt, L.nbh, G.rb_h, terms, G.stage_pairs, zeros, &empty[s]);
        named_sync(14 + group, kGroupThreads);
        if (work) gate_up_sums<CHAIN>(terms, G.stage_pairs, d.np, rs, tb.tile_hrow0[d.tile], d.pair0, xt, L.hbuf, FF, L.nbh);
      }
    }
  }
  ok = consumers_all(ok);                                   // (a wait that ran out in any thread ends the CTA's work)
  if (tid == 0) grid_arrive(gctr, ok);

  // ---- phase 4: quantise h (all rows, from L2), down rows of this CTA, combine in place ----
  const HTile hq = {smem + G.off_xh, L.nbf};
  const int f_lanes = __ffs(2 * next_pow2_cap32(L.nbf)) - 1, lpf = 1 << (f_lanes - 1);
  const int f_half = tid & 1, f_lr = (tid >> 1) & (lpf - 1), f_blk = min(f_lr, L.nbf - 1);
  const int dt = G.down_tiles, rounds = (T + dt - 1) / dt;
  bool first = true;
  // this thread's output element (as a rule it has one), its residual fetched ahead of the barrier
  const bool residual = L.add_residual && L.x_f16 != nullptr;
  const int o_t = tid / max(nr, 1);
  const size_t o_at = static_cast<size_t>(o_t) * H + r0 + (tid - o_t * nr);
  const uint16_t res = residual && tid < n * nr ? L.x_f16[o_at] : 0;
#pragma unroll 1
  for (int rd = 0; rd < rounds && ok; ++rd) {
    const int j0 = rd * dt, j1 = min(T, j0 + dt);
    const unsigned char* from = (rd & 1) ? ring : dn;
    if (rd == 0 && has_shared && !mbar_wait(shdn_full, 0)) ok = false;
    if (ok && !mbar_wait(&dn_full[rd & 1], (rd >> 1) & 1)) ok = false;
    ok = __all_sync(0xFFFFFFFFu, ok) != 0;
    if constexpr (MMA) {
      if (rd == 0) {
        const bool met = mbar_wait(passed, 0) && *reinterpret_cast<volatile int*>(flag + 1) != 0;
        quantize_h_rows<5>(hq, tb.n_hrows, L.hbuf, warp, lane);
        if (!consumers_all(met && ok)) {
          if (tid == 0) atomicExch(L.status, ok ? 5 : 3);
          return;
        }
      }
      // A warp per tile, or per tile and block where the blocks' terms are added as a tree of more than two; sixteen output rows at a time
      const int gid = lane >> 2, tig = lane & 3, tasks = ok ? (j1 - j0) * (APART ? L.nbf : 1) : 0;
#pragma unroll 1
      for (int q = warp; q < tasks; q += kWarps) {
        const int j = j0 + (APART ? q / L.nbf : q), b0 = APART ? q % L.nbf : 0, b1 = APART ? b0 + 1 : L.nbf;
        if (tb.tile_mode[j] == 1) continue;
        const int hrow0 = tb.tile_hrow0[j], rows = __popc(tb.tile_mask[j]);
        const int row = hrow0 + min((lane & 7) >> 1, rows - 1), row_m = hrow0 + min(gid >> 1, rows - 1), row_t = hrow0 + min(tig, rows - 1);
        float* y = ysm + (b0 * y_plane + hrow0 + tig) * G.nr_max;
#pragma unroll 1
        for (int m0 = 0; m0 < nr; m0 += 16) {
          const unsigned char* w = from + static_cast<size_t>(j - j0) * G.slot_bytes + b0 * kW4;
          const int ra = min(m0 + (lane & 15), nr - 1), q0 = m0 + gid, q1 = q0 + 8;
          float acc[2] = {CHAIN ? 0.f : -0.f, CHAIN ? 0.f : -0.f};       // (-0 + v is v)
#pragma unroll 1
          for (int b = b0; b < b1; ++b, w += kW4) {
            const float xd = *reinterpret_cast<const float*>(hq.blk(row_t, b) + 136);
            mma_terms(w + ra * G.rb_f + 16 + (lane >> 4) * 16, w + min(q0, nr - 1) * G.rb_f, w + min(q1, nr - 1) * G.rb_f, hq.blk(row, b), hq.blk(row_m, b),
                      zeros, lane, [] {}, [&](int r, float v) { acc[r] = CHAIN ? fmaf(xd, v, acc[r]) : __fadd_rn(acc[r], __fmul_rn(xd, v)); });
          }
          if (tig < rows) {
            if (q0 < nr) y[q0] = acc[0];
            if (q1 < nr) y[q1] = acc[1];
          }
        }
      }
    } else {
      const int tasks = (j1 - j0) * nr << f_lanes;
      int base = 0;
#pragma unroll 1
      do {
        // a task's weights go into registers first, at the first task while the other CTAs finish their gate / up
        const int q = base + tid;
        const int jr = q >> f_lanes;
        const int js = jr / max(nr, 1), r = jr - js * nr;
        const int tile = min(j0 + js, T - 1);
        const bool live = q < tasks && tb.tile_mode[tile] != 1;
        const int hrow0 = tb.tile_hrow0[tile];
        const RowSet rs = ONE ? RowSet{live ? hrow0 : 0, 0, 0, 0, 1} : rows_of(live ? tb.tile_mask[tile] : 0, live ? hrow0 : 0, false);   // h rows are stored per tile
        const int rows = ONE ? 1 : __reduce_max_sync(0xFFFFFFFFu, rs.n);
        const unsigned char* const w[1] = {from + (live ? js * G.slot_bytes + r * G.rb_f + f_blk * kW4 : 0)};
        HalfW<1> W;
        load_half<1>(W, w, f_half);
        if (first) {
          first = false;
          const bool met = mbar_wait(passed, 0) && *reinterpret_cast<volatile int*>(flag + 1) != 0;
          quantize_h_rows<2>(hq, tb.n_hrows, L.hbuf, warp, lane);
          if (!consumers_all(met && ok)) {
            if (tid == 0) atomicExch(L.status, ok ? 5 : 3);
            return;
          }
        }
        float v[kMaxTok];
        half_dots<1, CHAIN>(W, f_half, hq, f_blk, f_lr, L.nbf, rs, rows, v);
        const int at = CHAIN ? L.nbf - 1 : 0;
#pragma unroll
        for (int t = 0; t < kMaxTok; ++t) {
          if (t >= rows) break;                    // warp-uniform
          const float y = CHAIN ? v[t] : reduce_pairs(f_lr < L.nbf ? v[t] : 0.f, lpf);
          if (live && f_half == 0 && f_lr == at && t < rs.n) ysm[(hrow0 + t) * G.nr_max + r] = y;
        }
        base += kConsumers;
      } while (base < tasks && ok);
    }
    __syncwarp();
    if (lane == 0 && rd + 2 < rounds) mbar_arrive_one(&dn_empty[rd & 1]);
  }
  if (!consumers_all(ok)) {
    if (tid == 0) atomicExch(L.status, 3);
    return;
  }
  if constexpr (APART) {
    for (int i = tid; i < tb.n_hrows * nr; i += kConsumers) {
      const int hr = i / nr;
      float* p = ysm + hr * G.nr_max + (i - hr * nr);
      p[0] = blocks_tree(p, y_plane * G.nr_max, L.nbf);
    }
    consumers_sync();
  }
  for (int i = tid; i < n * nr; i += kConsumers) {
    const int t = i / nr, rr = i - t * nr;
    const size_t o = static_cast<size_t>(t) * H + r0 + rr;
    float acc = residual ? h2f(i == tid ? res : L.x_f16[o]) : 0.f;
#pragma unroll 4
    for (int kk = 0; kk <= K; ++kk) {
      const int hr = tb.route_hrow[t][kk];
      const float wk = tb.sel_w[t][kk], y = ysm[max(hr, 0) * G.nr_max + rr];
      if (hr >= 0) acc += wk * y;
    }
    if (L.out_f32 != nullptr) L.out_f32[o] = acc;
    if (residual) L.x_f16[o] = f2h(acc);
  }
}

}  // namespace tk
