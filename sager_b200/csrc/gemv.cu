// gemv.cu - the Q4_K x Q8_K GEMV family behind the reference's launchers
// (src/kernels/cuda/q4_k.cu:1534-1562, 1660-1849, 1926-1985 and
// src/kernels/cuda/mmq.cu:368-378 of the reference): dense single-row and
// multi-token, pointer-table, host-plan grouped and device-plan grouped with
// the null-pointer mailbox. One kernel template, four planners, all of which end in
// tile_run_staged (tile.cuh); dense matrices of up to eight tokens have kernels of their own.
#include <algorithm>

#include "api_util.cuh"
#include "tile.cuh"

namespace sgr {
namespace {

enum Mode : int { kDense = 0, kPtrs = 1, kGrouped = 2, kTab = 3, kMulti = 4 };

struct GemvArgs {
  const unsigned char* w[2];            // dense: matrix bases
  const unsigned char* const* tab[2];   // ptrs / grouped / tab: per-job or per-expert bases
  const unsigned char* xq;              // packed Q8_K rows, nb blocks each
  void* y[2];
  int n_rows, nb, n_tokens, tok_tile, rows_per, n_expert;
  const int *off, *m, *tile_base, *job_of_tile;   // grouped (host plan)
  const int *toff, *meta;                          // tab (device plan)
  int *mail, *mail_n;
  int* status;
  uint16_t* res;                        // dense, one token, fp16 out: residual row updated in place
  // multi: up to three matrices of the same k with their own outputs, one token row
  const unsigned char* wm[3];
  uint16_t* ym[3];
  int rows_cum[3];                      // rows of matrices 0..m inclusive
};

// last e with toff[e] <= tile (toff is the E+1 exclusive prefix of tiles per expert)
__device__ __forceinline__ int expert_of_tile(const int* toff, int n_expert, int tile) {
  int lo = 0, hi = n_expert - 1, res = n_expert - 1;
  while (lo <= hi) {
    const int mid = (lo + hi) >> 1;
    if (toff[mid + 1] <= tile) lo = mid + 1;
    else { res = mid; hi = mid - 1; }
  }
  return res;
}

template <bool F16>
__device__ __forceinline__ void store_out(void* y, size_t i, float v) {
  if constexpr (F16) reinterpret_cast<uint16_t*>(y)[i] = f2h(v);
  else reinterpret_cast<float*>(y)[i] = v;
}
// fp16 store followed by the residual add of the rounded value (add_kernel's semantics,
// src/kernels/cuda/mmq.cu:870-876 of the reference): res = f16(f32(res) + f32(f16(v)))
__device__ __forceinline__ void store_out_resadd(uint16_t* y, uint16_t* res, size_t i, float v) {
  const uint16_t h = f2h(v);
  y[i] = h;
  res[i] = f2h(h2f(res[i]) + h2f(h));
}

template <int NMAT, int TT, int MODE, bool F16>
__global__ void __launch_bounds__(kTileThreads) gemv_tile_kernel(const GemvArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int nb = a.nb;
  const int rc = tile_rows(nb);
  int row0 = blockIdx.x * rc;
  // plans and pointer tables may come from the kernel before this one; matrices named in the
  // arguments are fixed, so their copies start first and the wait sits just before the
  // activations are read (tile_run_staged's before_x hook)
  if constexpr (MODE != kDense && MODE != kMulti) {
    pdl_wait();
    pdl_launch_dependents();
  }
  int mat = 0;                           // multi: which matrix this CTA works on
  const size_t row_bytes = static_cast<size_t>(nb) * kW4;
  const size_t xrow_bytes = static_cast<size_t>(nb) * kX8;

  const unsigned char* wsrc[NMAT];
  int nrows, ntok;
  size_t xbase;          // first activation row of this tile
  size_t ybase;          // output row index of token slot 0 (multiplied by n_rows below)
  int ncols = a.n_rows;  // output row length

  if constexpr (MODE == kDense) {
    nrows = min(rc, a.n_rows - row0);
    const int tok0 = blockIdx.y * a.tok_tile;
    ntok = min(a.tok_tile, a.n_tokens - tok0);
#pragma unroll
    for (int m = 0; m < NMAT; ++m) wsrc[m] = a.w[m] + row0 * row_bytes;
    xbase = tok0;
    ybase = tok0;
  } else if constexpr (MODE == kMulti) {
    // tiles of matrix 0, then of matrix 1, then of matrix 2
    const int t0 = (a.rows_cum[0] + rc - 1) / rc;
    const int t1 = t0 + (a.rows_cum[1] - a.rows_cum[0] + rc - 1) / rc;
    int tile = blockIdx.x, rows_m = a.rows_cum[0];
    if (tile >= t1) { mat = 2; tile -= t1; rows_m = a.rows_cum[2] - a.rows_cum[1]; }
    else if (tile >= t0) { mat = 1; tile -= t0; rows_m = a.rows_cum[1] - a.rows_cum[0]; }
    row0 = tile * rc;
    nrows = min(rc, rows_m - row0);
    ntok = 1;
    wsrc[0] = (mat == 0 ? a.wm[0] : (mat == 1 ? a.wm[1] : a.wm[2])) + row0 * row_bytes;
    xbase = 0;
    ybase = 0;
    ncols = 0;
  } else if constexpr (MODE == kPtrs) {
    // y[e * rows_per + r]; every expert reads the SAME activation row, as the
    // reference kernel does (q4_k.cu:184-213 indexes xq[blk] only).
    const int e = blockIdx.y;
    nrows = min(rc, a.rows_per - row0);
    ntok = 1;
    wsrc[0] = a.tab[0][e] + row0 * row_bytes;
    xbase = 0;
    ybase = 0;
    ncols = 0;
  } else if constexpr (MODE == kGrouped) {
    const int job = a.job_of_tile[blockIdx.y];
    const int joff = a.off[job];
    const int tok0 = (blockIdx.y - a.tile_base[job]) * a.tok_tile;
    ntok = min(a.tok_tile, a.m[job] - tok0);
    nrows = min(rc, a.n_rows - row0);
    if (ntok <= 0) return;
#pragma unroll
    for (int m = 0; m < NMAT; ++m) wsrc[m] = a.tab[m][job] + row0 * row_bytes;
    xbase = joff + tok0;
    ybase = joff + tok0;
  } else {
    if (static_cast<int>(blockIdx.y) >= a.meta[1]) return;      // meta = {rows, tiles, bad}
    const int e = expert_of_tile(a.toff, a.n_expert, blockIdx.y);
    const int joff = a.off[e];
    const int tok0 = (blockIdx.y - a.toff[e]) * a.tok_tile;
    ntok = min(a.tok_tile, a.off[e + 1] - joff - tok0);
    nrows = min(rc, a.n_rows - row0);
    if (ntok <= 0) return;
    bool absent = false;
#pragma unroll
    for (int m = 0; m < NMAT; ++m) {
      const unsigned char* base = a.tab[m][e];
      absent = absent || (base == nullptr);
      wsrc[m] = base + row0 * row_bytes;
    }
    if (absent) {
      // Absent expert: its rows read as zero in the combine; the gate/up launch
      // posts the expert id once per tile for the host-side patch
      // (q4_k.cu:697-710 of the reference).
      for (int i = threadIdx.x; i < nrows * ntok; i += kTileThreads) {
        const int r = i % nrows, t = i / nrows;
#pragma unroll
        for (int m = 0; m < NMAT; ++m)
          reinterpret_cast<uint16_t*>(a.y[m])[static_cast<size_t>(joff + tok0 + t) * a.n_rows + row0 + r] = 0;
      }
      if (a.mail != nullptr && blockIdx.x == 0 && threadIdx.x == 0) {
        const int mi = atomicAdd(a.mail_n, 1);
        if (mi < a.n_expert) a.mail[mi] = e;
      }
      return;
    }
    xbase = joff + tok0;
    ybase = joff + tok0;
  }
  if (nrows <= 0 || ntok <= 0) return;

  tile_run_staged<NMAT, TT>(
      smem, wsrc, nrows, nb, ntok,
      [] {
        if constexpr (MODE == kDense || MODE == kMulti) {
          pdl_wait();
          pdl_launch_dependents();
        }
      },
      [&](const XTile& xt, int t0, int nt) {
        xtile_stage(xt, nt, [&](int t) { return a.xq + (xbase + t0 + t) * xrow_bytes; }, threadIdx.x, kTileThreads);
      },
      [&](int r, int t, const float (&v)[NMAT]) {
        if constexpr (MODE == kMulti) {
          uint16_t* ym = mat == 0 ? a.ym[0] : (mat == 1 ? a.ym[1] : a.ym[2]);
          ym[row0 + r] = f2h(v[0]);
          return;
        }
#pragma unroll
        for (int m = 0; m < NMAT; ++m) {
          size_t oi;
          if constexpr (MODE == kPtrs) oi = static_cast<size_t>(blockIdx.y) * a.rows_per + row0 + r;
          else oi = (ybase + t) * ncols + row0 + r;
          if constexpr (MODE == kDense && F16 && NMAT == 1) {
            if (a.res != nullptr) {
              store_out_resadd(reinterpret_cast<uint16_t*>(a.y[0]), a.res, oi, v[0]);
              continue;
            }
          }
          store_out<F16>(a.y[m], oi, v[m]);
        }
      },
      a.status);
}

template <int NMAT, int TT, int MODE, bool F16>
int launch_tile(const GemvArgs& a, dim3 grid, cudaStream_t stream) {
  const size_t smem = tile_smem(NMAT, a.nb, TT);
  if (smem > 200 * 1024) return kErrUnsupported;
  if (smem > 48 * 1024 && !opt_in_smem<gemv_tile_kernel<NMAT, TT, MODE, F16>>(static_cast<int>(smem))) return kErrLaunch;
  // (every launch of the family may start while the kernel before it drains; the kernels wait for that
  // one's results themselves, just before they first read anything it could have written)
  return launch_pdl(gemv_tile_kernel<NMAT, TT, MODE, F16>, grid, kTileThreads, smem, stream, a);
}

// ---- dense matrices far larger than the machine (the LM head): a persistent kernel ----------
// One CTA per SM walks stages of 256 consecutive super-blocks (36,864 contiguous bytes: a
// whole number of rows when nb divides 256), each stage one bulk copy into a five-deep
// ring issued by a producer warp. Thread t of the eight consumer warps owns block t of the
// stage: a quarter-warp reads eight consecutive 144-byte blocks, 16 bytes per lane per
// load, which spreads over all 32 banks without padding. The activations (at most two
// token rows) are staged once per CTA. The nb lanes of a row meet by shuffle.
constexpr int kStreamBlocks = 256;                       // super-blocks per stage = consumer threads
constexpr int kStreamStageBytes = kStreamBlocks * kW4;   // 36,864
constexpr int kStreamStages = 5;
constexpr int kStreamThreads = kStreamBlocks + 32;       // + the producer warp
inline size_t stream_gemv_smem(int nb, int tt) {
  return 128 + static_cast<size_t>(kStreamStages) * kStreamStageBytes + xtile_bytes(tt, nb);
}

template <int TT, bool F16>
__global__ void __launch_bounds__(kStreamThreads, 1) gemv_stream_kernel(const GemvArgs a) {
  extern __shared__ __align__(128) unsigned char smem[];
  uint64_t* full = reinterpret_cast<uint64_t*>(smem);
  uint64_t* empty = full + kStreamStages;
  unsigned char* ring = smem + 128;
  const int nb = a.nb;
  const XTile xt = xtile_at(ring + kStreamStages * kStreamStageBytes, TT, nb);
  const long long total_blocks = static_cast<long long>(a.n_rows) * nb;
  const int n_stages = static_cast<int>((total_blocks + kStreamBlocks - 1) / kStreamBlocks);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int i = 0; i < kStreamStages; ++i) {
      mbar_init(full + i, 1);
      mbar_init(empty + i, kStreamBlocks / 32);
    }
    fence_barrier_init();
    fence_proxy_async();
  }
  __syncthreads();

  bool ok = true;
  if (warp == kStreamBlocks / 32) {                      // producer
    if (lane == 0) {
      int it = 0;
      for (int st = blockIdx.x; st < n_stages; st += gridDim.x, ++it) {
        const int s = it % kStreamStages;
        if (it >= kStreamStages && !mbar_wait(empty + s, ((it / kStreamStages) - 1) & 1)) {
          ok = false;
          break;
        }
        const long long b0 = static_cast<long long>(st) * kStreamBlocks;
        const long long nblk = total_blocks - b0 < kStreamBlocks ? total_blocks - b0 : kStreamBlocks;
        const uint32_t bytes = static_cast<uint32_t>(nblk) * kW4;
        mbar_expect_tx(full + s, bytes);
        bulk_g2s_weights<true>(ring + s * kStreamStageBytes, a.w[0] + b0 * kW4, bytes, full + s);
      }
    }
  } else {
    pdl_wait();                                          // the weight stream above is already running
    pdl_launch_dependents();
    xtile_stage(xt, a.n_tokens, [&](int t) { return a.xq + static_cast<size_t>(t) * nb * kX8; },
                threadIdx.x, kStreamBlocks);
    asm volatile("bar.sync 1, %0;" ::"n"(kStreamBlocks) : "memory");
    const int blk = threadIdx.x & (nb - 1);              // nb is a power of two <= 16
    int it = 0;
    for (int st = blockIdx.x; st < n_stages && ok; st += gridDim.x, ++it) {
      const int s = it % kStreamStages;
      ok = mbar_wait(full + s, (it / kStreamStages) & 1);
      if (!__all_sync(0xFFFFFFFFu, ok)) { ok = false; break; }
      const long long b = static_cast<long long>(st) * kStreamBlocks + threadIdx.x;
      float acc[1][TT];
#pragma unroll
      for (int t = 0; t < TT; ++t) acc[0][t] = 0.f;
      if (b < total_blocks) {
        const uint4* wb[1] = {reinterpret_cast<const uint4*>(ring + s * kStreamStageBytes + threadIdx.x * kW4)};
        block_dot<1, TT>(wb, xt, blk, a.n_tokens, acc);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive_one(empty + s);          // this warp has read its blocks
#pragma unroll
      for (int t = 0; t < TT; ++t) acc[0][t] = reduce_lanes(acc[0][t], nb);
      if (blk == 0 && b < total_blocks) {
        const long long row = b / nb;
#pragma unroll
        for (int t = 0; t < TT; ++t)
          if (t < a.n_tokens) {
            if constexpr (F16 && TT == 1) {
              if (a.res != nullptr) {
                store_out_resadd(reinterpret_cast<uint16_t*>(a.y[0]), a.res, static_cast<size_t>(row), acc[0][t]);
                continue;
              }
            }
            store_out<F16>(a.y[0], static_cast<size_t>(t) * a.n_rows + row, acc[0][t]);
          }
      }
    }
  }
  if (!ok && lane == 0 && a.status != nullptr) atomicExch(a.status, 1);
}

template <int TT, bool F16>
int launch_stream(const GemvArgs& a, int sms, cudaStream_t stream) {
  const size_t smem = stream_gemv_smem(a.nb, TT);
  if (!opt_in_smem<gemv_stream_kernel<TT, F16>>(static_cast<int>(smem))) return kErrLaunch;
  return launch_pdl(gemv_stream_kernel<TT, F16>, dim3(sms), kStreamThreads, smem, stream, a);
}

// The persistent kernel pays off when every SM gets several stages and its dp4a dots keep up: one token row, and two of
// more than eight blocks (248,320 rows of 16 blocks, with norm and top-k: 176 us against 195 by the MMA kernel below; of
// eight blocks 103 against 99; four rows 288 against 231 and 169 against 125).
inline int stream_sms(const GemvArgs& a) {
  if (a.n_tokens > 2 || (a.n_tokens == 2 && a.nb <= 8) || a.nb > 16 || (a.nb & (a.nb - 1)) != 0) return 0;
  if (reinterpret_cast<uintptr_t>(a.w[0]) & 15u) return 0;
  const int sms = device_sms();
  if (sms <= 0) return 0;
  const long long stages = (static_cast<long long>(a.n_rows) * a.nb + kStreamBlocks - 1) / kStreamBlocks;
  return stages >= 8LL * sms ? sms : 0;
}

// ---- dense matrices below the streaming kernel's size, one to eight token rows -----------------
// A launch of a few microseconds: latency decides. A warp owns sixteen rows and every eighth block
// column (rows of fewer than eight blocks: the warps of a CTA take several row groups); each lane
// loads its share of the weight bytes straight into MMA fragment order - the order of k inside a
// sub-block is free as long as both operands use it - before the previous kernel is awaited, then its
// share of that block of the token rows, and ten int8 MMAs leave the exact integer sums of sixteen
// rows x eight tokens without a shuffle. The fp32 terms of a row's blocks meet in shared memory and
// are added in the order of the tile kernels' shuffle tree. dp4a takes 2.2 cycles a warp and
// scheduler for 128 products, this MMA 8 for 4096, a shuffle 4. One token fills an eighth of the MMA
// and goes the dp4a way below (2048 -> 4096 + 512 + 512: 3.1 us against 4.0), several tokens this one
// (2048 -> 4096 at 2 / 4 / 8 rows: 3.1 / 3.3 / 3.4 us, dp4a 3.8 / 5.2 / 8.9). Up to three matrices of the
// same k in one launch, their rows one after another.
constexpr int kDirectWarps = 8;

struct DirectArgs {
  const unsigned char* w[3];
  void* y[3];
  int rows_cum[3];                      // rows of matrices 0..m inclusive
  const unsigned char* xq;
  int nb, n_tokens;
  uint16_t* res;                        // one token, fp16 out: residual row updated in place
  __device__ __forceinline__ int matrix_of(int row) const { return row >= rows_cum[0] ? (row >= rows_cum[1] ? 2 : 1) : 0; }
  __device__ __forceinline__ int first_row(int m) const { return m == 0 ? 0 : (m == 1 ? rows_cum[0] : rows_cum[1]); }
};

// The terms of the NI block columns blk0, blk0 + 8, ... that are in registers: sixteen rows x eight tokens.
template <int NI, int NA>
__device__ __forceinline__ void direct_blocks(const DirectArgs& a, const uint4 (&hdr)[2][NI], const uint2 (&q)[2][NI][4], int blk0,
                                              int gid, int tig, float (&acc)[NA][4]) {
  const int zero[4] = {0, 0, 0, 0};
#pragma unroll
  for (int i = 0; i < NI; ++i) {
    // token gid's codes in the weights' order of k, its sums 4 tig .. 4 tig + 3, the scales of tokens 2 tig, 2 tig + 1
    uint32_t b[8][2] = {};
    uint32_t s01 = 0u, s23 = 0u;
    float xd[2] = {0.f, 0.f};
    const int blk = blk0 + 8 * i;
    if (gid < a.n_tokens) {
      const uint32_t* xb = reinterpret_cast<const uint32_t*>(a.xq + (static_cast<size_t>(gid) * a.nb + blk) * kX8);
#pragma unroll
      for (int sb = 0; sb < 8; ++sb) {
        b[sb][0] = __ldg(xb + 1 + 8 * sb + 2 * tig);
        b[sb][1] = __ldg(xb + 2 + 8 * sb + 2 * tig);
      }
      if (tig < 2) {
        s01 = __ldg(xb + 65 + 2 * tig);
        s23 = __ldg(xb + 66 + 2 * tig);
      }
    }
#pragma unroll
    for (int j = 0; j < 2; ++j)
      if (2 * tig + j < a.n_tokens) xd[j] = __ldg(reinterpret_cast<const float*>(a.xq + (static_cast<size_t>(2 * tig + j) * a.nb + blk) * kX8));
    const Scales6 sl = unpack_scales6(hdr[0][i].y, hdr[0][i].z, hdr[0][i].w), sh = unpack_scales6(hdr[1][i].y, hdr[1][i].z, hdr[1][i].w);
    int isum[4] = {0, 0, 0, 0};
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      const uint32_t raw[4] = {q[0][i][g].x, q[1][i][g].x, q[0][i][g].y, q[1][i][g].y};
      uint32_t lo[4], hi[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        lo[j] = raw[j] & 0x0F0F0F0Fu;
        hi[j] = raw[j] & 0xF0F0F0F0u;        // 16 q: the even sub-block's scale is taken 16-fold, d a sixteenth (exact)
      }
      const int shift = 16 * (g & 1);
      const int sc0_lo = ((sl.sc[g >> 1] >> shift) & 0xFF) << 4, sc1_lo = (sl.sc[g >> 1] >> (shift + 8)) & 0xFF;
      const int sc0_hi = ((sh.sc[g >> 1] >> shift) & 0xFF) << 4, sc1_hi = (sh.sc[g >> 1] >> (shift + 8)) & 0xFF;
      int e0[4], e1[4];
      mma_u8s8(e0, lo, b[2 * g][0], b[2 * g][1], zero);
      mma_u8s8(e1, hi, b[2 * g + 1][0], b[2 * g + 1][1], zero);
      isum[0] += sc0_lo * e0[0] + sc1_lo * e1[0];
      isum[1] += sc0_lo * e0[1] + sc1_lo * e1[1];
      isum[2] += sc0_hi * e0[2] + sc1_hi * e1[2];
      isum[3] += sc0_hi * e0[3] + sc1_hi * e1[3];
    }
    // min term: the eight min bytes of a row are k = 0..7, the sums split as 128 * hi + lo
    const uint32_t ma[4] = {tig == 0 ? sl.mn[0] : (tig == 1 ? sl.mn[1] : 0u), tig == 0 ? sh.mn[0] : (tig == 1 ? sh.mn[1] : 0u), 0u, 0u};
    int dl[4], dh[4];
    mma_u8s8(dl, ma, __byte_perm(s01 & 0x007F007Fu, s23 & 0x007F007Fu, 0x6420), 0u, zero);
    mma_u8s8(dh, ma, __byte_perm((s01 >> 7) & 0x00FF00FFu, (s23 >> 7) & 0x00FF00FFu, 0x6420), 0u, zero);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint4& hd = hdr[j >> 1][i];
      const float d = 0.0625f * h2f(static_cast<uint16_t>(hd.x & 0xFFFFu)), dmin = h2f(static_cast<uint16_t>(hd.x >> 16));
      acc[i % NA][j] += xd[j & 1] * (d * static_cast<float>(isum[j]) - dmin * static_cast<float>(dl[j] + 128 * dh[j]));
    }
  }
}

// STREAM: weights first to leave L2 (launch_direct)
// NI: block columns per warp (1 for rows of up to eight blocks); LONG: rows of more than 32 blocks, 32 at a time
template <int NI, bool F16, bool STREAM, bool LONG = false>
__global__ void __launch_bounds__(kDirectWarps * 32) gemv_direct_kernel(const DirectArgs a) {
  __shared__ float red[kDirectWarps][8][16];                // [warp][token][row]
  const int nb = a.nb, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int gid = lane >> 2, tig = lane & 3;
  const int wpg = NI > 1 ? kDirectWarps : min(nb, kDirectWarps);        // warps per row group
  const int groups = kDirectWarps / wpg, total = a.rows_cum[2];
  const int cta_row0 = blockIdx.x * groups * 16;
  const int row0 = cta_row0 + warp / wpg * 16, blk0 = warp & (wpg - 1);
  uint4 hdr[2][NI];
  uint2 q[2][NI][4];
  auto fetch = [&](int c0) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int row = min(row0 + gid + 8 * h, total - 1), m = a.matrix_of(row);
      const unsigned char* wb = (m == 0 ? a.w[0] : (m == 1 ? a.w[1] : a.w[2])) +
                                (static_cast<size_t>(row - a.first_row(m)) * nb + blk0 + c0) * kW4;
#pragma unroll
      for (int i = 0; i < NI; ++i) {
        hdr[h][i] = load_weights<STREAM>(reinterpret_cast<const uint4*>(wb + i * 8 * kW4));
#pragma unroll
        for (int g = 0; g < 4; ++g) q[h][i][g] = load_weights<STREAM>(reinterpret_cast<const uint2*>(wb + i * 8 * kW4 + 16 + 32 * g + 8 * tig));
      }
    }
  };
  fetch(0);
  pdl_wait();
  pdl_launch_dependents();
  constexpr int NA = NI > 2 ? 2 : 1;        // rows of 32 blocks: (t0 + t2) + (t1 + t3), the shuffle tree's order
  float acc[NA][4];
#pragma unroll
  for (int c = 0; c < NA; ++c)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[c][j] = 0.f;
  direct_blocks<NI, NA>(a, hdr, q, blk0, gid, tig, acc);
  if constexpr (LONG) {
    for (int c0 = 8 * NI; c0 < nb; c0 += 8 * NI) {
      fetch(c0);
      direct_blocks<NI, NA>(a, hdr, q, blk0 + c0, gid, tig, acc);
    }
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    float v = acc[0][j];
    if constexpr (NA > 1) v += acc[1][j];
    red[warp][2 * tig + (j & 1)][gid + 8 * (j >> 1)] = v;
  }
  __syncthreads();
  for (int o = threadIdx.x; o < groups * 16 * a.n_tokens; o += kDirectWarps * 32) {
    const int r = o & 15, t = (o >> 4) % a.n_tokens, grp = (o >> 4) / a.n_tokens;
    const int row = cta_row0 + grp * 16 + r;
    if (row >= total) continue;
    float v[kDirectWarps];
#pragma unroll
    for (int w = 0; w < kDirectWarps; ++w) v[w] = w < wpg ? red[grp * wpg + w][t][r] : 0.f;
    if (wpg == 8) {
#pragma unroll
      for (int w = 0; w < 4; ++w) v[w] += v[w + 4];
    }
    if (wpg >= 4) { v[0] += v[2]; v[1] += v[3]; }
    if (wpg >= 2) v[0] += v[1];
    const int m = a.matrix_of(row), first = a.first_row(m);
    void* y = m == 0 ? a.y[0] : (m == 1 ? a.y[1] : a.y[2]);
    const int m_rows = (m == 0 ? a.rows_cum[0] : (m == 1 ? a.rows_cum[1] : a.rows_cum[2])) - first;
    store_out<F16>(y, static_cast<size_t>(t) * m_rows + row - first, v[0]);
  }
}

// One token: a warp per row (rows of fewer than eight blocks: several), one lane per 32-byte nibble group,
// the token laid out in shared memory once per CTA so that a lane's 64 codes, two sums and scale are five
// conflict-free reads (a group is 80 bytes, a block 320). The integer partial sums of a super-block meet
// exactly by shuffle over its four lanes, the blocks' terms in the tile kernels' shuffle tree.
constexpr int kDirectGroup = 80, kDirectBlock = 4 * kDirectGroup;

// STREAM: weights first to leave L2 (launch_direct)
template <int NI, bool F16, bool STREAM>
__global__ void __launch_bounds__(kDirectWarps * 32) gemv_direct1_kernel(const DirectArgs a) {
  __shared__ __align__(16) unsigned char xs[32 * kDirectBlock];
  const int nb = a.nb, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int lpr = NI > 1 ? 32 : min(nb * 4, 32);           // lanes per row (a power of two >= 4)
  const int lr = lane & (lpr - 1), g = lr & 3, blk0 = lr >> 2;
  const int total = a.rows_cum[2];
  const int row_raw = (blockIdx.x * kDirectWarps + warp) * (32 / lpr) + lane / lpr;
  const int row = min(row_raw, total - 1), m = a.matrix_of(row), first = a.first_row(m);    // every lane runs the same loops
  const unsigned char* wb = (m == 0 ? a.w[0] : (m == 1 ? a.w[1] : a.w[2])) + (static_cast<size_t>(row - first) * nb + blk0) * kW4;
  uint4 hdr[NI], q0[NI], q1[NI];
#pragma unroll
  for (int i = 0; i < NI; ++i) {
    hdr[i] = load_weights<STREAM>(reinterpret_cast<const uint4*>(wb + i * 8 * kW4));
    q0[i] = load_weights<STREAM>(reinterpret_cast<const uint4*>(wb + i * 8 * kW4 + 16 + 32 * g));
    q1[i] = load_weights<STREAM>(reinterpret_cast<const uint4*>(wb + i * 8 * kW4 + 32 + 32 * g));
  }
  pdl_wait();
  pdl_launch_dependents();
  for (int b = warp; b < nb; b += kDirectWarps) {
    const uint32_t* src = reinterpret_cast<const uint32_t*>(a.xq + static_cast<size_t>(b) * kX8) + lane;
    const uint32_t v0 = __ldg(src), v1 = __ldg(src + 32), v2 = lane < 5 ? __ldg(src + 64) : 0u;
    unsigned char* dst = xs + b * kDirectBlock;            // word 0: scale; 1..64: codes; 65..68: sums
    auto put = [&](int w, uint32_t x) { *reinterpret_cast<uint32_t*>(dst + (w >> 4) * kDirectGroup + (w & 15) * 4) = x; };
    if (lane > 0) put(lane - 1, v0);
    put(lane + 31, v1);
    if (lane == 0) put(63, v2);
    else if (lane < 5) *reinterpret_cast<uint32_t*>(dst + (lane - 1) * kDirectGroup + 64) = v2;
    const uint32_t d = __shfl_sync(0xFFFFFFFFu, v0, 0);
    if (lane < 4) *reinterpret_cast<uint32_t*>(dst + lane * kDirectGroup + 68) = d;
  }
  __syncthreads();
  float acc[2] = {0.f, 0.f};                // rows of 32 blocks: (t0 + t2) + (t1 + t3), the shuffle tree's order
#pragma unroll
  for (int i = 0; i < NI; ++i) {
    const unsigned char* xb = xs + (blk0 + 8 * i) * kDirectBlock + g * kDirectGroup;
    const uint4 x0 = *reinterpret_cast<const uint4*>(xb), x1 = *reinterpret_cast<const uint4*>(xb + 16);
    const uint4 x2 = *reinterpret_cast<const uint4*>(xb + 32), x3 = *reinterpret_cast<const uint4*>(xb + 48);
    const uint2 sd = *reinterpret_cast<const uint2*>(xb + 64);
    const Scales6 s6 = unpack_scales6(hdr[i].y, hdr[i].z, hdr[i].w);
    const uint32_t scw = (g < 2 ? s6.sc[0] : s6.sc[1]) >> (16 * (g & 1)), mnw = (g < 2 ? s6.mn[0] : s6.mn[1]) >> (16 * (g & 1));
    const uint32_t raw[8] = {q0[i].x, q0[i].y, q0[i].z, q0[i].w, q1[i].x, q1[i].y, q1[i].z, q1[i].w};
    uint32_t lo[8], hi[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      lo[j] = raw[j] & 0x0F0F0F0Fu;
      hi[j] = (raw[j] >> 4) & 0x0F0F0F0Fu;
    }
    int isum = static_cast<int>(scw & 0xFF) * dot8(lo, x0, x1) + static_cast<int>((scw >> 8) & 0xFF) * dot8(hi, x2, x3);
    int msum = static_cast<int>(mnw & 0xFF) * static_cast<int16_t>(sd.x & 0xFFFFu) + static_cast<int>((mnw >> 8) & 0xFF) * static_cast<int16_t>(sd.x >> 16);
    isum += __shfl_xor_sync(0xFFFFFFFFu, isum, 1);
    msum += __shfl_xor_sync(0xFFFFFFFFu, msum, 1);
    isum += __shfl_xor_sync(0xFFFFFFFFu, isum, 2);
    msum += __shfl_xor_sync(0xFFFFFFFFu, msum, 2);
    const float d = h2f(static_cast<uint16_t>(hdr[i].x & 0xFFFFu)), dmin = h2f(static_cast<uint16_t>(hdr[i].x >> 16));
    acc[i & 1] += __uint_as_float(sd.y) * (d * static_cast<float>(isum) - dmin * static_cast<float>(msum));
  }
  float v = acc[0];
  if constexpr (NI > 1) v += acc[1];
  for (int off = lpr >> 1; off >= 4; off >>= 1) v += __shfl_down_sync(0xFFFFFFFFu, v, off);
  if (lr != 0 || row_raw >= total) return;
  void* y = m == 0 ? a.y[0] : (m == 1 ? a.y[1] : a.y[2]);
  if constexpr (F16) {
    if (a.res != nullptr) {
      store_out_resadd(reinterpret_cast<uint16_t*>(y), a.res, static_cast<size_t>(row - first), v);
      return;
    }
  }
  store_out<F16>(y, static_cast<size_t>(row - first), v);
}

// One to eight token rows, rows of a power of two of blocks (one token: up to 32), 16-byte aligned matrices.
inline bool direct_fits(const DirectArgs& a) {
  if (a.n_tokens < 1 || a.n_tokens > 8 || (a.n_tokens == 1 && a.nb > 32) || (a.nb & (a.nb - 1)) != 0) return false;
  for (int m = 0; m < 3; ++m)
    if (reinterpret_cast<uintptr_t>(a.w[m]) & 15u) return false;
  return true;
}
template <bool F16>
int launch_direct(const DirectArgs& a, cudaStream_t stream) {
  const int threads = kDirectWarps * 32;
  // Launches of four megabytes of weights and more - two for several rows - are taken for those of a model that L2 does not hold
  // between two steps: as the first to leave, its weights no longer push out the kernels' code and activations. What decides is
  // whether the weights are still in L2 at their next use, which a launch cannot know; both sides, in us per step from a
  // graph, ordinary lines / first to leave:
  //   projections of 4096 + 2 x 512 from 2048 and 2048 from 4096 with nothing in between, one row: 4 / 6 / 8 / 10 / 24 / 40 layers
  //   39.5 / 55.8 / 77 / 107 / 259 / 424 and 40.0 / 60.5 / 82 / 101 / 240 / 407 - six or eight such layers, which just fit, lose -,
  //   four rows: 4 / 8 / 24 layers 56 / 119 / 375 and 54 / 110 / 332;
  //   with a layer's experts in between, as a model has them (256 experts, 2048 / 512), one row: 2 / 4 / 8 / 12 layers
  //   49 / 108 / 215 / 319 and 49 / 100 / 198 / 302.
  // Below the line, where a model of many layers may stay in L2, the lines keep their place. 2048 + 2 x 512 from 2048 and 2048 from
  // 2048 (2.4 MB the largest), 8 / 12 / 16 / 24 layers: one row ordinary 63 / 96 / 138 / 224, first 71 / 105 / 130 / 203; four rows ordinary
  // 89 / 135 / 202 / 319, first 86 / 128 / 171 / 258, keeping their place 85 / 128 / 191 / 297. 2048 + 2 x 256 from 1024 and 1024 from
  // 2048 (1.2 MB), 24 layers, four rows: 219, 224, 211.
  const bool first = static_cast<long long>(a.rows_cum[2]) * a.nb * kW4 >= (a.n_tokens == 1 ? 4 : 2) << 20;
  auto launch = [&](auto stream_weights) {
    constexpr bool S = decltype(stream_weights)::value;
    if (a.n_tokens == 1) {
      const int rows_cta = kDirectWarps * std::max(1, 8 / a.nb);
      const dim3 grid((a.rows_cum[2] + rows_cta - 1) / rows_cta);
      if (a.nb <= 8) return launch_pdl(gemv_direct1_kernel<1, F16, S>, grid, threads, 0, stream, a);
      if (a.nb == 16) return launch_pdl(gemv_direct1_kernel<2, F16, S>, grid, threads, 0, stream, a);
      return launch_pdl(gemv_direct1_kernel<4, F16, S>, grid, threads, 0, stream, a);
    }
    const int rows_cta = 16 * std::max(1, kDirectWarps / a.nb);
    const dim3 grid((a.rows_cum[2] + rows_cta - 1) / rows_cta);
    if (a.nb <= 8) return launch_pdl(gemv_direct_kernel<1, F16, S>, grid, threads, 0, stream, a);
    if (a.nb == 16) return launch_pdl(gemv_direct_kernel<2, F16, S>, grid, threads, 0, stream, a);
    if (a.nb == 32) return launch_pdl(gemv_direct_kernel<4, F16, S>, grid, threads, 0, stream, a);
    return launch_pdl(gemv_direct_kernel<4, F16, S, true>, grid, threads, 0, stream, a);
  };
  return first ? launch(std::true_type{}) : launch(std::false_type{});
}

// Where the tile kernel's CTAs, which copy their rows by one bulk copy each, are faster than the direct ones (us, direct / tile):
// many rows of one or two blocks, whose lanes have little else in flight (one token, 24,000 / 60,000 rows of one block
// 2.3 / 2.6, 3.5 / 3.1; 32,000 / 100,000 of two 3.8 / 3.5, 8.0 / 6.0; five to eight tokens 60,000 rows of one block 5.7 / 5.0), and
// one token's rows of four or eight blocks that fill most of a single wave of them (20,000 of eight blocks 7.5 / 7.2, 16,000 6.5 /
// 7.0, 24,000 - a second wave - 8.9 / 10.0; 40,000 of four 7.0 / 6.4, 60,000 9.6 / 10.5).
inline bool tile_wins(const GemvArgs& a) {
  if (a.nb > 8 || (a.n_tokens != 1 && (a.nb > 1 || a.n_tokens < 5))) return false;
  const long long sms = device_sms(), rows = a.n_rows;
  if (a.nb <= 2) return rows > 190 * sms;
  const long long resident = 227 * 1024 / static_cast<long long>(tile_smem(1, a.nb, 1) + 1024), wave = sms * resident * tile_rows(a.nb);
  return rows <= wave && 100 * rows > 72 * wave;
}

// tokens per CTA of the dense multi-token kernels (walked in sub-tiles of 8)
constexpr int kDenseTokTile = 16;

template <int NMAT, bool F16>
int launch_dense(const void* w0, const void* w1, const void* xq, void* y0, void* y1, int n_rows,
                 int k, int n_tokens, cudaStream_t stream, uint16_t* res = nullptr) {
  if (n_tokens <= 0 || n_rows <= 0) return kOk;
  if (!w0 || !xq || !y0 || (NMAT == 2 && (!w1 || !y1)) || k <= 0 || k % kQK != 0) return kErrArg;
  if (reinterpret_cast<uintptr_t>(xq) & 3u) return kErrAlign;
  GemvArgs a{};
  a.w[0] = static_cast<const unsigned char*>(w0);
  a.w[1] = static_cast<const unsigned char*>(w1);
  a.xq = static_cast<const unsigned char*>(xq);
  a.y[0] = y0;
  a.y[1] = y1;
  a.n_rows = n_rows;
  a.nb = k / kQK;
  a.n_tokens = n_tokens;
  a.status = status_word();
  a.res = res;
  const int rc = tile_rows(a.nb);
  if constexpr (NMAT == 1) {
    if (const int sms = stream_sms(a)) {
      if (n_tokens == 1) return launch_stream<1, F16>(a, sms, stream);
      return launch_stream<2, F16>(a, sms, stream);
    }
  }
  if (NMAT == 2 || !tile_wins(a)) {
    DirectArgs d{{a.w[0], NMAT == 2 ? a.w[1] : nullptr, nullptr}, {y0, y1, nullptr}, {n_rows, NMAT * n_rows, NMAT * n_rows}, a.xq, a.nb, n_tokens, res};
    if (NMAT * static_cast<long long>(n_rows) <= 0x7FFFFFFF && direct_fits(d)) return launch_direct<F16>(d, stream);
  }
  if (n_tokens == 1) {
    a.tok_tile = 1;
    return launch_tile<NMAT, 1, kDense, F16>(a, dim3((n_rows + rc - 1) / rc, 1), stream);
  }
  if (n_tokens <= 4) {              // (block counts that are no power of two, matrices off a 16-byte boundary)
    a.tok_tile = 4;
    return launch_tile<NMAT, 4, kDense, F16>(a, dim3((n_rows + rc - 1) / rc, 1), stream);
  }
  a.tok_tile = kDenseTokTile;
  return launch_tile<NMAT, 8, kDense, F16>(
      a, dim3((n_rows + rc - 1) / rc, (n_tokens + kDenseTokTile - 1) / kDenseTokTile), stream);
}

template <int NMAT>
int launch_grouped(const void* const* t0, const void* const* t1, const int* off, const int* m,
                   const int* tile_base, const int* job_of_tile, int n_tiles, const void* xq,
                   void* y0, void* y1, int n_rows, int k, int tok_per, cudaStream_t stream) {
  if (n_tiles <= 0) return kOk;
  if (!t0 || (NMAT == 2 && (!t1 || !y1)) || !off || !m || !tile_base || !job_of_tile || !xq ||
      !y0 || n_rows <= 0 || k <= 0 || k % kQK != 0 || tok_per <= 0)
    return kErrArg;
  if (reinterpret_cast<uintptr_t>(xq) & 3u) return kErrAlign;
  GemvArgs a{};
  a.tab[0] = reinterpret_cast<const unsigned char* const*>(t0);
  a.tab[1] = reinterpret_cast<const unsigned char* const*>(t1);
  a.off = off; a.m = m; a.tile_base = tile_base; a.job_of_tile = job_of_tile;
  a.xq = static_cast<const unsigned char*>(xq);
  a.y[0] = y0; a.y[1] = y1;
  a.n_rows = n_rows; a.nb = k / kQK; a.tok_tile = tok_per;
  a.status = status_word();
  const int rc = tile_rows(a.nb);
  const dim3 grid((n_rows + rc - 1) / rc, n_tiles);
  return tok_per == 1 ? launch_tile<NMAT, 1, kGrouped, true>(a, grid, stream)
                      : launch_tile<NMAT, 8, kGrouped, true>(a, grid, stream);
}

template <int NMAT>
int launch_tab(const void* const* t0, const void* const* t1, const int* off, const int* toff,
               const int* meta, int* mail, int* mail_n, int tiles_max, const void* xq, void* y0,
               void* y1, int n_rows, int k, int n_expert, int tok_per, cudaStream_t stream) {
  if (tiles_max <= 0) return kOk;
  if (!t0 || (NMAT == 2 && (!t1 || !y1)) || !off || !toff || !meta || !xq || !y0 || n_rows <= 0 ||
      k <= 0 || k % kQK != 0 || tok_per <= 0 || n_expert <= 0 || (mail && !mail_n))
    return kErrArg;
  if (reinterpret_cast<uintptr_t>(xq) & 3u) return kErrAlign;
  GemvArgs a{};
  a.tab[0] = reinterpret_cast<const unsigned char* const*>(t0);
  a.tab[1] = reinterpret_cast<const unsigned char* const*>(t1);
  a.off = off; a.toff = toff; a.meta = meta; a.mail = mail; a.mail_n = mail_n;
  a.xq = static_cast<const unsigned char*>(xq);
  a.y[0] = y0; a.y[1] = y1;
  a.n_rows = n_rows; a.nb = k / kQK; a.tok_tile = tok_per; a.n_expert = n_expert;
  a.status = status_word();
  const int rc = tile_rows(a.nb);
  const dim3 grid((n_rows + rc - 1) / rc, tiles_max);
  return tok_per == 1 ? launch_tile<NMAT, 1, kTab, true>(a, grid, stream)
                      : launch_tile<NMAT, 8, kTab, true>(a, grid, stream);
}

// Raw int32 sub-block dots of token 0: out[(r*nb + blk)*8 + s]. Parity probe for
// the integer unit every kernel shares (block_dot).
__global__ void subblock_dots_kernel(const unsigned char* w, const unsigned char* xq, int* out,
                                     int n_rows, int nb) {
  extern __shared__ __align__(16) unsigned char smem[];
  unsigned char* wsm = smem;                       // one block per thread
  const XTile xt = xtile_at(smem + static_cast<size_t>(blockDim.x) * kW4, 1, nb);
  xtile_stage(xt, 1, [&](int) { return xq; }, threadIdx.x, blockDim.x);
  const int i = blockIdx.x * blockDim.x + threadIdx.x;   // (row, blk) pair
  const bool live = i < n_rows * nb;
  if (live) {
    const unsigned char* src = w + static_cast<size_t>(i) * kW4;
    for (int b = 0; b < kW4 / 2; ++b)
      reinterpret_cast<uint16_t*>(wsm + threadIdx.x * kW4)[b] = reinterpret_cast<const uint16_t*>(src)[b];
  }
  __syncthreads();
  if (!live) return;
  float acc[1][1] = {{0.f}};
  int dots[8];
  const uint4* wb[1] = {reinterpret_cast<const uint4*>(wsm + threadIdx.x * kW4)};
  block_dot<1, 1>(wb, xt, i % nb, 1, acc, dots);
  for (int s = 0; s < 8; ++s) out[static_cast<size_t>(i) * 8 + s] = dots[s];
}

}  // namespace
}  // namespace sgr

using namespace sgr;

SGR_API int sgr_gemv_q4_k_q8(const void* w, const void* x_q8, float* y, int n_rows, int k,
                             void* stream) {
  return launch_dense<1, false>(w, nullptr, x_q8, y, nullptr, n_rows, k, 1, as_stream(stream));
}

SGR_API int sgr_gemv_q4_k_q8_f16out(const void* w, const void* x_q8, uint16_t* y, int n_rows, int k,
                                    void* stream) {
  return launch_dense<1, true>(w, nullptr, x_q8, y, nullptr, n_rows, k, 1, as_stream(stream));
}

// cuda_ops.hpp:169-171 of the reference: the fp16 GEMV and, on the rounded result, the residual add.
// Same kernels as sgr_gemv_q4_k_q8_f16out, so y is bit-identical to it and res_inout to an add after it.
SGR_API int sgr_gemv_q4_k_q8_f16out_resadd(const void* w, const void* x_q8, uint16_t* y, uint16_t* res_inout,
                                           int n_rows, int k, void* stream) {
  if (n_rows > 0 && !res_inout) return kErrArg;
  return launch_dense<1, true>(w, nullptr, x_q8, y, nullptr, n_rows, k, 1, as_stream(stream), res_inout);
}

namespace {
// cuda_ops.hpp:156-164 of the reference: two or three projections of one token row in one launch.
int launch_multi(int nmat, const void* const (&w)[3], const void* xq, uint16_t* const (&y)[3], const int (&rows)[3],
                 int k, cudaStream_t stream) {
  int total = 0;
  for (int m = 0; m < nmat; ++m) {
    if (rows[m] < 0) return kErrArg;
    total += rows[m];
  }
  if (total == 0) return kOk;
  if (!xq || k <= 0 || k % kQK != 0) return kErrArg;
  for (int m = 0; m < nmat; ++m)
    if (rows[m] > 0 && (!w[m] || !y[m])) return kErrArg;
  if (reinterpret_cast<uintptr_t>(xq) & 3u) return kErrAlign;
  GemvArgs a{};
  int cum = 0, tiles = 0;
  DirectArgs d{};
  a.nb = k / kQK;
  const int rc = tile_rows(a.nb);
  for (int m = 0; m < 3; ++m) {
    const int r = m < nmat ? rows[m] : 0;
    a.wm[m] = m < nmat ? static_cast<const unsigned char*>(w[m]) : nullptr;
    a.ym[m] = m < nmat ? y[m] : nullptr;
    cum += r;
    a.rows_cum[m] = cum;
    d.w[m] = a.wm[m]; d.y[m] = a.ym[m]; d.rows_cum[m] = cum;
    tiles += (r + rc - 1) / rc;
  }
  a.xq = static_cast<const unsigned char*>(xq);
  a.n_rows = total;
  a.n_tokens = 1;
  a.tok_tile = 1;
  a.status = status_word();
  d.xq = a.xq; d.nb = a.nb; d.n_tokens = 1;
  if (direct_fits(d)) return launch_direct<true>(d, stream);
  return launch_tile<1, 1, kMulti, true>(a, dim3(tiles, 1), stream);
}
}  // namespace

SGR_API int sgr_gemv2m_q4_k_q8_f16out(const void* w1, const void* w2, const void* xq, uint16_t* y1, uint16_t* y2,
                                      int rows1, int rows2, int k, int slot, void* stream) {
  (void)slot;                              // the reference keys a per-layer parameter block by it; nothing to key here
  const void* const w[3] = {w1, w2, nullptr};
  uint16_t* const y[3] = {y1, y2, nullptr};
  const int rows[3] = {rows1, rows2, 0};
  return launch_multi(2, w, xq, y, rows, k, as_stream(stream));
}

SGR_API int sgr_gemv3m_q4_k_q8_f16out(const void* w1, const void* w2, const void* w3, const void* xq, uint16_t* y1,
                                      uint16_t* y2, uint16_t* y3, int rows1, int rows2, int rows3, int k, int slot,
                                      void* stream) {
  (void)slot;
  const void* const w[3] = {w1, w2, w3};
  uint16_t* const y[3] = {y1, y2, y3};
  const int rows[3] = {rows1, rows2, rows3};
  return launch_multi(3, w, xq, y, rows, k, as_stream(stream));
}

SGR_API int sgr_gemv_q4_k_q8_batched(const void* w, const void* x_q8, float* y, int n_rows, int k,
                                     int n_tokens, void* stream) {
  return launch_dense<1, false>(w, nullptr, x_q8, y, nullptr, n_rows, k, n_tokens, as_stream(stream));
}

SGR_API int sgr_gemv_q4_k_q8_f16out_batched(const void* w, const void* x_q8, uint16_t* y,
                                            int n_rows, int k, int n_tokens, void* stream) {
  return launch_dense<1, true>(w, nullptr, x_q8, y, nullptr, n_rows, k, n_tokens, as_stream(stream));
}

SGR_API int sgr_gemv_q4_k_q8_f16out_mtok(const void* w, const void* xq, uint16_t* y, int n_rows,
                                         int k, int n_tokens, void* stream) {
  return launch_dense<1, true>(w, nullptr, xq, y, nullptr, n_rows, k, n_tokens, as_stream(stream));
}

SGR_API int sgr_mmq_q4_k_q8_f16out(const void* w, const void* xq, uint16_t* y, int n_rows, int k,
                                   int n_tokens, void* stream) {
  return launch_dense<1, true>(w, nullptr, xq, y, nullptr, n_rows, k, n_tokens, as_stream(stream));
}

SGR_API int sgr_gemv2_q4_k_q8_f16out_mtok(const void* wg, const void* wu, const void* xq,
                                          uint16_t* yg, uint16_t* yu, int n_rows, int k,
                                          int n_tokens, void* stream) {
  return launch_dense<2, true>(wg, wu, xq, yg, yu, n_rows, k, n_tokens, as_stream(stream));
}

SGR_API int sgr_mmq2_q4_k_q8_f16out(const void* wg, const void* wu, const void* xq, uint16_t* yg,
                                    uint16_t* yu, int n_rows, int k, int n_tokens, void* stream) {
  return launch_dense<2, true>(wg, wu, xq, yg, yu, n_rows, k, n_tokens, as_stream(stream));
}

SGR_API int sgr_gemv_ptrs_q4_k_q8_f16out(const void* const* ptrs, const void* x_q8, uint16_t* y,
                                         int n_ptrs, int rows_per, int k, void* stream) {
  if (n_ptrs <= 0 || rows_per <= 0) return kOk;
  if (!ptrs || !x_q8 || !y || k <= 0 || k % kQK != 0) return kErrArg;
  if (reinterpret_cast<uintptr_t>(x_q8) & 3u) return kErrAlign;
  GemvArgs a{};
  a.tab[0] = reinterpret_cast<const unsigned char* const*>(ptrs);
  a.xq = static_cast<const unsigned char*>(x_q8);
  a.y[0] = y;
  a.rows_per = rows_per;
  a.n_rows = rows_per;
  a.nb = k / kQK;
  a.tok_tile = 1;
  a.status = status_word();
  const int rc = tile_rows(a.nb);
  return launch_tile<1, 1, kPtrs, true>(a, dim3((rows_per + rc - 1) / rc, n_ptrs), as_stream(stream));
}

SGR_API int sgr_gemv_grouped2_q4_k_q8_f16out_mtok(const void* const* wg, const void* const* wu,
                                                  const int* off, const int* m,
                                                  const int* tile_base, const int* job_of_tile,
                                                  int n_tiles, const void* xq, uint16_t* yg,
                                                  uint16_t* yu, int n_rows, int k, int tok_per,
                                                  void* stream) {
  return launch_grouped<2>(wg, wu, off, m, tile_base, job_of_tile, n_tiles, xq, yg, yu, n_rows, k,
                           tok_per, as_stream(stream));
}

SGR_API int sgr_gemv_grouped_q4_k_q8_f16out_mtok(const void* const* w, const int* off, const int* m,
                                                 const int* tile_base, const int* job_of_tile,
                                                 int n_tiles, const void* xq, uint16_t* y,
                                                 int n_rows, int k, int tok_per, void* stream) {
  return launch_grouped<1>(w, nullptr, off, m, tile_base, job_of_tile, n_tiles, xq, y, nullptr,
                           n_rows, k, tok_per, as_stream(stream));
}

SGR_API int sgr_gemv_grouped2_tab_q4_k_q8_f16out_mtok(
    const void* const* wg_tab, const void* const* wu_tab, const int* off, const int* toff,
    const int* meta, int* mail, int* mail_n, int tiles_max, const void* xq, uint16_t* yg,
    uint16_t* yu, int n_rows, int k, int n_expert, int tok_per, void* stream) {
  return launch_tab<2>(wg_tab, wu_tab, off, toff, meta, mail, mail_n, tiles_max, xq, yg, yu, n_rows,
                       k, n_expert, tok_per, as_stream(stream));
}

SGR_API int sgr_gemv_grouped_tab_q4_k_q8_f16out_mtok(const void* const* w_tab, const int* off,
                                                     const int* toff, const int* meta,
                                                     int tiles_max, const void* xq, uint16_t* y,
                                                     int n_rows, int k, int n_expert, int tok_per,
                                                     void* stream) {
  return launch_tab<1>(w_tab, nullptr, off, toff, meta, nullptr, nullptr, tiles_max, xq, y, nullptr,
                       n_rows, k, n_expert, tok_per, as_stream(stream));
}

SGR_API int sgr_q4k_subblock_dots(const void* w, const void* x_q8, int* out, int n_rows, int k,
                                  void* stream) {
  if (!w || !x_q8 || !out || n_rows <= 0 || k <= 0 || k % kQK != 0) return kErrArg;
  if (reinterpret_cast<uintptr_t>(x_q8) & 3u) return kErrAlign;
  const int nb = k / kQK;
  const int threads = 128;
  const size_t smem = static_cast<size_t>(threads) * kW4 + xtile_bytes(1, nb);
  if (smem > 48 * 1024) return kErrUnsupported;
  subblock_dots_kernel<<<(n_rows * nb + threads - 1) / threads, threads, smem, as_stream(stream)>>>(
      static_cast<const unsigned char*>(w), static_cast<const unsigned char*>(x_q8), out, n_rows, nb);
  return cudaPeekAtLastError() == cudaSuccess ? kOk : kErrLaunch;
}
