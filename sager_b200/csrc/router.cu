// router.cu - router logits (fp32 W x fp16 x) and the softmax / top-k selection.
//
// Arithmetic contracts restated from the reference:
//  * logits (src/kernels/cuda/q4_k.cu:133-149, 285-303, 1439-1495): lane l of a
//    warp accumulates w[i]*x[i] for i = l, l+32, ... ascending with one FMA per
//    term, then the shuffle-down tree 16,8,4,2,1. Kept exactly, so logits are
//    bit-identical to the reference kernels' and routing cannot flip.
//  * selection (src/kernels/cuda/moe.cu:25-85, 165-234; mmq.cu:420-510):
//    mx = max logit, z = sum of expf(l - mx) added serially in index order,
//    p = expf(l - mx)/z, K greedy argmax passes on p (NaN never picked, ties to
//    the lower index, picked entries masked with -1, an empty pass yields
//    kk % E), weights renormalised by the sum of the picked p, slot K =
//    shared_w. The exponentials are evaluated in parallel, the sum keeps the
//    serial order, the argmax is a warp reduction with the same tie rule.
#include <cooperative_groups.h>

#include "api_util.cuh"
#include "router_dev.cuh"

namespace cg = cooperative_groups;

namespace sgr {

namespace {

// ---- one token: a warp per expert row, straight from global memory ------------------
__global__ void router_logits_kernel(const float* __restrict__ w, const uint16_t* __restrict__ x,
                                     float* __restrict__ y, int n_rows, int k) {
  extern __shared__ __align__(16) unsigned char smem[];
  uint16_t* xs = reinterpret_cast<uint16_t*>(smem);
  for (int i = threadIdx.x; i < k; i += blockDim.x) xs[i] = x[i];
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= n_rows) return;
  float out[1];
  router_row_dot<1>(w + static_cast<size_t>(row) * k, xs, k, 1, lane, out);
  if (lane == 0) y[row] = out[0];
}

// ---- several tokens: a register-tiled fp32 product with the reference's sum order -----
// A warp owns TR expert rows x TT tokens; lane l holds their chain l (k = l, l + 32, ...), so an
// output's 32 partial sums live in the 32 lanes and every lane runs TR * TT independent FMA
// chains from TR + TT shared-memory operands. Two tokens share a packed fp32x2 FMA (the same
// rounding per component, half the issue slots). At the end the lanes exchange halves: in step
// 16, 8, 4, 2, 1 a lane adds the partner's half of the outputs to its own, which is the pairing
// of the reference's shuffle-down tree (addition commutes), in 31/32 of a shuffle per output
// instead of five. Bound by the fp32 pipes and the issue slots around them (1.07 G FMAs for 2048
// tokens x 256 rows x 2048: 29 us at 128 per clock and SM). (A warp per (row, eight tokens)
// with the fp16 values converted at every use took 534 / 212 / 33 us for 2048 / 777 / 96 tokens.)
__device__ __forceinline__ void fma2(unsigned long long& acc, float w, unsigned long long x) {
  unsigned long long ww;
  asm("mov.b64 %0, {%1, %1};" : "=l"(ww) : "f"(w));
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(ww), "l"(x));
}
// One step of the exchange: N outputs in, N / 2 out (the upper half in the lanes with `Bit` set), then the next.
template <int N, int Bit>
__device__ __forceinline__ void fold_lanes(float* f, int lane) {
  if constexpr (Bit > 0) {
    const bool up = (lane & Bit) != 0;
#pragma unroll
    for (int i = 0; i < N / 2; ++i) {
      const float keep = up ? f[i + N / 2] : f[i];
      const float send = up ? f[i] : f[i + N / 2];
      f[i] = keep + __shfl_xor_sync(0xFFFFFFFFu, send, Bit);
    }
    fold_lanes<N / 2, Bit / 2>(f, lane);
  }
}

// Fold the 32 lanes and store: output o = r * TT + t; after the five exchanges lane l holds the outputs whose bits above
// log2(TR * TT / 32) spell l's bits from bit 4 down.
template <int TR, int TT>
__device__ __forceinline__ void store_folded(const unsigned long long (&acc)[TR][TT / 2], float* __restrict__ y, int row0, int tok0,
                                             int n_rows, int n_tokens, int lane) {
  float f[TR * TT];
#pragma unroll
  for (int r = 0; r < TR; ++r)
#pragma unroll
    for (int p = 0; p < TT / 2; ++p)
      asm("mov.b64 {%0, %1}, %2;" : "=f"(f[r * TT + 2 * p]), "=f"(f[r * TT + 2 * p + 1]) : "l"(acc[r][p]));
  fold_lanes<TR * TT, 16>(f, lane);
  constexpr int kLeft = TR * TT / 32;
#pragma unroll
  for (int i = 0; i < kLeft; ++i) {
    const int o = i + kLeft * lane;           // step s split on output bit log2(TR*TT) - 1 - s and lane bit 4 - s
    const int row = row0 + o / TT, tok = tok0 + o % TT;
    if (row < n_rows && tok < n_tokens) y[static_cast<size_t>(tok) * n_rows + row] = f[i];
  }
}

// The product for rows of whole 16-byte pieces: a lane holds two neighbouring chains (columns 2 c, 2 c + 1 of every 32, c = lane % 16)
// of TR rows x TT tokens, and the packed FMA's two components are these chains, so that W and x are used as they lie: a row's two
// weights are one 8-byte read that both halves of the warp share, a token's two values one 4-byte read and two conversions.
// The raw columns arrive by cp.async, 128 to a stage, SLOTS - 1 stages ahead. 2048 / 1200 / 777 tokens x 256 rows of 2048 columns behind a
// top-k: 66.6 / 40.9 / 28.3 us, where a lane with one chain of two tokens - its weights spread over both components, x turned
// into token pairs in shared memory first - took 80.9 / 49.0 / 33.8. Neither pipe is full (at 2048 tokens FMA 66 %,
// shared memory 65 %): a packed FMA takes about three cycles and not two, and leaving out the conversions, either operand's loads or the
// copies gives 4 to 10 % each. (Scalar FMAs 75.8 for 57.6 back to back; the order of the products, the roles of the operands, W brought
// into L2 before the wait for the kernel before: nothing.)
// block: WR x WT warps; grid (row tiles, token tiles).
template <int TR, int TT, int WR, int WT, int SLOTS>
struct Logits {
  static constexpr int kWarps = WR * WT, kRows = TR * WR, kToks = 2 * TT * WT, kCols = 128, kSlots = SLOTS;
  static constexpr int kXPitch = kCols * 2 + 64;             // bytes of an x row: two tokens' 64 bytes in different banks
  static constexpr int kWBytes = kRows * kCols * 4, kXBytes = kToks * kXPitch;
  static constexpr int kSmem = kSlots * (kWBytes + kXBytes);
};
// One step of the exchange for lanes that hold two chains each: as fold_lanes.
template <int N, int Bit>
__device__ __forceinline__ void fold_pairs(float (*f)[2], int lane) {
  if constexpr (Bit > 0) {
    const bool up = (lane & Bit) != 0;
#pragma unroll
    for (int i = 0; i < N / 2; ++i)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float keep = up ? f[i + N / 2][h] : f[i][h];
        const float send = up ? f[i][h] : f[i + N / 2][h];
        f[i][h] = keep + __shfl_xor_sync(0xFFFFFFFFu, send, Bit);
      }
    fold_pairs<N / 2, Bit / 2>(f, lane);
  }
}
template <int TR, int TT, int WR, int WT, int SLOTS>
__global__ void __launch_bounds__(WR* WT * 32, (TR * TT >= 64 ? 8 : TR * TT >= 32 ? 16 : 20) / (WR * WT))
router_logits_staged_kernel(const float* __restrict__ w, const uint16_t* __restrict__ x, float* __restrict__ y,
                            int n_rows, int k, int n_tokens) {
  using T = Logits<TR, TT, WR, WT, SLOTS>;
  constexpr int kThreads = T::kWarps * 32;
  extern __shared__ __align__(16) unsigned char smem[];
  unsigned char* const w_raw = smem;                                           // [kSlots][kRows][128] fp32
  unsigned char* const x_raw = smem + T::kSlots * T::kWBytes;                  // [kSlots][kToks][kXPitch]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int row0 = blockIdx.x * T::kRows, tok0 = blockIdx.y * T::kToks;
  const int wr = warp % WR, wt = warp / WR;
  // rows and tokens past the end repeat the last one (never stored), columns past k are zero (add nothing)
  auto piece = [](uint32_t dst, const void* src, bool in) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(in ? 16 : 0) : "memory");
  };
  constexpr int kWPieces = T::kRows * 32 / kThreads, kXPieces = T::kToks * 16 / kThreads;
  static_assert(T::kRows * 32 % kThreads == 0 && T::kToks * 16 % kThreads == 0, "pieces");
  const int w_col = (tid & 31) * 4, x_col = (tid & 15) * 8;      // a thread's pieces lie in one column of pieces
  const float* w_at[kWPieces];
  const uint16_t* x_at[kXPieces];
#pragma unroll
  for (int i = 0; i < kWPieces; ++i) w_at[i] = w + static_cast<size_t>(min(row0 + (tid >> 5) + i * (kThreads / 32), n_rows - 1)) * k + w_col;
#pragma unroll
  for (int i = 0; i < kXPieces; ++i) x_at[i] = x + static_cast<size_t>(min(tok0 + (tid >> 4) + i * (kThreads / 16), n_tokens - 1)) * k + x_col;
  auto fill = [&](int c) {
    const int k0 = c * T::kCols;
    if (k0 < k) {
      const bool w_in = k0 + w_col < k, x_in = k0 + x_col < k;
      const uint32_t wd = smem_u32(w_raw + (c % T::kSlots) * T::kWBytes + tid * 16);
      const uint32_t xd = smem_u32(x_raw + (c % T::kSlots) * T::kXBytes + (tid >> 4) * T::kXPitch + (tid & 15) * 16);
#pragma unroll
      for (int i = 0; i < kWPieces; ++i) piece(wd + i * kThreads * 16, w_in ? w_at[i] + k0 : w, w_in);
#pragma unroll
      for (int i = 0; i < kXPieces; ++i) piece(xd + i * (kThreads / 16) * T::kXPitch, x_in ? x_at[i] + k0 : x, x_in);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  const int chunks = (k + T::kCols - 1) / T::kCols;
  pdl_wait();                                   // (a caller's kernel may have written W as well as x)
  pdl_launch_dependents();
#pragma unroll
  for (int c = 0; c < T::kSlots - 1; ++c) fill(c);
  unsigned long long acc[TT][TR];               // two chains' fp32 sums each
#pragma unroll
  for (int t = 0; t < TT; ++t)
#pragma unroll
    for (int r = 0; r < TR; ++r) acc[t][r] = 0ull;
#pragma unroll 1
  for (int c = 0; c < chunks; ++c) {
    asm volatile("cp.async.wait_group %0;" ::"n"(T::kSlots - 2) : "memory");     // chunk c has landed
    __syncthreads();                            // ... everybody's part of it; chunk c - 1 is no longer read
    fill(c + T::kSlots - 1);
    const unsigned char* wp = w_raw + (c % T::kSlots) * T::kWBytes + wr * TR * T::kCols * 4 + (lane & 15) * 8;
    const unsigned char* xp = x_raw + (c % T::kSlots) * T::kXBytes + (wt * 2 * TT + (lane >> 4)) * T::kXPitch + (lane & 15) * 4;
    // operands of 32 columns; the next ones are loaded under this one's products
    unsigned long long wv[2][TR];
    uint32_t xv[2][TT];
    auto load = [&](int j) {
#pragma unroll
      for (int r = 0; r < TR; ++r) wv[j & 1][r] = *reinterpret_cast<const unsigned long long*>(wp + (r * T::kCols + j * 32) * 4);
#pragma unroll
      for (int t = 0; t < TT; ++t) xv[j & 1][t] = *reinterpret_cast<const uint32_t*>(xp + 2 * t * T::kXPitch + j * 64);
    };
    load(0);
#pragma unroll
    for (int j = 0; j < T::kCols / 32; ++j) {
      if (j + 1 < T::kCols / 32) load(j + 1);
#pragma unroll
      for (int t = 0; t < TT; ++t) {
        const float2 v = __half22float2(*reinterpret_cast<const __half2*>(&xv[j & 1][t]));
        unsigned long long xx;
        asm("mov.b64 %0, {%1, %2};" : "=l"(xx) : "f"(v.x), "f"(v.y));
#pragma unroll
        for (int r = 0; r < TR; ++r) asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[t][r]) : "l"(wv[j & 1][r]), "l"(xx));
      }
    }
  }
  // fold: chains 16, 8, 4 and 2 apart are in lanes 8, 4, 2 and 1 apart, the last two in one lane
  float f[TT * TR][2];
#pragma unroll
  for (int t = 0; t < TT; ++t)
#pragma unroll
    for (int r = 0; r < TR; ++r) asm("mov.b64 {%0, %1}, %2;" : "=f"(f[t * TR + r][0]), "=f"(f[t * TR + r][1]) : "l"(acc[t][r]));
  fold_pairs<TT * TR, 8>(f, lane);
  constexpr int kLeft = TT * TR / 16;
#pragma unroll
  for (int i = 0; i < kLeft; ++i) {
    const int o = i + kLeft * (lane & 15);
    const int row = row0 + wr * TR + o % TR, tok = tok0 + wt * 2 * TT + 2 * (o / TR) + (lane >> 4);
    if (row < n_rows && tok < n_tokens) y[static_cast<size_t>(tok) * n_rows + row] = f[i][0] + f[i][1];
  }
}

// The same for rows off a 16-byte boundary.
// block: WR x WT warps; grid (row tiles, token tiles). KC columns per shared-memory stage, two
// stages: the next one is on its way to registers while this one is used, so a stage has to last a
// round trip to L2 (with 64 columns the trip showed: 124 us for 2048 tokens, 14 us for eight).
template <int TR, int TT, int WR, int WT, int KC>
__global__ void __launch_bounds__(WR* WT * 32, 8 / (WR * WT))
router_logits_tiled_kernel(const float* __restrict__ w, const uint16_t* __restrict__ x, float* __restrict__ y,
                           int n_rows, int k, int n_tokens) {
  constexpr int kWarps = WR * WT, kRows = TR * WR, kPairs = TT * WT / 2, kSteps = KC / 64;
  constexpr int kRowsPerWarp = kRows / kWarps, kPairsPerWarp = kPairs / kWarps;
  static_assert(kRows % kWarps == 0 && kPairs % kWarps == 0 && TR * TT >= 32 && KC % 64 == 0, "tile split");
  // a stage: two k steps of a lane lie together, [row][step][lane][2 k] and [pair][step][lane][2 k][2 tokens], so
  // that an operand is one 8- or 16-byte shared-memory access per two steps, without conflicts
  extern __shared__ __align__(16) unsigned char smem[];
  float2(*ws)[kRows][kSteps][32] = reinterpret_cast<float2(*)[kRows][kSteps][32]>(smem);
  float4(*xs)[kPairs][kSteps][32] =
      reinterpret_cast<float4(*)[kPairs][kSteps][32]>(smem + 2 * sizeof(float) * kRows * KC);
  pdl_wait();
  pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row0 = blockIdx.x * kRows, tok0 = blockIdx.y * (TT * WT);
  const int wr = warp % WR, wt = warp / WR;

  // the stage this warp copies: rows warp, warp + kWarps, ... and token pairs likewise; rows and
  // tokens past the end repeat the last one (never stored), columns past k are zero (add nothing)
  const float* wp[kRowsPerWarp];
  const uint16_t* xp[kPairsPerWarp][2];
#pragma unroll
  for (int i = 0; i < kRowsPerWarp; ++i)
    wp[i] = w + static_cast<size_t>(min(row0 + warp + i * kWarps, n_rows - 1)) * k + lane;
#pragma unroll
  for (int i = 0; i < kPairsPerWarp; ++i)
#pragma unroll
    for (int c = 0; c < 2; ++c)
      xp[i][c] = x + static_cast<size_t>(min(tok0 + 2 * (warp + i * kWarps) + c, n_tokens - 1)) * k + lane;
  float wreg[kRowsPerWarp][KC / 32];
  uint16_t xreg[kPairsPerWarp][KC / 32][2];
  auto fetch = [&](int k0) {
    if (k0 + KC <= k) {
#pragma unroll
      for (int j = 0; j < KC / 32; ++j) {
#pragma unroll
        for (int i = 0; i < kRowsPerWarp; ++i) wreg[i][j] = __ldg(wp[i] + k0 + 32 * j);
#pragma unroll
        for (int i = 0; i < kPairsPerWarp; ++i)
#pragma unroll
          for (int c = 0; c < 2; ++c) xreg[i][j][c] = __ldg(xp[i][c] + k0 + 32 * j);
      }
    } else {
#pragma unroll
      for (int j = 0; j < KC / 32; ++j) {
        const bool in = k0 + 32 * j + lane < k;
#pragma unroll
        for (int i = 0; i < kRowsPerWarp; ++i) wreg[i][j] = in ? __ldg(wp[i] + k0 + 32 * j) : 0.f;
#pragma unroll
        for (int i = 0; i < kPairsPerWarp; ++i)
#pragma unroll
          for (int c = 0; c < 2; ++c) xreg[i][j][c] = in ? __ldg(xp[i][c] + k0 + 32 * j) : static_cast<uint16_t>(0);
      }
    }
  };
  // (the conversions are pinned here: moved up to the loads they would wait for them)
  auto cvt = [](uint16_t h) { float f; asm volatile("cvt.f32.f16 %0, %1;" : "=f"(f) : "h"(h)); return f; };
  auto put = [&](int buf) {
#pragma unroll
    for (int j = 0; j < kSteps; ++j) {
#pragma unroll
      for (int i = 0; i < kRowsPerWarp; ++i)
        ws[buf][warp + i * kWarps][j][lane] = make_float2(wreg[i][2 * j], wreg[i][2 * j + 1]);
#pragma unroll
      for (int i = 0; i < kPairsPerWarp; ++i)
        xs[buf][warp + i * kWarps][j][lane] = make_float4(cvt(xreg[i][2 * j][0]), cvt(xreg[i][2 * j][1]),
                                                          cvt(xreg[i][2 * j + 1][0]), cvt(xreg[i][2 * j + 1][1]));
    }
  };

  unsigned long long acc[TR][TT / 2];           // two packed fp32 sums each
#pragma unroll
  for (int r = 0; r < TR; ++r)
#pragma unroll
    for (int p = 0; p < TT / 2; ++p) acc[r][p] = 0ull;
  fetch(0);
  put(0);
  __syncthreads();
  for (int k0 = 0, buf = 0; k0 < k; k0 += KC, buf ^= 1) {
    const bool more = k0 + KC < k;
    if (more) fetch(k0 + KC);
#pragma unroll
    for (int j = 0; j < kSteps; ++j) {
      float2 wv[TR];
      ulonglong2 xv[TT / 2];
#pragma unroll
      for (int r = 0; r < TR; ++r) wv[r] = ws[buf][wr * TR + r][j][lane];
#pragma unroll
      for (int p = 0; p < TT / 2; ++p)
        xv[p] = *reinterpret_cast<const ulonglong2*>(&xs[buf][wt * (TT / 2) + p][j][lane]);
#pragma unroll
      for (int r = 0; r < TR; ++r)
#pragma unroll
        for (int p = 0; p < TT / 2; ++p) fma2(acc[r][p], wv[r].x, xv[p].x);
#pragma unroll
      for (int r = 0; r < TR; ++r)
#pragma unroll
        for (int p = 0; p < TT / 2; ++p) fma2(acc[r][p], wv[r].y, xv[p].y);
    }
    if (more) put(buf ^ 1);       // the other buffer: every warp left it at the barrier below
    __syncthreads();
  }

  store_folded<TR, TT>(acc, y, row0 + wr * TR, tok0 + wt * TT, n_rows, n_tokens, lane);
}

template <int TR, int TT, int WR, int WT, int KC>
int launch_tiled(const float* w, const uint16_t* x, float* y, int n_rows, int k, int n_tokens, cudaStream_t stream) {
  constexpr int kSmem = 2 * KC * (TR * WR + TT * WT) * static_cast<int>(sizeof(float));
  if (kSmem > 48 * 1024 && !opt_in_smem<router_logits_tiled_kernel<TR, TT, WR, WT, KC>>(kSmem)) return kErrLaunch;
  const dim3 grid((n_rows + TR * WR - 1) / (TR * WR), (n_tokens + TT * WT - 1) / (TT * WT));
  return launch_pdl(router_logits_tiled_kernel<TR, TT, WR, WT, KC>, grid, WR * WT * 32, kSmem, stream, w, x, y, n_rows, k, n_tokens);
}

template <int TR, int TT, int WR, int WT, int SLOTS>
int launch_staged(const float* w, const uint16_t* x, float* y, int n_rows, int k, int n_tokens, cudaStream_t stream) {
  using T = Logits<TR, TT, WR, WT, SLOTS>;
  if (!opt_in_smem<router_logits_staged_kernel<TR, TT, WR, WT, SLOTS>>(T::kSmem)) return kErrLaunch;
  const dim3 grid((n_rows + T::kRows - 1) / T::kRows, (n_tokens + T::kToks - 1) / T::kToks);
  return launch_pdl(router_logits_staged_kernel<TR, TT, WR, WT, SLOTS>, grid, T::kWarps * 32, T::kSmem, stream, w, x, y, n_rows, k, n_tokens);
}

int launch_logits(const float* w, const uint16_t* x, float* y, int n_rows, int k, int n_tokens,
                  cudaStream_t stream) {
  if (n_tokens <= 0 || n_rows <= 0) return kOk;
  if (!w || !x || !y || k <= 0) return kErrArg;
  if (n_tokens == 1) {
    const int warps = 2;                           // 2 MB of W spread over >= 128 CTAs at E=256
    const size_t smem = static_cast<size_t>(k) * 2;
    if (smem > 48 * 1024) return kErrUnsupported;
    router_logits_kernel<<<(n_rows + warps - 1) / warps, warps * 32, smem, stream>>>(w, x, y, n_rows, k);
  } else if ((k & 7) == 0 && ((reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(x)) & 15u) == 0 &&
             (n_tokens + 15) / 16 <= 65535) {
    // Larger tiles read fewer operands per FMA, smaller ones spread over more warps; and with few outputs W's way out of DRAM is most
    // of the time, so a ring of eight stages or more asks for half of a CTA's rows at once. us of a prefill chunk with its experts (256 x
    // 2048; four layers of 65 / 96 / 130 / 200 / 300 / 500 rows, two of 777 / 1200 / 2048): 4 x 4 outputs a lane, two warps, eight stages 444 / 467 /
    // 494 / - / 615 / - / 493 / - / -; 8 x 4, four warps, eight 456 / 479 / 508 / 542 / 612 / 741 / 478 / 612 / 835 (with four stages 484 /
    // 505 / 540 / 576 / 629 / 747 / 476 / 608 / 826, with twelve 442 / 464 / 505 / 547 / 621 / 758 / 490 / 634 / 864); 16 x 4, four warps, four 483 /
    // 504 / 533 / 568 / 622 / 743 / 472 / 605 / 818; one chain to a lane 466 / 488 / 516 / 552 / 616 / 755 / 487 / 623 / 851. 64 experts, 300 rows:
    // 141.6, 148.3, 147.9 and 147.3. (592 rows, back to back and L2-hot: 8 x 4 21.3, 16 x 4 25.7 - three CTAs on an SM for little more than two.)
    // The lines are from 2048 columns. At 512 to 4096 columns, 16 to 256 rows and 2 to 4096 tokens the rule is ahead of the kernel with one chain to a
    // lane and its lines throughout: back to back by 1 to 110 %, 200 tokens x 256 rows of 4096 columns 25.4 -> 20.8, 4096 tokens x 128 of 512 21.5 -> 17.7.
    const long long outputs = static_cast<long long>(n_rows) * n_tokens;
    if (outputs >= 256LL * 620) return launch_staged<16, 4, 1, 4, 4>(w, x, y, n_rows, k, n_tokens, stream);
    if (outputs >= 256LL * 180) return launch_staged<8, 4, 2, 2, 8>(w, x, y, n_rows, k, n_tokens, stream);
    if (outputs > 64LL * 2 * device_sms()) return launch_staged<4, 4, 2, 1, 8>(w, x, y, n_rows, k, n_tokens, stream);
    // (all CTAs fit on the SMs at once with twelve stages as well: 80 rows x 64 experts 112.5 for 115.6, 100 x 128 123.7 for 125.6, 65 x 256 440
    // for 444; 96 x 256, where they do not, 474 for 467)
    return launch_staged<4, 4, 2, 1, 12>(w, x, y, n_rows, k, n_tokens, stream);
  } else if (static_cast<long long>(n_rows) * n_tokens >= 256LL * 592) {
    // 8 x 16 outputs per warp keep the FMA pipes fullest; below one such CTA per SM the smaller tile has more
    // warps to spread (at 256 x 592 the two take 41 and 38 us, and from there the larger one wins)
    return launch_tiled<8, 16, 2, 2, 128>(w, x, y, n_rows, k, n_tokens, stream);
  } else {
    return launch_tiled<4, 8, 4, 1, 256>(w, x, y, n_rows, k, n_tokens, stream);   // small: more warps to spread
  }
  return cudaPeekAtLastError() == cudaSuccess ? kOk : kErrLaunch;
}

// one warp per row, 4 rows per CTA; dynamic smem = 4 rows of n_expert floats at 16-byte steps
constexpr int kTopkWarps = 4;
__global__ void router_topk_kernel(const float* __restrict__ logits, int* __restrict__ idx,
                                   float* __restrict__ weight, int n_expert, int k, int stride,
                                   int n_rows, float shared_w) {
  extern __shared__ __align__(16) unsigned char smem[];
  pdl_wait();
  pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row = blockIdx.x * kTopkWarps + warp;
  if (row >= n_rows) return;
  float* prob = reinterpret_cast<float*>(smem) + static_cast<size_t>(warp) * ((n_expert + 3) & ~3);
  for (int i = lane; i < n_expert; i += 32) prob[i] = logits[static_cast<size_t>(row) * n_expert + i];
  __syncwarp();
  router_select_warp(prob, n_expert, k, idx + static_cast<size_t>(row) * stride,
                     weight + static_cast<size_t>(row) * stride, shared_w, true, lane);
}

// Fused single-token router: a cluster of 8 CTAs splits the rows of W, every
// CTA drops its logits into the leader's shared memory through DSMEM, and after
// one cluster barrier the leader's first warp selects. One launch, no global
// scratch. Slot K of `weight` is left untouched, as the reference's
// router_topk_fused does (mmq.cu:459-510).
constexpr int kFusedCluster = 8;
constexpr int kFusedThreads = 512;
__global__ void __cluster_dims__(kFusedCluster, 1, 1) __launch_bounds__(kFusedThreads)
router_topk_fused_kernel(const float* __restrict__ w, const uint16_t* __restrict__ x,
                         int* __restrict__ idx, float* __restrict__ weight, int n_expert, int k_used,
                         int hidden) {
  extern __shared__ __align__(16) unsigned char smem[];
  uint16_t* xs = reinterpret_cast<uint16_t*>(smem);
  float* logits = reinterpret_cast<float*>(smem + ((static_cast<size_t>(hidden) * 2 + 15) & ~size_t(15)));
  cg::cluster_group cluster = cg::this_cluster();
  const unsigned rank = cluster.block_rank();
  for (int i = threadIdx.x; i < hidden; i += blockDim.x) xs[i] = x[i];
  __syncthreads();
  float* leader_logits = cluster.map_shared_rank(logits, 0);
  const int lane = threadIdx.x & 31;
  const int gwarp = rank * (kFusedThreads / 32) + (threadIdx.x >> 5);
  for (int row = gwarp; row < n_expert; row += kFusedCluster * (kFusedThreads / 32)) {
    float out[1];
    router_row_dot<1>(w + static_cast<size_t>(row) * hidden, xs, hidden, 1, lane, out);
    if (lane == 0) leader_logits[row] = out[0];
  }
  cluster.sync();
  if (rank == 0 && threadIdx.x < 32)
    router_select_warp(logits, n_expert, k_used, idx, weight, 0.f, false, lane);
}

}  // namespace
}  // namespace sgr

using namespace sgr;

SGR_API int sgr_gemv_f32_out_f16x(const float* w_f32, const uint16_t* x_f16, float* y, int n_rows,
                                  int k, void* stream) {
  return launch_logits(w_f32, x_f16, y, n_rows, k, 1, as_stream(stream));
}
SGR_API int sgr_gemv_f32_out_f16x_batched(const float* w_f32, const uint16_t* x_f16, float* y,
                                          int n_rows, int k, int n_tokens, void* stream) {
  return launch_logits(w_f32, x_f16, y, n_rows, k, n_tokens, as_stream(stream));
}
SGR_API int sgr_gemv_f32_out_f16x_mtok(const float* w_f32, const uint16_t* x_f16, float* y,
                                       int n_rows, int k, int n_tokens, void* stream) {
  return launch_logits(w_f32, x_f16, y, n_rows, k, n_tokens, as_stream(stream));
}

SGR_API int sgr_router_topk_batched(const float* logits, int* idx, float* weight, int n_expert,
                                    int n_expert_used, int idx_stride, int n_rows, float shared_w,
                                    void* stream) {
  if (n_rows <= 0) return kOk;
  if (!logits || !idx || !weight || n_expert <= 0 || n_expert_used <= 0 ||
      idx_stride < n_expert_used + 1)
    return kErrArg;
  const size_t smem = static_cast<size_t>(kTopkWarps) * ((n_expert + 3) & ~3) * sizeof(float);
  if (smem > 48 * 1024) return kErrUnsupported;
  return launch_pdl(router_topk_kernel, dim3((n_rows + kTopkWarps - 1) / kTopkWarps), kTopkWarps * 32, smem,
                    as_stream(stream), logits, idx, weight, n_expert, n_expert_used, idx_stride, n_rows, shared_w);
}

SGR_API int sgr_router_topk(const float* logits, int* idx, float* weight, int n_expert,
                            int n_expert_used, float shared_w, void* stream) {
  return sgr_router_topk_batched(logits, idx, weight, n_expert, n_expert_used, n_expert_used + 1, 1,
                                 shared_w, stream);
}

SGR_API int sgr_router_topk_fused(const float* w_f32, const uint16_t* x_f16, int* idx, float* weight,
                                  int n_expert, int n_expert_used, int hidden, void* stream) {
  if (!w_f32 || !x_f16 || !idx || !weight || n_expert <= 0 || n_expert_used <= 0 || hidden <= 0)
    return kErrArg;
  const size_t smem = ((static_cast<size_t>(hidden) * 2 + 15) & ~size_t(15)) +
                      static_cast<size_t>(n_expert) * sizeof(float);
  if (smem > 48 * 1024) return kErrUnsupported;
  router_topk_fused_kernel<<<kFusedCluster, kFusedThreads, smem, as_stream(stream)>>>(
      w_f32, x_f16, idx, weight, n_expert, n_expert_used, hidden);
  return cudaPeekAtLastError() == cudaSuccess ? kOk : kErrLaunch;
}
