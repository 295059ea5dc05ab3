// router_dev.cuh - warp-level pieces of the router shared by router.cu and the
// fused layer: the lane-strided logit dot and the softmax / top-k selection.
// The arithmetic contracts are stated at the top of router.cu.
#pragma once

#include "q4k_common.cuh"

namespace sgr {

// One warp, one weight row, up to TT tokens whose fp16 rows sit in shared
// memory (xs[t*k + i]). Returns lane 0's tree sums in out[t].
template <int TT>
__device__ __forceinline__ void router_row_dot(const float* __restrict__ wrow,
                                               const uint16_t* __restrict__ xs, int k, int nt,
                                               int lane, float (&out)[TT]) {
  float acc[TT];
#pragma unroll
  for (int t = 0; t < TT; ++t) acc[t] = 0.f;
  int i = lane;
  // 32 independent loads in flight (a 2048-wide row is two round trips to memory),
  // FMAs issued in ascending index order
  for (; i + 31 * 32 < k; i += 32 * 32) {
    float wv[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) wv[j] = __ldg(wrow + i + j * 32);
#pragma unroll
    for (int j = 0; j < 32; ++j) {
#pragma unroll
      for (int t = 0; t < TT; ++t)
        if (t < nt) acc[t] = fmaf(wv[j], h2f(xs[t * k + i + j * 32]), acc[t]);
    }
  }
  for (; i + 7 * 32 < k; i += 8 * 32) {
    float wv[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) wv[j] = __ldg(wrow + i + j * 32);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
#pragma unroll
      for (int t = 0; t < TT; ++t)
        if (t < nt) acc[t] = fmaf(wv[j], h2f(xs[t * k + i + j * 32]), acc[t]);
    }
  }
  for (; i < k; i += 32) {
    const float wv = __ldg(wrow + i);
#pragma unroll
    for (int t = 0; t < TT; ++t)
      if (t < nt) acc[t] = fmaf(wv, h2f(xs[t * k + i]), acc[t]);
  }
#pragma unroll
  for (int t = 0; t < TT; ++t) {
    float a = acc[t];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) a += __shfl_down_sync(0xFFFFFFFFu, a, off);
    out[t] = a;
  }
}

// The logits of R router rows and T token rows by one warp, rows in shared memory: weights [R][k] as they lie in global
// memory, activations k-major fp16, xs[kk * T + t], so that a lane's T values of one k are one load. The FMAs of a (row,
// lane, token) chain run in the same order as in router_row_dot, and the shuffle tree adds the same pairs - each step also
// halves the number of sums a lane carries - so the logits are bit-identical. Lane l returns the sum of (row, token)
// number l / (32 / (R * T)), row-major.
template <int R, int T>
__device__ __forceinline__ float router_tile_dot(const float* ws, const uint16_t* xs, int k, int lane) {
  // two tokens share a packed fp32 FMA (each component rounds as the scalar instruction): 64 rows, 81.9 -> 81.4 us per layer
  unsigned long long sum[R * T / 2];
#pragma unroll
  for (int i = 0; i < R * T / 2; ++i) sum[i] = 0ull;
  // the loads of S steps are issued ahead of the FMAs of the S steps before (k is a multiple of 256: S divides the steps)
  constexpr int S = T == 2 ? 8 : 4;
  uint32_t raw[2][S][T / 2];
  float w[2][S][R];
  auto load = [&](int b, int kk) {
#pragma unroll
    for (int j = 0; j < S; ++j) {
      const uint16_t* x = xs + static_cast<size_t>(kk + 32 * j) * T;
      if constexpr (T == 8) {
        const uint4 q = *reinterpret_cast<const uint4*>(x);
        raw[b][j][0] = q.x; raw[b][j][1] = q.y; raw[b][j][2] = q.z; raw[b][j][3] = q.w;
      } else if constexpr (T == 4) {
        const uint2 q = *reinterpret_cast<const uint2*>(x);
        raw[b][j][0] = q.x; raw[b][j][1] = q.y;
      } else {
        raw[b][j][0] = *reinterpret_cast<const uint32_t*>(x);
      }
#pragma unroll
      for (int r = 0; r < R; ++r) w[b][j][r] = ws[static_cast<size_t>(r) * k + kk + 32 * j];
    }
  };
  auto add = [&](int b) {
#pragma unroll
    for (int j = 0; j < S; ++j)
#pragma unroll
      for (int t = 0; t < T / 2; ++t) {
        unsigned long long x, ww;
        asm("mov.b64 %0, {%1, %2};" : "=l"(x) : "f"(h2f(static_cast<uint16_t>(raw[b][j][t] & 0xFFFFu))), "f"(h2f(static_cast<uint16_t>(raw[b][j][t] >> 16))));
#pragma unroll
        for (int r = 0; r < R; ++r) {
          asm("mov.b64 %0, {%1, %1};" : "=l"(ww) : "f"(w[b][j][r]));
          asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(sum[r * T / 2 + t]) : "l"(ww), "l"(x));
        }
      }
  };
  load(0, lane);
#pragma unroll 1
  for (int kk = lane; kk < k; kk += 2 * S * 32) {
    if (kk + S * 32 < k) load(1, kk + S * 32);             // warp-uniform
    add(0);
    if (kk + 2 * S * 32 < k) load(0, kk + 2 * S * 32);
    if (kk + S * 32 < k) add(1);
  }
  float v[R * T];
#pragma unroll
  for (int i = 0; i < R * T / 2; ++i) asm("mov.b64 {%0, %1}, %2;" : "=f"(v[2 * i]), "=f"(v[2 * i + 1]) : "l"(sum[i]));
  int off = 16;
#pragma unroll
  for (int m = R * T / 2; m > 0; m >>= 1, off >>= 1) {
    const bool up = (lane & off) != 0;
#pragma unroll
    for (int i = 0; i < m; ++i) {
      const float send = up ? v[i] : v[i + m], keep = up ? v[i + m] : v[i];
      v[i] = keep + __shfl_xor_sync(0xFFFFFFFFu, send, off);
    }
  }
  for (; off > 0; off >>= 1) v[0] += __shfl_xor_sync(0xFFFFFFFFu, v[0], off);
  return v[0];
}

// Softmax + top-k of one row by one warp. `prob` is n_expert floats of shared
// memory that already hold the logits; it is overwritten.
__device__ __forceinline__ void router_select_warp(float* prob, int n_expert, int k, int* out_idx,
                                                   float* out_w, float shared_w, bool write_shared,
                                                   int lane) {
  if (n_expert <= 256 && k <= 32) {
    // Up to 256 experts: a lane keeps its eight values (experts lane, lane + 32, ...) in
    // registers from the logits to the picks. Same arithmetic as the general path below.
    float pr[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) pr[j] = lane + 32 * j < n_expert ? prob[lane + 32 * j] : -1e30f;
    float mx = -1e30f;
#pragma unroll
    for (int j = 0; j < 8; ++j) mx = fmaxf(mx, pr[j]);
    {                                            // warp maximum through an order-preserving integer key
      const int b = __float_as_int(mx);
      const int key = b ^ ((b >> 31) & 0x7FFFFFFF);
      const int mk = __reduce_max_sync(0xFFFFFFFFu, key);
      mx = __int_as_float(mk ^ ((mk >> 31) & 0x7FFFFFFF));
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      pr[j] = expf(pr[j] - mx);
      if (lane + 32 * j < n_expert) prob[lane + 32 * j] = pr[j];
    }
    __syncwarp();
    float z = 0.f;
    if (lane == 0) {                             // strictly in index order, loads ahead of the adds
      int i = 0;
#pragma unroll 4
      for (; i + 8 <= n_expert; i += 8) {
        const float4 a = *reinterpret_cast<const float4*>(prob + i), b = *reinterpret_cast<const float4*>(prob + i + 4);
        z += a.x; z += a.y; z += a.z; z += a.w; z += b.x; z += b.y; z += b.z; z += b.w;
      }
      for (; i < n_expert; ++i) z += prob[i];
    }
    z = __shfl_sync(0xFFFFFFFFu, z, 0);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float p = pr[j] / z;
      pr[j] = (lane + 32 * j < n_expert && p == p) ? p : -1.f;     // absent or NaN: never picked
    }
    float wsum = 0.f, my_w = 0.f;
    int my_i = 0;
    for (int kk = 0; kk < k; ++kk) {
      // this lane's best (lowest j on ties), then the warp's: largest value, lowest index
      float bv = pr[0];
      int bj = 0;
#pragma unroll
      for (int j = 1; j < 8; ++j)
        if (pr[j] > bv) { bv = pr[j]; bj = j; }
      const int vmax = __reduce_max_sync(0xFFFFFFFFu, __float_as_int(bv));      // values are >= 0 or -1
      const int cand = __float_as_int(bv) == vmax ? lane + 32 * bj : 0x7FFFFFFF;
      int bi = __reduce_min_sync(0xFFFFFFFFu, cand);
      float best = __int_as_float(vmax);
      if (best < 0.f) bi = kk % n_expert;          // nothing valid: deterministic filler
      if ((bi & 31) == lane && best >= 0.f) {
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (j == (bi >> 5)) pr[j] = -1.f;
      }
      wsum += best;
      if (lane == kk) { my_w = best; my_i = bi; }
    }
    if (lane < k) {
      out_idx[lane] = my_i;
      out_w[lane] = wsum > 0.f ? my_w / wsum : my_w;
    }
    if (lane == 0 && write_shared) out_w[k] = shared_w;
    return;
  }
  float mx = -1e30f;
  for (int i = lane; i < n_expert; i += 32) mx = fmaxf(mx, prob[i]);
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, off));
  for (int i = lane; i < n_expert; i += 32) prob[i] = expf(prob[i] - mx);
  __syncwarp();
  float z = 0.f;
  if (lane == 0) {
    int i = 0;
    for (; i + 8 <= n_expert; i += 8) {           // loads batched, adds strictly in order
      float e[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) e[j] = prob[i + j];
#pragma unroll
      for (int j = 0; j < 8; ++j) z += e[j];
    }
    for (; i < n_expert; ++i) z += prob[i];
  }
  z = __shfl_sync(0xFFFFFFFFu, z, 0);
  for (int i = lane; i < n_expert; i += 32) prob[i] = prob[i] / z;
  __syncwarp();

  // Every lane learns each pick (butterfly reduction); lane kk keeps pick kk in
  // registers, so the results reach global memory once, in parallel, already
  // renormalised. wsum is added in pick order in every lane (same rounding as the
  // reference's serial sum).
  float wsum = 0.f;
  float my_w = 0.f;
  int my_i = 0;
  // up to 256 experts: a lane keeps its eight probabilities in registers
  const bool in_regs = n_expert <= 256;
  float pr[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) pr[j] = (in_regs && lane + 32 * j < n_expert) ? prob[lane + 32 * j] : -1.f;
  for (int kk = 0; kk < k; ++kk) {
    float bv = -1.f;
    int bi = -1;
    if (in_regs) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float p = pr[j];
        if (p == p && p > bv) { bv = p; bi = lane + 32 * j; }
      }
    } else {
      for (int i = lane; i < n_expert; i += 32) {
        const float p = prob[i];
        if (p == p && p > bv) { bv = p; bi = i; }    // ascending scan: first strict max
      }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      const float ov = __shfl_xor_sync(0xFFFFFFFFu, bv, off);
      const int oi = __shfl_xor_sync(0xFFFFFFFFu, bi, off);
      const bool take = (oi >= 0) && (bi < 0 || ov > bv || (ov == bv && oi < bi));
      if (take) { bv = ov; bi = oi; }
    }
    if (bi < 0) bi = kk % n_expert;                // nothing valid: deterministic filler
    if (in_regs) {
      if ((bi & 31) == lane) {
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (j == (bi >> 5)) pr[j] = -1.f;
      }
    } else if (lane == 0) {
      prob[bi] = -1.f;
    }
    wsum += bv;
    if (k <= 32) {
      if (lane == kk) { my_w = bv; my_i = bi; }
    } else if (lane == 0) {
      out_idx[kk] = bi;
      out_w[kk] = bv;
    }
    __syncwarp();
  }
  if (k <= 32) {
    if (lane < k) {
      out_idx[lane] = my_i;
      out_w[lane] = wsum > 0.f ? my_w / wsum : my_w;
    }
  } else if (lane == 0 && wsum > 0.f) {
    for (int kk = 0; kk < k; ++kk) out_w[kk] /= wsum;
  }
  if (lane == 0 && write_shared) out_w[k] = shared_w;
}

static __device__ __noinline__ void router_select_general(float* prob, int E, int K, int* idx, float* w, float shared_w, int lane) {
  router_select_warp(prob, E, K, idx, w, shared_w, true, lane);
}

// Softmax and top-K of one token row by two warps (up to 256 experts, K < 32). The strictly serial sum of the
// exponentials - the reference's order - is long, so one warp picks the K + 1 largest exponentials and goes on to build
// what follows from them (`picked()`) while the other adds and makes the weights. Dividing by the sum keeps
// the order; only if it makes two of them equal, or something is not finite, the order of the quotients could be another
// one, and the adding warp runs the general selection on the quotients: it returns true, and the picks do not stand.
// logit(j) is the row's logit lane + 32 j; `prob` (E) and `pick_e` (K + 1) in shared memory, `bar` a barrier of the two warps.
template <typename Logit, typename Picked>
__device__ __forceinline__ bool router_select_pair(Logit logit, float* prob, float* pick_e, int* idx, float* w, int bar, bool adds, int E,
                                            int K, float shared_w, int lane, Picked picked) {
  float e[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) e[j] = lane + 32 * j < E ? logit(j) : -1e30f;
  float mx = -1e30f;
#pragma unroll
  for (int j = 0; j < 8; ++j) mx = fmaxf(mx, e[j]);
  {                                                // warp maximum through an order-preserving integer key
    const int b = __float_as_int(mx);
    const int mk = __reduce_max_sync(0xFFFFFFFFu, b ^ ((b >> 31) & 0x7FFFFFFF));
    mx = __int_as_float(mk ^ ((mk >> 31) & 0x7FFFFFFF));
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) e[j] = expf(e[j] - mx);
  if (!adds) {
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (lane + 32 * j >= E) e[j] = -1.f;
    // a lane's eight in descending order (Batcher's network), then the warp takes the largest head K + 1 times
    int sl[8] = {0, 1, 2, 3, 4, 5, 6, 7};
    auto ce = [&](int a, int b) {
      const bool sw = e[b] > e[a];
      const float x = fmaxf(e[a], e[b]), y = fminf(e[a], e[b]);
      const int i = sw ? sl[b] : sl[a], j = sw ? sl[a] : sl[b];
      e[a] = x; e[b] = y; sl[a] = i; sl[b] = j;
    };
    ce(0, 1); ce(2, 3); ce(4, 5); ce(6, 7);
    ce(0, 2); ce(1, 3); ce(4, 6); ce(5, 7);
    ce(1, 2); ce(5, 6); ce(0, 4); ce(3, 7);
    ce(1, 5); ce(2, 6);
    ce(1, 4); ce(3, 6);
    ce(2, 4); ce(3, 5);
    ce(3, 4);
    float my_e = -1.f;
    int my_i = 0;
#pragma unroll 1
    for (int kk = 0; kk <= K; ++kk) {
      const int top = __reduce_max_sync(0xFFFFFFFFu, __float_as_int(e[0]));        // values are >= 0 or -1
      const int win = __reduce_min_sync(0xFFFFFFFFu, __float_as_int(e[0]) == top ? lane + 32 * sl[0] : 0x7FFFFFFF);
      if ((win & 31) == lane) {
#pragma unroll
        for (int j = 0; j < 7; ++j) { e[j] = e[j + 1]; sl[j] = sl[j + 1]; }
        e[7] = -1.f;
      }
      if (lane == kk) { my_e = __int_as_float(top); my_i = win; }
    }
    my_i = min(my_i, E - 1);                     // (with NaNs about, a lane's filler could be picked: not fine below)
    if (lane < K) idx[lane] = my_i;
    if (lane <= K) pick_e[lane] = my_e;
    __syncwarp();
    asm volatile("bar.arrive %0, 64;" ::"r"(bar) : "memory");
    picked();
    return false;
  }
#pragma unroll
  for (int j = 0; j < 8; ++j)
    if (lane + 32 * j < E) prob[lane + 32 * j] = e[j];
  __syncwarp();
  float z = 0.f;                                 // every lane adds: the same broadcast reads
  int i = 0;
#pragma unroll 4
  for (; i + 8 <= E; i += 8) {
    const float4 a = *reinterpret_cast<const float4*>(prob + i), b = *reinterpret_cast<const float4*>(prob + i + 4);
    z += a.x; z += a.y; z += a.z; z += a.w; z += b.x; z += b.y; z += b.z; z += b.w;
  }
  for (; i < E; ++i) z += prob[i];
  asm volatile("bar.sync %0, 64;" ::"r"(bar) : "memory");
  const float my_e = lane <= K ? pick_e[lane] : -1.f;
  const float p = my_e / z;
  const float next = __shfl_down_sync(0xFFFFFFFFu, p, 1);
  const bool fine = z > 0.f && z <= 3.4e38f && __all_sync(0xFFFFFFFFu, lane >= K || (my_e >= 0.f && p > next));
  if (fine) {
    float wsum = 0.f;
    for (int kk = 0; kk < K; ++kk) wsum += __shfl_sync(0xFFFFFFFFu, p, kk);
    if (lane < K) w[lane] = wsum > 0.f ? p / wsum : p;
    if (lane == 0) w[K] = shared_w;
  } else {
    __syncwarp();
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (lane + 32 * j < E) prob[lane + 32 * j] = logit(j);
    __syncwarp();
    router_select_general(prob, E, K, idx, w, shared_w, lane);
  }
  return !fine;
}

}  // namespace sgr
