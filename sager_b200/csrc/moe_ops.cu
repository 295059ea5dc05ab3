// moe_ops.cu - the device-side plan, row movement, SwiGLU and combine kernels of
// the MoE half (src/kernels/cuda/moe.cu and src/kernels/cuda/norm_rotary.cu:
// 133-183 of the reference). All of them move or blend fp16 rows; they are
// written around 16-byte accesses (8 halves) with a scalar path for odd sizes.
#include <algorithm>

#include "api_util.cuh"
#include "q4k_common.cuh"

namespace sgr {
namespace {

__device__ __forceinline__ bool aligned16(const void* p) {
  return (reinterpret_cast<uintptr_t>(p) & 15u) == 0;
}

// ---- dispatch plan (moe.cu:366-434) ---------------------------------------------
// Every CTA reads the whole route list, counts it per expert and part of the list (shared-memory
// atomics) and builds the prefixes for itself, so nothing is exchanged; each of its warps then walks
// one part of the list for one expert of its own and hands the slots out by ballot. The slots inside
// an expert are in ascending (row, kk) order whatever the size. Bound by the latency of the phases:
// 3.9 us for 512 routes over 256 experts, 5.1 for 4,096. One CTA took 23 / 157 us (a thread per expert walking the
// list); counting and ranking by match_any in one CTA 48 us for 16,384.
// i / d for i below 2^31 by a multiplication (a division instruction sequence per route was half the time)
struct FastDiv {
  unsigned mul;
  int shift;                               // < 0: d is 1
  explicit FastDiv(unsigned d) : mul(0), shift(-1) {
    if (d <= 1) return;
    int l = 0;
    while ((1u << l) < d && l < 31) ++l;
    shift = l - 1;
    mul = static_cast<unsigned>(((1ull << (31 + l)) + d - 1) / d);
  }
  __device__ __forceinline__ int operator()(int i) const {
    return shift < 0 ? i : static_cast<int>(__umulhi(static_cast<unsigned>(i), mul) >> shift);
  }
};

constexpr int kScanThreads = 512, kScanWarps = kScanThreads / 32;
constexpr int kScanParts = 8;              // of the list
// With more experts or routes than this dispatch_scan_many_kernel (us for 256 experts, this kernel / that one: 4,096 routes 5.1 /
// 5.9, 6,216 7.2 / 6.1, 16,384 12.3 / 8.0; for 288 experts a single row 4.2 / 3.5, 512 experts 2,048 routes 6.2 / 6.0).
constexpr int kScanExperts = 256, kScanRoutes = 4096;

__global__ void __launch_bounds__(kScanThreads)
dispatch_scan_kernel(const int* __restrict__ idx, float* __restrict__ weight, int* __restrict__ gslot,
                     int* __restrict__ grows, int* __restrict__ off, int* __restrict__ toff,
                     int* __restrict__ meta, int* __restrict__ mail_n, int n_rows, int k,
                     int n_expert, int tok_per, int per, FastDiv by_k, FastDiv by_per) {
  constexpr int parts = kScanParts;
  extern __shared__ __align__(16) int cnt[];             // [parts][n_expert] counts, then first slots; ids after them
  uint16_t* ids = reinterpret_cast<uint16_t*>(cnt + static_cast<size_t>(parts) * n_expert);
  __shared__ int bad_sh;
  __shared__ int wsum[2][kScanWarps];
  __shared__ int carry[2];
  pdl_wait();
  pdl_launch_dependents();
  const int tid = threadIdx.x, lane = tid & 31, wp = tid >> 5;
  const int total = n_rows * k;
  if (tid == 0) bad_sh = carry[0] = carry[1] = 0;
  for (int e = tid; e < parts * n_expert; e += kScanThreads) cnt[e] = 0;
  __syncthreads();
  auto id_of = [&](int i) {
    const int e = __ldg(idx + i + by_k(i));                           // rows of k + 1
    return e >= 0 && e < n_expert ? e : 0xFFFF;
  };
  for (int b = tid; b < total; b += 8 * kScanThreads) {
    int e8[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) e8[q] = b + q * kScanThreads < total ? id_of(b + q * kScanThreads) : -1;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int i = b + q * kScanThreads;
      if (e8[q] < 0) continue;
      ids[i] = static_cast<uint16_t>(e8[q]);
      if (e8[q] != 0xFFFF) {
        atomicAdd(cnt + static_cast<size_t>(by_per(i)) * n_expert + e8[q], 1);
      } else if (blockIdx.x == 0) {
        // a corrupt id silences the whole row, shared-expert slot included
        float* wr = weight + static_cast<size_t>(by_k(i)) * (k + 1);
        for (int j = 0; j <= k; ++j) wr[j] = 0.f;
        gslot[i] = -1;
        atomicAdd(&bad_sh, 1);
      }
    }
  }
  __syncthreads();

  // exclusive prefixes of rows and of tiles over the experts: kScanThreads experts per round, scans
  // inside the warps, the warps' totals and the running totals through shared memory
  for (int base = 0; base < n_expert; base += kScanThreads) {
    const int e = base + tid;
    int c = 0;
    if (e < n_expert) {
      for (int w = 0; w < parts; ++w) {                               // the expert's routes, part after part
        const int v = cnt[static_cast<size_t>(w) * n_expert + e];
        cnt[static_cast<size_t>(w) * n_expert + e] = c;
        c += v;
      }
    }
    const int t = (c + tok_per - 1) / tok_per;
    int ic = c, it = t;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int uc = __shfl_up_sync(0xFFFFFFFFu, ic, o), ut = __shfl_up_sync(0xFFFFFFFFu, it, o);
      if (lane >= o) { ic += uc; it += ut; }
    }
    if (lane == 31) { wsum[0][wp] = ic; wsum[1][wp] = it; }
    __syncthreads();
    int pc = carry[0], pt = carry[1];
    for (int w = 0; w < wp; ++w) { pc += wsum[0][w]; pt += wsum[1][w]; }
    if (e < n_expert) {
      const int o0 = pc + ic - c;
      if (blockIdx.x == 0) {
        off[e] = o0;
        toff[e] = pt + it - t;
      }
      for (int w = 0; w < parts; ++w) cnt[static_cast<size_t>(w) * n_expert + e] += o0;
    }
    __syncthreads();
    if (tid == kScanThreads - 1) { carry[0] = pc + ic; carry[1] = pt + it; }
    __syncthreads();
  }
  if (blockIdx.x == 0 && tid == 0) {
    off[n_expert] = carry[0];
    toff[n_expert] = carry[1];
    meta[0] = carry[0];
    meta[1] = carry[1];
    meta[2] = bad_sh;
    if (mail_n != nullptr) *mail_n = 0;
  }

  const int e = blockIdx.x * (kScanWarps / parts) + wp / parts, part = wp % parts;
  if (e >= n_expert) return;
  int pos = cnt[static_cast<size_t>(part) * n_expert + e];
  const int i1 = min((part + 1) * per, total);
  for (int b = part * per; b < i1; b += 256) {
    int e8[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int i = b + 32 * q + lane;
      e8[q] = i < i1 ? ids[i] : -1;
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const unsigned hit = __ballot_sync(0xFFFFFFFFu, e8[q] == e);
      if (hit == 0) continue;
      if (e8[q] == e) {
        const int i = b + 32 * q + lane, slot = pos + __popc(hit & ((1u << lane) - 1u));
        gslot[i] = slot;
        grows[slot] = by_k(i);
      }
      pos += __popc(hit);
    }
  }
}

// More experts or routes: what every CTA does per expert (clear, prefix) and per route (its warps' walks) would be repeated by
// too many CTAs. Here a CTA takes a part of the route list: it counts the whole list, what lies before its part apart from
// the rest, builds the prefixes - a thread takes a run of experts -, and one warp hands out the part's slots 32 routes at a time,
// equal ids by match. Bound by the counting of the whole list, a shared-memory atomic per route: 16,384 routes 8.0 us over 256
// experts, 12.0 over 5,000; 131,072 routes 37.6 (one CTA 20 / 26 / 135).
constexpr int kManyThreads = 1024, kManyWarps = kManyThreads / 32;

__global__ void __launch_bounds__(kManyThreads)
dispatch_scan_many_kernel(const int* __restrict__ idx, float* __restrict__ weight, int* __restrict__ gslot,
                          int* __restrict__ grows, int* __restrict__ off, int* __restrict__ toff,
                          int* __restrict__ meta, int* __restrict__ mail_n, int n_rows, int k,
                          int n_expert, int tok_per, int per, FastDiv by_k) {
  extern __shared__ __align__(16) int before[];          // [n_expert] routes before this CTA's part, then its next slots
  int* rest = before + n_expert;                         // [n_expert] the other routes
  __shared__ int bad_sh;
  __shared__ int wsum[2][kManyWarps];
  pdl_wait();
  pdl_launch_dependents();
  const int tid = threadIdx.x, lane = tid & 31, wp = tid >> 5;
  const int total = n_rows * k, first = blockIdx.x * per, last = min(first + per, total);
  if (tid == 0) bad_sh = 0;
  for (int e = tid; e < 2 * n_expert; e += kManyThreads) before[e] = 0;
  __syncthreads();
  auto id_of = [&](int i) {
    const int e = __ldg(idx + i + by_k(i));              // rows of k + 1
    return e >= 0 && e < n_expert ? e : -1;
  };
  for (int b = tid; b < total; b += 8 * kManyThreads) {
    int e8[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) e8[q] = b + q * kManyThreads < total ? id_of(b + q * kManyThreads) : -2;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int i = b + q * kManyThreads;
      if (e8[q] >= 0) {
        atomicAdd((i < first ? before : rest) + e8[q], 1);
      } else if (e8[q] == -1 && blockIdx.x == 0) {
        // a corrupt id silences the whole row, shared-expert slot included
        float* wr = weight + static_cast<size_t>(by_k(i)) * (k + 1);
        for (int j = 0; j <= k; ++j) wr[j] = 0.f;
        gslot[i] = -1;
        atomicAdd(&bad_sh, 1);
      }
    }
  }
  __syncthreads();

  // exclusive prefixes of rows and of tiles: a thread takes a run of experts
  const int span = (n_expert + kManyThreads - 1) / kManyThreads, e0 = min(tid * span, n_expert), e1 = min(e0 + span, n_expert);
  int c = 0, t = 0;
  for (int e = e0; e < e1; ++e) {
    const int v = before[e] + rest[e];
    c += v;
    t += (v + tok_per - 1) / tok_per;
  }
  int ic = c, it = t;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int uc = __shfl_up_sync(0xFFFFFFFFu, ic, o), ut = __shfl_up_sync(0xFFFFFFFFu, it, o);
    if (lane >= o) { ic += uc; it += ut; }
  }
  if (lane == 31) { wsum[0][wp] = ic; wsum[1][wp] = it; }
  __syncthreads();
  int pc = ic - c + __reduce_add_sync(0xFFFFFFFFu, lane < wp ? wsum[0][lane] : 0);
  int pt = it - t + __reduce_add_sync(0xFFFFFFFFu, lane < wp ? wsum[1][lane] : 0);
  for (int e = e0; e < e1; ++e) {
    const int v = before[e] + rest[e];
    if (blockIdx.x == 0) { off[e] = pc; toff[e] = pt; }
    before[e] += pc;
    pc += v;
    pt += (v + tok_per - 1) / tok_per;
  }
  if (blockIdx.x == 0 && tid == kManyThreads - 1) {
    off[n_expert] = pc;
    toff[n_expert] = pt;
    meta[0] = pc;
    meta[1] = pt;
    meta[2] = bad_sh;
    if (mail_n != nullptr) *mail_n = 0;
  }
  __syncthreads();

  if (wp != 0) return;
  for (int b = first; b < last; b += 256) {
    int e8[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) e8[q] = b + 32 * q + lane < last ? id_of(b + 32 * q + lane) : -1;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int e = e8[q], i = b + 32 * q + lane;
      const unsigned same = __match_any_sync(0xFFFFFFFFu, e);
      const int rank = __popc(same & ((1u << lane) - 1u));
      if (e >= 0) {
        const int slot = before[e] + rank;
        gslot[i] = slot;
        grows[slot] = by_k(i);
      }
      __syncwarp();
      if (e >= 0 && rank == 0) before[e] += __popc(same);
      __syncwarp();
    }
  }
}

// ---- row movement ------------------------------------------------------------------
// dst row r <- src row src_rows[r]; rows of `row_bytes` bytes (multiple of 4).
// grid.x = rows (bounded by *meta when meta != nullptr), grid.y = chunks of a row.
__global__ void gather_rows_kernel(unsigned char* __restrict__ dst,
                                   const unsigned char* __restrict__ src,
                                   const int* __restrict__ src_rows, const int* __restrict__ meta,
                                   int row_bytes) {
  const int r = blockIdx.x;
  if (meta != nullptr && r >= *meta) return;
  const unsigned char* s = src + static_cast<size_t>(src_rows[r]) * row_bytes;
  unsigned char* d = dst + static_cast<size_t>(r) * row_bytes;
  if (aligned16(s) && aligned16(d) && (row_bytes & 15) == 0) {
    for (int i = blockIdx.y * blockDim.x + threadIdx.x; i < row_bytes / 16; i += gridDim.y * blockDim.x)
      reinterpret_cast<uint4*>(d)[i] = reinterpret_cast<const uint4*>(s)[i];
  } else if (((reinterpret_cast<uintptr_t>(s) | reinterpret_cast<uintptr_t>(d)) & 3u) == 0) {
    for (int i = blockIdx.y * blockDim.x + threadIdx.x; i < row_bytes / 4; i += gridDim.y * blockDim.x)
      reinterpret_cast<uint32_t*>(d)[i] = reinterpret_cast<const uint32_t*>(s)[i];
  } else {
    for (int i = blockIdx.y * blockDim.x + threadIdx.x; i < row_bytes / 2; i += gridDim.y * blockDim.x)
      reinterpret_cast<uint16_t*>(d)[i] = reinterpret_cast<const uint16_t*>(s)[i];
  }
}

// dst[dst_rows[i]] = src[i] (fp16 rows of `hidden`); grid.x = rows
__global__ void scatter_rows_kernel(uint16_t* __restrict__ dst, const uint16_t* __restrict__ src,
                                    const int* __restrict__ dst_rows, int hidden) {
  const int i = blockIdx.x;
  const uint16_t* s = src + static_cast<size_t>(i) * hidden;
  uint16_t* d = dst + static_cast<size_t>(dst_rows[i]) * hidden;
  if (aligned16(s) && aligned16(d) && (hidden & 7) == 0) {
    for (int j = blockIdx.y * blockDim.x + threadIdx.x; j < hidden / 8; j += gridDim.y * blockDim.x)
      reinterpret_cast<uint4*>(d)[j] = reinterpret_cast<const uint4*>(s)[j];
  } else {
    for (int j = blockIdx.y * blockDim.x + threadIdx.x; j < hidden; j += gridDim.y * blockDim.x)
      d[j] = s[j];
  }
}

// expert_y[row][kk][:] = grouped_out[gslot[row*n_used + kk]][:] (slab has n_used+1 slots
// per row; gslot < 0: slot left as is); grid (rows, chunks, n_used)
__global__ void scatter_routed_kernel(uint16_t* __restrict__ expert_y,
                                      const uint16_t* __restrict__ grouped_out,
                                      const int* __restrict__ gslot, int n_used, int hidden) {
  const int row = blockIdx.x, kk = blockIdx.z;
  const int gs = gslot[static_cast<size_t>(row) * n_used + kk];
  if (gs < 0) return;
  const uint16_t* s = grouped_out + static_cast<size_t>(gs) * hidden;
  uint16_t* d = expert_y + (static_cast<size_t>(row) * (n_used + 1) + kk) * hidden;
  if (aligned16(s) && aligned16(d) && (hidden & 7) == 0) {
    for (int j = blockIdx.y * blockDim.x + threadIdx.x; j < hidden / 8; j += gridDim.y * blockDim.x)
      reinterpret_cast<uint4*>(d)[j] = reinterpret_cast<const uint4*>(s)[j];
  } else {
    for (int j = blockIdx.y * blockDim.x + threadIdx.x; j < hidden; j += gridDim.y * blockDim.x)
      d[j] = s[j];
  }
}

// expert_out[k][:] = fp16(miss_y[slot_of_k[k]][:]) for slot >= 0; grid (k_rows, chunks)
__global__ void scatter_miss_kernel(uint16_t* __restrict__ expert_out,
                                    const int* __restrict__ slot_of_k,
                                    const float* __restrict__ miss_y, int hidden) {
  const int k = blockIdx.x;
  const int slot = slot_of_k[k];
  if (slot < 0) return;
  for (int i = blockIdx.y * blockDim.x + threadIdx.x; i < hidden; i += gridDim.y * blockDim.x)
    expert_out[static_cast<size_t>(k) * hidden + i] = f2h(miss_y[static_cast<size_t>(slot) * hidden + i]);
}

// dst[dst_flat[i] + j] = fp16(src[i][j]); dst_flat holds element offsets; grid (n_list, chunks)
__global__ void scatter_rows_generic_kernel(uint16_t* __restrict__ dst, const float* __restrict__ src,
                                            const int* __restrict__ dst_flat, int hidden) {
  const int i = blockIdx.x;
  const size_t base = static_cast<size_t>(dst_flat[i]);
  for (int j = blockIdx.y * blockDim.x + threadIdx.x; j < hidden; j += gridDim.y * blockDim.x)
    dst[base + j] = f2h(src[static_cast<size_t>(i) * hidden + j]);
}

// ---- SwiGLU and gates (norm_rotary.cu:133-183) ------------------------------------
__global__ void silu_mul_kernel(uint16_t* __restrict__ out, const uint16_t* __restrict__ g,
                                const uint16_t* __restrict__ u, long long total,
                                const int* __restrict__ d_rows, int n_ff) {
  if (d_rows != nullptr) total = min(total, static_cast<long long>(*d_rows) * n_ff);
  const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
  const long long t0 = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (aligned16(out) && aligned16(g) && aligned16(u)) {
    const long long n8 = total / 8;
    for (long long i = t0; i < n8; i += stride) {
      const uint4 gv = reinterpret_cast<const uint4*>(g)[i];
      const uint4 uv = reinterpret_cast<const uint4*>(u)[i];
      const uint32_t gw[4] = {gv.x, gv.y, gv.z, gv.w}, uw[4] = {uv.x, uv.y, uv.z, uv.w};
      uint32_t ow[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint16_t lo = f2h(silu_mul(h2f(gw[j] & 0xFFFF), h2f(uw[j] & 0xFFFF)));
        const uint16_t hi = f2h(silu_mul(h2f(gw[j] >> 16), h2f(uw[j] >> 16)));
        ow[j] = lo | (static_cast<uint32_t>(hi) << 16);
      }
      reinterpret_cast<uint4*>(out)[i] = make_uint4(ow[0], ow[1], ow[2], ow[3]);
    }
    for (long long i = n8 * 8 + t0; i < total; i += stride) out[i] = f2h(silu_mul(h2f(g[i]), h2f(u[i])));
  } else {
    for (long long i = t0; i < total; i += stride) out[i] = f2h(silu_mul(h2f(g[i]), h2f(u[i])));
  }
}

// out[row][i] *= sigmoid(g[row]); grid (rows, chunks)
__global__ void sigmoid_gate_scalar_kernel(uint16_t* __restrict__ out, const float* __restrict__ g,
                                           int hidden) {
  const int row = blockIdx.x;
  const float sig = 1.f / (1.f + expf(-g[row]));
  uint16_t* p = out + static_cast<size_t>(row) * hidden;
  for (int i = blockIdx.y * blockDim.x + threadIdx.x; i < hidden; i += gridDim.y * blockDim.x)
    p[i] = f2h(h2f(p[i]) * sig);
}

// ---- combine (moe.cu:88-100, 265-280, 503-518) --------------------------------------
// out[row][i] = f16( f32(out[row][i]) + sum_kk w[kk] * f32(y[row][kk][i]) ), kk ascending.
// idx != nullptr: single-row form, slots with idx[kk] < 0 are skipped and the slab has
// `slots` rows; idx == nullptr: batched positional form with `slots` = n_used + 1.
__global__ void combine_kernel(uint16_t* __restrict__ out, const uint16_t* __restrict__ expert_y,
                               const int* __restrict__ idx, const float* __restrict__ weight,
                               int slots, int hidden) {
  extern __shared__ float wsm[];       // [slots] weights of this row, then [slots] skip flags
  int* skip_sm = reinterpret_cast<int*>(wsm + slots);
  const int row = blockIdx.x;
  for (int kk = threadIdx.x; kk < slots; kk += blockDim.x) {
    wsm[kk] = weight[static_cast<size_t>(row) * slots + kk];
    skip_sm[kk] = (idx != nullptr && idx[kk] < 0) ? 1 : 0;   // slot not delivered (yet)
  }
  __syncthreads();
  uint16_t* o = out + static_cast<size_t>(row) * hidden;
  const uint16_t* y = expert_y + static_cast<size_t>(row) * slots * hidden;
  if (aligned16(o) && aligned16(y) && (hidden & 7) == 0) {
    for (int j = blockIdx.y * blockDim.x + threadIdx.x; j < hidden / 8; j += gridDim.y * blockDim.x) {
      const uint4 rv = reinterpret_cast<const uint4*>(o)[j];
      const uint32_t rw[4] = {rv.x, rv.y, rv.z, rv.w};
      float acc[8];
#pragma unroll
      for (int q = 0; q < 4; ++q) { acc[2 * q] = h2f(rw[q] & 0xFFFF); acc[2 * q + 1] = h2f(rw[q] >> 16); }
      for (int kk = 0; kk < slots; ++kk) {
        const float w = wsm[kk];
        if (skip_sm[kk]) continue;
        const uint4 yv = reinterpret_cast<const uint4*>(y + static_cast<size_t>(kk) * hidden)[j];
        const uint32_t yw[4] = {yv.x, yv.y, yv.z, yv.w};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          acc[2 * q] += w * h2f(yw[q] & 0xFFFF);
          acc[2 * q + 1] += w * h2f(yw[q] >> 16);
        }
      }
      uint32_t ow[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) ow[q] = f2h(acc[2 * q]) | (static_cast<uint32_t>(f2h(acc[2 * q + 1])) << 16);
      reinterpret_cast<uint4*>(o)[j] = make_uint4(ow[0], ow[1], ow[2], ow[3]);
    }
  } else {
    for (int i = blockIdx.y * blockDim.x + threadIdx.x; i < hidden; i += gridDim.y * blockDim.x) {
      float acc = h2f(o[i]);
      for (int kk = 0; kk < slots; ++kk) {
        const float w = wsm[kk];
        if (skip_sm[kk]) continue;
        acc += w * h2f(y[static_cast<size_t>(kk) * hidden + i]);
      }
      o[i] = f2h(acc);
    }
  }
}

// Late add of patched slots, one after another inside each thread so that the
// read-modify-write of a row never races (moe.cu:497-518).
__global__ void combine_add_slots_kernel(uint16_t* __restrict__ out,
                                         const uint16_t* __restrict__ expert_y,
                                         const float* __restrict__ weight, const int* __restrict__ rk,
                                         int n_used, int hidden, int n_list) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < hidden; i += gridDim.x * blockDim.x) {
    for (int li = 0; li < n_list; ++li) {
      const size_t slot = static_cast<size_t>(rk[li]);
      const size_t row = slot / (n_used + 1);
      const float acc = h2f(out[row * hidden + i]) + weight[slot] * h2f(expert_y[slot * hidden + i]);
      out[row * hidden + i] = f2h(acc);
    }
  }
}

// chunks of a row (grid.y) for kernels that put rows in grid.x: `units` work items per row,
// `threads` per CTA; few rows get more chunks so a single-row call still spreads out
inline int row_chunks(int units, int threads, int rows) {
  const int full = (units + threads - 1) / threads;
  return rows >= 64 ? 1 : (full < 1 ? 1 : (full > 64 ? 64 : full));
}
inline int ok_or_launch() { return cudaPeekAtLastError() == cudaSuccess ? kOk : kErrLaunch; }

}  // namespace
}  // namespace sgr

using namespace sgr;

SGR_API int sgr_moe_dispatch_scan(const int* idx, float* weight, int* gslot, int* grows, int* off,
                                  int* toff, int* meta, int* mail, int* mail_n, int n_rows, int k,
                                  int n_expert, int tok_per, void* stream) {
  (void)mail;
  if (!idx || !weight || !gslot || !grows || !off || !toff || !meta || n_rows < 0 || k <= 0 ||
      n_expert <= 0 || tok_per <= 0)
    return kErrArg;
  if (static_cast<long long>(n_rows) * k > 0x7FFFFF00) return kErrArg;
  if (n_expert > 12 * 1024) return kErrUnsupported;
  const int total = n_rows * k;
  cudaStream_t st = as_stream(stream);
  if (n_expert > kScanExperts || total > kScanRoutes) {
    const int sms = device_sms();
    if (sms <= 0) return kErrLaunch;
    const int per = std::max(256, (total + sms - 1) / sms);
    const size_t smem = 2 * static_cast<size_t>(n_expert) * sizeof(int);
    if (smem > 40 * 1024 && !opt_in_smem<dispatch_scan_many_kernel>(static_cast<int>(smem))) return kErrLaunch;
    return launch_pdl(dispatch_scan_many_kernel, dim3(std::max(1, (total + per - 1) / per)), kManyThreads, smem, st, idx, weight, gslot, grows,
                      off, toff, meta, mail_n, n_rows, k, n_expert, tok_per, per, FastDiv(k));
  }
  const int per = ((total + kScanParts - 1) / kScanParts + 31) / 32 * 32;       // routes per part
  const size_t smem = static_cast<size_t>(kScanParts) * n_expert * sizeof(int) + static_cast<size_t>(total) * 2;
  constexpr int per_cta = kScanWarps / kScanParts;
  return launch_pdl(dispatch_scan_kernel, dim3((n_expert + per_cta - 1) / per_cta), kScanThreads, smem, st, idx, weight,
                    gslot, grows, off, toff, meta, mail_n, n_rows, k, n_expert, tok_per, per, FastDiv(k), FastDiv(per));
}

SGR_API int sgr_gather_rows_q8(void* dst, const void* src, const int* src_rows, int n_rows,
                               int row_blocks, void* stream) {
  if (n_rows <= 0 || row_blocks <= 0) return kOk;
  if (!dst || !src || !src_rows) return kErrArg;
  if ((reinterpret_cast<uintptr_t>(dst) | reinterpret_cast<uintptr_t>(src)) & 3u) return kErrAlign;
  const int row_bytes = row_blocks * kX8;
  gather_rows_kernel<<<dim3(n_rows, row_chunks(row_bytes / 16, 128, n_rows)), 128, 0, as_stream(stream)>>>(
      static_cast<unsigned char*>(dst), static_cast<const unsigned char*>(src), src_rows, nullptr,
      row_bytes);
  return ok_or_launch();
}

SGR_API int sgr_gather_rows_q8_n(void* dst, const void* src, const int* src_rows, const int* meta,
                                 int r_max, int row_blocks, void* stream) {
  if (r_max <= 0 || row_blocks <= 0) return kOk;
  if (!dst || !src || !src_rows || !meta) return kErrArg;
  if ((reinterpret_cast<uintptr_t>(dst) | reinterpret_cast<uintptr_t>(src)) & 3u) return kErrAlign;
  gather_rows_kernel<<<dim3(r_max, row_chunks(row_blocks * kX8 / 16, 128, r_max)), 128, 0,
                       as_stream(stream)>>>(static_cast<unsigned char*>(dst),
                                            static_cast<const unsigned char*>(src), src_rows, meta,
                                            row_blocks * kX8);
  return ok_or_launch();
}

SGR_API int sgr_gather_rows_f16_n(uint16_t* dst, const uint16_t* src, const int* src_rows,
                                  const int* meta, int r_max, int hidden, void* stream) {
  if (r_max <= 0 || hidden <= 0) return kOk;
  if (!dst || !src || !src_rows || !meta) return kErrArg;
  gather_rows_kernel<<<dim3(r_max, row_chunks(hidden / 8, 128, r_max)), 128, 0, as_stream(stream)>>>(
      reinterpret_cast<unsigned char*>(dst), reinterpret_cast<const unsigned char*>(src), src_rows,
      meta, hidden * 2);
  return ok_or_launch();
}

SGR_API int sgr_scatter_rows_f16(uint16_t* dst, const uint16_t* src, const int* dst_rows, int n_rows,
                                 int hidden, void* stream) {
  if (n_rows <= 0 || hidden <= 0) return kOk;
  if (!dst || !src || !dst_rows) return kErrArg;
  scatter_rows_kernel<<<dim3(n_rows, row_chunks(hidden / 8, 128, n_rows)), 128, 0, as_stream(stream)>>>(dst, src, dst_rows, hidden);
  return ok_or_launch();
}

SGR_API int sgr_scatter_routed_f16(uint16_t* expert_y, const uint16_t* grouped_out, const int* gslot,
                                   int n_rows, int n_used, int hidden, void* stream) {
  if (n_rows <= 0 || n_used <= 0 || hidden <= 0) return kOk;
  if (!expert_y || !grouped_out || !gslot) return kErrArg;
  if (n_used > 65535) return kErrUnsupported;
  scatter_routed_kernel<<<dim3(n_rows, row_chunks(hidden / 8, 128, n_rows), n_used), 128, 0,
                          as_stream(stream)>>>(
      expert_y, grouped_out, gslot, n_used, hidden);
  return ok_or_launch();
}

SGR_API int sgr_scatter_miss_f32(uint16_t* expert_out, const int* d_slot_of_k, const float* miss_y,
                                 int k_rows, int hidden, void* stream) {
  if (k_rows <= 0 || hidden <= 0) return kOk;
  if (!expert_out || !d_slot_of_k || !miss_y) return kErrArg;
  scatter_miss_kernel<<<dim3(k_rows, row_chunks(hidden, 256, k_rows)), 256, 0, as_stream(stream)>>>(
      expert_out, d_slot_of_k, miss_y, hidden);
  return ok_or_launch();
}

SGR_API int sgr_scatter_rows_generic_f16(uint16_t* dst, const float* src, const int* dst_flat,
                                         int n_list, int hidden, void* stream) {
  if (n_list <= 0 || hidden <= 0) return kOk;
  if (!dst || !src || !dst_flat) return kErrArg;
  scatter_rows_generic_kernel<<<dim3(n_list, row_chunks(hidden, 256, n_list)), 256, 0, as_stream(stream)>>>(
      dst, src, dst_flat, hidden);
  return ok_or_launch();
}

SGR_API int sgr_silu_mul_f16(uint16_t* out, const uint16_t* g, const uint16_t* u, int rows, int n_ff,
                             void* stream) {
  const long long total = static_cast<long long>(rows) * n_ff;
  if (total <= 0) return kOk;
  if (!out || !g || !u) return kErrArg;
  const int blocks = static_cast<int>(std::min<long long>((total / 8 + 255) / 256 + 1, 148 * 8));
  silu_mul_kernel<<<blocks, 256, 0, as_stream(stream)>>>(out, g, u, total, nullptr, n_ff);
  return ok_or_launch();
}

SGR_API int sgr_silu_mul_f16_n(uint16_t* out, const uint16_t* g, const uint16_t* u, const int* d_rows,
                               int rows_max, int n_ff, void* stream) {
  const long long total = static_cast<long long>(rows_max) * n_ff;
  if (total <= 0) return kOk;
  if (!out || !g || !u || !d_rows) return kErrArg;
  const int blocks = static_cast<int>(std::min<long long>((total / 8 + 255) / 256 + 1, 148 * 8));
  silu_mul_kernel<<<blocks, 256, 0, as_stream(stream)>>>(out, g, u, total, d_rows, n_ff);
  return ok_or_launch();
}

SGR_API int sgr_sigmoid_gate_scalar_f16(uint16_t* out, const float* g, int n, void* stream) {
  if (n <= 0) return kOk;
  if (!out || !g) return kErrArg;
  sigmoid_gate_scalar_kernel<<<dim3(1, row_chunks(n, 256, 1)), 256, 0, as_stream(stream)>>>(out, g, n);
  return ok_or_launch();
}

SGR_API int sgr_sigmoid_gate_scalar_batched_f16(uint16_t* out, const float* g, int n_rows, int hidden,
                                                void* stream) {
  if (n_rows <= 0 || hidden <= 0) return kOk;
  if (!out || !g) return kErrArg;
  sigmoid_gate_scalar_kernel<<<dim3(n_rows, row_chunks(hidden, 256, n_rows)), 256, 0, as_stream(stream)>>>(
      out, g, hidden);
  return ok_or_launch();
}

SGR_API int sgr_moe_combine_f16(uint16_t* out, const uint16_t* expert_out, const int* idx,
                                const float* weight, int n_expert_used, int hidden, void* stream) {
  if (n_expert_used <= 0 || hidden <= 0) return kOk;
  if (!out || !expert_out || !idx || !weight) return kErrArg;
  combine_kernel<<<dim3(1, row_chunks(hidden / 8, 64, 1)), 64, n_expert_used * 8,
                   as_stream(stream)>>>(out, expert_out, idx, weight, n_expert_used, hidden);
  return ok_or_launch();
}

SGR_API int sgr_moe_combine_batched_f16(uint16_t* out, const uint16_t* expert_y, const float* weight,
                                        int n_used, int hidden, int n_rows, void* stream) {
  if (n_rows <= 0 || hidden <= 0) return kOk;
  if (!out || !expert_y || !weight || n_used < 0) return kErrArg;
  combine_kernel<<<dim3(n_rows, row_chunks(hidden / 8, 64, n_rows)), 64, (n_used + 1) * 8,
                   as_stream(stream)>>>(out, expert_y, nullptr, weight, n_used + 1, hidden);
  return ok_or_launch();
}

SGR_API int sgr_moe_combine_add_slots_f16(uint16_t* out, const uint16_t* expert_y,
                                          const float* weight, const int* rk, int n_used, int hidden,
                                          int n_list, void* stream) {
  if (n_list <= 0 || hidden <= 0) return kOk;
  if (!out || !expert_y || !weight || !rk) return kErrArg;
  combine_add_slots_kernel<<<(hidden + 255) / 256, 256, 0, as_stream(stream)>>>(
      out, expert_y, weight, rk, n_used, hidden, n_list);
  return ok_or_launch();
}
