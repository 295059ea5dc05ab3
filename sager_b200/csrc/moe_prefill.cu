// moe_prefill.cu - one MoE layer over a prefill chunk behind one call.
//
// The sequence is the one Session::moe_dispatch_device of the reference runs for a
// chunk (src/core/session.cpp:2482-3030): quantize_q8_k -> gemv_f32_out_f16x_mtok ->
// router_topk_batched -> moe_dispatch_scan -> gather_rows_q8_n -> gate / up ->
// silu_mul_f16_n -> quantize_q8_k_n -> down -> scatter_routed_f16 -> shared expert
// (gemv2 mtok, silu_mul, quantize, gemv mtok, strided copy into slot K of the combine
// slab) -> moe_combine_batched_f16, on the caller's scratch buffers
// (src/core/session.cpp:207-257). What is joined here, with the same values in the same order:
//   * gate, up and the shared expert's gate, up are one tensor-core launch (grouped_gemm_i8.cu) that
//     reads its activation rows through the plan (no gather), down and the shared down another -
//     where the reference dequantises to fp16 and calls a library GEMM per expert
//     (src/core/session.cpp:2643-2760);
//   * SwiGLU and the requantisation of both row sets are one launch, which writes the rows as ready
//     GEMM operands; so does the input quantiser. They lie in the combine slab, unused otherwise;
//   * scatter, strided copy and combine are one kernel that reads the grouped and the shared rows
//     where they lie.
// Stream-ordered, no host synchronisation, nothing allocated: legal inside stream capture.
#include <algorithm>

#include "api_util.cuh"
#include "q4k_common.cuh"

using namespace sgr;

namespace {
// Up to this many routed rows per expert on average the row-streaming GEMM takes the expert stage: its work grows with the rows,
// the tcgen05 form's with the weights. Two layers (hidden / FFN / experts / top-k), us, against the tcgen05 form, evenly spread rows:
//   2048 / 512 / 256 / 8: 12 rows per expert 298 / 433, 20 376 / 469, 25 424 / 481, 28 462 / 485, 31 511 / 496
//   1024 / 512 / 128 / 8: 12 132 / 163, 20 152 / 173, 25 168 / 176, 28 178 / 180, 31 189 / 184
//   2048 / 256 / 64 / 8:  12 101 / 111, 20 109 / 122, 25 122 / 123, 26 143 / 123 (passes past 32 rows begin a second wave of items)
//   1024 / 512 / 16 / 4:  12 69 / 72, 20 74 / 80, 25 76 / 77, 28 79 / 77;  512 / 256 / 128 / 8: 20 86 / 96, 25 93 / 97, 28 99 / 98
// The mean is what the host knows; hot experts move the line up, since both forms then work in passes, these of 32 rows and
// those of 80 (a fifth of the experts in 70 % of the routes: 25 rows 464 / 690, 183 / 281, 140 / 159; 31 rows 533 / 764, 198 / 324, 145 / 174).
constexpr int kFewRows = 25;
// x[row] += sum_k w[row][k] * y_grouped[gslot[row][k]] (k = 0 .. K-1, in this order; a route that was
// not computed, gslot < 0, adds nothing) + w[row][K] * sh_y[row] (when there is a shared expert):
// scatter_routed_f16 + the strided copy + moe_combine_batched_f16 of the reference's sequence
// (src/core/session.cpp:2890-2930) without the slab in between. fp32 sums, one rounding to fp16.
// grid (rows, column chunks), 128 threads, 8 columns per thread; dynamic smem: (K+1) floats + K ints.
__global__ void combine_grouped_kernel(uint16_t* __restrict__ x, const uint16_t* __restrict__ y_grouped,
                                       const int* __restrict__ gslot, const uint16_t* __restrict__ sh_y,
                                       const float* __restrict__ weight, int K, int H) {
  extern __shared__ float wsm[];       // [K+1] weights of this row, then [K] grouped slots
  int* slot_sm = reinterpret_cast<int*>(wsm + K + 1);
  pdl_wait();
  pdl_launch_dependents();
  const int row = blockIdx.x;
  for (int kk = threadIdx.x; kk <= K; kk += blockDim.x) {
    wsm[kk] = weight[static_cast<size_t>(row) * (K + 1) + kk];
    if (kk < K) slot_sm[kk] = gslot[static_cast<size_t>(row) * K + kk];
  }
  __syncthreads();
  uint16_t* o = x + static_cast<size_t>(row) * H;
  for (int j = blockIdx.y * blockDim.x + threadIdx.x; j < H / 8; j += gridDim.y * blockDim.x) {
    const uint4 rv = reinterpret_cast<const uint4*>(o)[j];
    const uint32_t rw[4] = {rv.x, rv.y, rv.z, rv.w};
    float acc[8];
#pragma unroll
    for (int q = 0; q < 4; ++q) { acc[2 * q] = h2f(rw[q] & 0xFFFF); acc[2 * q + 1] = h2f(rw[q] >> 16); }
    for (int k0 = 0; k0 < K; k0 += 8) {             // eight routes' rows requested together
      uint4 yv[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int gs = k0 + u < K ? slot_sm[k0 + u] : -1;
        yv[u] = gs >= 0 ? __ldg(reinterpret_cast<const uint4*>(y_grouped + static_cast<size_t>(gs) * H) + j)
                        : make_uint4(0u, 0u, 0u, 0u);
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        if (k0 + u < K && slot_sm[k0 + u] >= 0) {
          const float w = wsm[k0 + u];
          const uint32_t yw[4] = {yv[u].x, yv[u].y, yv[u].z, yv[u].w};
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            acc[2 * q] += w * h2f(yw[q] & 0xFFFF);
            acc[2 * q + 1] += w * h2f(yw[q] >> 16);
          }
        }
      }
    }
    if (sh_y != nullptr) {
      const float w = wsm[K];
      const uint4 sv = __ldg(reinterpret_cast<const uint4*>(sh_y + static_cast<size_t>(row) * H) + j);
      const uint32_t yw[4] = {sv.x, sv.y, sv.z, sv.w};
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
}

inline bool has_shared(const sgr_moe_prefill* a) { return a->shared_gate && a->shared_up && a->shared_down; }

// The rows the GEMMs read lie in the combine slab's memory when they fit there: Q8_K rows in padded blocks for the kernel of few
// token rows per expert, ready operands for the tcgen05 one (FFN up to about 0.8 x hidden at top-8); otherwise Q8_K rows from
// which the tcgen05 GEMMs make their operands themselves. In front of them lie the hand-out counters and, where the slab holds
// those too (some 400 bytes per expert: buffers of a few rows for many experts have no room), the experts' descriptors.
enum class Rows { kPadded, kOperands, kPacked };
struct OperandRows {
  Rows form;
  unsigned char *x, *h, *s;       // layer input, routed h, shared expert's h
  unsigned char* maps;            // null: none
  unsigned* counters;
};
OperandRows operand_rows(const sgr_moe_prefill* a) {
  const long long nbh = a->hidden / kQK, nbf = a->n_ff / kQK, room = static_cast<long long>(a->n_max) * (a->n_used + 1) * a->hidden * 2;
  unsigned char* slab = reinterpret_cast<unsigned char*>(a->expert_y);
  const uintptr_t at = reinterpret_cast<uintptr_t>(slab);
  const long long pad = -at & 127u, map_bytes = (a->n_expert + 1LL) * kExpertMapBytes;
  OperandRows r{};
  auto fits = [&](Rows form, long long blk) {
    const long long x = a->n * nbh * blk, h = static_cast<long long>(a->n) * a->n_used * nbf * blk, s = a->n * nbf * blk;
    for (const bool with_maps : {true, false}) {
      const long long maps_end = with_maps ? pad + ((map_bytes + 15) & ~15LL) : 0;
      const long long front = maps_end + (with_maps || form == Rows::kPadded ? 16 : 0);
      if (front + x + h + s > room) continue;
      unsigned char* base = slab + front;
      r = {form, base, base + x, base + x + h, with_maps ? slab + pad : nullptr, reinterpret_cast<unsigned*>(slab + maps_end)};
      return true;
    }
    return false;
  };
  const uintptr_t outs = reinterpret_cast<uintptr_t>(a->g) | reinterpret_cast<uintptr_t>(a->y_grouped) |
                         reinterpret_cast<uintptr_t>(a->sh_g) | reinterpret_cast<uintptr_t>(a->sh_y);
  if ((at & 15u) == 0) {
    if ((outs & 3u) == 0 && static_cast<long long>(a->n) * a->n_used <= static_cast<long long>(kFewRows) * a->n_expert && fits(Rows::kPadded, kRowBlk))
      return r;
    if (fits(Rows::kOperands, kOpBlk)) return r;
  }
  return {Rows::kPacked, static_cast<unsigned char*>(a->xq), static_cast<unsigned char*>(a->hq), static_cast<unsigned char*>(a->sh_q), nullptr, nullptr};
}

// the combine reads the grouped rows in place when every buffer allows 16-byte accesses
bool combines_in_place(const sgr_moe_prefill* a) {
  return (a->hidden & 7) == 0 && a->n_used <= 1024 &&
         ((reinterpret_cast<uintptr_t>(a->x_f16) | reinterpret_cast<uintptr_t>(a->y_grouped) |
           (has_shared(a) ? reinterpret_cast<uintptr_t>(a->sh_y) : 0)) & 15u) == 0;
}

ExpertMaps expert_maps(const sgr_moe_prefill* a, const OperandRows& op) {
  return {reinterpret_cast<const unsigned char* const*>(a->w_tab), a->tab_stride > 0 ? a->tab_stride : a->n_expert, op.maps, op.counters,
          {a->shared_gate, a->shared_up, a->shared_down}, a->n_expert, a->hidden, a->n_ff};
}

// gate / up, SwiGLU, requantise, down of the routed experts and of the shared one
int expert_stage(const sgr_moe_prefill* a, const OperandRows& op, cudaStream_t stream) {
  const int n = a->n, H = a->hidden, F = a->n_ff, E = a->n_expert, K = a->n_used;
  const bool shared = has_shared(a);
  const long long ts = a->tab_stride > 0 ? a->tab_stride : E, R = static_cast<long long>(a->n_max) * K;
  // (with descriptors: the addresses that these were made from, not what the table says by now)
  auto tab = [&](int m) {
    return op.maps != nullptr ? map_addresses(op.maps, E, m) : reinterpret_cast<const unsigned char* const*>(a->w_tab + m * ts);
  };
  ExpertGemm up{};
  up.tab = tab(0); up.off = a->off; up.rows = a->grows; up.xq = op.x; up.operand_rows = op.form == Rows::kOperands;
  up.y = a->g; up.n_rows = F; up.k = H; up.n_expert = E;
  ExpertGemm down{};
  down.tab = tab(2); down.off = a->off; down.xq = op.h; down.operand_rows = up.operand_rows;
  up.maps = down.maps = op.maps;
  up.counters = down.counters = op.counters;
  up.stream = down.stream = streams_weights(H, F, E);
  up.routes = down.routes = static_cast<long long>(n) * K;
  down.y = a->y_grouped; down.n_rows = H; down.k = F; down.n_expert = E;
  if (shared) {
    up.shared_w = a->shared_gate; up.shared_xq = op.x; up.shared_y = a->sh_g; up.shared_rows = n;
    down.shared_w = a->shared_down; down.shared_xq = op.s; down.shared_y = a->sh_y; down.shared_rows = n;
  }
  int rc;
  if (op.form == Rows::kPadded) {              // SwiGLU happens in the GEMM
    rc = gemm_rows_gate_up(up, tab(1), a->shared_up, stream);
    if (rc == kOk)
      rc = quantize_rows(a->g, op.h, static_cast<long long>(n) * K, a->meta, a->sh_g, op.s, shared ? n : 0, F, expert_maps(a, op), false, stream);
    return rc == kOk ? gemm_rows_down(down, stream) : rc;
  }
  rc = gemm_gate_up(up, tab(1), a->u, a->shared_up, a->sh_u, stream);
  if (rc != kOk) return rc;
  if (op.form == Rows::kOperands) {
    rc = quantize_operand(a->g, a->u, op.h, static_cast<long long>(n) * K, a->meta, a->sh_g, a->sh_u, op.s, shared ? n : 0, F, expert_maps(a, op), false,
                          stream);
  } else {
    rc = sgr_silu_mul_f16_n(a->g, a->g, a->u, a->meta, static_cast<int>(R), F, stream);
    if (rc == kOk) rc = sgr_quantize_q8_k_n(a->g, a->hq, a->meta, F, static_cast<int>(R * (F / kQK)), stream);
    if (rc == kOk && shared) rc = sgr_silu_mul_f16(a->sh_g, a->sh_g, a->sh_u, n, F, stream);
    if (rc == kOk && shared) rc = sgr_quantize_q8_k(a->sh_g, a->sh_q, static_cast<long long>(n) * F, stream);
  }
  return rc == kOk ? gemm_grouped(down, stream) : rc;
}
}  // namespace

// Diagnostics (sager_b200_diag.h): the expert stage of a finished call once more, for timing.
SGR_API int sgr_moe_prefill_expert_stage(const sgr_moe_prefill* a, void* stream) {
  if (a == nullptr) return kErrArg;
  const OperandRows op = operand_rows(a);
  if (op.form != Rows::kPacked && !combines_in_place(a)) return kErrUnsupported;      // the combine's slab lies where the operand rows were
  if (op.maps != nullptr) {                    // the weights are those of the table given here
    const int rc = op.form == Rows::kPadded
        ? quantize_rows(nullptr, nullptr, 0, nullptr, nullptr, nullptr, 0, a->hidden, expert_maps(a, op), true, as_stream(stream))
        : quantize_operand(nullptr, nullptr, nullptr, 0, nullptr, nullptr, nullptr, nullptr, 0, a->hidden, expert_maps(a, op), true, as_stream(stream));
    if (rc != kOk) return rc;
  }
  return expert_stage(a, op, as_stream(stream));
}

SGR_API int sgr_moe_layer_prefill(const sgr_moe_prefill* a, void* stream) {
  if (a == nullptr) return kErrArg;
  if (a->n <= 0) return kOk;
  const int n = a->n, H = a->hidden, F = a->n_ff, E = a->n_expert, K = a->n_used;
  if (H <= 0 || H % kQK || F <= 0 || F % kQK || E <= 0 || K <= 0 || K > E || a->n_max < n) return kErrGeometry;
  if (!a->xn || !a->x_f16 || !a->w_tab || !a->xq || !a->route_idx || !a->route_w || !a->gslot || !a->grows ||
      !a->off || !a->toff || !a->meta || !a->mail || !a->mail_n || !a->xqg || !a->g || !a->u || !a->hq ||
      !a->y_grouped || !a->expert_y)
    return kErrArg;
  if (!a->logits_in && (!a->router_w || !a->logits)) return kErrArg;
  const bool shared = has_shared(a);
  if (shared && (!a->sh_g || !a->sh_u || !a->sh_q || !a->sh_y)) return kErrArg;
  const long long ts = a->tab_stride > 0 ? a->tab_stride : E;
  if (ts < E) return kErrArg;
  const int tok_per = a->tok_per > 0 ? a->tok_per : 16;
  const long long R = static_cast<long long>(a->n_max) * K;
  if (R > 0x7FFFFFFF / (F / kQK)) return kErrUnsupported;
  // as the launchers of the sequence refuse them
  auto off_by = [](const void* p, unsigned mask) { return (reinterpret_cast<uintptr_t>(p) & mask) != 0; };
  if (off_by(a->xn, 1) || off_by(a->xq, 3) || off_by(a->xqg, 15) || off_by(a->hq, 15) || off_by(a->g, 1) ||
      (shared && (off_by(a->sh_g, 1) || off_by(a->sh_q, 3))))
    return kErrAlign;
  int rc;
#define SGR_STEP(call) do { rc = (call); if (rc != kOk) return rc; } while (0)
  const OperandRows op = operand_rows(a);
  if (op.form == Rows::kPadded) {
    SGR_STEP(quantize_rows(a->xn, op.x, n, nullptr, nullptr, nullptr, 0, H, expert_maps(a, op), true, as_stream(stream)));
  } else if (op.form == Rows::kOperands) SGR_STEP(quantize_operand(a->xn, nullptr, op.x, n, nullptr, nullptr, nullptr, nullptr, 0, H, expert_maps(a, op), true, as_stream(stream)));
  else SGR_STEP(sgr_quantize_q8_k(a->xn, a->xq, static_cast<long long>(n) * H, stream));
  const float* logits = a->logits_in;
  if (logits == nullptr) {
    SGR_STEP(sgr_gemv_f32_out_f16x_mtok(a->router_w, a->xn, a->logits, E, H, n, stream));
    logits = a->logits;
  }
  SGR_STEP(sgr_router_topk_batched(logits, a->route_idx, a->route_w, E, K, K + 1, n,
                                   shared ? a->shared_w : 0.f, stream));
  SGR_STEP(sgr_moe_dispatch_scan(a->route_idx, a->route_w, a->gslot, a->grows, a->off, a->toff, a->meta,
                                 a->mail, a->mail_n, n, K, E, tok_per, stream));
  SGR_STEP(expert_stage(a, op, as_stream(stream)));
  const bool direct = combines_in_place(a);
  if (!direct) SGR_STEP(sgr_scatter_routed_f16(a->expert_y, a->y_grouped, a->gslot, n, K, H, stream));
  if (shared) {
    if (a->shared_gate_w != nullptr) {           // scalar gate sigmoid(w_sg . x) on the shared rows (layer.cpp:128-134)
      if (a->sgate == nullptr) return kErrArg;
      SGR_STEP(sgr_gemv_f32_out_f16x_batched(a->shared_gate_w, a->xn, a->sgate, 1, H, n, stream));
      SGR_STEP(sgr_sigmoid_gate_scalar_batched_f16(a->sh_y, a->sgate, n, H, stream));
    }
    // slot K of every row of the combine slab (the reference's strided copy, src/core/session.cpp:2911-2916)
    if (!direct && cudaMemcpy2DAsync(a->expert_y + static_cast<size_t>(K) * H, static_cast<size_t>(K + 1) * H * 2, a->sh_y,
                          static_cast<size_t>(H) * 2, static_cast<size_t>(H) * 2, n, cudaMemcpyDeviceToDevice,
                          as_stream(stream)) != cudaSuccess)
      return kErrLaunch;
  }
  if (direct) {
    SGR_STEP(launch_pdl(combine_grouped_kernel, dim3(n, (H / 8 + 127) / 128), 128, (2 * K + 1) * sizeof(float), as_stream(stream),
                        a->x_f16, a->y_grouped, a->gslot, shared ? a->sh_y : nullptr, a->route_w, K, H));
  } else {
    SGR_STEP(sgr_moe_combine_batched_f16(a->x_f16, a->expert_y, a->route_w, K, H, n, stream));
  }
#undef SGR_STEP
  return kOk;
}
