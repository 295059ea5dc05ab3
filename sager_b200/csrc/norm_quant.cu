// norm_quant.cu - RMS norm fused with the Q8_K activation quantiser: the step
// that produces the MoE half's input rows (xn fp16 and their Q8_K blocks) from the
// residual stream. Replaces rmsnorm_quant_f16 of the reference
// (src/kernels/cuda/mmq.cu:533-641; call site src/core/session.cpp:1020-1023) and is
// held to its contract: bit-identical to the RMS norm followed by the quantiser.
//
// What fixes the bits:
//   sum of squares  thread t of a b-thread block (b = n rounded up to 32, at most
//                   1024) adds x[t]^2, x[t + b]^2, ... with FMA; a warp folds with
//                   shfl_down 16..1; thread 0 adds the warp sums in warp order
//   scale           rsqrtf(sum / n + eps)
//   out[i]          f16((f32(x[i]) * scale) * f32(w[i]))
//   Q8_K blocks     of the fp16 values just written: amax (order-free), d = amax/127,
//                   id = 1/d, codes rint(v * id) clamped to +-127, int16 sub-block sums
// Only the first line constrains the shape of the kernel; it is kept (one CTA per
// row, the same thread-to-element map). The quantiser runs warp-per-block on the
// normalised row held in shared memory instead of the reference's 256-thread
// groups with four CTA barriers per block.
#include "api_util.cuh"
#include "quantize_dev.cuh"

namespace sgr {
namespace {

// PER values per thread kept in registers (0: any number, read twice). Few rows are a chain of latencies -
// load, warp fold, the warp sums in order, normalise, quantise -, and the PER variants shorten it: the norm weights are
// requested before the previous kernel is awaited, and every thread adds the warp sums itself instead of waiting for one to
// do it (one barrier and about a microsecond less). With two CTAs on an SM, or rows of many values, the issue slots
// decide, and 32 warps that add 32 sums each cost more than the barrier: one thread adds (512 rows of 4096: 8.2 us, by
// all threads 9.9; one row of 8192: 4.35 / 4.61).
template <int PER>
__global__ void __launch_bounds__(1024) rmsnorm_quant_kernel(uint16_t* __restrict__ out, const uint16_t* __restrict__ x,
                                                            const uint16_t* __restrict__ w,
                                                            unsigned char* __restrict__ xq, int n, float eps) {
  extern __shared__ __align__(16) uint16_t row_sh[];        // the normalised row, fp16
  __shared__ __align__(16) float red[32];
  const int tid = threadIdx.x, stride = blockDim.x;
  const int lane = tid & 31, warp = tid >> 5;
  constexpr int N = PER > 0 ? PER : 1;
  float v[N], wv[N];
  if constexpr (PER > 0) {
#pragma unroll
    for (int j = 0; j < N; ++j) wv[j] = tid + j * stride < n ? h2f(__ldg(w + tid + j * stride)) : 0.f;
  }
  pdl_wait();                                               // x comes from the previous kernel
  pdl_launch_dependents();
  const size_t row = static_cast<size_t>(blockIdx.x) * n;
  float acc = 0.f;
  if constexpr (PER > 0) {
#pragma unroll
    for (int j = 0; j < N; ++j) v[j] = tid + j * stride < n ? h2f(x[row + tid + j * stride]) : 0.f;
#pragma unroll
    for (int j = 0; j < N; ++j) acc = fmaf(v[j], v[j], acc);
  } else {
    for (int i = tid; i < n; i += stride) {
      const float t = h2f(x[row + i]);
      acc = fmaf(t, t, acc);
    }
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) acc += __shfl_down_sync(0xFFFFFFFFu, acc, off);
  if (lane == 0) red[warp] = acc;
  __syncthreads();
  const int nw = blockDim.x >> 5;
  float scale;
  if constexpr (PER > 0) {
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < 32; i += 4) {
      const float4 r = *reinterpret_cast<const float4*>(red + i);
      if (i < nw) s += r.x;
      if (i + 1 < nw) s += r.y;
      if (i + 2 < nw) s += r.z;
      if (i + 3 < nw) s += r.w;
    }
    scale = rsqrtf(s / static_cast<float>(n) + eps);
  } else {
    if (tid == 0) {
      float s = 0.f;
      for (int i = 0; i < nw; ++i) s += red[i];
      red[0] = rsqrtf(s / static_cast<float>(n) + eps);
    }
    __syncthreads();
    scale = red[0];
  }
  if constexpr (PER > 0) {
#pragma unroll
    for (int j = 0; j < N; ++j)
      if (const int i = tid + j * stride; i < n) {
        const uint16_t h = f2h(v[j] * scale * wv[j]);
        out[row + i] = h;
        row_sh[i] = h;
      }
  } else {
    for (int i = tid; i < n; i += stride) {
      const uint16_t h = f2h(h2f(x[row + i]) * scale * h2f(w[i]));
      out[row + i] = h;
      row_sh[i] = h;
    }
  }
  __syncthreads();
  const int nb = n / kQK;
  for (int blk = warp; blk < nb; blk += nw)
    quantize_block_f16(row_sh + blk * kQK, xq + (static_cast<size_t>(blockIdx.x) * nb + blk) * kX8, lane);
}

}  // namespace
}  // namespace sgr

using namespace sgr;

// cuda_ops.hpp:149-151 of the reference. n must be a multiple of 256 (the reference falls back to
// its unfused norm kernel otherwise; that kernel is not part of this library).
SGR_API int sgr_rmsnorm_quant_f16(uint16_t* out, const uint16_t* x, const uint16_t* w, void* xq, int n, float eps,
                                  int n_rows, void* stream) {
  if (n_rows <= 0) return kOk;
  if (!out || !x || !w || !xq || n <= 0) return kErrArg;
  if (n % kQK != 0 || n > 16384) return kErrUnsupported;
  if (reinterpret_cast<uintptr_t>(xq) & 3u) return kErrAlign;
  int b = ((n + 31) / 32) * 32;
  if (b > 1024) b = 1024;
  const size_t smem = static_cast<size_t>(n) * 2;
  auto launch = [&](auto kern) {
    return launch_pdl(kern, dim3(n_rows), b, smem, as_stream(stream), out, x, w, static_cast<unsigned char*>(xq), n, eps);
  };
  if (n_rows <= device_sms()) {                 // one CTA per SM at most
    if (n <= b) return launch(rmsnorm_quant_kernel<1>);
    if (n <= 2 * b) return launch(rmsnorm_quant_kernel<2>);
    if (n <= 4 * b) return launch(rmsnorm_quant_kernel<4>);
  }
  return launch(rmsnorm_quant_kernel<0>);
}
