// api_util.cuh - conventions shared by the extern "C" entry points.
//
// Every entry point is stream-ordered and never synchronises, allocates or
// reads device memory on the host; it validates its arguments, launches, and
// returns 0 or one of the error codes in q4k_common.cuh. A failed device-side
// bounded wait raises the library's status word, which sgr_status() reads.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "opt_in.cuh"
#include "sager_b200.h"   // the public prototypes: definitions must agree with them
#include "sager_b200_diag.h"

#define SGR_API extern "C" __attribute__((visibility("default")))

namespace sgr {

inline cudaStream_t as_stream(void* s) { return static_cast<cudaStream_t>(s); }

// Device address of the library's status word on the current device.
int* status_word();

// SMs of the current device (0: none can be had), asked of the runtime once per device.
int device_sms();

// Opts kernel K in to `bytes` of dynamic shared memory on the current device; a call to the runtime only when it grows.
template <auto K>
bool opt_in_smem(int bytes) {
  static SmemGrant grant;
  int dev = 0;
  return cudaGetDevice(&dev) == cudaSuccess && grant.ensure(dev, bytes, [](int n) {
           return cudaFuncSetAttribute(K, cudaFuncAttributeMaxDynamicSharedMemorySize, n) == cudaSuccess;
         });
}

// Launch that may start while the kernel before it in the stream drains (programmatic dependent launch);
// the kernel waits for that one's results itself. CLUSTER: CTAs to a cluster, along x.
template <int CLUSTER = 1, typename... KArgs, typename... Args>
int launch_pdl(void (*kern)(KArgs...), dim3 grid, int threads, size_t smem, cudaStream_t stream, const Args&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = CLUSTER;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = CLUSTER > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kern, args...) == cudaSuccess ? 0 : 4 /* kErrLaunch */;
}

// Whether a layer's weights are read under the policy that makes them the first to leave L2. As ordinary lines they push out what
// every layer needs again. What a model keeps in L2 between two uses of a layer is not known here: a layer of more than an eighth
// of it (126 MB) is taken for one of many. us per step, ordinary lines / first to leave:
//   453 MB a layer (2048 / 512 / 256 experts), one layer: 64 / 8 / 4 / 1 rows 88.9 / 48.7 / 33.4 / 15.7, 81.5 / 44.1 / 32.8 / 15.4
//   113 MB (1024 / 512 / 128), 12 layers: 64 / 8 / 4 / 1 rows 669 / 420 / 275 / 162, 595 / 404 / 268 / 159
//   57 MB (2048 / 256 / 64), 12 layers: 588 / 444 / 264 / 160, 579 / 434 / 256 / 155
//   28 MB (1024 / 256 / 64), 12 layers: 459 / 363 / 233 / 151, 452 / 357 / 228 / 151; four, which L2 holds: 157 / 114 / 79 / 54, 154 / 118 / 79 / 54
//   14 MB (1024 / 256 / 32), 24 layers: 799 / 650 / 382 / 284, 788 / 635 / 375 / 284; four 133 / 108 / 64.5 / 51.8, 135 / 109 / 65.5 / 52.2
//   4 MB (512 / 256 / 16), 12 layers: 338 / 283 / 183 / 140, 345 / 287 / 185 / 142
// Below the line few layers lose as much as many would gain. In a prefill chunk the shared expert's weights are read once per 32
// or 80 of its rows, and a hot expert's once per pass, under the same policy: 96 / 777 / 2048 rows of the first geometry, four / two /
// two layers, 499 / 501 / 857 without the policy, 485 / 491 / 850 with it, 490 / 485 / 854 with the shared expert's copies left out of it.
inline bool streams_weights(int hidden, int n_ff, int n_expert) {
  return static_cast<long long>(hidden) * n_ff / 256 * 144 * 3 * n_expert > (16LL << 20);
}

// ---- tensor-core GEMM of Q4_K experts over their routed rows (grouped_gemm_i8.cu) ----
// Operand rows: the quantised activations as the GEMM's fp16 tiles want them, kOpBlk bytes per 256 values -
// 256 codes in K order (0, 2, 1, 3 of every four), eight low and eight high parts of the sub-block sums
// (bsum = 64 * hi + lo), the fp32 scale, 12 bytes of padding. 16-byte aligned.
constexpr int kOpBlk = 560;

// TMA descriptors of a layer's experts, which quantize_operand or quantize_rows makes: [n_expert + 1][3] of 128 bytes (gate, up,
// down; the shared expert's last), then the addresses they were made from, [3][n_expert + 1].
constexpr int kExpertMapBytes = 3 * (128 + 8);
inline const unsigned char* const* map_addresses(const void* maps, int n_expert, int m) {
  return reinterpret_cast<const unsigned char* const*>(static_cast<const unsigned char*>(maps) + (n_expert + 1LL) * 384) + m * (n_expert + 1LL);
}
struct ExpertMaps {
  const unsigned char* const* tab;     // [3][stride]
  long long stride;
  void* maps;                          // 128-byte aligned; null: no room for them
  unsigned* counters;                  // [4], cleared with every launch of quantize_rows
  const void* shared[3];
  int n_expert, hidden, n_ff;
};

// One more expert (shared_w) that every row of its own slab visits may ride along.
struct ExpertGemm {
  const unsigned char* const* tab;
  const int* off;
  const int* rows;              // activation row of each grouped slot, or null: the slot itself
  const unsigned char* xq;      // operand rows, or Q8_K rows (operand_rows false)
  uint16_t* y;
  int n_rows, k, n_expert;
  bool operand_rows;
  bool stream;                  // the weights' L2 policy (streams_weights)
  const void* maps;             // the descriptors (null: none); for operand rows n_rows is a multiple of 128
  unsigned* counters;           // gemm_rows_*: ExpertMaps'
  long long routes;             // routed rows at most (gemm_rows_*)
  const void* shared_w;
  const unsigned char* shared_xq;
  uint16_t* shared_y;
  int shared_rows;
};
int gemm_grouped(const ExpertGemm& g, cudaStream_t stream);
// ---- the same for few token rows per expert (grouped_gemm_rows.cu) ----
// Its activation rows: kRowBlk bytes per 256 values - fp32 scale, 12 bytes of padding, 256 codes, and the sub-block sums as
// bsum = 128 * hi + lo: lo of sub-blocks 0-3, hi of 0-3, lo of 4-7, hi of 4-7, a byte each. 16-byte aligned.
constexpr int kRowBlk = 288;
// n_rows and k multiples of 256, outputs 4-byte aligned.
// gate, up and SwiGLU: y receives h
int gemm_rows_gate_up(const ExpertGemm& g, const unsigned char* const* tab_up, const void* shared_up, cudaStream_t stream);
int gemm_rows_down(const ExpertGemm& g, cudaStream_t stream);
// rows of k fp16 values -> such rows; two slabs, the first of at most *d_rows rows when that is given.
// Clears the counters of the two GEMM launches; with make_maps the descriptors are made as well.
int quantize_rows(const uint16_t* x0, void* out0, long long rows0, const int* d_rows, const uint16_t* x1, void* out1, long long rows1,
                  int k, const ExpertMaps& em, bool make_maps, cudaStream_t stream);
// gate and up in one pass (g holds the gate side)
int gemm_gate_up(const ExpertGemm& g, const unsigned char* const* tab_up, uint16_t* y_up, const void* shared_up,
                 uint16_t* shared_y_up, cudaStream_t stream);
// rows of k fp16 values (SwiGLU of x and u where u is given) -> operand rows; two slabs, the first of at most
// *d_rows rows when that is given; with make_maps the descriptors are made as well
int quantize_operand(const uint16_t* x0, const uint16_t* u0, void* out0, long long rows0, const int* d_rows,
                     const uint16_t* x1, const uint16_t* u1, void* out1, long long rows1, int k, const ExpertMaps& em, bool make_maps,
                     cudaStream_t stream);

}  // namespace sgr
