// tmap_dev.cuh - TMA descriptors that are patched on the device, shared by the row-streaming expert kernels and the tcgen05 GEMM
// (expert_rows.cuh, grouped_gemm_rows.cu, grouped_gemm_i8.cu): expert addresses live in a pointer table on the device, so a descriptor is
// encoded on the host for a placeholder address and gets its base there.
#pragma once

#include "api_util.cuh"
#include "q4k_common.cuh"

namespace sgr {

// A 2-D descriptor over a Q4_K matrix seen as bytes, [rows][row_bytes], with boxes of one super-block column (144 bytes) x
// 128 rows, encoded for a placeholder address. Encoded once per geometry. (moe_layer.cu)
bool matrix_tmap(int row_bytes, int rows, const void* placeholder, uint32_t* out128);

__device__ __forceinline__ void tmap_replace_addr(void* smem_map, const void* gaddr) {
  asm volatile("tensormap.replace.tile.global_address.shared::cta.b1024.b64 [%0], %1;" ::"r"(smem_u32(smem_map)), "l"(gaddr) : "memory");
}
// whole warp: copy the patched 128-byte descriptor to global memory for the TMA unit
__device__ __forceinline__ void tmap_publish(void* gmem_map, void* smem_map) {
  asm volatile("tensormap.cp_fenceproxy.global.shared::cta.tensormap::generic.release.gpu.sync.aligned [%0], [%1], 128;"
               ::"l"(gmem_map), "r"(smem_u32(smem_map)) : "memory");
}
__device__ __forceinline__ void tmap_acquire(const void* gmem_map) {
  asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(gmem_map) : "memory");
}
// box (144 bytes x 128 rows) at byte column x, row y; dst 128-byte aligned, x a multiple of 16; STREAM: evict_first_policy
template <bool STREAM>
__device__ __forceinline__ void tma_load_box(void* dst, const void* gmem_map, int x, int y, uint64_t* bar) {
  if constexpr (STREAM)
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%2, %3}], [%4], %5;"
                 ::"r"(smem_u32(dst)), "l"(gmem_map), "r"(x), "r"(y), "r"(smem_u32(bar)), "l"(evict_first_policy()) : "memory");
  else
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(smem_u32(dst)), "l"(gmem_map), "r"(x), "r"(y), "r"(smem_u32(bar)) : "memory");
}

// One warp: what tma_load_box copies, where there is no descriptor - `rows` (a multiple of 32) rows' blocks from src, the first
// row's, 16-byte aligned - by cp.async. Each lane's copies add an arrival of their own to the barrier's phase, so the caller's
// arrival counts as with the other form and comes after a __syncwarp. (By a bulk copy per block it is issue-bound:
// 5 rows, 1024 / 512 / 256 experts, 122 us instead of 45; 30 rows, 3584 / 2560 / 4 198 instead of 75. Not inlined: its registers beside the
// TMA copies made the copies of unaligned weights spill, 500 rows of 1024 / 512 / 64 two bytes off 277 -> 410 us.)
static __device__ __noinline__ void cp_load_box(unsigned char* dst, const unsigned char* src, int rows, int row_bytes, uint64_t* bar, int lane) {
  int offs[9];                                   // 16-byte piece q * 32 + lane of 32 rows
#pragma unroll
  for (int q = 0; q < 9; ++q) offs[q] = (q * 32 + lane) / 9 * row_bytes + (q * 32 + lane) % 9 * 16;
  uint32_t d = smem_u32(dst) + lane * 16;
#pragma unroll 1
  for (int r = 0; r < rows; r += 32, d += 9 * 512, src += static_cast<size_t>(32) * row_bytes)
#pragma unroll
    for (int q = 0; q < 9; ++q) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d + q * 512), "l"(src + offs[q]) : "memory");
  asm volatile("cp.async.mbarrier.arrive.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// The descriptors of a layer's experts (ExpertMaps, api_util.cuh), made by CTAs of a launch before the GEMMs, with the addresses
// that they were made from: the GEMMs take absence, alignment and plain copies' sources from those, since the table may be
// rewritten in between, and an entry that was null when the descriptors were made has none. And the counters, cleared.
struct MapArgs {
  unsigned* counters;
  const unsigned char* const* tab;     // [3][stride]
  long long stride;
  unsigned char* maps;
  const unsigned char* shared[3];
  int n_expert;
  alignas(16) uint32_t up[32], down[32];
};
// false: the driver has no encoder
inline bool map_args(const ExpertMaps& em, bool make, MapArgs* m) {
  m->counters = em.counters;
  if (!make || em.maps == nullptr) return true;
  m->tab = em.tab; m->stride = em.stride; m->maps = static_cast<unsigned char*>(em.maps); m->n_expert = em.n_expert;
  for (int i = 0; i < 3; ++i) m->shared[i] = static_cast<const unsigned char*>(em.shared[i]);
  return matrix_tmap(em.hidden / kQK * kW4, em.n_ff, em.maps, m->up) && matrix_tmap(em.n_ff / kQK * kW4, em.hidden, em.maps, m->down);
}
// One warp: the three descriptors of expert e (n_expert: the shared one); `patch` is 384 bytes of shared memory, 128-byte aligned.
// A base that is absent or off a 16-byte boundary keeps the placeholder: its descriptor is not used.
__device__ __forceinline__ void make_maps(const MapArgs& m, int e, unsigned char* patch, int lane) {
  const unsigned char* w[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    w[i] = e == m.n_expert ? m.shared[i] : m.tab[i * m.stride + e];
    reinterpret_cast<uint32_t*>(patch + 128 * i)[lane] = i < 2 ? m.up[lane] : m.down[lane];
  }
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 3; ++i)
    if (lane == i && w[i] != nullptr && (reinterpret_cast<uintptr_t>(w[i]) & 15u) == 0) tmap_replace_addr(patch + 128 * i, w[i]);
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    tmap_publish(m.maps + (static_cast<size_t>(e) * 3 + i) * 128, patch + 128 * i);
    if (lane == i) reinterpret_cast<const unsigned char**>(m.maps + (m.n_expert + 1LL) * 384)[i * (m.n_expert + 1LL) + e] = w[i];
  }
}

}  // namespace sgr
