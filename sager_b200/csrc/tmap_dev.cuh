// tmap_dev.cuh - TMA descriptors that are patched on the device, shared by the row-streaming expert kernels
// (expert_rows.cuh, grouped_gemm_rows.cu): expert addresses live in a pointer table on the device, so a descriptor is
// encoded on the host for a placeholder address and gets its base there.
#pragma once

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
// box (144 bytes x 128 rows) at byte column x, row y; dst 128-byte aligned, x a multiple of 16
__device__ __forceinline__ void tma_load_box(void* dst, const void* gmem_map, int x, int y, uint64_t* bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
               ::"r"(smem_u32(dst)), "l"(gmem_map), "r"(x), "r"(y), "r"(smem_u32(bar)) : "memory");
}

}  // namespace sgr
