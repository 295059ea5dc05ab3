/*
 * sager_b200_diag.h - entry points of libsager_b200.so that serve tests and
 * measurements only. None of them replaces a launcher of the reference
 * (include/sager/kernels/cuda_ops.hpp) and a caller of the library never needs them.
 */
#ifndef SAGER_B200_DIAG_H_
#define SAGER_B200_DIAG_H_

#ifdef __cplusplus
extern "C" {
#endif

/* Operand tile layout of the fp16 tensor-core GEMM kernel behind the sgr_tc_* entries: 0 = 128-byte
 * swizzled tiles (default), 1 = unswizzled core matrices. Same results either way; process-global. */
int sgr_tc_set_operand_layout(int layout);

/* Byte offset of a region inside the workspace of sgr_moe_layer_decode (same geometry arguments as
 * sgr_moe_layer_workspace_bytes), so that a test can read the intermediate rows a finished call
 * left there. which: 0 = fp32 h rows [n_max*K + n_max][n_ff] (routed rows in grouped order, then
 * the shared expert's), 1 = fp32 y rows [..][hidden], 2 = gslot [n_max*K] (route -> grouped row,
 * -1 = not computed), 3 = grows, 4 = plan records, 5 = meta, 6 = counters (uint32; words 12 and 13 are the 64-bit arrival
 * counter of the one-launch layers, CTAs that gave up counted in its top byte), 7 = the logits that these exchange
 * [16 copies][n][n_expert], the launch's number in a word's upper half. -1 for a refused geometry. */
long long sgr_moe_layer_workspace_offset(int n_max, int hidden, int n_ff, int n_expert, int n_used,
                                         int which);

/* How sgr_gemv_q6_k_q8 streams a matrix of k columns (host arithmetic, no device): plan[0] = rows to a stage, plan[1] =
 * stages of the ring (fewer than 2: always the plain kernel), plan[2] = groups of warps that take the stages in turn. */
int sgr_gemv_q6_k_plan(int* plan, int k);

/* How sgr_tc_gemm_q4_k_f16 splits a product over `sms` SMs (host arithmetic, no device): plan[0] = CTAs that share a unit (1, or 2 of a
 * cluster), [1] = token rows of a unit, [2] = token tiles, [3] = units, [4] = CTAs that work on them, [5] = CTAs per row tile that only
 * write the scratch, [6] = the scratch is written by the dequantisation kernel ahead. */
int sgr_tc_gemm_q4_k_plan(int* plan, int sms, int n_rows, int k, int n_tokens);

/* Residency handle in host-only mode: mark an arena slot as "its copy is still in flight" (what an
 * unfinished event says on the device), so that the rule "an in-flight slot is never evicted" can be
 * exercised without a GPU. */
int sgr_residency_test_set_inflight(void* handle, int slot, int on);

/* The expert stage (gate, up, SwiGLU, requantise, down) of a finished sgr_moe_layer_prefill call once more, on
 * the plan and the operand rows that call left in its buffers, with the weights that args names now (their descriptors are
 * made anew: one short launch). For timing. SGR_EUNSUPPORTED where the combine
 * has used the slab that held those rows (x_f16, y_grouped or sh_y off a 16-byte boundary). */
struct sgr_moe_prefill;
int sgr_moe_prefill_expert_stage(const struct sgr_moe_prefill* args, void* stream);

#ifdef __cplusplus
}
#endif
#endif /* SAGER_B200_DIAG_H_ */
