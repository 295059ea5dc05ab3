"""CPU checks of the C boundary: the library builds for sm_100a, loads without a
GPU and exports every symbol the header declares; the shim header compiles."""
import ctypes as C
import os
import subprocess

from sager_b200 import build as sbuild
from sager_b200 import capi

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_library_builds_and_exports_header_symbols():
    path = sbuild.build()
    assert os.path.exists(path)
    lib = capi.Lib(path)            # raises if a declared symbol is missing
    assert len(lib.protos) >= 39
    assert lib.raw("sgr_abi_version")() == 4
    out = subprocess.run(["nm", "-D", "--defined-only", path], capture_output=True, text=True).stdout
    exported = {ln.split()[-1] for ln in out.splitlines() if " T " in ln}
    assert set(lib.protos) <= exported


def test_argument_validation_needs_no_gpu():
    lib = capi.lib()
    # null pointers and bad sizes are refused before any CUDA call
    assert lib.raw("sgr_gemv_q4_k_q8")(None, None, None, 8, 2048, None) == 1
    assert lib.raw("sgr_gemv_q4_k_q8")(16, 16, 16, 8, 2000, None) == 1      # k % 256 != 0
    assert lib.raw("sgr_gemv_q4_k_q8")(16, 18, 16, 8, 2048, None) == 2      # x_q8 not 4-byte aligned
    assert lib.raw("sgr_quantize_q8_k")(16, 16, 100, None) == 1
    assert lib.raw("sgr_router_topk_batched")(16, 16, 16, 256, 8, 8, 1, 1.0, None) == 1  # stride < K+1
    assert lib.raw("sgr_gemv_q4_k_q8")(16, 16, 16, 0, 2048, None) == 0      # empty: nothing to do
    # the tensor-core family refuses what the reference refuses, before any CUDA call
    assert lib.raw("sgr_tc_gemm_f16_raw")(16, 16, 16, 8, 100, 4, None) == 3          # k % 64 != 0
    assert lib.raw("sgr_tc_gemm_f16_raw")(18, 16, 16, 8, 64, 4, None) == 2           # operand not 16-byte aligned
    assert lib.raw("sgr_tc_gemm_q4_k_f16")(16, 16, 16, 16, 8, 768, 4, None) == 3     # k not a power of two
    assert lib.raw("sgr_tc_gemm_q4_k_f16")(16, 16, 17, 16, 8, 512, 4, None) == 2     # output not 2-byte aligned
    assert lib.raw("sgr_tc_scratch_elems")(512, 2048) == 512 * 2048


def test_static_scratch_takes_and_refuses_the_shapes_of_its_rule():
    lib = capi.lib()
    size, limit = lib.raw("sgr_moe_layer_workspace_bytes"), lib.raw("sgr_moe_layer_static_limit")()

    def call(n_max, hidden, n_ff, E, k):
        a = capi.MoeLayerArgs()
        a.n, a.n_max, a.hidden, a.n_ff, a.n_expert, a.n_used = 1, n_max, hidden, n_ff, E, k        # (no buffers: refused further on)
        return lib.raw("sgr_moe_layer_decode_static")(C.byref(a), None)

    for n_max in (1, 3, 4, 15, 16, 17, 24):
        for shape in ((2048, 512, 256, 8), (512, 256, 16, 4), (1024, 256, 1024, 2)):
            logits = (128 * min(n_max, 4) * shape[2] + 255) // 256 * 256
            assert (call(n_max, *shape) == 6) == (size(n_max, *shape) - logits > limit), (n_max, shape)
    assert call(16, 2048, 512, 256, 8) != 6 and call(17, 2048, 512, 256, 8) == 6
    assert call(1, 256, 256, 1025, 2) == 3                   # more experts than the layer takes


def test_head_ring_slots_belong_to_one_group_of_warps():
    """A wait by parity tells a phase from the one before only if that one was waited for: the ring's stages are a multiple of the
    groups that take them in turn, for every row length."""
    lib, plan, depths = capi.lib(), (C.c_int * 3)(), set()
    for k in range(256, 1 << 17, 256):
        assert lib.raw("sgr_gemv_q6_k_plan")(plan, k) == 0
        rows, stages, groups = plan
        assert stages % groups == 0
        if stages >= 2:
            depths.add((stages, groups))
            assert rows > 0 and stages * ((rows * (k // 256) * 210 + 127) // 128 * 128) + 128 + k // 256 * 324 <= 227 * 1024
    assert depths == {(2, 1), (3, 1), (4, 2)}
    assert lib.raw("sgr_gemv_q6_k_plan")(plan, 100) == 1


def test_projection_plans_are_shapes_that_the_tensor_cores_take():
    """M = 128 with N a multiple of 16 for one CTA, M = 256 with N a multiple of 32 for a pair; every token in one tile; whole pairs."""
    lib, plan, seen = capi.lib(), (C.c_int * 7)(), set()
    for sms in (148, 132, 7):
        for rows in (1, 128, 129, 1000, 2048, 3201, 4096, 8192, 100000):
            for k in (256, 512, 2048, 8192):
                for tok in (*range(1, 100, 9), 255, 256, 257, 300, 512, 777, 1154, 1457, 2047, 2048, 2049, 5000, 70001):
                    assert lib.raw("sgr_tc_gemm_q4_k_plan")(plan, sms, rows, k, tok) == 0
                    cg, bn, tiles, units, workers, spare, ahead = plan
                    row_tiles = (rows + 127) // 128
                    assert cg in (1, 2) and bn % (16 * cg) == 0 and 16 * cg <= bn <= 256
                    assert (tiles - 1) * bn < tok <= tiles * bn and units == (row_tiles + cg - 1) // cg * tiles
                    assert workers % cg == 0 and cg <= workers <= min(sms // cg * cg, units * cg)
                    assert workers + spare * row_tiles <= sms and not (ahead and spare)
                    seen.add(cg)
    assert seen == {1, 2}


def test_prefill_chunk_refuses_unaligned_buffers():
    """What the launchers of the sequence refuse, the one call refuses, and before anything is launched."""
    lib = capi.lib()

    def call(**moved):
        a = capi.MoePrefillArgs()
        a.n, a.n_max, a.hidden, a.n_ff, a.n_expert, a.n_used = 4, 4, 512, 256, 8, 2
        for name, kind in capi.MoePrefillArgs._fields_:
            if kind is C.c_void_p:
                setattr(a, name, 4096)
        a.shared_gate_w = a.sgate = None
        for name, by in moved.items():
            setattr(a, name, 4096 + by if by is not None else None)
        return lib.raw("sgr_moe_layer_prefill")(C.byref(a), None)

    for name, by in (("xn", 1), ("xq", 2), ("xqg", 8), ("hq", 4), ("g", 1), ("sh_g", 1), ("sh_q", 2)):
        assert call(**{name: by}) == 2, name
    assert call(xn=None) == 1
    # the expert stage is not repeated on operand rows that the combine has overwritten
    a = capi.MoePrefillArgs()
    a.n, a.n_max, a.hidden, a.n_ff, a.n_expert, a.n_used = 4, 4, 512, 256, 8, 2
    for name, kind in capi.MoePrefillArgs._fields_:
        if kind is C.c_void_p:
            setattr(a, name, 4096)
    a.x_f16 = 4096 + 2
    assert lib.raw("sgr_moe_prefill_expert_stage")(C.byref(a), None) == 3


def test_shim_header_compiles_against_c_abi():
    shim = os.path.join(ROOT, "include", "sager_b200_shim.hpp")
    if not os.path.exists(shim):
        import pytest
        pytest.skip("shim header not written yet")
    src = '#include "sager_b200_shim.hpp"\nint main() { return 0; }\n'
    res = subprocess.run(["g++", "-std=c++17", "-fsyntax-only", "-I", os.path.join(ROOT, "include"),
                          "-x", "c++", "-"], input=src, capture_output=True, text=True)
    assert res.returncode == 0, res.stderr


def test_shim_defines_exactly_the_reference_launchers(tmp_path):
    """Link check against the reference's own header: a translation unit that only
    sees include/sager/kernels/cuda_ops.hpp takes the address of every launcher the
    shim claims to provide; it links only if the shim defines those exact
    signatures. Needs the reference tree and the CUDA headers."""
    import pytest
    from oracle.oracle import reference_root
    import shutil
    ref_inc = os.path.join(reference_root(), "include")
    nvcc = shutil.which("nvcc")
    cuda_home = os.environ.get("CUDA_HOME") or (os.path.dirname(os.path.dirname(os.path.realpath(nvcc))) if nvcc else "")
    cuda_inc = os.path.join(cuda_home, "include")
    if not (os.path.isdir(ref_inc) and os.path.isdir(cuda_inc)):
        pytest.skip("reference tree or CUDA headers not present")
    import re
    shim = open(os.path.join(ROOT, "include", "sager_b200_shim.hpp")).read()
    body = shim.split("int b200_last_error();", 1)[1].split("#ifdef SAGER_B200_SHIM_IMPLEMENTATION", 1)[0]
    # every launcher the shim declares, whatever it returns (void, bool, void*, size_t)
    names = re.findall(r"^(?:void|bool|void\*|size_t) (\w+)\(", body, flags=re.M)
    assert len(names) >= 41 and {"tc_gemm_q4_k_f16", "tc_handle", "tc_scratch_elems", "tc_gemm_f16_raw",
                                 "tc_gemm_f16_f32out_raw"} <= set(names)
    user = tmp_path / "user.cpp"
    user.write_text('#include "sager/kernels/cuda_ops.hpp"\n'
                    "const void* volatile sink[] = {\n" +
                    "".join(f"  reinterpret_cast<const void*>(&sager::cuda::{n}),\n" for n in names) +
                    "};\nint main() { return sink[0] != nullptr ? 0 : 1; }\n")
    impl = tmp_path / "impl.cpp"
    impl.write_text('#include "sager/kernels/cuda_ops.hpp"\n#define SAGER_B200_SHIM_IMPLEMENTATION\n'
                    '#include "sager_b200_shim.hpp"\n')
    lib = sbuild.build()
    exe = tmp_path / "a.out"
    cmd = ["g++", "-std=c++20", "-I", ref_inc, "-I", cuda_inc, "-I", os.path.join(ROOT, "include"),
           str(user), str(impl), lib, f"-Wl,-rpath,{os.path.dirname(lib)}", "-o", str(exe)]
    res = subprocess.run(cmd, capture_output=True, text=True)
    assert res.returncode == 0, res.stderr[-3000:]
