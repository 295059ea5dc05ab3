"""The prefill chunk's expert stage for few token rows per expert (row-streaming GEMM) against the launchers it joins: grouped
GEMM on gathered rows, SwiGLU, quantiser. Integer sums and fp32 steps are the same on both paths: equal to the bit."""
import ctypes as C

import numpy as np
import pytest
import torch

from sager_b200 import lib, ops, synth
from sager_b200.ops import stream_ptr
from sager_b200.layer import PrefillLayer
from tests.util import DEV, dev

pytestmark = pytest.mark.gpu


def quantize_dev(x16):
    n, k = x16.shape
    out = torch.zeros(n, k // 256 * 276, dtype=torch.uint8, device=DEV)
    ops.quantize_q8_k(x16, out, n * k)
    return out


def launchers(tabs, off, grows, x16, R, H, F, E):
    """y of the routed rows through the separate launchers; tabs: three [E] pointer tables."""
    xqg = torch.zeros(R, H // 256 * 276, dtype=torch.uint8, device=DEV)
    ops.gather_rows_q8(xqg, quantize_dev(x16), grows, R, H // 256)
    g, u, y = (torch.zeros(R, d, dtype=torch.float16, device=DEV) for d in (F, F, H))
    ops.moe_grouped_gemm_i8(tabs[0], off, xqg, g, F, H, E)
    ops.moe_grouped_gemm_i8(tabs[1], off, xqg, u, F, H, E)
    ops.silu_mul_f16(g, g, u, R, F)
    ops.moe_grouped_gemm_i8(tabs[2], off, quantize_dev(g), y, H, F, E)
    return y


def chosen_logits(counts, n, seed):
    """Router logits (top-1) that give expert e counts[e] of the rows, in shuffled order."""
    e = np.repeat(np.arange(len(counts)), counts)
    assert len(e) == n
    np.random.default_rng(seed).shuffle(e)
    logits = np.zeros((n, len(counts)), np.float32)
    logits[np.arange(n), e] = 5.0
    return dev(logits)


# rows per expert at the edges of the token groups (4, 8, 16, 24, 32), of the passes, none at all
EDGES = [1, 8, 9, 16, 17, 24, 25, 32, 33, 40, 0, 65, 2, 3, 4, 31, 5]


@pytest.mark.parametrize("H,F", [(512, 256), (256, 512), (2048, 512), (512, 768)])
@pytest.mark.parametrize("shift", [0, 2, 4])
def test_rows_per_expert(H, F, shift):
    """shift: bytes by which the experts' blobs lie off a 16-byte boundary."""
    E, K, n = len(EDGES), 1, sum(EDGES)
    n_max = n * (1 + 2 * F // H)                # room for the rows and the descriptors
    w = synth.MoeWeights(H, F, E, DEV, seed=81, std=0.05)
    big = torch.empty(w.blob.numel() + 16, dtype=torch.uint8, device=DEV)
    big[shift:shift + w.blob.numel()] = w.blob.reshape(-1)
    w.blob = big[shift:shift + w.blob.numel()].view(w.n_slots, -1)
    x16 = synth.normal_fp16((n, H), 82, DEV)
    L = PrefillLayer(n_max, H, F, E, K, DEV)
    x = x16.clone()
    absent = (3,)
    t = w.table(absent)
    L.run(n, x16, x, w, t, logits=chosen_logits(EDGES, n, 5))
    off = L.off.cpu().numpy()
    assert np.array_equal(np.diff(off), EDGES)
    y = launchers([t[m].contiguous() for m in range(3)], L.off, L.grows, x16, n, H, F, E)
    assert torch.equal(L.yg[:n].view(torch.int16), y.view(torch.int16))
    assert (L.yg[off[3]:off[4]] == 0).all()
    one = [ops.ptr_table([w.matrix(E, m)], DEV) for m in range(3)]
    sy = launchers(one, dev(np.int32([0, n])), dev(np.arange(n, dtype=np.int32)), x16, n, H, F, 1)
    assert torch.equal(L.sh_y[:n].view(torch.int16), sy.view(torch.int16))
    assert lib().raw("sgr_status")(0) == 0
    # the expert stage once more on what the call left behind (the hand-out counters start anew)
    want = L.yg.clone()
    L.yg.zero_()
    a = L.args(n, x16, x, w, t, logits=None)
    lib().call("sgr_moe_prefill_expert_stage", C.byref(a), stream_ptr())
    assert torch.equal(L.yg[:n].view(torch.int16), want[:n].view(torch.int16))


@pytest.mark.parametrize("E,K,n", [(300, 2, 77), (1, 1, 20), (257, 8, 65)])
def test_many_units(E, K, n):
    """More experts than a CTA's first round, one expert, no shared expert."""
    H, F = 512, 256
    w = synth.MoeWeights(H, F, E, DEV, seed=83, std=0.05, distinct=9)
    x16 = synth.normal_fp16((n, H), 84, DEV)
    L = PrefillLayer(4 * n, H, F, E, K, DEV)
    t = w.table()
    for shared in (True, False):
        x = x16.clone()
        L.run(n, x16, x, w, t, shared=shared)
        y = launchers([t[m].contiguous() for m in range(3)], L.off, L.grows, x16, n * K, H, F, E)
        assert torch.equal(L.yg[:n * K].view(torch.int16), y.view(torch.int16)), shared
    assert lib().raw("sgr_status")(0) == 0


def test_saturated_codes():
    """Codes, scales and nibbles near their largest: block sums beyond 2^24 stay exact integers here (one rounding to fp32 each),
    so the result is within the fp16 step of the exact one."""
    H, F, E, K, n = 512, 256, 4, 1, 40
    rng = np.random.default_rng(3)
    x = torch.from_numpy(rng.choice([-1.0, 1.0], (n, 1)) * rng.uniform(0.9, 1.0, (n, H))).half().to(DEV)
    w = synth.MoeWeights(H, F, E, DEV, seed=85, std=0.05)
    blob = w.blob.view(w.n_slots, -1, 144)
    blob[:, :, 0:4] = dev(np.frombuffer(np.float16([2.0 ** -14, 0.0]).tobytes(), np.uint8).copy())
    blob[:, :, 4:] = 0xFF
    L = PrefillLayer(4 * n, H, F, E, K, DEV)
    L.run(n, x, x.clone(), w, w.table(), logits=chosen_logits([10] * 4, n, 6))
    xq = quantize_dev(x).cpu().numpy().reshape(n, H // 256, 276)
    d = xq[..., 0:4].copy().view(np.float32)[..., 0].astype(np.float64)
    codes = xq[..., 4:260].view(np.int8).astype(np.int64)
    g = (d * codes.sum(2) * 63 * 15 * 2.0 ** -14).sum(1)         # gate and up alike, every row
    h = (g / (1 + np.exp(-g)) * g)
    got = L.g[:n].double().cpu().numpy()[np.argsort(L.grows[:n].cpu().numpy())]
    # g to fp16 (2^-11), h = silu(g) g: its relative error is at most (2 + |g|) times that of g, and rounded itself
    assert (np.abs(got - h[:, None]) <= (np.abs(h) * (3 + np.abs(g)) * 2.0 ** -11 + 1e-6)[:, None]).all()


@pytest.mark.parametrize("E,hot", [(70, {66: 301}), (70, {0: 130, 31: 97, 32: 65, 69: 33}), (300, {5: 1, 299: 260}), (33, {32: 400})])
def test_hot_experts(E, hot):
    """Passes of one expert are handed out one by one: hot experts at the edges of the 32-expert windows in which an item is
    looked up, windows without a row in between."""
    H, F = 512, 256
    counts = [hot.get(e, 0) for e in range(E)]
    n = sum(counts)
    w = synth.MoeWeights(H, F, E, DEV, seed=87, std=0.05, distinct=7)
    x16 = synth.normal_fp16((n, H), 88, DEV)
    L = PrefillLayer(4 * n, H, F, E, 1, DEV)
    t = w.table()
    L.run(n, x16, x16.clone(), w, t, logits=chosen_logits(counts, n, 9))
    assert np.array_equal(np.diff(L.off.cpu().numpy()), counts)
    y = launchers([t[m].contiguous() for m in range(3)], L.off, L.grows, x16, n, H, F, E)
    assert torch.equal(L.yg[:n].view(torch.int16), y.view(torch.int16))
    assert lib().raw("sgr_status")(0) == 0


def test_a_hot_expert_is_shared_out():
    """The same routes with one expert in all of them: as many dots and fewer weights than spread evenly, and so no slower as
    long as every SM gets its share (one CTA for an expert's passes took three times as long)."""
    H, F, E, K, n = 2048, 512, 256, 2, 1024
    w = synth.MoeWeights(H, F, E, DEV, seed=89, std=0.05, distinct=7)
    x16 = synth.normal_fp16((n, H), 90, DEV)
    L = PrefillLayer(2 * n, H, F, E, K, DEV)
    t = w.table()
    spread = torch.randn(n, E, generator=torch.Generator(device=DEV).manual_seed(1), device=DEV)
    hot = spread.clone()
    hot[:, 100:102] += 20.0
    us = []
    for logits in (spread, hot):
        x = torch.zeros_like(x16)
        best = []
        for rep in range(8):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            L.run(n, x16, x, w, t, logits=logits)
            b.record()
            b.synchronize()
            best.append(a.elapsed_time(b) * 1e3)
        us.append(min(best))
    assert L.off.cpu().numpy()[102] == 2 * n and L.off.cpu().numpy()[100] == 0
    assert us[1] < 1.2 * us[0], us


@pytest.mark.parametrize("n", [70, 200])
def test_the_table_is_read_once(n):
    """The expert cache may rewrite the table at any time: what counts for a chunk is the table as it was when the descriptors
    were made, for absent and present experts and for their alignment alike. A graph of the call with a copy of another
    table between its first kernel (which makes them) and the rest; row-streaming and tcgen05 form."""
    from cuda.bindings import runtime as rt
    H, F, E, K = 512, 256, 12, 4
    w, other = (synth.MoeWeights(H, F, E, DEV, seed=s, std=0.05) for s in (95, 96))
    before = w.table((2, 9)).clone()
    odd = torch.empty(other.blob.numel() + 16, dtype=torch.uint8, device=DEV)
    shifted = other.table() - other.blob.data_ptr() + odd.data_ptr() + 2
    after = other.table((4, 9)).clone()
    after[:, 6:8] = shifted[:, 6:8]
    x16 = synth.normal_fp16((n, H), 97, DEV)
    L = PrefillLayer(n, H, F, E, K, DEV)
    x = x16.clone()
    L.run(n, x16, x, w, before)
    want = x.clone()
    want_y = L.yg.clone()

    def ok(r):
        assert r[0] == rt.cudaError_t.cudaSuccess, r[0]
        return r[1] if len(r) > 1 else None

    table = before.clone()
    a = L.args(n, x16, x, w, table)
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    ok(rt.cudaStreamBeginCapture(s.cuda_stream, rt.cudaStreamCaptureMode.cudaStreamCaptureModeRelaxed))
    lib().call("sgr_moe_layer_prefill", C.byref(a), C.c_void_p(s.cuda_stream))
    graph = ok(rt.cudaStreamEndCapture(s.cuda_stream))
    count = rt.cudaGraphGetNodes(graph, 0)[2]
    nodes = rt.cudaGraphGetNodes(graph, count)[1][:count]
    firsts = rt.cudaGraphGetRootNodes(graph, 1)[1]
    rest = [v for v in nodes if int(v) != int(firsts[0])]
    copy = ok(rt.cudaGraphAddMemcpyNode1D(graph, firsts, 1, table.data_ptr(), after.data_ptr(), table.numel() * 8,
                                          rt.cudaMemcpyKind.cudaMemcpyDeviceToDevice))
    for v in rest:
        ok(rt.cudaGraphAddDependencies(graph, [copy], [v], 1))
    run = ok(rt.cudaGraphInstantiate(graph, 0))
    x.copy_(x16)
    L.yg.zero_()
    torch.cuda.synchronize()
    ok(rt.cudaGraphLaunch(run, s.cuda_stream))
    torch.cuda.synchronize()
    assert torch.equal(table, after)
    assert torch.equal(L.yg.view(torch.int16), want_y.view(torch.int16))
    assert torch.equal(x.view(torch.int16), want.view(torch.int16))
    assert lib().raw("sgr_status")(0) == 0
    ok(rt.cudaGraphExecDestroy(run))
    ok(rt.cudaGraphDestroy(graph))


# combine slabs with room for the operand rows but not for descriptors: few rows for many experts (row-streaming form), and the
# tcgen05 form's operands at exactly the slab's size (7 x 512 bytes a row and route against 64 blocks of 560)
@pytest.mark.parametrize("H,F,E,K,n", [(512, 256, 256, 8, 16), (512, 256, 256, 8, 5), (1024, 512, 256, 8, 9), (3584, 2560, 4, 4, 40)])
@pytest.mark.parametrize("shift", [0, 2, 8])
def test_no_room_for_descriptors(H, F, E, K, n, shift):
    w = synth.MoeWeights(H, F, E, DEV, seed=91, std=0.05, distinct=5)
    big = torch.empty(w.blob.numel() + 16, dtype=torch.uint8, device=DEV)
    big[shift:shift + w.blob.numel()] = w.blob.reshape(-1)
    w.blob = big[shift:shift + w.blob.numel()].view(w.n_slots, -1)
    x16 = synth.normal_fp16((n, H), 92, DEV)
    L = PrefillLayer(n, H, F, E, K, DEV)
    L.xq.fill_(0xA5)
    absent = (1,)
    t = w.table(absent)
    x = x16.clone()
    L.run(n, x16, x, w, t)
    assert (L.xq == 0xA5).all()                  # (the form that reads plain Q8_K rows would have written them there)
    y = launchers([t[m].contiguous() for m in range(3)], L.off, L.grows, x16, n * K, H, F, E)
    assert torch.equal(L.yg[:n * K].view(torch.int16), y.view(torch.int16))
    one = [ops.ptr_table([w.matrix(E, m)], DEV) for m in range(3)]
    sy = launchers(one, dev(np.int32([0, n])), dev(np.arange(n, dtype=np.int32)), x16, n, H, F, 1)
    assert torch.equal(L.sh_y[:n].view(torch.int16), sy.view(torch.int16))
    assert lib().raw("sgr_status")(0) == 0


@pytest.mark.parametrize("n", [70, 200])
def test_expert_stage_reads_the_table_it_is_given(n):
    """The stage once more with another layer's weights on the same buffers: row-streaming and tcgen05 form."""
    H, F, E, K = 512, 256, 12, 4
    w, other = (synth.MoeWeights(H, F, E, DEV, seed=s, std=0.05) for s in (97, 98))
    x16 = synth.normal_fp16((n, H), 99, DEV)
    L = PrefillLayer(n, H, F, E, K, DEV)
    for absent in ((), (5,)):
        L.run(n, x16, x16.clone(), w, w.table())
        t = other.table(absent)
        L.run(n, x16, x16.clone(), other, t, experts_only=True)
        y = launchers([t[m].contiguous() for m in range(3)], L.off, L.grows, x16, n * K, H, F, E)
        assert torch.equal(L.yg[:n * K].view(torch.int16), y.view(torch.int16))
