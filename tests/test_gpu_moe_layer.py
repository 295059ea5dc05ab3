"""GPU parity of the fused MoE layer (sgr_moe_layer_decode) against the oracle's
whole-layer restatement: router as the device computes it, every selected and
the shared expert through the CPU expert FFN, weighted sum in slot order.
Bars: selected experts exact in value and order, routing weights within 1e-6,
fp32 layer output within 1e-3 max relative error (the stated bound; the measured
figure is asserted an order of magnitude tighter)."""
import numpy as np
import pytest
import torch

from sager_b200 import lib, ops, synth
from sager_b200.layer import MoeLayerRunner, MoeStack
from tests.util import DEV, LAYER_TOL, dev, f16_close, rel

pytestmark = pytest.mark.gpu


def oracle_layer(oracle, w, x16_np, resid_np, k, absent=(), bias=None, n_threads=8, use_shared=True,
                 blob_np=None):
    """Run the oracle on the experts the routing needs only (the rest stay None). blob_np: a host
    copy of w.blob to slice the matrices from (saves one device copy per matrix)."""
    E = w.n_expert
    if blob_np is not None:
        o3 = [0, w.gu_bytes, 2 * w.gu_bytes, w.expert_bytes]
        mat = lambda e, m: blob_np[w.slot(e), o3[m]:o3[m + 1]]
    else:
        mat = lambda e, m: w.matrix(e, m).cpu().numpy()
    logits = np.stack([oracle.router_logits(w.router.cpu().numpy(), x16_np[t]) for t in range(x16_np.shape[0])])
    if bias is not None:
        logits = logits + bias[None, :]
    need = set()
    for t in range(x16_np.shape[0]):
        need |= set(oracle.router_topk(logits[t], k)[0][:k].tolist())
    experts = [None] * E
    for e in need:
        if e in absent:
            continue
        experts[e] = tuple(mat(e, m) for m in range(3))
    shared = tuple(mat(E, m) for m in range(3)) if use_shared else None
    router = w.router.cpu().numpy()
    if bias is not None:
        # the oracle computes logits itself: fold the bias in by routing on biased logits
        res = _oracle_with_logits(oracle, x16_np, logits, experts, shared, resid_np, k, w.n_ff, n_threads)
    else:
        res = oracle.moe_layer(x16_np, router, experts, shared, resid_np, k, w.n_ff, shared_w=1.0,
                               n_threads=n_threads)
    return res


def _oracle_with_logits(oracle, x16_np, logits, experts, shared, resid_np, k, n_ff, n_threads):
    n, H = x16_np.shape
    out = np.zeros((n, H), dtype=np.float32)
    idx = np.zeros((n, k + 1), dtype=np.int32)
    wts = np.zeros((n, k + 1), dtype=np.float32)
    jobs_w, jobs_x, slots = [], [], []
    for t in range(n):
        i, wv = oracle.router_topk(logits[t], k, shared_w=1.0)
        idx[t], wts[t] = i, wv
        idx[t, k] = -1
        for kk in range(k + 1):
            ex = experts[i[kk]] if kk < k else shared
            if ex is None:
                continue
            jobs_w += list(ex)
            jobs_x.append(x16_np[t].astype(np.float32))
            slots.append((t, kk))
    ys = oracle.expert_ffn_batch(jobs_w, np.stack(jobs_x), H, n_ff, n_threads)
    acc = resid_np.astype(np.float32).copy()
    per = {s: y for s, y in zip(slots, ys)}
    for t in range(n):
        for kk in range(k + 1):
            if (t, kk) in per:
                acc[t] = acc[t] + wts[t, kk] * per[(t, kk)]
    return dict(out=acc, idx=idx, w=wts, logits=logits)


def run_layer(w, n, k, x16_dev, n_max=None, absent=(), bias=None, use_shared=True, kernel=None):
    runner = MoeLayerRunner(n_max or n, w.hidden, w.n_ff, w.n_expert, k, DEV)
    x = x16_dev.clone()
    out32 = torch.zeros(n, w.hidden, dtype=torch.float32, device=DEV)
    a = runner.args(n, x16_dev, w.router, w.table(absent), w.shared_ptrs() if use_shared else None,
                    x_f16=x, out_f32=out32, bias=None if bias is None else dev(bias))
    runner.run(a, kernel=kernel)
    torch.cuda.synchronize()
    assert lib().raw("sgr_status")(0) == 0, "a bounded device-side wait gave up"
    return runner, x, out32


def check(oracle, w, n, k, seed, absent=(), bias=None, use_shared=True, n_max=None, tol=1e-4, kernel=None):
    x16 = synth.normal_fp16((n, w.hidden), seed, DEV)
    x_np = x16.cpu().numpy()
    runner, x_out, out32 = run_layer(w, n, k, x16, n_max=n_max, absent=absent, bias=bias,
                                     use_shared=use_shared, kernel=kernel)
    want = oracle_layer(oracle, w, x_np, x_np.astype(np.float32), k, absent=absent, bias=bias,
                        use_shared=use_shared)
    idx = runner.route_idx.cpu().numpy()[:n]
    wt = runner.route_w.cpu().numpy()[:n]
    assert np.array_equal(idx[:, :k], want["idx"][:, :k])
    assert np.abs(wt[:, :k] - want["w"][:, :k]).max() <= 1e-6
    assert np.all(wt[:, k] == 1.0)
    err = rel(out32.cpu().numpy(), want["out"])
    assert err < LAYER_TOL and err < tol, err
    assert f16_close(x_out.cpu().numpy(), want["out"], tol=tol)
    return runner, want, err


@pytest.fixture(scope="module")
def small_w():
    return synth.MoeWeights(512, 256, 16, DEV, seed=11, std=0.05)


@pytest.fixture(scope="module")
def full_w():
    # the benchmark geometry: hidden 2048, expert FFN 512, 256 experts + shared
    return synth.MoeWeights(2048, 512, 256, DEV, seed=20260718)


@pytest.mark.parametrize("kernel", ["items", "rows", None])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 17, 64])
def test_small_layer_all_row_counts(oracle, small_w, n, kernel):
    check(oracle, small_w, n, 4, seed=100 + n, n_max=64, kernel=kernel)


@pytest.mark.parametrize("kernel", ["items", "rows"])
def test_small_layer_without_shared_expert_and_with_bias(oracle, small_w, kernel):
    check(oracle, small_w, 3, 4, seed=7, use_shared=False, kernel=kernel)
    bias = synth.zipf_bias(16, seed=3, alpha=0.5)
    check(oracle, small_w, 9, 4, seed=8, bias=bias, kernel=kernel)
    # hot experts: full tiles of 16 rows and ragged ones. (The seed matters: h is requantised
    # to Q8_K between the projections, and when an h value sits on a rounding boundary the two
    # summation orders can pick different codes - one token row then moves by ~1e-3 of the
    # largest output on this 512-wide layer. This seed has no such value.)
    check(oracle, small_w, 40, 4, seed=12, bias=bias * 4, kernel=kernel)


@pytest.mark.parametrize("kernel", ["items", "rows"])
def test_absent_experts_contribute_zero_and_are_mailed(oracle, small_w, kernel):
    n, k = 6, 4
    x16 = synth.normal_fp16((n, 512), 55, DEV)
    r0, _, _ = run_layer(small_w, n, k, x16)
    used = sorted(set(r0.route_idx.cpu().numpy()[:n, :k].reshape(-1).tolist()))
    absent = (used[0], used[-1])
    runner, want, _ = check(oracle, small_w, n, k, seed=55, absent=absent, kernel=kernel)
    n_mail = int(runner.mail_n.item())
    mails = runner.mail.cpu().numpy()[:n_mail].tolist()
    assert sorted(set(mails)) == sorted(absent)


@pytest.mark.parametrize("kernel", ["items", "rows"])
@pytest.mark.parametrize("shift", [2, 4])
def test_weight_pointers_with_only_block_alignment(oracle, small_w, kernel, shift):
    """The pointer table only promises the alignment of the block struct (2 bytes): the
    same weights at addresses 2 and 4 bytes off a 16-byte boundary must give the same layer."""
    import copy
    w = copy.copy(small_w)
    big = torch.empty(small_w.blob.numel() + 16, dtype=torch.uint8, device=DEV)
    w.blob = big[shift:shift + small_w.blob.numel()].view(small_w.blob.shape)
    w.blob.copy_(small_w.blob)
    assert w.blob.data_ptr() % 16 == shift
    check(oracle, w, 21, 4, seed=77, kernel=kernel)


@pytest.mark.parametrize("kernel", ["items", "rows", None])
@pytest.mark.parametrize("n", [1, 2, 4, 64])
def test_benchmark_geometry(oracle, full_w, n, kernel):
    bias = synth.zipf_bias(256, seed=5, alpha=0.6) if n == 64 else None
    _, _, err = check(oracle, full_w, n, 8, seed=20260718 + n, bias=bias, n_max=64, kernel=kernel)
    print(f"n={n}: max relative error of the fp32 layer output = {err:.3e}")


def test_expert_ranges_partition_the_layer(full_w):
    """Expert parallelism on one device: two owner-side calls over disjoint expert
    ranges with the routing given, summed, reproduce the single call exactly up to
    fp32 addition order."""
    n, k = 16, 8
    w = full_w
    x16 = synth.normal_fp16((n, w.hidden), 77, DEV)
    runner, x_full, out_full = run_layer(w, n, k, x16, n_max=64)
    nb = w.hidden // 256
    xq = torch.zeros(n, nb * 276, dtype=torch.uint8, device=DEV)
    ops.quantize_q8_k(x16, xq, n * w.hidden)
    parts = []
    for lo, hi, sh in ((0, 128, (0, n)), (128, 256, None)):
        r = MoeLayerRunner(64, w.hidden, w.n_ff, w.n_expert, k, DEV, expert_lo=lo, expert_hi=hi)
        out = torch.zeros(n, w.hidden, dtype=torch.float32, device=DEV)
        a = r.args(n, None, None, w.table(), w.shared_ptrs() if sh else None, out_f32=out, xq_in=xq,
                   routing_given=True, no_residual=True, route_idx=runner.route_idx.clone(),
                   route_w=runner.route_w.clone())
        r.run(a)
        parts.append(out)
    torch.cuda.synchronize()
    total = x16.float() + parts[0] + parts[1]
    assert rel(total.cpu().numpy(), out_full.cpu().numpy()) < 1e-6


def test_stack_argument_blocks_belong_to_the_caller():
    """A block from layer_args may be changed without touching the stack's own steps, follows what the weights object says
    now, and asks no more of that object than its router, table and shared pointers."""
    class Weights:
        def __init__(self, w):
            self.hidden, self.n_ff, self.n_expert, self.router, self.w, self.shared = w.hidden, w.n_ff, w.n_expert, w.router, w, True

        def table(self):
            return self.w.table()

        def shared_ptrs(self):
            return self.w.shared_ptrs() if self.shared else None

    w = Weights(synth.MoeWeights(512, 256, 16, DEV, seed=230, std=0.05))
    x0 = synth.normal_fp16((2, 512), 231, DEV)
    st = MoeStack([w], 2, 4, DEV)

    def step():
        st.x.copy_(x0)
        st.step_eager(2)
        return st.x.clone()

    first = step()
    _, a = st.layer_args(0, 2)
    a.no_residual, a.x_f16 = 1, None
    assert torch.equal(step(), first)
    w.shared = False
    assert not torch.equal(step(), first)


def test_stack_graph_replay_is_deterministic(oracle):
    layers = [synth.MoeWeights(512, 256, 16, DEV, seed=200 + i, std=0.05) for i in range(3)]
    n, k = 4, 4
    x0 = synth.normal_fp16((n, 512), 9, DEV)
    st = MoeStack(layers, 8, k, DEV)
    st.x[:n] = x0
    st.step_eager(n)
    torch.cuda.synchronize()
    eager = st.x[:n].clone()
    idx_eager = st.idx.clone()
    st.x[:n] = x0
    st.capture(n)
    outs = []
    for _ in range(3):
        st.x[:n] = x0
        st.replay()
        torch.cuda.synchronize()
        outs.append(st.x[:n].clone())
    assert all(torch.equal(o, eager) for o in outs)
    assert torch.equal(st.idx, idx_eager)
    # and the chain matches the oracle layer by layer (fp16 residual stream between layers)
    x_np = x0.cpu().numpy()
    for li, w in enumerate(layers):
        want = oracle_layer(oracle, w, x_np, x_np.astype(np.float32), k)
        assert np.array_equal(st.idx[li].cpu().numpy()[:n, :k], want["idx"][:, :k])
        x_np = want["out"].astype(np.float16)
    assert f16_close(eager.cpu().numpy(), x_np.astype(np.float32), tol=2e-3)
    from sager_b200 import lib
    assert lib().raw("sgr_status")(0) == 0


@pytest.mark.parametrize("padded", [False, True])
@pytest.mark.parametrize("world,tokens", [(4, 16), (4, 64), (8, 64)])
def test_expert_parallel_record_path_on_one_device(full_w, padded, world, tokens):
    """The expert-parallel layer with its exchanges done by hand on one device: each
    emulated rank routes its home rows straight into dispatch records (strided Q8_K
    rows, ids, weights), every rank's owner call runs its expert range over all
    records, partial sums are added at home. Must reproduce the single call."""
    import ctypes as C
    from sager_b200 import lib
    from sager_b200.ep import record_layout
    from sager_b200.ops import stream_ptr
    w, k = full_w, 8
    n_home = tokens // world
    x16 = synth.normal_fp16((tokens, w.hidden), 91, DEV)
    _, x_full, out_full = run_layer(w, tokens, k, x16, n_max=64)
    rec, idx_off, w_off = record_layout(w.hidden, k, padded)      # padded: Q8 rows in 288-byte blocks, read in place
    records = torch.zeros(world, n_home, rec, dtype=torch.uint8, device=DEV)
    for r in range(world):                                    # home side of every rank
        home = MoeLayerRunner(n_home, w.hidden, w.n_ff, w.n_expert, k, DEV)
        a = home.args(n_home, x16[r * n_home:(r + 1) * n_home].contiguous(), w.router, w.table(), None,
                      x_f16=torch.zeros(n_home, w.hidden, dtype=torch.float16, device=DEV))
        base = records[r].data_ptr()
        a.xq_out, a.xq_stride = C.c_void_p(base), rec
        a.route_idx, a.route_w = C.c_void_p(base + idx_off), C.c_void_p(base + w_off)
        a.route_stride = rec // 4
        a.xq_padded = int(padded)
        lib().call("sgr_moe_layer_decode_stages", C.byref(a), 1 | 8, stream_ptr())
    torch.cuda.synchronize()
    total = x16.float().clone()
    per = w.n_expert // world
    for r in range(world):                                    # owner side of every rank
        owner = MoeLayerRunner(64, w.hidden, w.n_ff, w.n_expert, k, DEV, expert_lo=r * per,
                               expert_hi=(r + 1) * per)
        part = torch.zeros(tokens, w.hidden, dtype=torch.float32, device=DEV)
        b = owner.args(tokens, None, None, w.table(), w.shared_ptrs(), out_f32=part, xq_in=records,
                       routing_given=True, no_residual=True, shared_lo=r * n_home,
                       shared_hi=(r + 1) * n_home)
        b.xq_stride, b.route_stride = rec, rec // 4
        b.xq_padded = int(padded)
        b.route_idx = C.c_void_p(records.data_ptr() + idx_off)
        b.route_w = C.c_void_p(records.data_ptr() + w_off)
        lib().call("sgr_moe_layer_decode_stages", C.byref(b), 7, stream_ptr())
        torch.cuda.synchronize()
        total += part
    assert rel(total.cpu().numpy(), out_full.cpu().numpy()) < 1e-6
    # and the home-side reduction kernel
    xh = x16[:n_home].clone()
    parts = torch.randn(world, n_home, w.hidden, device=DEV)
    lib().call("sgr_ep_reduce_add_f16", C.c_void_p(xh.data_ptr()), C.c_void_p(parts.data_ptr()), world,
               n_home * w.hidden, n_home * w.hidden, stream_ptr())
    want = x16[:n_home].float()
    for p_ in range(world):
        want = want + parts[p_]
    assert torch.equal(xh, want.half())


def test_route_only_stage_repeats_on_one_workspace(full_w):
    """The home side of expert parallelism calls the route stage without the plan once per layer on
    one workspace: the second call must route its own rows (its per-tile counters start at zero
    again), not leave the first call's routing in place."""
    import ctypes as C
    from sager_b200.ops import stream_ptr
    w, k, n = full_w, 8, 32
    runner = MoeLayerRunner(n, w.hidden, w.n_ff, w.n_expert, k, DEV)
    picks = []
    for seed in (301, 302):
        x16 = synth.normal_fp16((n, w.hidden), seed, DEV)
        a = runner.args(n, x16, w.router, w.table(), None,
                        x_f16=torch.zeros(n, w.hidden, dtype=torch.float16, device=DEV))
        lib().call("sgr_moe_layer_decode_stages", C.byref(a), 1 | 8, stream_ptr())
        torch.cuda.synchronize()
        idx = runner.route_idx.cpu().numpy()[:n, :k].copy()
        want = (x16.float() @ w.router.t()).topk(k, dim=1).indices.cpu().numpy()
        assert np.array_equal(np.sort(idx, axis=1), np.sort(want, axis=1)), seed
        picks.append(idx)
    assert not np.array_equal(picks[0], picks[1])


def test_peer_memory_entry_points_with_one_rank():
    """sgr_ep_push / the waits / sgr_ep_step_advance with this device as its own only peer: the
    bytes arrive, the arrival word takes step * mul + add, a wait on a word that is already set
    returns, and the step counter advances in stream order."""
    import ctypes as C
    from sager_b200.ops import stream_ptr
    L, sp = lib(), stream_ptr()
    src = torch.arange(4096, dtype=torch.int32, device=DEV)
    dst = torch.zeros(2, 4096, dtype=torch.int32, device=DEV)
    flags = torch.zeros(2, dtype=torch.int32, device=DEV)
    step = torch.full((1,), 3, dtype=torch.int32, device=DEV)
    scratch = torch.zeros(1, dtype=torch.int32, device=DEV)
    dptr = torch.tensor([dst[0].data_ptr(), dst[1].data_ptr()], dtype=torch.int64, device=DEV)
    fptr = torch.tensor([flags.data_ptr(), flags.data_ptr() + 4], dtype=torch.int64, device=DEV)
    p = lambda t: C.c_void_p(t.data_ptr())
    L.call("sgr_ep_push", p(src), 0, src.numel() * 4, p(dptr), p(fptr), 2, p(step), 5, 2, p(scratch), sp)
    torch.cuda.synchronize()
    assert torch.equal(dst[0], src) and torch.equal(dst[1], src)
    assert flags.tolist() == [17, 17] and int(scratch.item()) == 0
    x = torch.ones(1024, dtype=torch.float16, device=DEV)
    parts = torch.full((2, 1024), 0.5, dtype=torch.float32, device=DEV)
    L.call("sgr_ep_reduce_add_f16_wait", p(x), p(parts), 2, 1024, 1024, p(flags), p(step), 5, 2, sp)
    L.call("sgr_ep_step_advance", p(step), sp)
    torch.cuda.synchronize()
    assert torch.all(x == 2.0) and int(step.item()) == 4
    assert lib().raw("sgr_status")(0) == 0


# ---- seed sweep at the benchmark geometry ---------------------------------------------------------
def _h_code_flips(oracle, w, blob_np, runner, x16_np, idx_row, t, k):
    """For token row t of a finished call: the Q8_K codes of h (the SwiGLU output that is
    requantised between the projections) as the device's fp32 h rows give them, against the codes
    the CPU path's h gives. -> (codes compared, codes that differ)."""
    H, F, E, n_max = w.hidden, w.n_ff, w.n_expert, runner.n_max
    off = lambda which: lib().raw("sgr_moe_layer_workspace_offset")(n_max, H, F, E, k, which)
    rows = n_max * k + n_max
    ws = runner.ws
    hbuf = ws[off(0):off(0) + rows * F * 4].view(torch.float32).view(rows, F)
    gslot = ws[off(2):off(2) + n_max * k * 4].view(torch.int32).cpu().numpy()
    o3 = [0, w.gu_bytes, 2 * w.gu_bytes]
    xq = oracle.quantize_q8k(x16_np[t].astype(np.float32)[None])[0]
    total = flips = 0
    for kk in range(k + 1):
        e = int(idx_row[kk]) if kk < k else E
        row = int(gslot[t * k + kk]) if kk < k else n_max * k + t
        g = oracle.gemv(blob_np[w.slot(e), o3[0]:o3[1]], xq, F, H)
        u = oracle.gemv(blob_np[w.slot(e), o3[1]:o3[2]], xq, F, H)
        h_cpu = (g / (np.float32(1) + np.exp(-g, dtype=np.float32)) * u).astype(np.float32)
        h_dev = hbuf[row].cpu().numpy()
        qa = oracle.quantize_q8k(h_cpu[None])[0].reshape(-1, 276)[:, 4:260]
        qb = oracle.quantize_q8k(h_dev[None])[0].reshape(-1, 276)[:, 4:260]
        total += qa.size
        flips += int((qa != qb).sum())
    return total, flips


@pytest.mark.parametrize("kernel", ["items", "rows", None])
def test_benchmark_geometry_seed_sweep(oracle, kernel):
    """32 seeded cases (4 weight sets x 8 input sets) x 1, 4 and 64 token rows, none of them picked:
    every case must meet the stated bound of 1e-3 against the CPU expert path, and the distribution
    is printed. Where a case is far from the typical 1e-7, the cause is counted, not assumed: h is
    requantised to Q8_K between the projections, and a value that sits on a rounding boundary can
    take another code on the device (other fp32 summation order, expf) than on the CPU."""
    k = 8
    errs = {1: [], 4: [], 64: []}
    worst = (0.0, None)
    for wi, wseed in enumerate((20260718, 11, 12, 13)):
        w = synth.MoeWeights(2048, 512, 256, DEV, seed=wseed)
        blob_np = w.blob.cpu().numpy()
        for xi in range(8):
            for n in (1, 4, 64):
                seed = 5000 + 100 * wi + 10 * xi + n
                bias = synth.zipf_bias(256, seed=seed, alpha=0.6) if n == 64 else None
                x16 = synth.normal_fp16((n, w.hidden), seed, DEV)
                x_np = x16.cpu().numpy()
                runner, _, out32 = run_layer(w, n, k, x16, n_max=64, bias=bias, kernel=kernel)
                want = oracle_layer(oracle, w, x_np, x_np.astype(np.float32), k, bias=bias, blob_np=blob_np,
                                    n_threads=16)
                idx = runner.route_idx.cpu().numpy()[:n]
                assert np.array_equal(idx[:, :k], want["idx"][:, :k]), (wseed, xi, n)
                got = out32.cpu().numpy()
                err = rel(got, want["out"])
                errs[n].append(err)
                if err > worst[0]:
                    t = int(np.abs(got - want["out"]).max(axis=1).argmax())
                    worst = (err, (wseed, xi, n, t) + _h_code_flips(oracle, w, blob_np, runner, x_np, idx[t], t, k))
        del w
    for n, v in errs.items():
        print(f"{kernel} kernel, {n:2d} rows: {len(v)} cases, max relative error median {np.median(v):.2e}, "
              f"max {np.max(v):.2e}")
    wseed, xi, n, t, total, flips = worst[1]
    print(f"worst case (weights {wseed}, inputs {xi}, {n} rows, row {t}): {worst[0]:.2e}; "
          f"{flips} of {total} Q8_K codes of h differ from the CPU path's")
    assert max(max(v) for v in errs.values()) <= LAYER_TOL


def test_strided_pointer_table_is_used_in_place(small_w):
    """The reference's decode table is [3][Lm][E] (src/core/session.cpp:3596-3598): a layer's
    gate / up / down slices are Lm * E pointers apart. tab_stride takes them where they are."""
    k, Lm, li = 4, 3, 2
    E = small_w.n_expert
    for kernel, n in (("items", 9), ("rows", 9), (None, 3)):
        x16 = synth.normal_fp16((n, small_w.hidden), 431, DEV)
        _, _, want = run_layer(small_w, n, k, x16, n_max=16, kernel=kernel)
        big = torch.zeros(3, Lm, E, dtype=torch.int64, device=DEV)
        big[:, li, :] = small_w.table()
        runner = MoeLayerRunner(16, small_w.hidden, small_w.n_ff, E, k, DEV)
        out32 = torch.zeros(n, small_w.hidden, dtype=torch.float32, device=DEV)
        a = runner.args(n, x16, small_w.router, big[0, li], small_w.shared_ptrs(), x_f16=x16.clone(), out_f32=out32)
        a.tab_stride = Lm * E
        runner.run(a, kernel=kernel)
        torch.cuda.synchronize()
        assert torch.equal(out32, want)
    assert lib().raw("sgr_status")(0) == 0


@pytest.mark.parametrize("hidden,n_ff", [(256, 2048), (2048, 256)])
def test_rows_kernel_with_one_block_column_per_group(oracle, hidden, n_ff):
    """hidden == 256 (gate / up groups) or n_ff == 256 (down groups) makes a group a single stage, so
    a CTA that draws several groups changes tile with every stage: more tiles than descriptor
    slots pass through a CTA while earlier copies are still in flight. 64 rows x top-8 over 64
    experts are about 70 tiles and several hundred single-stage groups, a handful per CTA."""
    E, k, n = 64, 8, 64
    w = synth.MoeWeights(hidden, n_ff, E, DEV, seed=77, std=0.05)
    for seed in (1, 2):
        check(oracle, w, n, k, seed=900 + seed, n_max=64, kernel="rows", tol=1e-3)


# ---- the single persistent launch for up to three token rows (kernel=None; four rows covered too,
# whichever path the library picks there) --------------------------------------------------------
@pytest.mark.parametrize("n", [1, 2, 3, 4])
def test_token_kernel_variants(oracle, small_w, n):
    """Without the shared expert, with a router bias, with absent experts (zero contribution, id
    mailed once), and with weight pointers that are only 2- or 4-byte aligned."""
    import copy
    k = 4
    check(oracle, small_w, n, k, seed=600 + n, use_shared=False)
    bias = synth.zipf_bias(16, seed=3, alpha=2.0)
    check(oracle, small_w, n, k, seed=610 + n, bias=bias)
    x16 = synth.normal_fp16((n, 512), 620 + n, DEV)
    r0, _, _ = run_layer(small_w, n, k, x16)
    used = sorted(set(r0.route_idx.cpu().numpy()[:n, :k].reshape(-1).tolist()))
    absent = (used[0], used[-1])
    runner, _, _ = check(oracle, small_w, n, k, seed=620 + n, absent=absent)
    n_mail = int(runner.mail_n.item())
    assert sorted(runner.mail.cpu().numpy()[:n_mail].tolist()) == sorted(absent)
    for shift in (2, 4):
        w = copy.copy(small_w)
        big = torch.empty(small_w.blob.numel() + 16, dtype=torch.uint8, device=DEV)
        w.blob = big[shift:shift + small_w.blob.numel()].view(small_w.blob.shape)
        w.blob.copy_(small_w.blob)
        check(oracle, w, n, k, seed=630 + n)


def test_token_kernel_agrees_with_the_two_launch_path(full_w):
    """Same routing bit for bit and the same layer to fp32 rounding as route + expert kernel, over
    repeated calls on one workspace (the grid barrier's counter carries over from call to call)."""
    k = 8
    for n in (1, 2, 3, 4):
        runner = MoeLayerRunner(4, full_w.hidden, full_w.n_ff, full_w.n_expert, k, DEV)
        for rep in range(3):
            x16 = synth.normal_fp16((n, full_w.hidden), 700 + 10 * n + rep, DEV)
            res = []
            for kernel in (None, "two_launch"):
                out32 = torch.zeros(n, full_w.hidden, dtype=torch.float32, device=DEV)
                x = x16.clone()
                a = runner.args(n, x16, full_w.router, full_w.table(), full_w.shared_ptrs(), x_f16=x, out_f32=out32)
                runner.run(a, kernel=kernel)
                torch.cuda.synchronize()
                res.append((out32.clone(), x.clone(), runner.route_idx.clone(), runner.route_w.clone()))
            assert torch.equal(res[0][2][:n], res[1][2][:n])
            assert torch.equal(res[0][3][:n], res[1][3][:n])
            assert rel(res[0][0].cpu().numpy(), res[1][0].cpu().numpy()) < 1e-5
    assert lib().raw("sgr_status")(0) == 0


@pytest.mark.parametrize("hidden,n_ff,E,k,n,ties", [
    (1280, 1024, 48, 8, 4, False),     # eight tiles' down rows at a time: five rounds in two regions
    (256, 256, 5, 4, 1, False),        # one block per row, fewer experts than lanes
    (768, 512, 300, 3, 2, False),      # more experts than one selecting warp holds
    (512, 256, 40, 4, 1, True),        # picks that do not stand: every logit twice, the lower expert goes first
    (512, 256, 40, 4, 3, True),
    (512, 256, 10, 4, 3, False),       # rows of probabilities that are no multiple of sixteen bytes
])
def test_token_kernel_edges(hidden, n_ff, E, k, n, ties):
    """The same routing and, to fp32 rounding of the same terms (1e-5), the same layer as route + expert kernel."""
    w = synth.MoeWeights(hidden, n_ff, E, DEV, seed=88, std=0.05)
    if ties:
        w.router[E // 2:] = w.router[:E // 2]
    x16 = synth.normal_fp16((n, hidden), 89, DEV)
    r0, _, o0 = run_layer(w, n, k, x16)
    r1, _, o1 = run_layer(w, n, k, x16, kernel="two_launch")
    assert torch.equal(r0.route_idx[:n], r1.route_idx[:n]) and torch.equal(r0.route_w[:n], r1.route_w[:n])
    assert rel(o0.cpu().numpy(), o1.cpu().numpy()) < 1e-5
    if ties:
        first = r0.route_idx[:n, 0].cpu().numpy()
        assert (first < E // 2).all() and (r0.route_idx[:n, 1].cpu().numpy() == first + E // 2).all()


@pytest.mark.parametrize("hidden,n_ff,E,k", [
    (2048, 512, 256, 8), (1024, 512, 128, 8), (2048, 256, 64, 8), (512, 256, 16, 4),      # 8, 4 and 2 block columns, down rows of 2 and 1
    (256, 256, 5, 4), (768, 768, 12, 3), (1280, 1024, 48, 8), (4096, 256, 20, 2),          # 1, 3, 5 and 16; 3 and 4
])
def test_four_rows_have_the_bits_of_the_row_streaming_kernel(hidden, n_ff, E, k):
    """From four rows on a layer's sums run block after block, whichever kernel takes it: no bit changes when a batch of four
    moves between the one-launch and the two-launch path. Hot experts (tiles of several rows), null experts, no shared one."""
    w = synth.MoeWeights(hidden, n_ff, E, DEV, seed=87, std=0.05)
    for i, (absent, use_shared) in enumerate((((), True), ((0, E - 1), True), ((), False))):
        x16 = synth.normal_fp16((4, hidden), 860 + i, DEV)
        x16[1:3] = x16[0] + 0.05 * x16[1:3]               # three rows that pick much the same experts
        r0, x0, o0 = run_layer(w, 4, k, x16, absent=absent, use_shared=use_shared)
        r1, x1, o1 = run_layer(w, 4, k, x16, absent=absent, use_shared=use_shared, kernel="two_launch")
        assert torch.equal(r0.route_idx, r1.route_idx) and torch.equal(r0.route_w, r1.route_w)
        assert torch.equal(o0.view(torch.int32), o1.view(torch.int32)) and torch.equal(x0.view(torch.int16), x1.view(torch.int16))


@pytest.mark.parametrize("hidden,n_ff,E,k", [(512, 256, 16, 4), (256, 256, 5, 4), (2048, 512, 32, 8)])
def test_one_launch_layers_back_to_back_on_one_workspace(hidden, n_ff, E, k):
    """The layers of a step share a workspace and its barrier counter, and each may start while the one before it drains:
    the bits of the same layers with a device synchronisation between them."""
    layers = [synth.MoeWeights(hidden, n_ff, E, DEV, seed=880 + i, std=0.05) for i in range(6)]
    for n in (1, 2, 4):
        x0 = synth.normal_fp16((n, hidden), 890 + n, DEV)
        ins = [synth.normal_fp16((n, hidden), 891 + 10 * n + i, DEV) for i in range(6)]
        st = MoeStack(layers, n, k, DEV, inputs=ins)
        st.x.copy_(x0)
        for li in range(6):
            r, a = st.layer_args(li, n)
            r.run(a)
            torch.cuda.synchronize()
        want, idx = st.x.clone(), st.idx.clone()
        st.capture(n)
        for _ in range(50):
            st.x.copy_(x0)
            st.replay()
            st.x.copy_(x0)
            st.step_eager(n)
        torch.cuda.synchronize()
        assert torch.equal(st.x.view(torch.int16), want.view(torch.int16)) and torch.equal(st.idx, idx)
    assert lib().raw("sgr_status")(0) == 0


@pytest.mark.parametrize("hidden,n_ff,E,k", [
    (2048, 512, 256, 8),     # two rows of a stage to a chunk, the last stage of a CTA one or none
    (1280, 1024, 48, 8),     # five block columns, eight tiles' down rows at a time, four blocks to a down row
    (1536, 768, 40, 7),      # six and three
    (2048, 256, 64, 8),      # two rows: the dp4a kernel
    (3072, 256, 24, 10),     # twelve, and one
    (1280, 2048, 24, 8),     # five, and eight
])
def test_several_rows_on_the_mma(hidden, n_ff, E, k):
    """Routed tiles on the int8 MMA: exact integer sums, and the fp32 terms of a row's blocks in the order of the kernels without it.
    Two and three rows have the bits that each row has by itself, four those of the row-streaming kernel, whichever form a
    geometry takes. Tiles of one row to all, null experts, no shared one, weights off a 16-byte boundary."""
    def same(a, b):
        return torch.equal(a.view(torch.int32 if a.dtype == torch.float32 else torch.int16), b.view(torch.int32 if b.dtype == torch.float32 else torch.int16))

    for shift in (0, 4):
        w = synth.MoeWeights(hidden, n_ff, E, DEV, seed=95, std=0.05)
        if shift:
            big = torch.zeros(w.blob.numel() + 16, dtype=torch.uint8, device=DEV)
            moved = big[shift:shift + w.blob.numel()]
            moved.copy_(w.blob.view(-1))
            w.blob = moved.view(w.blob.shape)
        for n in (2, 3, 4):
            for i, (absent, use_shared) in enumerate((((), True), ((0, E - 1), False))):
                x16 = synth.normal_fp16((n, hidden), 960 + 10 * n + i, DEV)
                x16[1:] = x16[0] + (0.05 if i else 0.4) * x16[1:]          # rows that pick much the same experts
                r0, x0, o0 = run_layer(w, n, k, x16, absent=absent, use_shared=use_shared)
                if n == 4:
                    r1, x1, o1 = run_layer(w, n, k, x16, absent=absent, use_shared=use_shared, kernel="rows")
                    assert torch.equal(r0.route_idx, r1.route_idx) and same(o0, o1) and same(x0, x1)
                    continue
                for t in range(n):
                    r1, x1, o1 = run_layer(w, 1, k, x16[t:t + 1], absent=absent, use_shared=use_shared)
                    assert torch.equal(r0.route_idx[t], r1.route_idx[0]) and same(o0[t], o1[0]) and same(x0[t], x1[0]), (n, i, t)


@pytest.mark.parametrize("hidden,n_ff,E,k", [(512, 256, 16, 4), (512, 256, 300, 4), (2048, 512, 64, 8)])
def test_one_workspace_through_changing_row_counts(hidden, n_ff, E, k):
    """The CTAs of a one-launch layer know each other's logits by the launch's number: whatever ran on the workspace before - more
    rows, fewer, the two-launch path - every layer has the bits that it has on a workspace of its own."""
    w = synth.MoeWeights(hidden, n_ff, E, DEV, seed=97, std=0.05)
    runner = MoeLayerRunner(6, hidden, n_ff, E, k, DEV)
    for step, n in enumerate((1, 4, 1, 6, 1, 2, 3, 5, 4, 2, 1, 1, 3)):
        x16 = synth.normal_fp16((n, hidden), 970 + step, DEV)
        if step % 3 == 0:
            x16.zero_()                                   # logits of zero, equal everywhere
        outs = []
        for r in (runner, MoeLayerRunner(6, hidden, n_ff, E, k, DEV)):
            out = torch.zeros(n, hidden, dtype=torch.float32, device=DEV)
            r.run(r.args(n, x16, w.router, w.table(), w.shared_ptrs(), x_f16=x16.clone(), out_f32=out))
            outs.append((out, r.route_idx[:n].clone(), r.route_w[:n].clone()))
        assert all(torch.equal(a, b) for a, b in zip(*outs)), (step, n)
    assert lib().raw("sgr_status")(0) == 0


@pytest.mark.parametrize("hidden,n_ff,E,k", [(512, 256, 16, 4), (512, 256, 300, 4), (2048, 512, 64, 8)])
def test_one_launch_layer_after_one_that_gave_up(hidden, n_ff, E, k):
    """A launch whose waits ran out leaves logits with its number behind and the arrival counter at a multiple of the grid, the
    CTAs that gave up counted in the top byte (written here by the host). The next launch has a number of its own: it
    takes none of those logits, and what was counted before is not its own failure."""
    w = synth.MoeWeights(hidden, n_ff, E, DEV, seed=98, std=0.05)
    grid = min(torch.cuda.get_device_properties(0).multi_processor_count, 160)
    offset = lib().raw("sgr_moe_layer_workspace_offset")
    for n in (1, 3):
        runner = MoeLayerRunner(4, hidden, n_ff, E, k, DEV)
        at, words = offset(4, hidden, n_ff, E, k, 6) + 48, offset(4, hidden, n_ff, E, k, 7)
        counter = runner.ws[at:at + 8].view(torch.int64)
        logits = runner.ws[words:words + 16 * n * E * 8].view(torch.int32).view(-1, 2)     # value, number
        x16 = synth.normal_fp16((n, hidden), 980 + n, DEV)
        outs = []
        for launch in range(3):
            out = torch.zeros(n, hidden, dtype=torch.float32, device=DEV)
            runner.run(runner.args(n, x16, w.router, w.table(), w.shared_ptrs(), x_f16=x16.clone(), out_f32=out))
            torch.cuda.synchronize()
            gave_up = 0 if launch == 0 else 3 * launch << 56
            assert counter.item() == (2 * launch + 1) * grid + gave_up and torch.all(logits[:, 1] == 2 * launch + 1)
            outs.append((out, runner.route_idx[:n].clone(), runner.route_w[:n].clone()))
            counter += grid + (3 << 56)                              # the launch that gives up: three of its CTAs
            logits[:, 0] = torch.randperm(logits.shape[0], device=DEV).to(torch.float32).view(torch.int32)
            logits[:, 1] += 1
        assert all(torch.equal(a, b) for o in outs[1:] for a, b in zip(outs[0], o)), n
    assert lib().raw("sgr_status")(0) == 0


def test_four_rows_on_a_workspace_for_the_item_kernel(full_w):
    """A workspace too small for the row-streaming kernel keeps four rows on the item kernel and its order of the sums."""
    x16 = synth.normal_fp16((4, full_w.hidden), 870, DEV)
    outs = []
    for kernel in (None, "items"):
        runner = MoeLayerRunner(4, full_w.hidden, full_w.n_ff, full_w.n_expert, 8, DEV)
        out = torch.zeros(4, full_w.hidden, dtype=torch.float32, device=DEV)
        a = runner.args(4, x16, full_w.router, full_w.table(), full_w.shared_ptrs(), x_f16=x16.clone(), out_f32=out)
        a.workspace_bytes -= 256                  # one alignment step short of the whole layout
        runner.run(a, kernel=kernel)
        torch.cuda.synchronize()
        outs.append(out)
    assert torch.equal(outs[0].view(torch.int32), outs[1].view(torch.int32))


@pytest.mark.parametrize("E,k,n", [
    (10, 4, 9),        # two experts per route CTA, a token tile of one row
    (40, 8, 33),       # two per CTA, five tiles
    (80, 8, 40),       # four per CTA
    (160, 6, 61),      # sixteen per CTA, a ragged last tile
    (256, 8, 30),      # eight per CTA
    (300, 3, 20),      # more experts than two selecting warps hold
])
def test_route_kernel_edges(oracle, E, k, n):
    """Every split of the logits over CTAs and warps: the oracle's picks, weights to its fp32 rounding."""
    w = synth.MoeWeights(512, 256, E, DEV, seed=90, std=0.05, distinct=4)
    x16 = synth.normal_fp16((n, 512), 91 + E, DEV)
    runner, _, _ = run_layer(w, n, k, x16, n_max=64, kernel="two_launch")
    idx, wt = runner.route_idx.cpu().numpy(), runner.route_w.cpu().numpy()
    for t in range(n):
        i, v = oracle.router_topk(oracle.router_logits(w.router.cpu().numpy(), x16.cpu().numpy()[t]), k)
        assert np.array_equal(idx[t, :k], i[:k]) and np.abs(wt[t, :k] - v[:k]).max() <= 1e-6


@pytest.mark.parametrize("own_plan", [False, True])
@pytest.mark.parametrize("tokens", [8, 64])
def test_fused_exchange_entry_points_with_one_rank(full_w, tokens, own_plan):
    """The expert-parallel layer with the exchanges done by its own kernels, this device being its
    own only peer: the route kernel stores the records into the 'owner's' receive slot and sets the
    arrival word, the owner call waits for it and stores its rows into the 'home rank's' return
    slot, the home reduction waits for that word. Must reproduce the single call."""
    import ctypes as C
    from sager_b200.ep import record_layout
    from sager_b200.ops import stream_ptr
    w, k, H = full_w, 8, full_w.hidden
    x16 = synth.normal_fp16((tokens, H), 191, DEV)
    _, x_full, _ = run_layer(w, tokens, k, x16, n_max=64)
    rec, idx_off, w_off = record_layout(H, k, True)
    send = torch.zeros(tokens, rec, dtype=torch.uint8, device=DEV)
    recv = torch.zeros(tokens, rec, dtype=torch.uint8, device=DEV)
    back = torch.zeros(1, tokens, H, dtype=torch.float32, device=DEV)
    flags = torch.zeros(2, dtype=torch.int32, device=DEV)
    step = torch.full((1,), 5, dtype=torch.int32, device=DEV)
    p64 = lambda *addr: torch.tensor(list(addr), dtype=torch.int64, device=DEV)
    dst_recv, dst_back = p64(recv.data_ptr()), p64(back.data_ptr())
    fl_d, fl_r = p64(flags.data_ptr()), p64(flags.data_ptr() + 4)
    ptr = lambda t, off=0: C.c_void_p(t.data_ptr() + off)
    L, sp = lib(), stream_ptr()
    home = MoeLayerRunner(tokens, H, w.n_ff, w.n_expert, k, DEV)
    x = x16.clone()
    tab = w.table()                               # kept alive: the calls hold its device address only
    a = home.args(tokens, x16, w.router, tab, None, x_f16=x)
    a.xq_out, a.xq_stride, a.xq_padded = ptr(send), rec, 1
    a.route_idx, a.route_w, a.route_stride = ptr(send, idx_off), ptr(send, w_off), rec // 4
    a.ep_dst, a.ep_flags, a.ep_step = ptr(dst_recv), ptr(fl_d), ptr(step)
    a.ep_world, a.ep_rec_bytes, a.ep_mul, a.ep_add = 1, rec, 3, 2
    owner = MoeLayerRunner(64, H, w.n_ff, w.n_expert, k, DEV)
    if own_plan:
        # the owner call plans inside its expert kernel (stage bit 7, no plan launch); the home call's
        # route stage re-arms the owner workspace's counters
        a.rearm_workspace, a.rearm_mail_n, a.rearm_n_max = ptr(owner.ws), ptr(owner.mail_n), 64
    L.call("sgr_moe_layer_decode_stages", C.byref(a), 1 | 8, sp)
    b = owner.args(tokens, None, None, tab, w.shared_ptrs(), xq_in=recv, routing_given=True, no_residual=True)
    b.xq_stride, b.route_stride, b.xq_padded = rec, rec // 4, 1
    b.route_idx, b.route_w = ptr(recv, idx_off), ptr(recv, w_off)
    b.wait_flags, b.wait_step, b.wait_count, b.wait_mul, b.wait_add = ptr(flags), ptr(step), 1, 3, 2
    b.ep_out, b.ep_flags, b.ep_step = ptr(dst_back), ptr(fl_r), ptr(step)
    b.ep_world, b.ep_home_rows, b.ep_mul, b.ep_add = 1, tokens, 3, 2
    def issue():
        L.call("sgr_moe_layer_decode_stages", C.byref(a), 1 | 8, sp)
        L.call("sgr_moe_layer_decode_stages", C.byref(b), (6 | 16 | 128) if own_plan else (7 | 16), sp)
        L.call("sgr_ep_reduce_add_f16_wait", ptr(x), ptr(back), 1, tokens * H, tokens * H, ptr(flags, 4), ptr(step), 3, 2, sp)
    L.call("sgr_moe_layer_decode_stages", C.byref(b), (6 | 16 | 128) if own_plan else (7 | 16), sp)
    L.call("sgr_ep_reduce_add_f16_wait", ptr(x), ptr(back), 1, tokens * H, tokens * H, ptr(flags, 4), ptr(step), 3, 2, sp)
    torch.cuda.synchronize()
    assert flags.tolist() == [17, 17]
    if own_plan:                                  # a second layer on the same workspaces: the re-armed counters hold
        x_once = x.clone()
        x.copy_(x16)
        step.fill_(6)
        issue()
        torch.cuda.synchronize()
        assert flags.tolist() == [20, 20]
        assert torch.equal(x, x_once)
    assert torch.equal(recv, send)
    assert rel(x.float().cpu().numpy(), x_full.float().cpu().numpy()) <= 2.0 ** -10      # fp16 store after another add order
    assert lib().raw("sgr_status")(0) == 0


def picks_of(meet, n):
    """Experts of each row, eight apiece, so that tiles of the wanted numbers of rows arise."""
    if meet == "all":
        return [list(range(8)) for _ in range(n)]
    own = [list(range(8 + 8 * t, 16 + 8 * t)) for t in range(n)]          # experts no other row has
    if meet == "none":
        return own
    if meet == "pair":
        return [list(range(8)) if t < 2 else own[t] for t in range(n)]
    # tiles of one to four rows beside one another
    common = {0: range(4), 1: range(4), 2: (0, 1, 2), 3: (1, 2, 3), 4: (0, 1), 5: (2, 3), 6: (0, 2)}
    return [([e for e, rows in common.items() if t in rows] + own[t])[:8] for t in range(n)]


@pytest.mark.parametrize("n", [3, 4])
@pytest.mark.parametrize("meet", ["all", "pair", "none", "mixed", "absent"])
def test_token_layer_shares_by_cost(oracle, n, meet):
    """Layers of three and four rows whose CTAs take more pairs than a pass of both groups: tiles of one to four rows in one
    layer, every tile with all rows, no two rows in a tile, an absent expert among them. Every (tile, pair) has to be in exactly
    one CTA's share: a pair left out or taken by a neighbour shows in h. The router's first columns hold the logits wanted, the
    rows' first values name the column."""
    H, F, E, K = 2048, 768, 40, 8
    w = synth.MoeWeights(H, F, E, DEV, seed=91, std=0.05)
    x16 = synth.normal_fp16((n, H), 92 + n, DEV)
    x16[:, :n] = torch.eye(n, dtype=torch.float16, device=DEV)
    picks = picks_of(meet, n)
    w.router.zero_()
    for t, chosen in enumerate(picks):
        w.router[chosen, t] = 3.0 - 0.125 * torch.arange(K, dtype=torch.float32, device=DEV)
    distinct = {e for chosen in picks for e in chosen}
    # (the line of the kernel's rule: a pass of both groups is 2 x 16 pairs at hidden 2048)
    assert len(distinct) * F > 2 * 16 * torch.cuda.get_device_properties(0).multi_processor_count
    if meet in ("mixed", "absent"):
        assert {sum(e in chosen for chosen in picks) for e in distinct} == set(range(1, n + 1))
    x_np = x16.cpu().numpy()
    absent = (0, 3) if meet == "absent" else ()
    want = oracle_layer(oracle, w, x_np, x_np.astype(np.float32), K, absent=absent)
    assert [sorted(r) for r in want["idx"][:, :K].tolist()] == [sorted(chosen) for chosen in picks]
    for rep in range(2):                         # (the second call finds the first one's h rows)
        runner, x_out, out32 = run_layer(w, n, K, x16, absent=absent)
        assert np.array_equal(runner.route_idx.cpu().numpy()[:n, :K], want["idx"][:, :K])
        assert rel(out32.cpu().numpy(), want["out"]) < LAYER_TOL
    # the row-streaming kernel adds a row's blocks in the same order from four rows on
    if n == 4:
        other = run_layer(w, n, K, x16, absent=absent, kernel="rows")[2]
        assert torch.equal(out32, other)
