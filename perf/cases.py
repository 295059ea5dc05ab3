"""The work that a program built on this library has it do on one GPU, as cases that can be timed.

  decode   one decode step through the MoE halves of a stack of layers (MoeStack): 1 to 64 token rows, replayed
           from the CUDA graph that a serving loop keeps, or issued call by call where the row count changes from
           step to step
  prefill  a prompt chunk through the MoE half of a few layers (PrefillLayer), router included
  dense    the Q4_K projections around attention in a decode step (norm + quantise, q / k / v, output projection),
           for one token row or a window of a few
  head     the final norm, the LM head (Q4_K or Q6_K weights) and the top-k after it
  project  a dense Q4_K projection of a prefill chunk on the fp16 tensor-core entry

Weights, inputs and routing have the benchmark's distributions: activations N(0, 1), weights N(0, 0.02), router
logits optionally skewed by a Zipf(s = 1.1) bias over expert rank of the strength that gives 20 % of the experts
about 70 % of the picks.
"""
import numpy as np
import torch

from sager_b200 import ops, synth
from sager_b200.layer import MoeStack, PrefillLayer

DEV = "cuda:0"
ZIPF_ALPHA = 0.36            # bench.py's calibration for 256 experts
Q8_BYTES, Q4_BYTES, Q6_BYTES = 276, 144, 210          # per 256 values

# (hidden, expert FFN, experts, top-k): the benchmark's layer, the tests' small layer, two between
FULL, MID, NARROW, SMALL = (2048, 512, 256, 8), (1024, 512, 128, 8), (2048, 256, 64, 8), (512, 256, 16, 4)


def _geometry(g):
    return dict(zip(("hidden", "ff", "experts", "top_k"), g))


def _decode(rows, layers, zipf, graph, geometry, **kw):
    return dict(kw, kind="decode", rows=rows, layers=layers, zipf=zipf, graph=graph, **_geometry(geometry))


def _prefill(rows, layers, geometry, **kw):
    return dict(kw, kind="prefill", rows=rows, layers=layers, **_geometry(geometry))


def _dense(rows, layers, graph, hidden=2048, q_rows=4096, kv_rows=512, **kw):
    return dict(kw, kind="dense", rows=rows, layers=layers, graph=graph, hidden=hidden, q_rows=q_rows, kv_rows=kv_rows)


def _head(rows, vocab, hidden, weights, k, **kw):
    return dict(kw, kind="head", rows=rows, vocab=vocab, hidden=hidden, weights=weights, k=k)


def _project(rows, n_out, n_in, **kw):
    return dict(kw, kind="project", rows=rows, n_out=n_out, n_in=n_in)


def listed():
    return [
        # a single user's token through the whole 40-layer stack: every layer is a chain of short launches
        _decode(1, 40, False, True, FULL, name="decode_1row"),
        # two rows issued layer by layer, as a loop does whose row count changes: host time per call counts
        _decode(2, 8, False, False, FULL, name="decode_2rows_calls"),
        # a speculative-verify window (three drafts and one token), hot experts
        _decode(4, 40, True, True, FULL, name="decode_4rows_verify"),
        # a ragged batch on a smaller model
        _decode(19, 12, True, True, MID, name="decode_19rows_mid"),
        # the headline: 64 concurrent tokens
        _decode(64, 40, True, True, FULL, name="decode_64rows"),
        # a short prompt, just past what the decode entry takes: a few rows per expert, bound by the weights
        _prefill(96, 4, FULL, name="prefill_96rows"),
        # a prompt's ragged tail
        _prefill(777, 2, FULL, name="prefill_777rows"),
        # a full chunk
        _prefill(2048, 2, FULL, name="prefill_2048rows"),
        # attention's projections of one token through 40 layers, from the step's graph
        _dense(1, 40, True, name="dense_1row"),
        # the same for a verify window, call by call
        _dense(4, 8, False, name="dense_4rows_calls"),
        # logits and candidates of one token on the Q6_K head
        _head(1, 151936, 2048, "q6", 40, name="head_q6"),
        # one projection of a full prefill chunk
        _project(2048, 4096, 2048, name="project_2048rows"),
    ]


def _log(rng, lo, hi):
    """A whole number, its logarithm spread evenly."""
    return min(hi, max(lo, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choice(("decode", "decode", "decode", "prefill", "prefill", "dense", "head", "project"))
    if kind == "decode":
        geometry = rng.choice((FULL, FULL, MID, NARROW, SMALL))
        return _decode(_log(rng, 1, 64), rng.randint(4, 12), rng.random() < 0.5, rng.random() < 0.7, geometry)
    if kind == "prefill":
        return _prefill(_log(rng, 65, 2048), rng.randint(1, 2), rng.choice((FULL, FULL, MID, NARROW)))
    if kind == "dense":
        return _dense(_log(rng, 1, 8), rng.randint(4, 24), rng.random() < 0.5, rng.choice((1024, 2048, 4096)),
                      rng.choice((2048, 4096, 8192)), rng.choice((256, 512, 1024)))
    if kind == "head":
        weights = rng.choice(("q4", "q6"))
        return _head(rng.randint(1, 4) if weights == "q4" else 1, _log(rng, 8000, 248320), rng.choice((1024, 2048, 4096)),
                     weights, rng.choice((1, 8, 20, 40, 64)))
    return _project(_log(rng, 64, 2048), rng.choice((512, 1000, 2048, 4096)), rng.choice((512, 2048, 4096)))


# ---- what a program has in hand -----------------------------------------------------------------------------

def _normal(g, *shape):
    return torch.randn(*shape, generator=g, device=DEV).half()


def _q4(g, rows, k):
    """Q4_K bytes of a [rows][k] matrix drawn from N(0, 0.02)."""
    q = torch.empty(rows, k // 256 * Q4_BYTES, dtype=torch.uint8, device=DEV)
    for r0 in range(0, rows, 16384):
        r1 = min(rows, r0 + 16384)
        q[r0:r1] = synth.quantize_q4k(torch.randn(r1 - r0, k, generator=g, device=DEV) * 0.02)
    return q


def _q6(g, rows, k):
    """Q6_K bytes of a [rows][k] matrix of about N(0, 0.02): 6-bit codes around 32, int8 scales, one fp16 scale."""
    nb = k // 256
    q = torch.empty(rows, nb, Q6_BYTES, dtype=torch.uint8, device=DEV)
    for r0 in range(0, rows, 16384):
        n = min(rows, r0 + 16384) - r0
        code = (32 + 10 * torch.randn(n, nb, 2, 128, generator=g, device=DEV)).round().clamp(0, 63).to(torch.uint8)
        lo, hi = code & 15, code >> 4                # low nibbles: 32 apart in pairs; high bits: four runs of 32 in a byte
        ql = (lo[..., 0:64] | (lo[..., 64:128] << 4)).reshape(n, nb, 128)
        qh = (hi[..., 0:32] | (hi[..., 32:64] << 2) | (hi[..., 64:96] << 4) | (hi[..., 96:128] << 6)).reshape(n, nb, 64)
        sc = torch.randint(60, 128, (n, nb, 16), generator=g, device=DEV, dtype=torch.int32).to(torch.uint8)
        d = torch.full((n, nb, 1), 0.02 / 940, device=DEV).half()
        q[r0:r0 + n] = torch.cat((ql, qh, sc, d.view(torch.uint8)), dim=2)
    return q.reshape(rows, nb * Q6_BYTES)


def _empty_q8(rows, k):
    return torch.zeros(rows, k // 256 * Q8_BYTES, dtype=torch.uint8, device=DEV)


def _captured(issue):
    """`issue` as a graph, the way a serving loop keeps its step."""
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        issue()
    torch.cuda.current_stream().wait_stream(s)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        issue()
    return g


def prepare(case, seed):
    g = torch.Generator(device=DEV).manual_seed(seed * 7919 + 17)
    state = dict(case=case)
    kind, rows = case["kind"], case["rows"]
    if kind in ("decode", "prefill"):
        H, F, E, K, n_layers = case["hidden"], case["ff"], case["experts"], case["top_k"], case["layers"]
        # 32 experts' bytes are drawn for each layer, the others hold copies of them at addresses of their own
        weights = [synth.MoeWeights(H, F, E, DEV, seed=seed * 1009 + li, distinct=32) for li in range(n_layers)]
        inputs = [_normal(g, rows, H) for _ in range(n_layers)]
        state.update(x0=_normal(g, rows, H), weights=weights, inputs=inputs)
    if kind == "decode":
        biases = None
        if case["zipf"]:
            biases = [torch.from_numpy(synth.zipf_bias(E, seed * 31 + li, ZIPF_ALPHA)).to(DEV) for li in range(n_layers)]
        stack = MoeStack(weights, rows, K, DEV, biases=biases, inputs=inputs)
        if case["graph"]:
            stack.capture(rows)
        state.update(stack=stack)
    elif kind == "prefill":
        state.update(layer=PrefillLayer(rows, H, F, E, K, DEV), tables=[w.table() for w in weights],
                     x=torch.empty_like(state["x0"]))
    elif kind == "dense":
        H, Q, KV = case["hidden"], case["q_rows"], case["kv_rows"]
        state["layers"] = [dict(
            norm=(1 + 0.1 * torch.randn(H, generator=g, device=DEV)).half(), wq=_q4(g, Q, H), wk=_q4(g, KV, H),
            wv=_q4(g, KV, H), wo=_q4(g, H, Q), x=_normal(g, rows, H), attn=_normal(g, rows, Q),
            q=torch.empty(rows, Q, dtype=torch.float16, device=DEV), k=torch.empty(rows, KV, dtype=torch.float16, device=DEV),
            v=torch.empty(rows, KV, dtype=torch.float16, device=DEV), o=torch.empty(rows, H, dtype=torch.float16, device=DEV))
            for _ in range(case["layers"])]
        state.update(x0=_normal(g, rows, H), x=torch.zeros(rows, H, dtype=torch.float16, device=DEV),
                     xn=torch.empty(rows, H, dtype=torch.float16, device=DEV), xq=_empty_q8(rows, H), aq=_empty_q8(rows, Q))
        state["graph"] = _captured(lambda: _dense_step(state)) if case["graph"] else None
    elif kind == "head":
        H, V, k = case["hidden"], case["vocab"], case["k"]
        slots = (V + 2047) // 2048 * k
        state.update(
            w=_q6(g, V, H) if case["weights"] == "q6" else _q4(g, V, H), x=_normal(g, rows, H),
            norm=(1 + 0.1 * torch.randn(H, generator=g, device=DEV)).half(),
            xn=torch.empty(rows, H, dtype=torch.float16, device=DEV), xq=_empty_q8(rows, H), slots=slots,
            logits=torch.empty(rows, V, dtype=torch.float32, device=DEV), seg_v=torch.empty(slots, device=DEV),
            seg_i=torch.empty(slots, dtype=torch.int32, device=DEV), top_v=torch.empty(rows, k, device=DEV),
            top_i=torch.empty(rows, k, dtype=torch.int32, device=DEV))
    else:
        n_out, n_in = case["n_out"], case["n_in"]
        state.update(w=_q4(g, n_out, n_in), x=_normal(g, rows, n_in),
                     y=torch.empty(rows, n_out, dtype=torch.float16, device=DEV),
                     scratch=torch.empty(n_out * n_in, dtype=torch.float16, device=DEV))
    return state


# ---- one pass -----------------------------------------------------------------------------------------------

def _dense_step(s):
    c = s["case"]
    rows, H, Q, KV = c["rows"], c["hidden"], c["q_rows"], c["kv_rows"]
    for li in s["layers"]:
        if rows == 1:                # the residual stream goes through the layers
            ops.rmsnorm_quant_f16(s["xn"], s["x"], li["norm"], s["xq"], H, 1e-6, 1)
            ops.gemv3m_q4_k_q8_f16out(li["wq"], li["wk"], li["wv"], s["xq"], li["q"], li["k"], li["v"], Q, KV, KV, H, 0)
            ops.quantize_q8_k(li["attn"], s["aq"], Q)
            ops.gemv_q4_k_q8_f16out_resadd(li["wo"], s["aq"], li["o"], s["x"], H, Q)
        else:                        # a window of rows; adding to the residual is not this library's launch there
            ops.rmsnorm_quant_f16(s["xn"], li["x"], li["norm"], s["xq"], H, 1e-6, rows)
            ops.gemv_q4_k_q8_f16out_mtok(li["wq"], s["xq"], li["q"], Q, H, rows)
            ops.gemv2_q4_k_q8_f16out_mtok(li["wk"], li["wv"], s["xq"], li["k"], li["v"], KV, H, rows)
            ops.quantize_q8_k(li["attn"], s["aq"], rows * Q)
            ops.gemv_q4_k_q8_f16out_mtok(li["wo"], s["aq"], li["o"], H, Q, rows)


def run(state):
    s, c = state, state["case"]
    kind, rows = c["kind"], c["rows"]
    if kind == "decode":
        stack = s["stack"]
        stack.x.copy_(s["x0"])       # the step's residual rows
        if c["graph"]:
            stack.replay()
        else:
            stack.step_eager(rows)
        return {"x": stack.x, "idx": stack.idx, "w": stack.w}
    if kind == "prefill":
        s["x"].copy_(s["x0"])
        for w, table, xn in zip(s["weights"], s["tables"], s["inputs"]):
            s["layer"].run(rows, xn, s["x"], w, table)
        return {"x": s["x"], "idx": s["layer"].idx, "w": s["layer"].w}
    if kind == "dense":
        s["x"].copy_(s["x0"])
        if s["graph"] is not None:
            s["graph"].replay()
        else:
            _dense_step(s)
        last = s["layers"][-1]
        return [s["x"], s["xq"]] + [last[n] for n in "qkvo"] + [li["o"] for li in s["layers"][:-1]]
    if kind == "head":
        H, V, k = c["hidden"], c["vocab"], c["k"]
        ops.rmsnorm_quant_f16(s["xn"], s["x"], s["norm"], s["xq"], H, 1e-6, rows)
        if c["weights"] == "q6":
            ops.gemv_q6_k_q8(s["w"], s["xq"], s["logits"], V, H)
        elif rows == 1:
            ops.gemv_q4_k_q8(s["w"], s["xq"], s["logits"], V, H)
        else:
            ops.gemv_q4_k_q8_batched(s["w"], s["xq"], s["logits"], V, H, rows)
        for r in range(rows):
            ops.topk_select_f32_2p(s["logits"][r], s["seg_v"], s["seg_i"], s["slots"], s["top_v"][r], s["top_i"][r], V, k)
        return {"logits": s["logits"], "top_v": s["top_v"], "top_i": s["top_i"]}
    ops.tc_gemm_q4_k_f16(s["w"], s["x"], s["y"], s["scratch"], c["n_out"], c["n_in"], rows)
    return s["y"]


# ---- what a pass cannot do without --------------------------------------------------------------------------

def _experts_hit(case):
    """Distinct routed experts of a layer: the mean over eight drawn layers of the case's rows and skew."""
    E, K, rows = case["experts"], case["top_k"], case["rows"]
    rng = np.random.default_rng(5)
    hit = []
    for i in range(8):
        logits = rng.standard_normal((rows, E)) * 0.02 * case["hidden"] ** 0.5
        if case.get("zipf"):
            logits += synth.zipf_bias(E, i, ZIPF_ALPHA)
        hit.append(len(np.unique(np.argpartition(-logits, K - 1, axis=1)[:, :K])))
    return sum(hit) / len(hit)


def work(case):
    kind, rows = case["kind"], case["rows"]
    if kind in ("decode", "prefill"):
        H, F, E, K = case["hidden"], case["ff"], case["experts"], case["top_k"]
        weights = (_experts_hit(case) + 1) * 3 * H * F // 256 * Q4_BYTES + E * H * 4
        rows_io = rows * (H * 2 + 8 * (K + 1))                        # input rows, ids and weights
        flops = rows * (2 * E * H + (K + 1) * 6 * H * F)
        return {"bytes": case["layers"] * (weights + rows_io) + rows * H * 4, "flops": case["layers"] * flops}
    if kind == "dense":
        H, Q, KV = case["hidden"], case["q_rows"], case["kv_rows"]
        macs = 2 * H * (Q + KV)
        io = rows * 2 * ((H if rows > 1 else 0) + 2 * Q + 2 * KV + H) + 2 * H
        return {"bytes": case["layers"] * (macs // 256 * Q4_BYTES + io) + (4 * H if rows == 1 else 0),
                "flops": case["layers"] * 2 * rows * macs}
    if kind == "head":
        H, V = case["hidden"], case["vocab"]
        return {"bytes": V * H // 256 * (Q6_BYTES if case["weights"] == "q6" else Q4_BYTES) + rows * (V * 4 + 2 * H + 8 * case["k"]),
                "flops": 2 * rows * V * H}
    n_out, n_in = case["n_out"], case["n_in"]
    return {"bytes": n_out * n_in // 256 * Q4_BYTES + 2 * rows * (n_in + n_out), "flops": 2 * rows * n_out * n_in}


def tolerance(case):
    # The head's logits are fp32 sums; every other result is a row of fp16 values, and inside a layer an activation
    # that sits on a rounding boundary of the 8-bit quantiser may take the code next to it.
    return {"rel": 1e-5} if case["kind"] == "head" else {"rel": 1e-3}
