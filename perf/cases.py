"""Performance cases: the work that a serving host has the Seedless decode core do, through the package's public calls.

One full-size model (the synthetic 40-layer 35B-A3B-shaped geometry of the benchmark) serves every engine case of a
process, as it does in a server; what differs from case to case, and from seed to seed, are the prompts, the streams and
the calls.  The kinds of case:

  matmul   the 4-bit group-64 product on device buffers (the operator a micro-benchmark or a host's own graph calls)
  small    one decode step of the two-layer test geometry in the checkpoint's data layout (8-bit router and shared gate,
           f32 GDN norm): nothing but launches and latency
  step     one greedy decode step of one stream, token in and token out: the single-user case
  chain    greedy steps chained on the device, at long context
  verify   a speculative verify call of several rows that ends in a rejection (snapshot, rows, rollback)
  sample   a speculative-sampling call: rows, nucleus, penalties, draft tokens, then the rollback
  batch    one greedy step of many streams at once (continuous batching)
  prompt   a prompt in prefill mode, in calls of at most 1024 tokens, and its first token
  strict   a prompt through the strict forward (the form whose rows equal single steps bit for bit)
  prefix   a stream's state saved to a host blob and restored into another stream (the prefix cache's traffic)
"""
import math

import numpy as np
import torch

import qwisp_b200 as Q

H, I, V, E, TOPK, LAYERS = 2048, 512, 151936, 256, 8, 40
N_GDN, N_ATT = 30, 10
Q4 = 0.5625                                        # bytes of a 4-bit weight with its group-64 scale and bias
GDN_IN, GDN_VAL, ATT_IN, ATT_OUT = 12352, 4096, 9216, 4096
STATE_BYTES = 32 * 128 * 128 * 4                   # fp32 GDN state of one layer
HIST_BYTES = 3 * 8192 * 2                          # conv history of one layer
KV_BYTES = 2 * 2 * 256 * 2                         # K and V of one position and attention layer
CHUNK = 1024                                       # rows of the largest call
MAX_LEN = 65536                                    # positions a decoding stream may grow to

#: the two-layer geometry of the repository's tests, real head and hidden sizes
SMALL = dict(hidden=2048, n_layers=2, attn_every=2, vocab=1024, n_experts=16, top_k=8, moe_inter=512,
             gdn_k_heads=16, gdn_v_heads=32, attn_heads=16, attn_kv_heads=2)

_engines = {}


def _model():
    """The served model: made once per process, as in a server."""
    if "full" not in _engines:
        cfg = Q.config(n_layers=LAYERS, max_rows=CHUNK, max_streams=208, kv_page_size=64, kv_pages=8192)
        _engines["full"] = Q.Engine.synthetic(cfg, seed=0, norm_jitter=0.0, conv_std=0.02)
    return _engines["full"]


def _q8(w):
    """fp16 rows -> the checkpoint's 8-bit group-64 layout (bytes, fp16 scales, fp16 biases)."""
    g = w.astype(np.float32).reshape(w.shape[0], -1, 64)
    lo, hi = g.min(axis=2), g.max(axis=2)
    s = np.maximum((hi - lo) / 255.0, 1e-7).astype(np.float16)
    b = lo.astype(np.float16)
    q = np.rint((g - b.astype(np.float32)[..., None]) / s.astype(np.float32)[..., None])
    return np.clip(q, 0, 255).astype(np.uint8).reshape(w.shape), s, b


def _small_model():
    """The small model loaded by name from host tensors, router and GDN norm as a checkpoint stores them."""
    if "small" not in _engines:
        room = dict(max_rows=64, max_streams=16, kv_page_size=64, kv_pages=4096)
        src = Q.Engine.synthetic(Q.config(**SMALL, **{**room, "max_streams": 1, "kv_pages": 1}), seed=1, norm_jitter=0.1, conv_std=0.5)
        q4 = lambda base: [f"{base}.{p}" for p in "wsb"]  # noqa: E731
        names = ["embed", "final_norm"] + q4("lm_head")
        for i in range(SMALL["n_layers"]):
            p = f"L{i}."
            names += [p + "in_norm", p + "post_norm", p + "moe.router", p + "moe.shared_gate"]
            for m in ("gate_proj", "up_proj", "down_proj", "shared_gate_proj", "shared_up_proj", "shared_down_proj"):
                names += q4(p + "moe." + m)
            if (i + 1) % SMALL["attn_every"]:
                names += [p + "gdn.conv_w", p + "gdn.A_log", p + "gdn.dt_bias", p + "gdn.norm"]
                for m in ("in_proj_qkv", "in_proj_z", "in_proj_b", "in_proj_a", "out_proj"):
                    names += q4(p + "gdn." + m)
            else:
                names += [p + "attn.q_norm", p + "attn.k_norm"]
                for m in ("q_proj", "k_proj", "v_proj", "o_proj"):
                    names += q4(p + "attn." + m)
        t = {n: src.read_tensor(n) for n in names}
        src.close()
        for i in range(SMALL["n_layers"]):
            p = f"L{i}."
            for n, rows in (("moe.router", SMALL["n_experts"]), ("moe.shared_gate", 1)):
                w, s, b = _q8(t.pop(p + n).view(np.float16).reshape(rows, -1))
                t.update({p + n + ".w": w, p + n + ".s": s, p + n + ".b": b})
            if p + "gdn.norm" in t:
                t[p + "gdn.norm.f32"] = t.pop(p + "gdn.norm").view(np.float16).astype(np.float32) * np.float32(1.0003)
        _engines["small"] = Q.Engine.from_tensors(Q.config(**SMALL, **room), t)
    return _engines["small"]


# ---------------------------------------------------------------------------------------------- the cases
def listed():
    return [
        # the operator alone at the size of the reference's kernel test: one decode row, 2048 -> 4096
        {"name": "matmul_1", "kind": "matmul", "rows": 1, "k": 2048, "n": 4096},
        # a two-layer model's decode step: all latency
        {"name": "small_step", "kind": "small", "context": 64},
        # the headline: single-stream greedy decode after a 512-token prompt
        {"name": "step_512", "kind": "step", "context": 512},
        # the same at long context, chained on the device as a host does between stop checks
        {"name": "chain_8192", "kind": "chain", "context": 8192, "steps": 8},
        # speculative sampling of a short draft (4 rows), nucleus 0.95 with penalties
        {"name": "sample_4", "kind": "sample", "rows": 4, "context": 700, "top_p": 0.95, "penalties": True},
        # the longest verify call of the speculative loop
        {"name": "verify_17", "kind": "verify", "rows": 17, "context": 1000},
        # a server under light load, an odd number of streams
        {"name": "batch_7", "kind": "batch", "streams": 7, "context": 200},
        # the full batch of the continuous-batching configuration
        {"name": "batch_64", "kind": "batch", "streams": 64, "context": 192},
        # a short chat turn, odd length
        {"name": "prompt_129", "kind": "prompt", "tokens": 129},
        # a long ragged prompt: two whole calls and a remainder
        {"name": "prompt_2900", "kind": "prompt", "tokens": 2900},
        # the benchmark's prompt through the strict forward
        {"name": "strict_512", "kind": "strict", "tokens": 512},
        # a 1024-token prefix saved and restored (the shared prefix of the continuous-batching configuration)
        {"name": "prefix_1024", "kind": "prefix", "tokens": 1024},
    ]


def draw(rng):
    def size(lo, hi):
        return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.5)))))))

    kind = rng.choice(["matmul", "small", "step", "chain", "sample", "verify", "batch", "batch", "prompt", "prompt", "strict", "prefix"])
    if kind == "matmul":
        return {"kind": kind, "rows": size(1, 64), "k": rng.choice([512, 1024, 2048, 4096]), "n": 16 * size(32, 1024)}
    if kind == "small":
        return {"kind": kind, "context": size(2, 4000)}
    if kind == "step":
        return {"kind": kind, "context": size(2, 8192)}
    if kind == "chain":
        return {"kind": kind, "context": size(64, 8192), "steps": size(2, 32)}
    if kind == "sample":
        return {"kind": kind, "rows": size(1, 12), "context": size(16, 4096), "top_p": rng.choice([0.8, 0.9, 0.95, 1.0]), "penalties": rng.random() < 0.5}
    if kind == "verify":
        return {"kind": kind, "rows": size(2, 33), "context": size(16, 4096)}
    if kind == "batch":
        return {"kind": kind, "streams": size(2, 64), "context": size(16, 256)}
    if kind == "prompt":
        return {"kind": kind, "tokens": size(5, 2900)}
    if kind == "strict":
        return {"kind": kind, "tokens": size(9, 512)}
    return {"kind": kind, "tokens": size(16, 1500)}


# ---------------------------------------------------------------------------------------------- inputs
def _tokens(seed, name, n, vocab=V):
    return Q.ops.synth_tokens(seed, "perf." + name, n, vocab)


def _filled(eng, tokens):
    """A stream that has taken a prompt in prefill mode, as a server's streams have."""
    st = eng.stream(MAX_LEN)
    step = min(CHUNK, eng.cfg.max_rows)
    for i in range(0, len(tokens), step):
        st.forward_hybrid(tokens[i:i + step], want_hidden=False)
    return st


def _matmul_weights(gen, n, k):
    """N(0, 0.02) weights quantised to 4 bits per group of 64 and packed eight to a word, low nibble first."""
    w = (torch.randn(n, k // 64, 64, generator=gen, device="cuda") * 0.02).half().float()
    lo, hi = w.amin(dim=2, keepdim=True), w.amax(dim=2, keepdim=True)
    s, b = ((hi - lo) / 15.0).half(), lo.half()
    q = ((w - b.float()) / s.float()).round_().clamp_(0, 15).to(torch.int64).view(n, k // 8, 8)
    packed = (q << (4 * torch.arange(8, device="cuda"))).sum(dim=2)
    packed = torch.where(packed >= 1 << 31, packed - (1 << 32), packed).to(torch.int32).contiguous()
    return packed, s.view(n, k // 64).contiguous(), b.view(n, k // 64).contiguous()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "matmul":
        m, k, n = case["rows"], case["k"], case["n"]
        gen = torch.Generator(device="cuda").manual_seed(seed)
        w, s, b = _matmul_weights(gen, n, k)
        wr = torch.empty(n // 16 * (k // 128) * 1024, dtype=torch.uint8, device="cuda")
        sr = torch.empty(n // 16 * (k // 128) * 128, dtype=torch.uint8, device="cuda")
        rc = Q.lib().sl_op_repack_q4_device(w.data_ptr(), s.data_ptr(), b.data_ptr(), k, n, wr.data_ptr(), sr.data_ptr(),
                                            torch.cuda.current_stream().cuda_stream)
        if rc != 0:
            raise Q.SeedlessError(rc, "sl_op_repack_q4_device")
        x = torch.randn(m, k, generator=gen, device="cuda").half()
        torch.cuda.synchronize()                   # the unpacked weights go away here
        return {"kind": kind, "m": m, "k": k, "n": n, "wr": wr, "sr": sr, "x": x, "y": torch.empty(m, n, dtype=torch.float16, device="cuda")}
    if kind == "small":
        eng = _small_model()
        st = _filled(eng, _tokens(seed, "small", case["context"], SMALL["vocab"]))
        return {"kind": "step", "stream": st, "last": [int(_tokens(seed, "small.next", 1, SMALL["vocab"])[0])]}
    eng = _model()
    if kind == "step":
        st = _filled(eng, _tokens(seed, "step", case["context"]))
        return {"kind": kind, "stream": st, "last": [int(_tokens(seed, "step.next", 1)[0])]}
    if kind == "chain":
        st = _filled(eng, _tokens(seed, "chain", case["context"]))
        return {"kind": kind, "stream": st, "steps": case["steps"], "last": int(_tokens(seed, "chain.next", 1)[0])}
    if kind in ("sample", "verify"):
        rows = case["rows"]
        s = {"kind": kind, "stream": _filled(eng, _tokens(seed, kind, case["context"])), "tokens": _tokens(seed, kind + ".rows", rows)}
        if kind == "sample":
            s["draft"] = np.concatenate([s["tokens"][1:], np.array([-1], dtype=np.int32)]).astype(np.int32)
            s["adj"] = None
            if case["penalties"]:                  # a repetition penalty on the tokens seen so far
                s["adj"] = np.zeros(V, dtype=np.float32)
                s["adj"][_tokens(seed, kind, case["context"])] = -0.5
            s.update(top_p=case["top_p"], seed=seed & 0xFFFFFFFF, pos=case["context"])
        return s
    if kind == "batch":
        # prompts around the stated length, all different (half to one and a half of it)
        b, c = case["streams"], case["context"]
        lens = [max(1, c // 2 + (37 * g + seed) % (c + 1)) for g in range(b)]
        streams = [_filled(eng, _tokens(seed, f"batch.{g}", n)) for g, n in enumerate(lens)]
        return {"kind": kind, "engine": eng, "streams": streams, "last": _tokens(seed, "batch.next", b)}
    if kind in ("prompt", "strict"):
        n = case["tokens"]
        return {"kind": kind, "engine": eng, "stream": eng.stream(n + 64), "tokens": _tokens(seed, kind, n)}
    if kind == "prefix":
        n = case["tokens"]
        return {"kind": kind, "from": _filled(eng, _tokens(seed, "prefix", n)), "to": eng.stream(n + 64)}
    raise ValueError(kind)


# ---------------------------------------------------------------------------------------------- one pass
def run(state):
    kind = state["kind"]
    if kind == "matmul":
        rc = Q.lib().sl_op_qmm4_device(state["x"].data_ptr(), state["wr"].data_ptr(), state["sr"].data_ptr(), state["m"], state["k"], state["n"],
                                       state["y"].data_ptr(), torch.cuda.current_stream().cuda_stream)
        if rc != 0:
            raise Q.SeedlessError(rc, "sl_op_qmm4_device")
        return state["y"]
    if kind == "step":                             # the stream goes on with the token it has just produced
        state["last"] = state["stream"].step_argmax(state["last"])
        return state["last"]
    if kind == "chain":
        out = state["stream"].chained_step_argmax(state["last"], state["steps"])
        state["last"] = int(out[-1])
        return out
    if kind == "verify":                           # the draft is rejected: back to where the call began
        st = state["stream"]
        snap = st.snapshot()
        out = st.step_argmax(state["tokens"])
        st.rollback(snap)
        return out
    if kind == "sample":
        st = state["stream"]
        snap = st.snapshot()
        out = st.step_sample_rows(state["tokens"], state["draft"], 1.0 / 0.7, state["top_p"], state["seed"], 7, state["pos"], logit_adj=state["adj"])
        st.rollback(snap)
        return out
    if kind == "batch":
        state["last"] = state["engine"].batch_step_argmax(state["streams"], state["last"])
        return state["last"]
    if kind == "prompt":
        st, toks = state["stream"], state["tokens"]
        st.reset()
        hidden = None
        for i in range(0, len(toks), CHUNK):
            hidden = st.forward_hybrid(toks[i:i + CHUNK], want_hidden=i + CHUNK >= len(toks))
        return {"hidden": hidden, "token": state["engine"].lm_head_argmax(hidden[-1:])}
    if kind == "strict":
        st = state["stream"]
        st.reset()
        return {"hidden": st.forward(state["tokens"])}
    if kind == "prefix":
        blob = state["from"].state_save()
        if not state["to"].state_restore(blob):
            raise RuntimeError("the blob was refused")
        return blob
    raise ValueError(kind)


# ---------------------------------------------------------------------------------------------- what a pass cannot do without
def _step_work(rows, streams, context, head_rows, layers=LAYERS):
    """One call of `rows` rows over `streams` streams at a mean context: weights once (the experts that the rows are
    expected to touch), GDN state and history read and written, keys and values read, outputs of the head."""
    gdn = (GDN_IN + GDN_VAL) * H
    att = (ATT_IN + ATT_OUT) * H
    expert = 3 * I * H
    touched = E * (1.0 - (1.0 - TOPK / E) ** rows)
    f = layers / LAYERS
    weights = Q4 * (N_GDN * gdn + N_ATT * att + LAYERS * (touched + 1) * expert) + LAYERS * (E + 1) * H * 2
    state = streams * N_GDN * 2 * (STATE_BYTES + HIST_BYTES)
    kv = N_ATT * KV_BYTES * (streams * context + rows)
    b = f * (weights + state + kv) + (V * H * Q4 if head_rows else 0) + rows * H * 2
    per_row = N_GDN * (gdn + 3 * 32 * 128 * 128) + N_ATT * (att + 2 * 16 * 256 * context) + LAYERS * ((TOPK + 1) * expert + E * H)
    return {"bytes": b, "flops": 2.0 * (f * rows * per_row + head_rows * V * H)}


def work(case):
    kind = case["kind"]
    if kind == "matmul":
        m, k, n = case["rows"], case["k"], case["n"]
        return {"bytes": n * k * Q4 + 2 * m * (k + n), "flops": 2.0 * m * n * k}
    if kind == "small":                            # one GDN and one attention layer, 8 of 16 experts and the shared one each
        b = Q4 * ((GDN_IN + GDN_VAL + ATT_IN + ATT_OUT) * H + 2 * 9 * 3 * I * H + SMALL["vocab"] * H) + 2 * (STATE_BYTES + HIST_BYTES) + KV_BYTES * case["context"]
        return {"bytes": b + 2 * 17 * H, "flops": 4.0 * b}
    if kind == "step":
        return _step_work(1, 1, case["context"], 1)
    if kind == "chain":
        one = _step_work(1, 1, case["context"] + case["steps"] / 2, 1)
        return {k: v * case["steps"] for k, v in one.items()}
    if kind == "verify":
        return _step_work(case["rows"], 1, case["context"], case["rows"])
    if kind == "sample":
        w = _step_work(case["rows"], 1, case["context"], case["rows"])
        return {"bytes": w["bytes"] + (4 * V if case["penalties"] else 0), "flops": w["flops"]}
    if kind == "batch":
        return _step_work(case["streams"], case["streams"], case["context"], case["streams"])
    if kind == "prompt":
        return _step_work(case["tokens"], 1, case["tokens"] / 2, 1)
    if kind == "strict":
        return _step_work(case["tokens"], 1, case["tokens"] / 2, 0)
    blob = N_GDN * (STATE_BYTES + HIST_BYTES) + N_ATT * KV_BYTES * case["tokens"]
    return {"bytes": 4.0 * blob, "flops": 0.0}     # read and written by the save, and again by the restore


def tolerance(case):
    if case["kind"] in ("matmul", "prompt", "strict"):
        return {"rel": 2e-3, "max": 2e-2}          # fp16 outputs of f32 sums
    return "exact"                                 # tokens and bytes
