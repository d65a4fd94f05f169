"""The work that this package is used for, as cases that can be timed and compared.

A case names one call of the public surface and its sizes: a request through `Engine`
(`generate`, `generate_spec`, `sequence_logits`), one of the operators that a host calls directly
(`_w4.gemv`, `_w4.gemm`, `_C.gemv_bf16`), or the packing of a checkpoint's matrices
(`W4Linear.prepare`, `prepare_gate_up`). `listed()` holds the cases that are always looked at,
`draw()` gives others of the same ranges.

Models are seeded random weights of the repository's configurations, with one thing made as it is
in a trained model: the next token stands out. Row t + 1 of the lm_head is the direction of
embedding row t, so the model counts upwards, with a margin between the best and the second-best
logit that rounding does not close (on plain random weights the best two logits are often equal in
bf16, and everything behind such a tie is a matter of luck). The draft layer passes its token's
embedding on, so its drafts are good and verify passes keep several rows, as they do in use.
"""
import math

import torch

from qengine_b200 import _C, _w4, synth
from qengine_b200.engine import Engine, W4Linear
from qengine_b200.quant import W4Packed, dequantize_w4, quantize_w4

DEV = "cuda"
BF16 = torch.bfloat16
PER_WEIGHT = 0.5 + 2.0 / 128  # bytes: a nibble, and a 2-byte scale per 128
SCALE = 0.002      # W4 scales ~ |N(0, 1)| * SCALE: a sub-layer adds a few tenths to the residual stream
EMBED_STD = 24.0   # of the embedding rows: what 128 sub-layers add up to does not drown the token
DRAFT_STD = 12.0   # of the draft layer's input


# ---- the cases ------------------------------------------------------------------------------------
def _request(name=None, model="27b", layers=16, prompt=24, new=24, k=0, wide=False, context=0):
    """One request to an engine: `prompt` tokens behind `context` cached positions, then `new`
    tokens; k drafts per cycle (0: plain decoding); wide: the prompt in 64-row passes."""
    c = {"kind": "request", "model": model, "layers": layers, "prompt": prompt, "new": new, "k": k, "wide": wide,
         "context": context}
    return {"name": name, **c} if name else c


def _score(name=None, model="27b", layers=16, tokens=200):
    c = {"kind": "score", "model": model, "layers": layers, "tokens": tokens}
    return {"name": name, **c} if name else c


def _op(kind, name=None, **sizes):
    c = {"kind": kind, **sizes}
    return {"name": name, **c} if name else c


def listed():
    return [
        # The CPU-sized model (4 layers, hidden 512), 32-token prompt, 64 tokens: nothing but launches
        # and latency; what a test, a demo or a tiny draft model sees.
        _request("tiny_generate", model="tiny", layers=4, prompt=32, new=64),
        # Batch-1 greedy decoding of the whole 27B-shape model: the headline use.
        _request("decode_27b", layers=64, prompt=24, new=32),
        # The same model with the draft layer, 4 drafts per cycle, in the middle of a chat (3,000
        # positions cached): verify passes of 5 rows, draft passes of 5 and 1, rollback bookkeeping.
        _request("spec4_27b_chat", layers=64, prompt=17, new=60, k=4, context=3000),
        # Decoding behind a long document: the K/V caches are most of what a token reads. 16 layers of
        # the 27B shape (every layer is like every fourth one; only the depth is less).
        _request("decode_32k", prompt=9, new=24, context=32000),
        # Reading a prompt of about a thousand tokens in wide passes, up to the first token.
        _request("prompt_1k_wide", prompt=1021, new=1, wide=True),
        # Teacher-forced scoring of a text (perplexity): 8-row passes, the logits of every position.
        _score("score_203", tokens=203),
        # The operators by themselves, as a host that brings its own engine calls them. The smallest
        # matrix: the cost of a call.
        _op("gemv", "gemv_small", rows=1, M=512, K=512, swiglu=False),
        # Five rows (a verify pass) on a matrix whose sides are no multiple of anything.
        _op("gemv", "gemv_ragged", rows=5, M=5001, K=3407, swiglu=False),
        # 64 rows of a prompt through the 27B gate/up matrix.
        _op("gemm", "gemm_gate_up_64", rows=64, M=17408, K=5120, swiglu=True),
        # An lm_head left in bf16 (a quarter of the vocabulary, the shard of one of four ranks).
        _op("gemv_bf16", "bf16_head", rows=3, M=62080, K=5120),
        # Packing a checkpoint: the gate and up matrices of one layer.
        _op("pack", "pack_gate_up", M=17408, K=5120, gate_up=True, dtype="bf16"),
    ]


def _spread(rng, lo, hi):
    """A whole number whose logarithm is spread evenly over [lo, hi]."""
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    kind = rng.choice(["request"] * 5 + ["score", "gemv", "gemv", "gemm", "gemv_bf16", "pack"])
    if kind == "request":
        model = rng.choice(["tiny", "small", "27b", "27b", "27b"])
        layers = 4 if model != "27b" else rng.choice([4, 8, 12, 16])
        wide = rng.random() < 0.4
        return _request(model=model, layers=layers, prompt=_spread(rng, 8, 1200 if wide else 160),
                        new=_spread(rng, 4, 80), k=rng.choice([0, 0, 1, 2, 3, 4, 5]), wide=wide,
                        context=rng.choice([0, 0, _spread(rng, 100, 4000), _spread(rng, 4000, 33000)]))
    if kind == "score":
        return _score(model=rng.choice(["small", "27b"]), layers=rng.choice([4, 8]), tokens=_spread(rng, 9, 300))
    if kind == "gemv":
        return _op(kind, rows=rng.randint(1, 8), M=_spread(rng, 200, 34816), K=_spread(rng, 256, 17408),
                   swiglu=rng.random() < 0.3)
    if kind == "gemm":
        return _op(kind, rows=_spread(rng, 9, 64), M=_spread(rng, 512, 17408), K=128 * _spread(rng, 4, 136),
                   swiglu=rng.random() < 0.3)
    if kind == "gemv_bf16":
        return _op(kind, rows=rng.randint(1, 8), M=_spread(rng, 500, 124160), K=8 * _spread(rng, 64, 640))
    return _op(kind, M=_spread(rng, 200, 17408), K=_spread(rng, 200, 8192), gate_up=rng.random() < 0.4,
               dtype=rng.choice(["bf16", "bf16", "fp32"]))


# ---- models -----------------------------------------------------------------------------------------
def _config(case):
    if case["model"] == "tiny":
        return synth.tiny_config()
    if case["model"] == "small":
        return synth.shardable8_config()
    return synth.qwen27b_config(layers=case["layers"])


def _centre(p):
    """Code 0 becomes code 8 (the number zero) in every nibble: uniform codes 0..15 have the mean -1/2,
    which no trained matrix has, and which 64 layers add up to one large common vector."""
    w = p.qw
    zero = w | (w >> 1)
    zero |= zero >> 2
    w |= ((zero & 0x11111111) ^ 0x11111111) << 3


@torch.no_grad()
def _counting_model(cfg, seed, mtp):
    """Seeded random weights whose greedy continuation of token t is t + 1."""
    W = synth.build_model(cfg, seed=seed, device=DEV, scale_std=SCALE, mtp=mtp)
    head, V, H = W["lm_head"], cfg.vocab, cfg.hidden
    for L in W["layers"] + [W] + ([W["mtp"]] if mtp else []):
        for m in L.values():
            if isinstance(m, W4Packed):
                _centre(m)
    gain = EMBED_STD / (SCALE * math.sqrt(17.5))  # 17.5: mean square of such a code minus 8
    for r0 in range(0, V, 8192):
        r1 = min(V, r0 + 8192)
        part = W4Packed(head.qw[r0 // 16:r1 // 16], head.scales[r0 // 16:r1 // 16], r1 - r0, H)
        rows = (dequantize_w4(part) * gain).to(BF16)
        if r0 == 0:
            W["embed"][V - 1].copy_(rows[0])
            rows = rows[1:]
        W["embed"][r1 - 1 - rows.shape[0]:r1 - 1].copy_(rows)
    if mtp:
        fc = torch.zeros(H, 2 * H, device=DEV)
        g = torch.Generator(device=DEV).manual_seed(seed + 1)
        fc[:, H:] = torch.randn(H, H, generator=g, device=DEV) * (0.1 / math.sqrt(H))
        fc[:, :H].fill_diagonal_(DRAFT_STD)
        W["mtp"]["fc"] = quantize_w4(fc)
    return W


def _engine(case, seed):
    cfg = _config(case)
    k = case.get("k", 0)
    need = case.get("context", 0) + case.get("prompt", case.get("tokens", 0)) + case.get("new", 0) + 64
    eng = Engine(cfg, _counting_model(cfg, seed, mtp=k > 0), max_len=max(4096, -(-need // 256) * 256))
    if case.get("context"):
        eng.set_context(case["context"], seed=seed)
    return cfg, eng


def _normal(seed, *shape):
    return torch.randn(*shape, generator=torch.Generator(device=DEV).manual_seed(seed), device=DEV)


def _random_packed(case, seed):
    """A packed matrix of any size (through the packer, which pads it), and rows to multiply."""
    M, K = case["M"], case["K"]
    if case["swiglu"]:
        p = W4Linear().prepare_gate_up(_normal(seed, M, K) * 0.02, _normal(seed + 1, M, K) * 0.02)
    else:
        p = W4Linear().prepare(_normal(seed, M, K) * 0.02)
    return p, _normal(seed + 2, case["rows"], K).to(BF16)


# ---- prepare / run ----------------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind in ("request", "score"):
        cfg, eng = _engine(case, seed)
        n = case["prompt"] if kind == "request" else case["tokens"]
        state = {"kind": kind, "case": case, "eng": eng, "ids": synth.prompt_ids(n, cfg.vocab - 256, seed=seed)}
        # a serving program has answered requests of this size before: its graphs are captured
        warm = dict(state, ids=synth.prompt_ids(n, cfg.vocab - 256, seed=seed + 7))
        run(warm)
        return state
    if kind in ("gemv", "gemm"):
        p, x = _random_packed(case, seed)
        return {"kind": kind, "p": p, "x": x, "out": torch.empty(case["rows"], case["M"], dtype=BF16, device=DEV)}
    if kind == "gemv_bf16":
        w = torch.empty(case["M"], case["K"], dtype=BF16, device=DEV)
        w.normal_(0.0, 0.02, generator=torch.Generator(device=DEV).manual_seed(seed))
        return {"kind": kind, "w": w, "x": _normal(seed + 1, case["rows"], case["K"]).to(BF16),
                "out": torch.empty(case["rows"], case["M"], dtype=BF16, device=DEV)}
    dt = BF16 if case["dtype"] == "bf16" else torch.float32
    mats = [(_normal(seed + i, case["M"], case["K"]) * 0.02).to(dt) for i in range(2 if case["gate_up"] else 1)]
    return {"kind": kind, "mats": mats, "lin": W4Linear()}


def run(state):
    kind = state["kind"]
    if kind == "request":
        return _run_request(state["eng"], state["case"], state["ids"])
    if kind == "score":
        return state["eng"].sequence_logits(state["ids"])
    if kind == "gemv":
        p, x, out = state["p"], state["x"], state["out"]
        (_w4.gemv_swiglu if p.gate_up else _w4.gemv)(x, p.qw, p.scales, out, p.M)
        return out
    if kind == "gemm":
        p, x, out = state["p"], state["x"], state["out"]
        _w4.gemm(x, p.qw, p.scales, out, p.M, swiglu=p.gate_up)
        return out
    if kind == "gemv_bf16":
        _C.gemv_bf16(state["w"], state["x"], state["out"])
        return state["out"]
    p = (state["lin"].prepare_gate_up if len(state["mats"]) == 2 else state["lin"].prepare)(*state["mats"])
    return {"qw": p.qw, "scales": p.scales}


def _run_request(eng, case, ids):
    if case["k"]:
        tokens = eng.generate_spec(ids, case["new"], case["k"], wide=case["wide"])
    else:
        tokens = eng.generate(ids, case["new"], wide=case["wide"])
    out = {"tokens": torch.tensor(tokens), "logits": eng.logits[:case["k"] + 1]}
    # what the request leaves behind: DeltaNet states and K/V caches, layer by layer (64 outputs at most)
    for i, L in enumerate(eng.layers):
        for name in ("S",) if len(eng.layers) > 40 else ("S", "kc", "vc"):
            if name in L:
                out[f"layer{i:02d}.{name}"] = L[name]
    return out


# ---- what a pass cannot do without ------------------------------------------------------------------
def _model_sizes(case):
    """(packed bytes of the decoder, of the lm_head, of the draft layer; K/V bytes per cached position;
    bytes of the DeltaNet states)."""
    cfg = _config(case)
    per = PER_WEIGHT
    mlp = 3 * cfg.hidden * cfg.inter
    lin = cfg.hidden * cfg.gdn_proj_rows + cfg.hidden * cfg.value_dim
    att = cfg.hidden * cfg.attn_proj_rows + cfg.hidden * cfg.hq * cfg.head_dim
    n_att = sum(t == "full_attention" for t in cfg.layer_types)
    n_lin = len(cfg.layer_types) - n_att
    kv = cfg.hkv * cfg.head_dim * 2 * 2
    return {"decoder": per * (n_lin * lin + n_att * att + len(cfg.layer_types) * mlp), "head": per * cfg.vocab * cfg.hidden,
            "draft": per * (att + mlp + 2 * cfg.hidden * cfg.hidden), "kv": n_att * kv, "kv_draft": kv,
            "state": n_lin * cfg.hv * cfg.dk * cfg.dv * 4, "vocab": cfg.vocab}


def work(case):
    kind = case["kind"]
    if kind == "request":
        s, k, P, new = _model_sizes(case), case["k"], case["prompt"], case["new"]
        length = case["context"] + P + new / 2
        # the prompt in one pass over the weights, then a pass per token (per k + 1 tokens with drafts)
        later = new - 1 if k == 0 else -(-(new - 1) // (k + 1))
        one = s["decoder"] + s["head"] + s["kv"] * length + 2 * s["state"]
        drafts = k * (s["draft"] + s["head"] + s["kv_draft"] * length)
        rows = P + (k + 1) * later
        flops = 2.0 / PER_WEIGHT * (rows * s["decoder"] + (1 + (k + 1) * later) * s["head"] + k * (1 + later) * (s["draft"] + s["head"]))
        return {"bytes": (1 + later) * (one + drafts), "flops": flops}
    if kind == "score":
        s, T = _model_sizes(case), case["tokens"]
        return {"bytes": s["decoder"] + s["head"] + 2 * s["state"] + s["kv"] * T + 2.0 * T * s["vocab"],
                "flops": 2.0 / PER_WEIGHT * T * (s["decoder"] + s["head"])}
    M, K = case["M"], case["K"]
    if kind in ("gemv", "gemm"):
        mats = 2 if case["swiglu"] else 1
        return {"bytes": mats * M * K * PER_WEIGHT + 2.0 * case["rows"] * (M + K), "flops": 2.0 * mats * M * K * case["rows"]}
    if kind == "gemv_bf16":
        return {"bytes": 2.0 * M * K + 2.0 * case["rows"] * (M + K), "flops": 2.0 * M * K * case["rows"]}
    mats, size = (2 if case["gate_up"] else 1), (2 if case["dtype"] == "bf16" else 4)
    return {"bytes": mats * M * K * (size + PER_WEIGHT), "flops": 3.0 * mats * M * K}


def tolerance(case):
    """What the order of the sums alone does, times four. Measured: requests with half the warps per
    block in every W4 GEMV (another split of every sum), prompts in 8-row against wide passes; rel over
    the outputs with the largest figure (the states of the deepest layers). Operators against fp64,
    rounded to bf16: a few outputs in a thousand are one bf16 step apart."""
    kind = case["kind"]
    if kind == "pack":
        return "exact"
    if kind == "request":  # 64 layers: 0.0094 and 0.28; 16 layers: 0.0055 and 0.12
        return {"rel": 0.03, "max": 0.9} if case["layers"] > 16 else {"rel": 0.022, "max": 0.5}
    if kind == "score":  # 0.0027 and 0.019
        return {"rel": 0.011, "max": 0.08}
    return {"rel": 2e-4, "max": 0.027}  # 3e-5 and 0.0067
