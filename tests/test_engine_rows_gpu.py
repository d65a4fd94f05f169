"""Passes of up to 128 rows (Engine._row_blocks) leave, bit for bit, what passes of 8 rows leave."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


def build(kind, **kw):
    from qengine_b200 import synth
    from qengine_b200.engine import Engine, W4Linear
    cfg = {"tiny": synth.tiny_config, "small": synth.shardable8_config, "27b": lambda: synth.qwen27b_config(layers=4)}[kind]()
    W = synth.build_model(cfg, seed=5, device="cuda")
    if "warps" in kw:
        kw["linear"] = W4Linear(warps=kw.pop("warps"))
    return cfg, Engine(cfg, W, **{"max_len": 512, **kw})


def snapshot(eng, P):
    out = {"ctl": eng.ctl.clone(), "logits": eng.logits.clone(), "hid": eng.hid.clone(), "drafts": eng.drafts.clone(),
           "next": eng.next_tok.clone(), "log": eng.log[P:].clone()}
    for i, L in enumerate(eng.layers + ([eng.mtp] if eng.has_mtp else [])):
        for name in ("S", "st_k", "st_v", "st_g", "ring"):
            if name in L:
                out[f"{i}.{name}"] = L[name].clone()
        for name in ("kc", "vc"):
            if name in L:
                out[f"{i}.{name}"] = L[name][:, :P].clone()
    return out


def run(eng, prompt, exact, mtp, k, **kw):
    eng.rows_ok = (lambda: True) if exact else (lambda: False)
    assert bool(eng._row_blocks(len(prompt))) == exact
    eng._need_prompt(len(prompt), mtp, k, 8, None, set())
    eng.reset()
    if eng.start_pos:
        eng.set_context(eng.start_pos, seed=3)
    eng.prefill(prompt, mtp=mtp, k=k, **kw)
    torch.cuda.synchronize()
    eng._check_device_errors()
    return snapshot(eng, eng.start_pos + len(prompt))


@pytest.mark.parametrize("kind,P,kw", [("tiny", 33, {}), ("tiny", 129, {}), ("tiny", 300, {}), ("small", 211, {}),
                                       ("27b", 40, {}), ("27b", 153, {}), ("tiny", 150, {"warps": 8}),
                                       ("tiny", 140, {"attn_splits": 300}), ("27b", 145, {"max_len": 9000, "context": 1000})])
def test_state_after_a_prompt(kind, P, kw):
    from qengine_b200 import synth
    kw = dict(kw)
    context = kw.pop("context", 0)
    cfg, eng = build(kind, **kw)
    assert eng.rows_ok()
    if context:
        eng.set_context(context, seed=3)
    prompt = synth.prompt_ids(P, cfg.vocab, seed=6)
    for mtp, k in ((True, 2), (False, 0)):
        want, got = run(eng, prompt, False, mtp, k), run(eng, prompt, True, mtp, k)
        for name in want:
            a, b = want[name], got[name]
            assert torch.equal(a.view(torch.int16) if a.dtype == torch.bfloat16 else a,
                               b.view(torch.int16) if b.dtype == torch.bfloat16 else b), (name, mtp)


@pytest.mark.parametrize("kind,T", [("tiny", 32), ("tiny", 33), ("small", 203), ("27b", 137)])
def test_sequence_logits(kind, T):
    from qengine_b200 import synth
    cfg, eng = build(kind, mtp=False)
    seq = synth.prompt_ids(T, cfg.vocab, seed=7)
    got, best = eng.sequence_logits(seq), eng.sequence_logits(seq, keep="argmax")
    assert bool(eng._row_blocks(T)) == (T > 32) == any(key[0] == "rows" for key in eng.graphs)
    eng.rows_ok = lambda: False
    want = eng.sequence_logits(seq)
    assert torch.equal(got.view(torch.int16), want.view(torch.int16))
    assert torch.equal(best, eng.sequence_logits(seq, keep="argmax"))


def test_requests():
    """Whole requests, plain, speculative and wide; options that leave the 8-row passes alone."""
    from qengine_b200 import synth
    cfg, eng = build("tiny")
    prompt = synth.prompt_ids(293, cfg.vocab, seed=8)
    plain = eng.generate(prompt, 40)
    assert ("rows", 128, False, False) in eng.graphs and ("rows", 32, False, False) in eng.graphs  # 128 + 128 + 32
    assert eng.generate_spec(prompt, 40, 3) == plain and eng.generate(prompt, 40, chunk=5) == plain
    assert eng._row_blocks(293, 5) == [] and eng._row_blocks(293, 8, True) == [128, 128] and eng._row_blocks(32) == []
    wide = eng.generate(prompt, 40, wide=True)
    assert eng.generate_spec(prompt, 40, 4, wide=True) == wide
    _, plainer = build("tiny", fuse=False)
    assert not plainer.rows_ok() and plainer._row_blocks(293) == []
