"""The mixers of a prefill pass (up to 64 rows per launch) against the 8-row calls they stand for.

Both are the same arithmetic in the same order, so everything is compared bit for bit.
"""
from __future__ import annotations

import pytest
import torch

from test_mixers_gpu import BF, GdnLayer, dev, gdn_cfg, gdn_rows, gdn_weights

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def C():
    from qengine_b200 import _C
    return _C


def steps(L, rows):
    return torch.cat([L.run(rows[i:i + 8], 8) for i in range(0, rows.shape[0], 8)])


def prefill(L, rows):
    cfg, n = L.cfg, rows.shape[0]
    c0, c1 = cfg.conv_dim, cfg.conv_dim + cfg.value_dim
    r = rows.to(dev)[:, :c1 + 2 * cfg.hv]
    out = torch.empty(n, cfg.value_dim, dtype=BF, device=dev)
    L.C.gdn_prefill(r[:, :c0], r[:, c0:c1], r[:, c1:c1 + cfg.hv], r[:, c1 + cfg.hv:], L.ring, L.W["conv_w"],
                    L.W["A_log"], L.W["dt_bias"], L.W["norm_w"], L.S, *L.st, L.ctl, out, cfg.hk, 1e-6)
    L.ctl[0] += n
    L.ctl[1] = 8
    return out


def split(L, rows, wire):
    """`gdn_rows`: the same in four launches."""
    from qengine_b200 import _w4
    cfg, n = L.cfg, rows.shape[0]
    c0, c1 = cfg.conv_dim, cfg.conv_dim + cfg.value_dim
    r = rows.to(dev)[:, :c1 + 2 * cfg.hv]
    out = torch.empty(n, cfg.value_dim, dtype=BF, device=dev)
    size = L.C.gdn_rows_workspace(n, cfg.hk, cfg.hv, cfg.dk)
    ws = torch.full((size + 64,), 255, dtype=torch.uint8, device=dev)
    L.C.gdn_rows(r[:, :c0], r[:, c0:c1], r[:, c1:c1 + cfg.hv], r[:, c1 + cfg.hv:], L.ring, L.W["conv_w"],
                 L.W["A_log"], L.W["dt_bias"], L.W["norm_w"], L.S, *L.st, L.ctl, out, cfg.hk, 1e-6, ws[:size], wire)
    assert (ws[size:] == 255).all()
    L.ctl[0] += n
    L.ctl[1] = 8
    return _w4.wire_order(out) if wire else out


@pytest.mark.parametrize("hk,hv,d", [(16, 48, 128), (2, 4, 64), (1, 1, 128), (1, 3, 64)])
@pytest.mark.parametrize("before,n", [(0, 8), (3, 24), (21, 40), (8, 64), (5, 72), (1, 128)])
def test_deltanet_rows_equal_the_8_row_steps(C, hk, hv, d, before, n):
    cfg, g = gdn_cfg(hk, hv, d), torch.Generator().manual_seed(before * 100 + n)
    W = gdn_weights(cfg, seed=d)
    A, B = GdnLayer(C, cfg, W), GdnLayer(C, cfg, W)
    first, rows, last = (gdn_rows(cfg, k, g) for k in (before, n, 5))
    for L in (A, B):
        for i in range(0, before, 8):
            L.run(first[i:i + 8], min(8, before - i))
    want, got = steps(A, rows), split(B, rows, wire=n % 16 == 0)
    assert torch.equal(want, got)
    for a, b in zip((A.S, A.ring, A.ctl, *A.st), (B.S, B.ring, B.ctl, *B.st)):
        assert torch.equal(a, b)
    assert torch.equal(A.run(last, 5), B.run(last, 5))


@pytest.mark.parametrize("hk,hv,d", [(16, 48, 128), (2, 4, 64), (1, 1, 128)])
@pytest.mark.parametrize("before,n", [(0, 8), (0, 16), (3, 24), (8, 64), (21, 40), (1, 64)])
def test_deltanet_prefill_equals_the_8_row_steps(C, hk, hv, d, before, n):
    """Empty and non-empty history (conv ring, 1 .. 8 pending rows), then n rows in one launch, then an
    ordinary step on what they left (checkpoints, ring, state)."""
    cfg, g = gdn_cfg(hk, hv, d), torch.Generator().manual_seed(before * 100 + n)
    W = gdn_weights(cfg, seed=d)
    A, B = GdnLayer(C, cfg, W), GdnLayer(C, cfg, W)
    first, rows, last = (gdn_rows(cfg, k, g) for k in (before, n, 5))
    for L in (A, B):
        for i in range(0, before, 8):
            L.run(first[i:i + 8], min(8, before - i))
    want, got = steps(A, rows), prefill(B, rows)
    assert torch.equal(want, got)
    for a, b in zip((A.S, A.ring, A.ctl, *A.st), (B.S, B.ring, B.ctl, *B.st)):
        assert torch.equal(a, b)
    assert torch.equal(A.run(last, 5), B.run(last, 5))


@pytest.mark.parametrize("n", [0, 4, 12, 72])
def test_deltanet_prefill_refuses_other_row_counts(C, n):
    cfg = gdn_cfg(1, 1, 64)
    with pytest.raises(RuntimeError):
        prefill(GdnLayer(C, cfg, gdn_weights(cfg)), gdn_rows(cfg, n, torch.Generator().manual_seed(1)))


@pytest.mark.parametrize("hq,hkv,hd,NS", [(24, 4, 256, 16), (4, 2, 64, 6), (5, 1, 128, 7)])
@pytest.mark.parametrize("pos,n", [(0, 8), (0, 64), (37, 40), (300, 33), (470, 64)])
def test_attention_rows_equal_the_8_row_calls(C, hq, hkv, hd, NS, pos, n):
    """The last case runs past the end of the cache (512 positions)."""
    g = torch.Generator(device=dev).manual_seed(pos + n)
    max_len, rd = 512, 32
    rand = lambda *s: torch.randn(*s, generator=g, device=dev).to(BF)
    width = hq * 2 * hd + 2 * hkv * hd
    proj = rand(n, width + 8)[:, :width]
    nq, nk = hq * 2 * hd, hq * 2 * hd + hkv * hd
    qn, kn = rand(hd) * 0.1, rand(hd) * 0.1
    inv = 1e4 ** (-torch.arange(0, rd, 2, device=dev).float() / rd)
    kc0, vc0 = rand(hkv, max_len, hd), rand(hkv, max_len, hd)
    res = []
    for rows in (8, 64):
        kc, vc = kc0.clone(), vc0.clone()
        q, out = (torch.zeros(n, hq * hd, dtype=BF, device=dev) for _ in range(2))
        po, ml = torch.zeros(rows, hq, NS, hd, device=dev), torch.zeros(rows, hq, NS, 2, device=dev)
        prep, dec = (C.attn_prep, C.attn_decode) if rows == 8 else (C.attn_prep_rows, C.attn_decode_rows)
        for i in range(0, n, rows):
            p = torch.tensor([pos + i], dtype=torch.int32, device=dev)
            r = proj[i:i + rows]
            prep(r[:, :nq], r[:, nq:nk], r[:, nk:], qn, kn, inv, p, q[i:i + rows], kc, vc, 1e-6)
            dec(q[i:i + rows], kc, vc, p, r[:, :nq], po, ml, out[i:i + rows])
        res.append((q, out, kc, vc))
    for a, b in zip(*res):
        assert torch.equal(a.view(torch.int16), b.view(torch.int16))


def test_attention_rows_refuse_the_tensor_core_split(C):
    z = lambda *s, dt=BF: torch.zeros(*s, dtype=dt, device=dev)
    p = torch.zeros(1, dtype=torch.int32, device=dev)
    with pytest.raises(RuntimeError):
        C.attn_decode_rows(z(16, 256), z(1, 64, 256), z(1, 64, 256), p, z(16, 512), z(16, 1, 6, 256, dt=torch.float32),
                           z(16, 1, 6, 2, dt=torch.float32), z(16, 256))
