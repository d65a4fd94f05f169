"""`_w4.gemv` / `gemv_swiglu` with default options take a short way to the launch (qe_w4_gemv_call);
the general way (`job` + `_launch`) is what it is compared with, bit for bit, over the forms both
accept, and what is refused there is refused here. Also: the two-row BF16 GEMV against single rows, and the
small merge of attention splits against the large one's arithmetic, at the sizes where they begin and end."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV, BF = "cuda", torch.bfloat16


@pytest.fixture(scope="module")
def w4():
    from qengine_b200 import _w4
    return _w4


def rand(*s, seed=0):
    return torch.randn(*s, generator=torch.Generator(device=DEV).manual_seed(seed), device=DEV)


@pytest.mark.parametrize("M,K,N", [(1, 8, 1), (16, 128, 8), (17, 130, 3), (512, 512, 1), (1000, 3407, 5), (5120, 6144, 2)])
@pytest.mark.parametrize("swiglu", [False, True])
def test_short_way_equals_the_general_one(w4, M, K, N, swiglu):
    from qengine_b200.quant import quantize_w4, quantize_w4_gate_up
    p = quantize_w4_gate_up(rand(M, K) * 0.02, rand(M, K, seed=1) * 0.02) if swiglu else quantize_w4(rand(M, K) * 0.02)
    fn = w4.gemv_swiglu if swiglu else w4.gemv
    for pad, first in ((0, 0), (8, 8), (3, 1)):  # contiguous; aligned rows; rows of any alignment
        x = rand(N, K + pad + first, seed=2).to(BF)[:, first:first + K]
        got = torch.full((N, M + pad), 7.0, dtype=BF, device=DEV)
        want = got.clone()
        before = w4.launches[0]
        fn(x, p.qw, p.scales, got[:, :M], p.M)
        assert w4.launches[0] == before + 1
        w4._launch([w4.job(x, p.qw, p.scales, want[:, :M], p.M, swiglu=swiglu)], w4._cfg(*w4._DEFAULTS), "gemv_w4")
        assert torch.equal(got.view(torch.int16), want.view(torch.int16))


def test_scratch_grows_through_the_general_way(w4):
    from qengine_b200.quant import quantize_w4
    p, x = quantize_w4(rand(5120, 6144) * 0.02), rand(1, 6144, seed=3).to(BF)
    a, b = (torch.empty(1, 5120, dtype=BF, device=DEV) for _ in range(2))
    w4.gemv(x, p.qw, p.scales, a, 5120)
    kept = w4._per_device.pop(torch.cuda.current_device())
    try:
        w4.gemv(x, p.qw, p.scales, b, 5120)  # no workspace yet
        assert torch.equal(a, b)
        W = w4._per_device[torch.cuda.current_device()]
        W.keep += [W.ws, W.counters]
        W.ws, W.counters = torch.zeros(1, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
        b.zero_()
        w4.gemv(x, p.qw, p.scales, b, 5120)  # too small a one
        assert torch.equal(a, b)
    finally:
        torch.cuda.synchronize()
        w4._per_device[torch.cuda.current_device()] = kept


def test_refusals(w4):
    from qengine_b200.quant import quantize_w4
    p = quantize_w4(rand(64, 256) * 0.02)
    x, out = rand(2, 256).to(BF), torch.empty(2, 64, dtype=BF, device=DEV)
    bad = [(x.float(), p.qw, p.scales, out, 64), (x, p.qw.long(), p.scales, out, 64), (x, p.qw, p.scales.float(), out, 64),
           (x, p.qw, p.scales, out.float(), 64), (x[:, :100], p.qw, p.scales, out, 64), (x, p.qw, p.scales, out[:1], 64),
           (x, p.qw, p.scales, out, 48), (x.cpu(), p.qw, p.scales, out, 64), (rand(9, 256).to(BF), p.qw, p.scales, out, 64),
           (x[0], p.qw, p.scales, out, 64), (x, p.qw[:2], p.scales, out, 64), (x.t(), p.qw, p.scales, out, 64),
           (x[:0], p.qw, p.scales, out[:0], 64), (None, p.qw, p.scales, out, 64)]
    for a in bad:
        with pytest.raises(RuntimeError):
            w4.gemv(*a)
    w4.gemv(x, p.qw, p.scales, out, 64)


@pytest.mark.parametrize("N", [1, 2, 7, 8, 9, 4097])
@pytest.mark.parametrize("nr,K", [(1, 8), (2, 264), (3, 1024), (8, 1032)])
def test_bf16_gemv_tile_edges(N, nr, K):
    """One weight row per warp (1, 2, 3 activation rows at these sizes) and two (8): odd last rows, and lanes
    with zero to two packets. Bound: one rounding to bf16 and K fp32 additions."""
    from qengine_b200 import _C
    W, x = rand(N, K).to(BF), rand(nr, K, seed=1).to(BF)
    ob = torch.full((nr, N + 3), 7.0, dtype=BF, device=DEV)
    _C.gemv_bf16(W, x, ob[:, :N])
    ref = x.double() @ W.double().T
    bnd = 2.0 ** -8 * ref.abs() + K * 2.0 ** -23 * (x.double().abs() @ W.double().abs().T) + 1e-30
    assert ((ob[:, :N].double() - ref).abs() <= bnd).all() and (ob[:, N:] == 7).all()


@pytest.mark.parametrize("nr,per_sm,K", [(nr, b, 72) for nr in (2, 3, 4, 5, 6, 7, 8) for b in (4, 5, 6, 7, 8, 10)] +
                         [(2, b, 1536) for b in (10, 14, 15)] + [(nr, 9, 648) for nr in (2, 3, 4)] +
                         [(3, 10, 1536), (4, 12, 1536), (5, 3, 4096), (5, 4, 4096), (5, 8, 2048), (6, 5, 3584),
                          (6, 7, 3584), (7, 5, 2048), (7, 7, 2048)])
def test_bf16_gemv_on_both_sides_of_each_rule(nr, per_sm, K):
    """The number of weight rows per warp changes with the blocks (of 8 rows) per SM and with K: a last block
    that is full, one row short, and one row alone, each with the bits of one activation row at a time."""
    from qengine_b200 import _C
    from qengine_b200._lib import lib
    edge = 8 * per_sm * lib.qe_sm_count()
    W, x = rand(edge + 8, K).to(BF), rand(nr, K, seed=1).to(BF)
    one = torch.empty(nr, edge + 8, dtype=BF, device=DEV)
    for r in range(nr):
        _C.gemv_bf16(W, x[r:r + 1], one[r:r + 1])
    for N in (edge - 8, edge - 1, edge, edge + 1, edge + 8):
        ob = torch.full((nr, N + 3), 7.0, dtype=BF, device=DEV)
        _C.gemv_bf16(W[:N], x, ob[:, :N])
        assert torch.equal(ob[:, :N].view(torch.int16), one[:, :N].view(torch.int16)) and (ob[:, N:] == 7).all()


def _large_merge(po, ml, gate):
    """attn_merge_kernel on the partials a call left, for at most 16 splits: then each of its 16 warps has one
    split at most, the warps are added in ascending order, and L is the butterfly sum of one warp."""
    m, l = ml[..., 0], ml[..., 1]
    f = torch.where(m == -torch.inf, 0.0, torch.exp(m - m.amax(-1, keepdim=True)))
    lanes = torch.nn.functional.pad(l * f, (0, 32 - m.size(-1)))
    for o in (16, 8, 4, 2, 1):
        lanes = lanes + lanes[..., torch.arange(32, device=DEV) ^ o]
    O = torch.zeros_like(po[..., 0, :])
    for s in range(po.size(-2)):
        O = O + po[..., s, :] * f[..., s, None]
    o = (O / lanes[..., :1]).to(BF).float()
    return (o * (1.0 / (1.0 + torch.exp(-gate.float()))).to(BF).float()).to(BF)


@pytest.mark.parametrize("hd", [64, 128, 256])
@pytest.mark.parametrize("NS", [1, 5, 15, 16, 17])
@pytest.mark.parametrize("pos", [0, 3, 200])
def test_merge_of_few_splits(hd, NS, pos):
    """At most 16 splits merge without shared memory, more with it: up to there the bits are those of the
    large merge. The reference sums in fp64 over the prefix; 2 bf16 ulps cover the rounding of O / L, of
    the gate and of their product."""
    from qengine_b200 import _C
    hq, hkv, L, n = 4, 2, 256, 3
    q, qg = rand(n, hq * hd).to(BF), rand(n, hq * 2 * hd, seed=1).to(BF)
    kc, vc = rand(hkv, L, hd, seed=2).to(BF), rand(hkv, L, hd, seed=3).to(BF)
    out = torch.empty(n, hq * hd, dtype=BF, device=DEV)
    po, ml = torch.empty(n, hq, NS, hd, device=DEV), torch.empty(n, hq, NS, 2, device=DEV)
    _C.attn_decode(q, kc, vc, torch.tensor([pos], dtype=torch.int32, device=DEV), qg, po, ml, out)
    if NS <= 16:
        want = _large_merge(po, ml, qg.view(n, hq, 2 * hd)[..., hd:]).reshape(n, hq * hd)
        assert torch.equal(out.view(torch.int16), want.view(torch.int16))
    for t in range(n):
        for h in range(hq):
            k, v = (c[h // 2, :pos + t + 1].double() for c in (kc, vc))
            p = torch.softmax(k @ q[t, h * hd:(h + 1) * hd].double() * hd ** -0.5, 0)
            gate = torch.sigmoid(qg[t, h * 2 * hd + hd:(h + 1) * 2 * hd].double())
            ref = (p @ v) * gate
            got = out[t, h * hd:(h + 1) * hd].double()
            assert ((got - ref).abs() <= 2.0 ** -6 * ref.abs() + 1e-3).all()
