"""The GPU packer (qe_w4_pack behind quant.quantize_w4 / quantize_w4_gate_up) against the torch packer, which
the golden vectors of the reference pin: every bit of codes and scales. (The scale of a group with a NaN in
it is a NaN on both sides; its payload is 0x7fff on the GPU and 0x7e00 on the CPU, for torch as well.)"""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


def _w(M, K, dtype, seed):
    g = torch.Generator().manual_seed(seed)
    w = torch.randn(M, K, generator=g) * torch.rand(M, 1, generator=g)
    w[0] = 0.0                                    # a row of zeros: scale 0, code 8
    if M > 3 and K > 3:
        w[1] = torch.randint(-15, 16, (K,), generator=g) / 2.0   # quotients on the middle between two codes
        w[1, 0] = 7.5
        w[2] *= 1e-9                              # scale below fp16's smallest number
        w[3] *= 3e-6                              # scale a denormal fp16
        w[-1] *= 1e6                              # scale beyond fp16: infinite
        w[M // 2, K // 2] = float("nan")
    return w.to(dtype)


def _same(a, b):
    sa, sb = a.scales.cpu(), b.scales
    assert torch.equal(a.qw.cpu(), b.qw) and torch.equal(sa.isnan(), sb.isnan())
    assert torch.equal(sa.nan_to_num(-1.0), sb.nan_to_num(-1.0))
    assert (a.M, a.K, a.gate_up) == (b.M, b.K, b.gate_up)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("M,K", [(16, 128), (1, 1), (15, 127), (17, 129), (200, 1000), (512, 640), (333, 2056)])
def test_bits_of_the_torch_packer(M, K, dtype):
    from qengine_b200 import quant
    w = _w(M, K, dtype, seed=M + K)
    w[~w.isfinite() & ~w.isnan()] = 1.0           # fp16 cannot hold the 1e6 row
    _same(quant.quantize_w4(w.cuda()), quant.quantize_w4(w))
    u = _w(M, K, dtype, seed=M + K + 1)
    u[~u.isfinite() & ~u.isnan()] = 1.0
    _same(quant.quantize_w4_gate_up(w.cuda(), u.cuda()), quant.quantize_w4_gate_up(w, u))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
def test_infinite_weights(dtype):
    """An infinite weight makes its group's scale infinite: its own quotient is no number and gets code 0, the
    finite ones of the group get code 8. As torch's operators have it on the GPU and on the CPU."""
    from qengine_b200 import quant
    w = _w(40, 300, torch.float32, seed=8)
    w[~w.isfinite() | (w.abs() > 6e4)] = 1.0
    w[5, 7], w[6, 140], w[7, 0], w[7, 1] = torch.inf, -torch.inf, torch.inf, -torch.inf
    w = w.to(dtype)
    p = quant.quantize_w4(w.cuda())
    _same(p, quant.quantize_w4(w))
    _same(p, quant._quantize_pack(w.cuda(), 40, 300, False).to("cpu"))
    codes, _ = quant.unpack_codes(p)
    assert codes[5, 7] == 0 and codes[6, 140] == 0 and (codes[7, :2] == 0).all() and (codes[5, :7] == 8).all()


def test_views_and_misaligned_rows():
    from qengine_b200 import quant
    big = torch.randn(300, 1030, generator=torch.Generator().manual_seed(5)).to(torch.bfloat16)
    dev = big.cuda()
    for rows, cols in ((slice(0, 256), slice(0, 1024)), (slice(3, 200), slice(1, 900)), (slice(0, 300, 2), slice(8, 776))):
        _same(quant.quantize_w4(dev[rows, cols]), quant.quantize_w4(big[rows, cols]))
    _same(quant.quantize_w4(dev.T), quant.quantize_w4(big.T))                    # no unit stride along K: torch path
    _same(quant.quantize_w4(dev.double()), quant.quantize_w4(big.double()))


def test_lazily_negated_and_traced_matrices():
    """A lazy negation is not in memory yet, and a trace must hold the packing, not its first result."""
    from torch.fx.experimental.proxy_tensor import make_fx

    from qengine_b200 import quant
    a, b = (torch.randn(48, 256, generator=torch.Generator().manual_seed(s)).to(torch.bfloat16) for s in (6, 7))
    _same(quant.quantize_w4(torch._neg_view(a.cuda())), quant.quantize_w4(-a))
    traced = make_fx(lambda w: quant.quantize_w4(w).qw)(a.cuda())
    assert torch.equal(traced(b.cuda()).cpu(), quant.quantize_w4(b).qw)


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
def test_quotients_half_way_between_codes(dt):
    """Rows whose quotients are exact halves or next to one (a maximum that 15 divides has an exact scale; a
    negative one then is the quotient -7.5): the codes are those of a division, ties to even."""
    from qengine_b200.quant import quantize_w4
    g = torch.Generator().manual_seed(3)
    top = 256 if dt == torch.bfloat16 else 2048
    m = torch.randint(1, top, (4096, 1), generator=g).float()
    m[:1024] = 15 * torch.randint(1, top // 15, (1024, 1), generator=g)
    w = torch.randint(-top, top + 1, (4096, 256), generator=g).float().clamp(-m, m)
    w[:, 1::2] = (torch.randint(-15, 16, (4096, 128), generator=g) * m / 15).round()  # at and around k + 1/2
    w[:, 0], w[:, 128] = -m[:, 0], m[:, 0]
    w = (w * 2.0 ** torch.randint(-9, 2, (4096, 1), generator=g)).to(dt)
    a, b = quantize_w4(w.cuda()), quantize_w4(w)
    assert torch.equal(a.scales.cpu().view(torch.int16), b.scales.view(torch.int16)) and torch.equal(a.qw.cpu(), b.qw)
