"""The product of up to 128 rows (w4_rows.cu) against the GEMV: the same bits, row by row."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def packed(M, K, seed):
    from qengine_b200.quant import W4Packed
    g = torch.Generator(device=DEV).manual_seed(seed)
    Mp = -(-M // 16) * 16
    qw = torch.randint(-2**31, 2**31 - 1, (Mp // 16, K // 64, 32, 4), dtype=torch.int32, device=DEV, generator=g)
    sc = (torch.randn(Mp // 16, K // 128, 16, device=DEV, generator=g) * 0.01).half()
    return W4Packed(qw, sc, M, K)


def rand_x(n, K, seed, wild=False):
    g = torch.Generator(device=DEV).manual_seed(seed)
    x = torch.randn(n, K, device=DEV, generator=g)
    if wild:  # exponents far apart: the order of every addition shows
        x *= torch.exp2(torch.randint(-12, 12, (n, K), device=DEV, generator=g).float())
    return x.bfloat16()


def by_gemv(x, p, swiglu=False, **kw):
    from qengine_b200 import _w4
    M = p.M // 2 if swiglu else p.M
    out = torch.empty(x.size(0), M, dtype=torch.bfloat16, device=DEV)
    for r in range(0, x.size(0), 8):
        (_w4.gemv_swiglu if swiglu else _w4.gemv)(x[r:r + 8], p.qw, p.scales, out[r:r + 8], M, **kw)
    return out


def same(a, b):
    return torch.equal(a.view(torch.int16), b.view(torch.int16))


# 27B matrices (whole tiles per CTA; cut tiles), few and ragged super-tiles, groups that are no multiple of four
SHAPES = [(16480, 5120), (5120, 6144), (34816, 5120), (5120, 17408), (16, 128), (128, 256), (200, 896), (5008, 384),
          (1040, 3456), (4096, 4096), (148 * 128 + 48, 640)]


@pytest.mark.parametrize("M,K", SHAPES)
@pytest.mark.parametrize("n", [1, 16, 23, 64, 65, 128])
def test_bits_of_the_gemv(M, K, n):
    from qengine_b200 import _w4
    p, x = packed(M, K, 1), rand_x(n, K, 2, wild=True)
    out = torch.full((n, M), 7.0, dtype=torch.bfloat16, device=DEV)
    _w4.rows(_w4.wire_order(x), p.qw, p.scales, out, M)
    assert same(out, by_gemv(x, p)) and _w4.ring_error() == 0


@pytest.mark.parametrize("n", [9, 40, 128])
@pytest.mark.parametrize("opts", [{}, {"warps": 8}, {"min_units": 1}, {"ksplit": 4}])
def test_swiglu_wire_order_options_and_sums(n, opts):
    from qengine_b200 import _w4
    p, x = packed(2 * 1088, 1280, 3), rand_x(n, 1280, 4)
    wide = torch.full((n, 1088 + 24), 7.0, dtype=torch.bfloat16, device=DEV)  # strided rows in and out
    xs = torch.zeros(n, 1280 + 8, dtype=torch.bfloat16, device=DEV)
    xs[:, :1280] = _w4.wire_order(x)
    _w4.rows(xs[:, :1280], p.qw, p.scales, wide[:, :1088], 1088, swiglu=True, wire_out=True, **opts)
    want = by_gemv(x, p, swiglu=True, **opts)
    assert same(_w4.wire_order(wide[:, :1088]), want) and (wide[:, 1088:] == 7).all()
    q = packed(720, 1280, 5)
    sums, one = torch.empty(n, 720, device=DEV), torch.empty(n, 720, device=DEV)
    _w4.rows(xs[:, :1280], q.qw, q.scales, sums, 720, **opts)
    for r in range(0, n, 8):
        _w4.gemv_partial(x[r:r + 8], q.qw, q.scales, one[r:r + 8], 720, **opts)
    assert torch.equal(sums.view(torch.int32), one.view(torch.int32))


@pytest.mark.parametrize("M,K", [(5120, 17408), (5120, 6144), (4096, 4096), (1040, 3456), (1008, 16384), (72, 8064)])
@pytest.mark.parametrize("n", [1, 16, 49, 67, 128])
@pytest.mark.parametrize("limit", [1 << 20, 0, 3])
def test_split_along_k(M, K, n, limit):
    """With scratch a matrix of few rows is split along K: the bits of the unsplit product, nothing outside of the
    scratch and the output, and a way out when waits run out."""
    import ctypes as C

    from qengine_b200 import _w4
    from qengine_b200._lib import W4Cfg, W4Params, lib
    p, x = packed(M, K, 12), _w4.wire_order(rand_x(n, K, 13, wild=True))
    want, got = (torch.full((n, M), 7.0, dtype=torch.bfloat16, device=DEV) for _ in range(2))
    cfg, stream = W4Cfg(0, 0, 0, 1, 0, -1, 0, 4), torch.cuda.current_stream().cuda_stream
    a = W4Params(p.qw.data_ptr(), p.scales.data_ptr(), x.data_ptr(), want.data_ptr(), None, None, M, K, 16 * p.qw.size(0),
                 K, n, K, M, 0, 0, 0)
    assert lib.qe_w4_rows(C.byref(a), C.byref(cfg), 0, stream) == 0
    floats = lib.qe_w4_rows_ws_floats(C.byref(a), C.byref(cfg))
    assert floats > 0 if M > 2000 else floats >= 0
    ws = torch.full((floats + 64,), float("nan"), device=DEV)
    a.ws, a.out = ws.data_ptr(), got.data_ptr()
    assert lib.qe_w4_rows_bounded(C.byref(a), C.byref(cfg), 0, limit, stream) == 0
    error = _w4.ring_error()
    assert error == 0 if limit > 3 else error > 0 if limit == 0 else error >= 0
    assert error or same(got, want)
    assert ws[floats:].isnan().all()
    assert lib.qe_w4_clear_error() == 0
    assert lib.qe_w4_rows(C.byref(a), C.byref(cfg), 0, stream) == 0
    assert _w4.ring_error() == 0 and same(got, want)
    a.ws = ws.data_ptr() + 4
    assert lib.qe_w4_rows(C.byref(a), C.byref(cfg), 0, stream) == -22


def test_special_values():
    """Rows of zeros, infinities and NaN stay what the GEMV makes of them, and among themselves."""
    from qengine_b200 import _w4
    p, x = packed(5120, 6144, 6), rand_x(24, 6144, 7)
    x[3] = 0
    x[5, 100] = float("inf")
    x[7, 6000] = float("nan")
    out = torch.empty(24, 5120, dtype=torch.bfloat16, device=DEV)
    _w4.rows(_w4.wire_order(x), p.qw, p.scales, out, 5120)
    want = by_gemv(x, p)
    assert torch.equal(out.isnan(), want.isnan()) and torch.equal(out.nan_to_num(1.5), want.nan_to_num(1.5))
    assert not out[[r for r in range(24) if r not in (5, 7)]].isnan().any()


def test_refused():
    from qengine_b200 import _w4
    p, x = packed(64, 512, 8), rand_x(16, 512, 9)
    out = torch.empty(16, 64, dtype=torch.bfloat16, device=DEV)
    for bad in (lambda: _w4.rows(rand_x(129, 512, 1), p.qw, p.scales, torch.empty(129, 64, dtype=torch.bfloat16, device=DEV), 64),
                lambda: _w4.rows(x[:, :500], p.qw, p.scales, out, 64),
                lambda: _w4.rows(rand_x(1, 2048, 1)[0].as_strided((16, 512), (8, 1)), p.qw, p.scales, out, 64),
                lambda: _w4.rows(x, p.qw, p.scales, out[:, :56], 56, wire_out=True)):
        with pytest.raises(RuntimeError):
            bad()


@pytest.mark.parametrize("limit", [0, 1, 3, 20, 100])
@pytest.mark.parametrize("M,K,n", [(148 * 128 + 77, 640, 128), (5120, 6144, 48)])
def test_waits_that_run_out(M, K, n, limit):
    """Few polls per wait: the launch ends, says so and leaves the device as before."""
    import ctypes as C

    from qengine_b200 import _w4
    from qengine_b200._lib import W4Cfg, W4Params, lib
    p, x = packed(M, K, 10), rand_x(n, K, 11)
    want, xw, got = by_gemv(x, p), _w4.wire_order(x), torch.empty(n, M, dtype=torch.bfloat16, device=DEV)
    a = W4Params(p.qw.data_ptr(), p.scales.data_ptr(), xw.data_ptr(), got.data_ptr(), None, None, M, K, 16 * p.qw.size(0),
                 K, n, K, M, 0, 0, 0)
    cfg, stream = W4Cfg(0, 0, 0, 1, 0, -1, 0, 4), torch.cuda.current_stream().cuda_stream
    assert lib.qe_w4_rows_bounded(C.byref(a), C.byref(cfg), 0, -1, stream) == -22
    assert lib.qe_w4_rows_bounded(C.byref(a), C.byref(cfg), 0, limit, stream) == 0
    error = _w4.ring_error()
    assert error > 0 if limit == 0 else error >= 0
    assert error > 0 or same(got, want)
    assert lib.qe_w4_clear_error() == 0
    assert lib.qe_w4_rows(C.byref(a), C.byref(cfg), 0, stream) == 0
    assert _w4.ring_error() == 0 and same(got, want)
