"""Index arithmetic of the product that keeps the GEMV's bits for up to 128 rows (w4_rows_kernel in
qengine_b200/csrc/w4_rows.cu), restated in Python and checked on the CPU: the unpacking warps meet every unit
once and in the order of the products, and the partial sums are closed exactly where the warps and CTAs of the GEMV hand over."""
from __future__ import annotations

import random

import pytest

from test_gemm_split_cpu import SMS, share_begin


class Deal:
    """w4::Deal as resolve() in w4_gemv.cu fills it, for 16 warps per CTA and min_units 4."""

    def __init__(self, tiles, G, nw=16, min_units=4, sms=SMS):
        units, q = tiles * G, 4 if G % 4 == 0 else 1
        want = -(-units // min_units)
        self.nctas = max(1, min(sms, want, units // q))
        per_cta = -(-units // self.nctas)
        self.nwarps = max(1, min(nw, -(-per_cta // min_units)))
        self.q, self.total, self.G = q, units, G
        tiles_max = -(-tiles // self.nctas)
        whole = self.nctas > 1 and tiles >= self.nctas and (tiles_max * self.nctas - tiles) * G <= 26 * self.nctas
        self.qc = G if whole else q
        self.per, self.rem = divmod(units // self.qc, self.nctas)

    def warp_ranges(self):
        """[(CTA, first unit, end)] of the warps that own units, in the order of the stream."""
        out = []
        for c in range(self.nctas):
            b, e = (self.qc * share_begin(self.total // self.qc, self.nctas, c + i) for i in (0, 1))
            for w in range(self.nwarps):
                u0, u1 = (b + self.q * share_begin((e - b) // self.q, self.nwarps, w + i) for i in (0, 1))
                if u1 > u0:
                    out.append((c, u0, u1))
        return out

    # range_at, range_next and range_bounds in w4_dev.cuh
    def bounds(self, c, w):
        more = int(c < self.rem)
        b = self.qc * (c * self.per + min(c, self.rem))
        per, rem = divmod((self.per + more) * (self.qc // self.q), self.nwarps)
        return b, per, rem, b + self.q * ((w + 1) * per + min(w + 1, rem)), b + self.qc * (self.per + more)

    def range_at(self, u):
        Q, big = u // self.qc, self.rem * (self.per + 1)
        c = Q // (self.per + 1) if Q < big else self.rem + (Q - big) // self.per
        b, per, rem, _, _ = self.bounds(c, 0)
        i, cut = (u - b) // self.q, rem * (per + 1)
        return c, i // (per + 1) if i < cut else rem + (i - cut) // per

    def range_next(self, c, w):
        _, _, _, end, cta_end = self.bounds(c, w)
        return (c + 1, 0) if end == cta_end else (c, w + 1)


SHAPES = [(1030, 40), (320, 48), (2176, 40), (320, 136), (1, 1), (3, 7), (200, 4), (32, 4), (17, 5), (5, 3), (148, 4),
          (149, 8), (40, 1), (313, 27), (7, 131)]


@pytest.mark.parametrize("tiles,G", SHAPES + [(random.Random(7).randint(1, 900), g) for g in (2, 6, 12, 20, 33)])
def test_partial_sums_close_where_the_gemv_hands_over(tiles, G):
    d = Deal(tiles, G)
    ranges = d.warp_ranges()
    assert ranges[0][1] == 0 and all(a[2] == b[1] for a, b in zip(ranges, ranges[1:])) and ranges[-1][2] == tiles * G
    it = iter(ranges)
    c, u0, u1 = next(it)
    for T in range(tiles):
        # the kernel's walk over the tile: closing points, and whether the CTA ends there
        closes, at = [], d.range_at(T * G)
        for i in range(G):
            end, cta_end = d.bounds(*at)[3:]
            if T * G + i == end:
                closes.append((i, end == cta_end))
                at = d.range_next(*at)
        want = []
        for g in range(G):
            u = T * G + g
            while u >= u1:
                last = c
                c, u0, u1 = next(it)
                if g:
                    want.append((g, c != last))
        assert closes == want, (T, closes, want)
        if d.qc == G:  # whole tiles per CTA: no second level of sums, which has no room at 128 columns
            assert not any(e for _, e in closes)


def jobs(tiles, N, whole, cta):
    ST, n16 = (tiles + 7) // 8, (N + 15) // 16
    parts = 1 if ST * 2 > SMS else min(SMS // ST, n16)
    if not whole:
        parts = max(parts, (n16 + 3) // 4)
    cols = 16 * -(-n16 // parts)
    cparts = -(-N // cols)
    J = ST * cparts
    nctas = min(SMS, J)
    return [((cta + j * nctas) // cparts * 8, (cta + j * nctas) % cparts * cols) for j in
            range((J - cta + nctas - 1) // nctas if cta < J else 0)], cols, nctas


@pytest.mark.parametrize("tiles,G,N", [(t, g, n) for t, g in SHAPES for n in (1, 16, 40, 64, 65, 128)])
def test_walk(tiles, G, N):
    whole = Deal(tiles, G).qc == G
    seen = set()
    for cta in range(jobs(tiles, N, whole, 0)[2]):
        mine, cols, _ = jobs(tiles, N, whole, cta)
        assert cols % 16 == 0 and cols <= (128 if whole else 64)
        order = [(t, c, g) for t, c in mine for g in range(G)]
        for t0, c0 in mine:
            assert c0 < N
            for t in range(t0, min(t0 + 8, tiles)):
                for n in range(c0, min(c0 + cols, N)):
                    assert (t, n) not in seen
                    seen.add((t, n))
        U, P = (1, 3) if cols > 64 else (2, 2) if cols > 48 else (3, 1)
        for grp in range(U):  # the cursor of a group of unpacking warps
            cj, cg, out = 0, grp, []
            while True:
                while cg >= G:
                    cg, cj = cg - G, cj + 1
                if cj >= len(mine):
                    break
                out.append((*mine[cj], cg))
                cg += U
            assert out == order[grp::U]
        for _, c0 in mine:  # the drain warps of a quarter share the 16-column blocks of a job
            nb = -(-min(cols, N - c0) // 16)
            each = (nb + P - 1) // P
            mine3 = [(each * h, min(each, max(0, nb - each * h))) for h in range(P)]
            assert [b for b0, n in mine3 for b in range(b0, b0 + n)] == list(range(nb)) and each <= (2 if P == 2 else 3)
            assert whole or 16 * (mine3[-1][0] + mine3[-1][1]) <= 64 or nb <= 4
    assert len(seen) == tiles * N


def test_wire_order():
    from qengine_b200.quant import quantize_w4  # noqa: F401  (the format's home)

    def pos(k):
        return (k & ~60) | (k & 12) << 2 | (k >> 2 & 12)

    assert [pos(64 * c + 16 * t + 4 * s + j) for c in range(3) for t in range(4) for s in range(4) for j in range(4)] == \
        [64 * c + 16 * s + 4 * t + j for c in range(3) for t in range(4) for s in range(4) for j in range(4)]
    assert all(pos(pos(k)) == k for k in range(256))
