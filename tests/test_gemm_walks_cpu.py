"""Index arithmetic of the tensor-memory prefill GEMM (w4_gemm_tc_kernel in
qengine_b200/csrc/w4_gemm.cu), restated in Python and checked on the CPU: the unpacking groups'
cursors meet every unit once and in the order in which the products are issued, two steps share a
load of activations whose stage is free by then, and scales are requested before they are read."""
from __future__ import annotations

import pytest

from test_gemm_split_cpu import SHAPES, SMS, kparts, share_begin

STAGES, CHUNK = 8, 28  # kTcB, kTcChunk


def cta_jobs(tiles, G, cta):
    KP = kparts(tiles, G)
    J = (tiles + 7) // 8 * KP
    nctas = min(SMS, J)
    nj = (J - cta + nctas - 1) // nctas if cta < J else 0
    g0, g1 = (share_begin(G, KP, cta % KP), share_begin(G, KP, cta % KP + 1)) if KP > 1 else (0, G)
    return [(cta + j * nctas) // KP * 8 for j in range(nj)], g0, g1, nctas


def issue_order(tile0s, g0, g1):
    """(first tile, group, padded step) per micro-step, in the order of the products."""
    walk, out = (g1 - g0 + 1) & ~1, []
    for w, j in enumerate(range(0, len(tile0s), 2)):
        for i in range(g1 - g0):
            out += [(t, g0 + i, w * walk + i) for t in tile0s[j:j + 2]]
    return out


def cursor(tile0s, g0, g1, grp):
    """enter / load_next of an unpacking group: the micro-steps it fetches."""
    j, nj, out = 0, len(tile0s), []
    while j < nj:
        pair = j + 1 < nj
        g = g0 + (0 if pair else grp)
        while g < g1:
            out.append((tile0s[j + grp] if pair else tile0s[j], g))
            g += 1 if pair else 2
        j += 2
    return out


@pytest.mark.parametrize("tiles,G", SHAPES + [(148 * 8 * 3 + 19, 1), (148 * 8 * 4 + 5, 3), (148 * 8 * 2, 5), (8, 57)])
def test_walks(tiles, G):
    seen = set()
    for cta in range(cta_jobs(tiles, G, 0)[3]):
        tile0s, g0, g1, _ = cta_jobs(tiles, G, cta)
        order = issue_order(tile0s, g0, g1)
        for grp in (0, 1):
            assert cursor(tile0s, g0, g1, grp) == [(t, g) for t, g, _ in order[grp::2]]
        for t0, g, _ in order:
            for t in range(t0, min(t0 + 8, tiles)):
                assert (t, g) not in seen
                seen.add((t, g))
        # loads of activations: unit u holds the padded steps 2 u, 2 u + 1; drain warp u % 8 requests it
        # at the first of its own micro-steps in a step z with 2 u < z + STAGES - 1 (the first STAGES / 2
        # units at the start), when the products of all steps before z are complete
        units = (len(tile0s) + 1) // 2 * (((g1 - g0 + 1) & ~1) // 2)
        pairs = len(tile0s) // 2 * 2 * (g1 - g0)
        real = sorted({z for _, _, z in order})
        for wd in range(8):
            own = [z for v, (_, _, z) in enumerate(order) if v >= pairs or v % 2 == wd // 4]
            nxt = wd + 8 if wd < STAGES // 2 else wd
            for z in own:
                if 2 * nxt < z + STAGES - 1:
                    for step in (2 * nxt, 2 * nxt + 1):
                        assert step - STAGES < z, "stage still in use"
                    if nxt < units and 2 * nxt in real:
                        assert z <= 2 * nxt, "requested after the step that needs it"
                    nxt += 8
            assert nxt >= units, "a load of activations is never requested"
    assert len(seen) == tiles * G
    assert CHUNK * 32 % 16 == 0
