"""Index arithmetic of the tensor-memory prefill GEMM (w4_gemm_tc_kernel in
qengine_b200/csrc/w4_gemm.cu), restated in Python and checked on the CPU: the unpacking groups'
cursors meet every unit once and in the order in which the products are issued, two steps share a
load of activations whose stage is free by then, scales are requested before they are read and into a
slot nobody reads, and a warp that gives a wait up leaves no copy behind that it has not waited for."""
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


class GivenUp(Exception):
    pass


class Scales:
    """A drain warp's requests of scales (request_scales) and their barriers s_full[wd][2]."""

    def __init__(self, nj, per_job):
        self.nj, self.per_job, self.j, self.g, self.next = nj, per_job, 0, 0, 0
        self.content, self.busy, self.landed = {}, set(), set()  # by number; slots being read; numbers waited for

    def request(self):
        if self.j >= self.nj:
            return
        assert self.next & 1 not in self.busy, "slot is still being read"
        assert self.next < 2 or self.next - 2 in self.landed, "barrier armed again before its phase was waited for"
        self.content[self.next] = (self.j, self.g, min(CHUNK, self.per_job - self.g))
        self.next += 1
        self.g += CHUNK
        if self.g >= self.per_job:
            self.j, self.g = self.j + 2, 0

    def wait(self, number):
        assert number in self.content, "waits for scales that were never requested"
        self.landed.add(number)


def drain_warp(nj, per_job, wd, give_up):
    """The waits and requests of drain warp `wd` in their order, up to its wait number `give_up` (-1: none
    fails). Returns the scales, the last unit of activations requested and the padded step reached."""
    walk, half = (per_job + 1) & ~1, STAGES // 2
    steps = (nj + 1) // 2 * walk
    sc, waits, unit = Scales(nj, per_job), 0, wd + 8 if wd < half else wd
    sc.request()
    sc.request()
    zb = chunk = z = 0

    def wait():
        nonlocal waits
        waits += 1
        if waits - 1 == give_up:
            raise GivenUp

    try:
        for j in range(0, nj, 2):
            i = 0
            for c0 in range(0, per_job, CHUNK):
                wait()
                sc.wait(chunk)
                assert sc.content[chunk] == (j, c0, min(CHUNK, per_job - c0)), "scales of other groups"
                sc.busy.add(chunk & 1)
                while i < min(c0 + CHUNK, per_job):
                    z = zb + i
                    wait()  # a pair: this group's micro-step; a lone super-tile: the only one
                    if 2 * unit < z + STAGES - 1:
                        unit += 8
                    i += 1
                sc.busy.discard(chunk & 1)
                sc.request()
                chunk += 1
            zb += walk
    except GivenUp:
        pass
    return sc, unit - 8, z, steps, waits


@pytest.mark.parametrize("nj,per_job", [(1, 1), (1, 8), (1, 45), (2, 28), (2, 29), (3, 27), (3, 57), (5, 1), (6, 3)])
def test_a_warp_that_gives_up_has_waited_for_its_copies(nj, per_job):
    """Every wait in turn is the one that runs out. What is in flight then is what the waits on the way
    out cover: the last two requests of scales, the warp's last unit of activations."""
    total = drain_warp(nj, per_job, 0, -1)[4]
    for wd in (0, 3, 4, 7):
        for give_up in (-1, *range(total)):
            sc, u, z, steps, _ = drain_warp(nj, per_job, wd, give_up)
            flying = set(sc.content) - sc.landed
            if give_up < 0:
                assert not flying and sc.j >= nj
                continue
            assert flying <= set(range(max(sc.next - 2, 0), sc.next))
            # own units before the last one: their products are complete, so they have landed. Parity: when the
            # warp asked for u, unit u - 4 of the same barrier was multiplied, and no unit after u + 4 is asked for
            if u >= 8:
                assert 2 * (u - 8) + 1 < z and 2 * (u - 4) + 1 < z


@pytest.mark.parametrize("nj,per_job", [(1, 1), (1, 8), (2, 5), (3, 57), (5, 3)])
def test_rows_without_a_tensor_map(nj, per_job):
    """load_b: the steps in order, the group each holds, and no stage written before its products are."""
    walk = (per_job + 1) & ~1
    steps = (nj + 1) // 2 * walk
    held, bi = [], 0

    def load():
        nonlocal bi
        if len(held) >= steps:
            return
        held.append(bi if bi < per_job else None)
        bi = 0 if bi + 1 == walk else bi + 1

    for _ in range(STAGES - 1):
        load()
    for z in range(steps):
        if z % walk >= per_job:
            continue
        assert len(held) > z and held[z] == z % walk, "multiplied before it is asked for"
        while len(held) < min(steps, z + STAGES):
            assert len(held) - STAGES < z, "stage still in use"
            load()
    assert len(held) == steps
