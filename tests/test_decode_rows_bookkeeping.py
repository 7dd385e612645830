"""The bookkeeping of csrc/decode_rows.cu on the CPU: what its source promises about barriers, which CTA has which tiles, its ring of weights and its words with flags as
state machines that run in random order.  The rules are restated from the kernel, the constants read from its source."""
import pathlib
import random
import re

import numpy as np
import pytest

SOURCE = (pathlib.Path(__file__).resolve().parents[1] / "nano-qwen3tts-vllm_b200" / "csrc" / "decode_rows.cu").read_text()
CODE = re.sub(r"//[^\n]*", "", SOURCE)


def test_warps_meet_between_polling_and_the_next_barrier():
    """Lanes of a warp leave a polling loop one by one; an aligned barrier, a vote or a shuffle behind it wants all of them."""
    marks = [(m.start(), m.group(1)) for m in re.finditer(r"(dr_wait(?:_all)?(?=[(<])|dr_sync\(\)|__syncwarp\(\)|__syncthreads\(\)|__all_sync\(|warp_sum\()", CODE)]
    waits, open_wait = 0, None
    for at, name in marks:
        line = CODE[:at].count("\n") + 1
        if name.startswith("dr_wait"):
            if re.search(r"__forceinline__ \w+ $", CODE[:at]):
                continue                                         # its definition
            waits, open_wait = waits + 1, line
        elif name == "__syncwarp()":
            open_wait = None
        else:
            assert open_wait is None, f"{name} in line {line} follows the polling of line {open_wait}"
    assert waits >= 6


# ---------------------------------------------------------------- who does what, restated from the kernel; its constants come from the source
def _const(name):
    return int(re.search(rf"{name} = (\d+)", SOURCE).group(1))


CTAS, UNIT, STAGES, WARPS, MAX_TILES, SUMS = 148, _const("DR_UNIT"), _const("DR_STAGES"), _const("DR_WARPS"), _const("DR_MAX_TILES"), _const("DR_SUMS")
Q, GROUP = _const("DR_Q"), _const("DR_GROUP")
KVH = Q // GROUP // 128
FORMS = {2048: (6144, 8, 2), 1024: (3072, 8, 4)}                 # hidden: inner width, slices of K of gate_up and of the others (gemm.cu's, which dr_form() compares)
ceil = lambda a, b: -(-a // b)


def _group(tiles, ctas=CTAS):
    most = ceil(tiles, ctas)
    return 4 if ceil(ceil(tiles, 4), ctas) * 4 <= most + 1 else 2 if ceil(ceil(tiles, 2), ctas) * 2 <= most else 1


def _span(tiles, cta, ctas=CTAS):
    g = _group(tiles, ctas)
    n = ceil(tiles, g)
    return min(tiles, cta * n // ctas * g), min(tiles, (cta + 1) * n // ctas * g)


def _plan(hidden, cta):
    inter = FORMS[hidden][0]
    o = _span(hidden // 8, cta)
    return [_span((Q + 2 * Q // GROUP) // 8, cta), o, _span(2 * inter // 8, cta), o]


def _phases(hidden):
    """(slices, steps of 64 columns of a slice, steps a stage) of qkv, o, gate_up, down"""
    inter, sq, sg = FORMS[hidden][0], FORMS[hidden][1], FORMS[hidden][2]
    return [(sq, hidden // 64 // sq, 1), (sq, Q // 64 // sq, 2), (sg, hidden // 64 // sg, 2), (sq, inter // 64 // sq, 2)]


def _units(hidden, rows):
    wide = max(FORMS[hidden][0], Q)
    xs = max(rows * wide * 2, GROUP * 32 * (2 + 128) * 4)
    return (222 * 1024 - xs - 2 * SUMS * 64 * 4 - 4096) // UNIT // 16 * 16


@pytest.mark.parametrize("hidden", FORMS)
def test_every_tile_has_one_cta_and_every_cta_has_tiles_of_gate_up(hidden):
    inter = FORMS[hidden][0]
    for phase, tiles in enumerate(((Q + 2 * Q // GROUP) // 8, hidden // 8, 2 * inter // 8, hidden // 8)):
        spans = [_plan(hidden, c)[phase] for c in range(CTAS)]
        assert [t for a, b in spans for t in range(a, b)] == list(range(tiles))
        slices, steps, per_stage = _phases(hidden)[phase]
        for a, b in spans:
            assert (b - a) * slices <= SUMS and ceil(b - a, WARPS // slices) <= MAX_TILES and steps % 2 == 0 and steps % per_stage == 0
        if phase == 2:
            assert all(b > a for a, b in spans)                  # see the head of the source: a step of padding rows has nothing else to hold a CTA back
    assert re.search(r"< n\) return 0;\s*\n\s*if \(!fits", CODE)      # ... which dr_form() asks for


# ---------------------------------------------------------------- the stream of weights
@pytest.mark.parametrize("hidden,rows", [(2048, 2), (2048, 4), (1024, 2), (1024, 4), (1024, 8)])
@pytest.mark.parametrize("seed", range(4))
def test_ring(hidden, rows, seed):
    """The copying warp and eight readers in random order: no copy lands on a stage that a reader still wants, no barrier is armed twice, readers find their
    stages where the copies went, and both come to their ends."""
    r, units, layers = random.Random(seed), _units(hidden, rows), 3
    for cta in r.sample(range(CTAS), 12):
        plan, phases, todo = _plan(hidden, cta), _phases(hidden), []
        for i in range(4 * layers):
            (t0, t1), (slices, steps, per) = plan[i & 3], phases[i & 3]
            if t1 == t0:
                continue
            copied = sorted((s, t) for lane in range(32) for s in [lane // (32 // slices)] for first in [(t0 & ~3) + 4 * (lane % (32 // slices))]
                            for t in range(max(t0, first), min(t1, first + 4)))
            assert copied == [(s, t) for s in range(slices) for t in range(t0, t1)]
            todo += [(t1 - t0) * slices * per] * (steps // per)
        assert max(todo) <= units
        head = count = oldest = 0
        begin, read = {}, [0] * WARPS                            # where stage k lies; stages that a reader is done with
        places = []                                              # as the readers work them out
        at = 0
        for size in todo:
            at = 0 if at + size > units else at
            places.append(at)
            at += size
        while min(read) < len(todo):
            who = r.randrange(WARPS + 1) if r.random() < 0.7 else WARPS
            if who < WARPS:                                      # a reader: its next stage, if that has been copied
                if read[who] < count and read[who] - min(read) < STAGES:
                    assert begin[read[who]] == places[read[who]]
                    read[who] += 1
                continue
            if count == len(todo):
                continue
            size = todo[count]
            place = 0 if head + size > units else head
            blocked = False
            while oldest < count:
                b = begin[oldest]
                free = (place == head or size <= b) if head > b else (place == head and head + size <= b)
                if free and count - oldest < STAGES:
                    break
                if min(read) <= oldest:                          # its barrier is not complete
                    blocked = True
                    break
                oldest += 1
            if blocked:
                continue
            for k in range(min(read), count):                    # stages that somebody still wants
                assert place + size <= begin[k] or begin[k] + todo[k] <= place
            assert count - min(read) < STAGES
            begin[count], head = place, place + size
            count += 1


# ---------------------------------------------------------------- words with flags
def _cta_program(hidden, cta, m, lens, parts, layers):
    """What a CTA reads and writes, in order: ("r" | "w", buffer, places, number of the layer).  A place is eight columns of a row (of act: four), or a part of a unit."""
    inter, plan, out = FORMS[hidden][0], _plan(hidden, cta), []
    part, row, head = cta // (m * KVH), cta % (m * KVH) // KVH, cta % KVH
    L = lens[row] if part < parts else 0
    mine = part < (parts if L > 0 else 1)
    rows = lambda width, cols: (np.arange(m)[:, None] * width + np.asarray(cols)[None, :]).ravel()
    widths = {"qkv": (Q + 2 * Q // GROUP) // 8, "att": Q // 8, "res1": hidden // 8, "res2": hidden // 8, "act": 2 * inter // 8}
    tiles = lambda buffer, phase: rows(widths[buffer], range(*plan[phase]))
    everything = {b: rows(w, range(w)) for b, w in widths.items()}
    unit = (row * KVH + head) * 32
    for l in range(layers):
        if plan[0][0] < plan[0][1]:
            if l:
                out.append(("r", "res2", everything["res2"], l - 1))
            out.append(("w", "qkv", tiles("qkv", 0), l))
        if mine:
            if L > 0:
                cols = [head * GROUP * 16 + i for i in range(GROUP * 16)] + [Q // 8 + head * 16 + i for i in range(16)] + [Q // 8 + Q // GROUP // 8 + head * 16 + i for i in range(16)]
                out.append(("r", "qkv", row * widths["qkv"] + np.array(cols), l))
            if part:
                out.append(("w", "part", np.array([unit + part]), l))
            else:
                if L > 0 and parts > 1:
                    out.append(("r", "part", unit + np.arange(1, parts), l))
                out.append(("w", "att", row * widths["att"] + head * GROUP * 16 + np.arange(GROUP * 16), l))
        if plan[1][0] < plan[1][1]:
            out.append(("r", "att", everything["att"], l))
            if l:
                out.append(("r", "res2", tiles("res2", 1), l - 1))
            out.append(("w", "res1", tiles("res1", 1), l))
        out += [("r", "res1", everything["res1"], l), ("w", "act", tiles("act", 2), l)]
        if plan[3][0] < plan[3][1]:
            out += [("r", "act", everything["act"], l), ("r", "res1", tiles("res1", 3), l), ("w", "res2", tiles("res2", 3), l)]
    if cta < m:
        out.append(("r", "res2", cta * widths["res2"] + np.arange(widths["res2"]), layers - 1))
    return out, dict(widths, part=KVH * 32)


def _play(programs, sizes, slow, r):
    step, left, running, idle = [0] * CTAS, [None] * CTAS, set(range(CTAS)), 0
    flag = {b: np.full(n, -1) for b, n in sizes.items()}
    while running:
        moved = False
        for c in r.sample(sorted(running), len(running)):
            if c in slow and r.random() < 0.7:
                continue
            while step[c] < len(programs[c]):
                kind, buffer, places, number = programs[c][step[c]]
                if kind == "w":
                    flag[buffer][places] = number
                else:
                    todo = places if left[c] is None else left[c]
                    now = flag[buffer][todo]
                    assert (now <= number).all(), f"a word of {buffer} was written again before CTA {c} had read it"
                    waiting = now < number
                    if c in slow and r.random() < 0.5:
                        waiting[len(waiting) // 2:] = True       # stops in the middle of its rows
                    moved |= not waiting.all()
                    left[c] = todo[waiting]
                    if len(left[c]):
                        break
                left[c], step[c], moved = None, step[c] + 1, True
            if step[c] == len(programs[c]):
                running.discard(c)
        idle = 0 if moved else idle + 1
        assert idle < 50, "nobody can go on"


@pytest.mark.parametrize("hidden,lens,parts", [(2048, [97], 1), (2048, [3000], 8), (1024, [0], 1), (1024, [5, 0], 1), (1024, [0, 0], 8)])
@pytest.mark.parametrize("slow", [0, 20, 147])
def test_no_word_is_overwritten_before_its_readers(hidden, lens, parts, slow):
    """CTAs run in random order, some far behind; a word is read when it carries its layer's number.  A word that carries a later one when a reader comes would be waited for
    until the tries run out: that, and a wait that nothing ends, fail here."""
    m, r = len(lens), random.Random(hidden + sum(lens) + slow)
    programs = [_cta_program(hidden, c, m, lens, parts, 4) for c in range(CTAS)]
    _play([p for p, _ in programs], {b: m * n for b, n in programs[0][1].items()}, set(r.sample(range(CTAS), slow)), r)


def test_padding_rows_would_be_overwritten_without_gate_up():
    """What the play is there to see: in a step of padding rows a CTA without tiles of gate_up, o and down writes qkv, and its part of attention, whenever it likes."""
    programs = [_cta_program(1024, c, 1, [0], 1, 4) for c in range(CTAS)]
    idle = next(c for c in range(KVH) if c)                      # it has a unit of attention
    mine = [[op for op in p if c != idle or op[1] == "att" and op[0] == "w"] for c, (p, _) in enumerate(programs)]
    with pytest.raises(AssertionError, match="written again"):
        for seed in range(20):
            _play(mine, dict(programs[0][1]), set(range(CTAS)) - {idle}, random.Random(seed))
