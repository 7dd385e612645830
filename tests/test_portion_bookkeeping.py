"""The bookkeeping of csrc/portion_attn.cu played on the CPU: which CTA takes which items, and its warps' barriers, ring slots and TMEM columns as
state machines that run in random order.  A product that reads what is not there, a copy that lands on what is still needed, an item taken twice
or a wait that nothing ends fails here.  The rules are restated from the kernel; its constants are read from the source, so that a
change of either shows."""
import pathlib
import random
import re

import pytest

SOURCE = (pathlib.Path(__file__).resolve().parents[1] / "nano-qwen3tts-vllm_b200" / "csrc" / "portion_attn.cu").read_text()
DEEP, ITEMS = (int(re.search(rf"{name} = (\d+)", SOURCE).group(1)) for name in ("PO_DEEP", "PO_ITEMS"))
KEYS = int(re.search(r"PO_N = (\d+)", SOURCE).group(1))
SLOTS = re.search(r"po_slots\(\) \{ return MODE == PO_SIGMOID \? (\d+) : NS == 1 \? (\d+) : NS == 2 \? (\d+) : (\d+); \}", SOURCE)
SIGMOID_SLOTS, *NS_SLOTS = (int(x) for x in SLOTS.groups())
ceil = lambda a, b: -(-a // b)


# ---------------------------------------------------------------- the list of a CTA's items
def _lists(lens, pos0, per, groups, mask, max_new, sms, least=2):
    """(items of every launched CTA, tokens an item); an item is (first token, end, sequence, group)."""
    count = lambda f: sum(f(n, p) for n, p in zip(lens, pos0) if n >= least)
    bound = lambda tiles: ceil(max_new, tiles * per) * groups * len(lens)
    grid = max(min(bound(1), sms), ceil(bound(2), ITEMS))
    span, g = per, grid
    if bound(1) > sms:
        span, items = 2 * per, groups * count(lambda n, p: ceil(n, 2 * per))
        if items < sms:
            keys = max([n + p for n, p in zip(lens, pos0) if n >= least], default=0)
            far = (min(keys, mask) if mask else keys) // 3 * 2
            if groups * count(lambda n, p: max(ceil(n, per) - max(far - p, 0) // per, 0)) <= sms:
                span, items = per, groups * count(lambda n, p: ceil(n, per))
        g = max(min(items, sms), ceil(items, ITEMS))
    assert g <= grid
    order = [(t * span, min(n, (t + 1) * span), b, hg) for t in reversed(range(ceil(max_new, span))) for b, n in enumerate(lens)
             if n >= least and t * span < n for hg in range(groups)]
    out = []
    for c in range(grid):
        mine, k, want = [], 0, c
        while c < g and want < len(order) and k < ITEMS:
            mine.append(order[want])
            k += 1
            want = k * g + (g - 1 - c if (k + 1) // 2 % 2 else c)
        out.append(mine)
    return out, span


@pytest.mark.parametrize("seed", range(60))
def test_every_item_is_taken_once(seed):
    r = random.Random(seed)
    n_seqs, per, groups = r.choice([1, 2, 5, 40, 200]), r.choice([16, 32, 64, 128]), r.choice([1, 2, 8, 32])
    lens = [r.choice([0, 1, 1, r.randint(2, 90), r.randint(2, 5000)]) for _ in range(n_seqs)]
    pos0, max_new = [r.choice([0, r.randint(1, 3000)]) for _ in lens], max(lens) + r.choice([0, 0, 700])
    lists, span = _lists(lens, pos0, per, groups, r.choice([0, 100, 1024]), max(max_new, 1), 148)
    got = sorted(i for mine in lists for i in mine)
    assert got == sorted((t, min(n, t + span), b, g) for b, n in enumerate(lens) if n > 1 for t in range(0, n, span) for g in range(groups))
    assert span in (per, 2 * per) and max(len(mine) for mine in lists) <= ITEMS


# ---------------------------------------------------------------- an item's key list
class Item:
    def __init__(self, t0, end, pos0, per, box, kind, mask, keep):
        low = lambda i: 0 if mask <= 0 else max(0, i - mask + 1) if kind == "window" else i // mask * mask
        keep_r, j_lo, j_hi = ceil(keep, box) * box, low(pos0 + t0), pos0 + end - 1
        pre = 0 < keep and keep_r <= j_lo
        n_pre, pre_r, keep_in = (keep, keep_r, 0) if pre else (0, 0, keep)
        jl = j_lo // box * box if pre or keep == 0 else 0
        self.tiles = ceil(pre_r + j_hi - jl + 1, KEYS)
        self.key = lambda v: v if v < pre_r else jl + v - pre_r
        self.listed = [v for v in range(self.tiles * KEYS) if v < n_pre or pre_r <= v <= pre_r + j_hi - jl]
        self.spans, self.sees = [None, None], [set(), set()]
        for g in range(2):
            t = t0 + g * per
            if t >= end:
                continue
            first, last = (max(low(pos0 + t) - jl, 0) + pre_r) // KEYS, (pos0 + min(end, t + per) - 1 - jl + pre_r) // KEYS
            self.spans[g] = (min(ceil(n_pre + keep_in, KEYS), last + 1), first, last)
            for i in range(pos0 + t, pos0 + min(end, t + per)):
                self.sees[g] |= {j for j in range(i + 1) if j >= low(i) or (mask > 0 and j < keep)}

    def has(self, g, j):
        s = self.spans[g]
        return s is not None and (j < s[0] or s[1] <= j <= s[2])


def _items(r, per):
    out = []
    for _ in range(r.randint(1, 5)):
        t0, mask = r.choice([0, per, 2 * per * r.randint(1, 6)]), r.choice([0, 60, 300, 1000])
        out.append(Item(t0, t0 + r.randint(1, 2 * per), r.choice([0, r.randint(1, 900)]), per, r.choice([16, 32, 64]), r.choice(["window", "chunk"]), mask,
                        r.choice([0, 0, 4, 17, 200]) if mask else 0))
    return out


@pytest.mark.parametrize("seed", range(40))
def test_every_visible_key_is_in_a_tile_of_its_rows(seed):
    r = random.Random(seed)
    for m in _items(r, r.choice([16, 64, 128])):
        where = {}
        for v in m.listed:
            assert m.key(v) not in where, "a key twice"
            where[m.key(v)] = v // KEYS
        for g in range(2):
            assert all(m.has(g, where[j]) for j in m.sees[g])


# ---------------------------------------------------------------- the warps of a CTA
class Cta:
    """Barriers as counts of completed phases.  A role is a generator that yields what it waits for: (barrier, completions)."""

    def __init__(self, items, ns, nv, slots, rng):
        self.items, self.ns, self.nv, self.slots, self.rng = items, ns, nv, slots, rng
        self.done, self.ring, self.q, self.s, self.o = {}, [None] * slots, [None, None], [None, None], [None, None]
        self.copies, self.products, self.results = [], [], []

    def arrive(self, bar):
        self.done[bar] = self.done.get(bar, 0) + 1

    def fill(self, t, keys, slot):
        n = self.ns if keys else self.nv
        old = t * (self.ns + self.nv) + (0 if keys else self.ns) + n - 1 - self.slots
        if old >= 0:
            ot = (old + self.nv) // (self.ns + self.nv)
            yield ("empty", ot % DEEP), ot // DEEP + 1
        where = [(slot + i) % self.slots for i in range(n)]
        for w in where:
            self.ring[w] = None                                      # from its issue on, the copy may land at any time
        self.copies.append((where, ("K" if keys else "V", t), ("k" if keys else "v", t % DEEP)))

    def loader(self):
        t = slot = 0
        uses = [0, 0]
        for x, m in enumerate(self.items):
            for j in range(m.tiles):
                yield from self.fill(t, True, slot)
                for g in range(2):
                    if j == 0 and m.spans[g]:
                        if uses[g]:
                            yield ("q_empty", g), uses[g]
                        self.q[g] = None
                        self.copies.append((g, x, ("q", g)))
                        uses[g] += 1
                yield from self.fill(t, False, (slot + self.ns) % self.slots)
                slot, t = (slot + self.ns + self.nv) % self.slots, t + 1

    def cleaner(self):
        t = 0
        for m in self.items:
            for _ in range(m.tiles):
                yield ("v", t % DEEP), t // DEEP + 1
                slot = t * (self.ns + self.nv) + self.ns
                assert all(self.ring[(slot + i) % self.slots] == ("V", t) for i in range(self.nv))
                self.arrive(("clean", t % DEEP))
                t += 1

    def issuer(self):
        t, q_uses, p_uses = 0, [0, 0], [0, 0]
        for x, m in enumerate(self.items):
            was, begun = [False, False], [False, False]
            for j in range(m.tiles + 1):
                if j > 0:
                    yield ("clean", (t - 1) % DEEP), (t - 1) // DEEP + 1
                if j < m.tiles:
                    yield ("k", t % DEEP), t // DEEP + 1
                for g in range(2):
                    now = j < m.tiles and m.has(g, j)
                    if was[g]:
                        yield ("p", g), p_uses[g] + 1
                        p_uses[g] += 1
                    if now and not begun[g]:
                        yield ("q", g), q_uses[g] + 1
                    if was[g]:
                        self.products.append(("pv", g, x, j - 1, t - 1, begun[g]))
                        if m.spans[g][2] == j - 1:
                            self.products.append(("commit", ("o", g)))
                    if now:
                        self.products.append(("s", g, x, j, t))
                        self.products.append(("commit", ("s", g)))
                        if m.spans[g][2] == j:
                            self.products.append(("commit", ("q_empty", g)))
                            q_uses[g] += 1
                    if g == 1 and j < m.tiles:
                        self.products.append(("commit", ("empty", t % DEEP)))
                    begun[g], was[g] = begun[g] or was[g], now
                t += j < m.tiles

    def softmax(self, g):
        s_uses = o_uses = 0
        for x, m in enumerate(self.items):
            if not m.spans[g]:
                continue
            tiles = [j for j in range(m.spans[g][2] + 1) if m.has(g, j)]
            for j in tiles:
                yield ("s", g), s_uses + 1
                s_uses += 1
                assert self.s[g] == ("S", x, j)
                self.s[g] = ("P", x, j)
                self.arrive(("p", g))
            yield ("o", g), o_uses + 1
            o_uses += 1
            assert self.o[g] == [(x, j) for j in tiles]
            self.results.append((x, g))

    def land(self):
        where, what, bar = self.copies.pop(self.rng.randrange(len(self.copies)))
        if bar[0] == "q":
            self.q[where] = what
        else:
            for w in where:
                self.ring[w] = what
        self.arrive(bar)

    def multiply(self):
        op, *a = self.products.pop(0)                                # in the order of their issue
        per = self.ns + self.nv
        if op == "commit":
            self.arrive(a[0])
        elif op == "s":
            g, x, j, t = a
            assert self.q[g] == x and all(self.ring[(t * per + i) % self.slots] == ("K", t) for i in range(self.ns))
            assert self.s[g] is None or self.s[g][0] == "used"
            self.s[g] = ("S", x, j)
        else:
            g, x, j, t, more = a
            assert self.s[g] == ("P", x, j) and all(self.ring[(t * per + self.ns + i) % self.slots] == ("V", t) for i in range(self.nv))
            self.s[g] = ("used",)
            self.o[g] = (self.o[g] if more else []) + [(x, j)]

    def run(self):
        roles = [self.loader(), self.cleaner(), self.issuer(), self.softmax(0), self.softmax(1)]
        waits = {i: None for i in range(len(roles))}                 # None: ready
        while waits or self.copies or self.products:
            ready = [i for i, w in waits.items() if w is None or self.done.get(w[0], 0) >= w[1]]
            steps = ready + ["copy"] * bool(self.copies) + ["product"] * bool(self.products)
            assert steps, f"nothing can go on: {waits}"
            at = self.rng.choice(steps)
            if at == "copy":
                self.land()
            elif at == "product":
                self.multiply()
            else:
                w = waits[at]
                # a parity tells phases apart only while the barrier is not a whole turn ahead
                assert w is None or self.done.get(w[0], 0) <= w[1], w
                try:
                    waits[at] = next(roles[at])
                except StopIteration:
                    del waits[at]


@pytest.mark.parametrize("ns,nv,slots", [(1, 1, NS_SLOTS[0]), (1, 2, NS_SLOTS[0]), (2, 1, NS_SLOTS[1]), (2, 2, NS_SLOTS[1]), (3, 1, NS_SLOTS[2]), (3, 2, NS_SLOTS[2]),
                                         (1, 1, SIGMOID_SLOTS), (2, 2, SIGMOID_SLOTS)])
@pytest.mark.parametrize("seed", range(12))
def test_roles_in_any_order(ns, nv, slots, seed):
    r = random.Random(seed * 100 + slots + ns)
    items = _items(r, r.choice([16, 64, 128]))
    cta = Cta(items, ns, nv, slots, r)
    cta.run()
    assert sorted(cta.results) == sorted((x, g) for x, m in enumerate(items) for g in range(2) if m.spans[g])
