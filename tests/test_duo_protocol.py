"""CPU: the protocol of the persistent two-tile kernel (csrc/attention_duo.cu) -- order of the copies, numbering of the K / V
blocks, phases of the barriers, turns of the two tiles -- as coroutines in random interleavings.  A copy or a multiplication
takes effect some time after it was asked for, in the order of its engine, and finds there what it was meant for."""
import random

import pytest

SLOTS, ITEMS, ORDERS = 2, 2, 8


class Bar:
    """mbarrier: a wait sees the parity of the completed phases only."""

    def __init__(self, count):
        self.count, self.left, self.phases = count, count, 0

    def arrive(self):
        self.left -= 1
        assert self.left >= 0
        if self.left == 0:
            self.left, self.phases = self.count, self.phases + 1

    def done(self, parity):
        return self.phases & 1 != parity & 1


class Tile:
    def __init__(self, name, group, first, blocks):
        self.name, self.group, self.first, self.blocks = name, group, first, blocks     # group: (head, class)


def stream(a, b):
    """shared, first block, number of the entries of an item"""
    shared = a.blocks > 0 and b.blocks > 0 and a.group == b.group and a.first <= b.first + b.blocks and b.first <= a.first + a.blocks
    first = min(a.first, b.first)
    return shared, first, (max(a.first + a.blocks, b.first + b.blocks) - first) if shared else a.blocks + b.blocks


class Model:
    def __init__(self, items, rng, asks_s_free=True):
        self.items, self.rng, self.asks_s_free = items, rng, asks_s_free
        pair = lambda count: [Bar(count), Bar(count)]
        self.q_full, self.q_free, self.o_full, self.s_full, self.pv_done = (pair(1) for _ in range(5))
        self.p_full = [pair(1), pair(1)]                 # (the four warps of a tile are one here)
        self.s_free = Bar(1)
        self.k_full, self.v_full, self.k_free, self.v_free = pair(1), pair(1), pair(2), pair(2)
        self.order_full = [Bar(1) for _ in range(ORDERS)]
        self.item_full, self.item_free = pair(1), pair(2 + 2 + 1)
        self.item, self.order = [None] * ITEMS, [None] * ORDERS
        self.q, self.k, self.v = [None] * 2, [None] * SLOTS, [None] * SLOTS     # what the memory holds
        self.s, self.p, self.o, self.p_out = None, [[None] * 2, [None] * 2], [None, None], [-1, -1]
        self.reads_p = [[0, 0], [0, 0]]                  # multiplications asked for that have yet to read P
        self.copies, self.tensor, self.out = [], [], {}
        self.early = 0                                   # two S in a row, the first not half exponentiated

    # a role yields a condition to wait for, or None for "some time passes"
    def plan(self):
        for n, it in enumerate(self.items + [None]):
            slot = n % ITEMS
            if n >= ITEMS:
                yield lambda: self.item_free[slot].done((n // ITEMS & 1) ^ 1)
            self.item[slot] = it
            self.item_full[slot].arrive()
            yield None

    def copy(self, memory, slot, tag, bar):
        def land():
            memory[slot] = tag
            bar.arrive()
        self.copies.append(land)

    def tma(self):
        entry, asked = 0, [0, 0]
        for n in range(len(self.items) + 1):
            slot = n % ITEMS
            yield lambda: self.item_full[slot].done(n // ITEMS & 1)
            it = self.item[slot]
            if it is None:
                return
            self.item_free[slot].arrive()
            shared, first, count = stream(*it)
            twice = 2 * min(it[0].blocks, it[1].blocks)
            for i in range(count):
                if shared:
                    x, block = 0, first + i
                    need_q = [t for t in (0, 1) if block == it[t].first]
                else:
                    k = i >> 1 if i < twice else i - twice // 2
                    x = i & 1 if i < twice else int(it[0].blocks <= it[1].blocks)
                    block, need_q = it[x].first + k, [x] if k == 0 else []
                for t in need_q:
                    if asked[t]:
                        yield lambda: self.q_free[t].done((asked[t] & 1) ^ 1)
                    self.copy(self.q, t, it[t].name, self.q_full[t])
                    asked[t] += 1
                st, parity = entry % SLOTS, (entry // SLOTS & 1) ^ 1
                for memory, full, free in ((self.k, self.k_full, self.k_free), (self.v, self.v_full, self.v_free)):
                    if entry >= SLOTS:
                        yield lambda: free[st].done(parity)
                    self.copy(memory, st, (it[x].group, block), full[st])
                    yield None
                entry += 1

    def qk(self):
        class Pipe:
            items = n = k = base = count = next = tiles = scores = first_entry = 0
            done = shared = False
            tile = other = None
        pipes, x, last_x, issued = [Pipe(), Pipe()], 0, -1, 0
        while not (pipes[0].done and pipes[1].done):
            me, other = pipes[x], pipes[x ^ 1]
            while not me.done and me.k == me.n:
                slot = me.items % ITEMS
                if not self.item_full[slot].done(me.items // ITEMS & 1):
                    break
                it = self.item[slot]
                self.item_free[slot].arrive()
                if it is None:
                    me.done, me.next = True, 1 << 30
                    break
                me.tile, me.other = it[x], it[x ^ 1]
                me.base += me.count
                me.shared, first, me.count = stream(*it)
                me.n, me.k, me.first_entry = me.tile.blocks, 0, me.tile.first - first
                me.next = me.base + (me.count if me.n == 0 else me.first_entry if me.shared else 0 if me.other.blocks == 0 else x)
                me.items += 1
            yield None
            go = me.k < me.n
            if go:
                k, m = me.k, me.other.blocks
                e = me.base + (me.first_entry + k if me.shared else 2 * k + x if k < m else m + k)
                st = e % SLOTS
                go = e - SLOTS < other.next and (k > 0 or self.q_full[x].done(me.tiles & 1)) and self.k_full[st].done(e // SLOTS & 1)
                if go and last_x == x:
                    go = (not self.asks_s_free or self.s_free.done((issued - 1) & 1)) and self.p_full[x][0].done((me.scores - 1) & 1)
                    if go and self.p_out[x] < me.scores - 1:
                        self.early += 1
            if go:
                block, last = me.tile.first + me.k, me.k + 1 == me.n
                both = me.shared and me.other.first <= block < me.other.first + me.other.blocks
                if issued:
                    want = issued - 1 & 1
                    yield lambda: self.s_free.done(want)
                self.tensor.append(self.multiply_s(x, me.scores, me.tile, block, st, last))
                if not both:
                    self.k_free[st].arrive()
                self.order[issued % ORDERS] = (x, me.scores, me.tile, block, st, e, me.k == 0, last, both)
                self.order_full[issued % ORDERS].arrive()
                issued, last_x = issued + 1, x
                me.tiles += last
                me.next = me.base + me.count if last else e + 1
                me.k, me.scores = me.k + 1, me.scores + 1
            x ^= 1
        self.order[issued % ORDERS] = None
        self.order_full[issued % ORDERS].arrive()

    def multiply_s(self, x, step, tile, block, st, last):
        def act():
            assert self.q[x] == tile.name and self.k[st] == (tile.group, block)
            self.s = (x, step, tile.name, block)
            self.s_full[x].arrive()
            self.k_free[st].arrive()
            if last:
                self.q_free[x].arrive()
        return act

    def pv(self):
        n, phase = 0, [0, 0]
        while True:
            slot = n % ORDERS
            yield lambda: self.order_full[slot].done(n // ORDERS & 1)
            if self.order[slot] is None:
                return
            x, step, tile, block, st, e, first, last, both = self.order[slot]
            yield lambda: self.v_full[st].done(e // SLOTS & 1)
            for half in (0, 1):
                yield lambda: self.p_full[x][half].done(phase[x])
                self.tensor.append(self.multiply_o(x, step, tile, block, st, half, first and half == 0))
            self.tensor.append(self.commit_o(x, st, last))
            if not both:
                self.v_free[st].arrive()
            phase[x] ^= 1
            n += 1

    def multiply_o(self, x, step, tile, block, st, half, overwrite):
        self.reads_p[x][half] += 1

        def act():
            self.reads_p[x][half] -= 1
            assert self.v[st] == (tile.group, block) and self.p[x][half] == (step, block)
            if overwrite:
                self.o[x] = (tile.name, [])
            assert self.o[x][0] == tile.name
            if half:
                self.o[x][1].append(block)
        return act

    def commit_o(self, x, st, last):
        def act():
            self.pv_done[x].arrive()
            self.v_free[st].arrive()
            if last:
                self.o_full[x].arrive()
        return act

    def softmax(self, x):
        g, tiles, now, n = 0, 0, None, 0
        while True:
            for k in range(now.blocks if now else 0):
                yield lambda: self.s_full[x].done(g & 1)
                assert self.s == (x, g, now.name, now.first + k)
                yield None
                assert self.s == (x, g, now.name, now.first + k)
                self.s_free.arrive()
                yield None
                if g:
                    yield lambda: self.pv_done[x].done((g - 1) & 1)
                for half in (0, 1):
                    yield None
                    assert self.reads_p[x][half] == 0
                    self.p[x][half] = (g, now.first + k)
                    if half == 0:
                        self.p_out[x] = g
                    self.p_full[x][half].arrive()
                g += 1
            was = now
            yield lambda: self.item_full[n % ITEMS].done(n // ITEMS & 1)
            it = self.item[n % ITEMS]
            self.item_free[n % ITEMS].arrive()
            now = it[x] if it else None
            if was:
                if was.blocks:
                    yield lambda: self.o_full[x].done(tiles & 1)
                    tiles += 1
                    yield None
                    assert self.o[x][0] == was.name
                    self.out[was.name] = list(self.o[x][1])
                    yield None
                    assert self.o[x][0] == was.name
                else:
                    self.out[was.name] = []
            if it is None:
                return
            n += 1

    def run(self):
        roles = [self.plan(), self.tma(), self.qk(), self.pv(), self.softmax(0), self.softmax(1)]
        pace = [self.rng.choice([1, 1, 3, 10]) for _ in range(len(roles) + 2)]
        waits = [None] * len(roles)
        idle = 0
        while any(r is not None for r in roles):
            i = self.rng.choices(range(len(pace)), pace)[0]
            moved = False
            if i >= len(roles):
                queue = (self.copies, self.tensor)[i - len(roles)]
                if queue:
                    queue.pop(0)()
                    moved = True
            elif roles[i] is not None and (waits[i] is None or waits[i]()):
                try:
                    waits[i] = next(roles[i])
                    moved = i != 2                       # (the QK role polls)
                except StopIteration:
                    roles[i] = None
                    moved = True
            idle = 0 if moved else idle + 1
            assert idle < 20000, "nobody moves"
        assert not self.copies and not self.tensor
        for it in self.items:
            for t in it:
                assert self.out[t.name] == list(range(t.first, t.first + t.blocks))


def _items(rng):
    items, name = [], 0
    for _ in range(rng.randint(1, 6)):
        it = []
        for x in range(2):
            near = it and it[0].blocks and rng.random() < 0.7
            blocks = 0 if rng.random() < 0.1 else rng.randint(1, 5)
            first = max(0, it[0].first + rng.randint(-1, it[0].blocks + 1)) if near else rng.randint(0, 9)
            it.append(Tile(name, it[0].group if near else ("head", name), first, blocks))
            name += 1
        items.append(it)
    return items


@pytest.mark.parametrize("seed", range(300))
def test_every_interleaving_computes_every_tile(seed):
    rng = random.Random(seed)
    m = Model(_items(rng), rng)
    m.run()
    assert m.early == 0


def test_a_parity_alone_does_not_tell_whose_turn_it_is():
    """Without a look at s_free first, the test of p_full reads the phase two steps back as complete."""
    early = 0
    for seed in range(300):
        rng = random.Random(seed)
        m = Model(_items(rng), rng, asks_s_free=False)
        m.run()
        early += m.early
    assert early > 0
