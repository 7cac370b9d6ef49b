"""CPU models of the mbarrier protocols of the warp-specialised kernels: every role is
a generator of waits, arrivals and asynchronous completions (a copy that lands, MMAs
that finish), run in random interleavings. A parity wait must never meet a barrier two
phases past the awaited one (it reads as not yet there), no role may stay stuck, and a
buffer must not be rewritten before its readers are done (checked at every write).

Operations: ("wait", bar, phase), ("arrive", bar), ("async", bar) (arrives later),
("touch", name, op, key): op "w" claims the buffer for content `key`, "r" asserts it
holds `key`, so a write under a reader or a read of newer content shows."""
import random

import pytest


class Model:
    def __init__(self, counts, rng):
        self.counts, self.rng = counts, rng
        self.arrived, self.done, self.content = {}, {}, {}

    def arrive(self, bar):
        n = self.arrived.get(bar, 0) + 1
        if n == self.counts.get(bar, 1):
            self.done[bar] = self.done.get(bar, 0) + 1
            n = 0
        self.arrived[bar] = n

    def run(self, roles):
        current = [next(r, None) for r in roles]
        pending = []
        while any(c is not None for c in current) or pending:
            movable = [i for i, c in enumerate(current) if c is not None and not (
                c[0] == "wait" and self.done.get(c[1], 0) <= c[2])]
            choices = [("role", i) for i in movable] + [("land", i) for i in range(len(pending))]
            assert choices, f"stuck at {current}"
            kind, i = self.rng.choice(choices)
            if kind == "land":
                op = pending.pop(i)
                for touch in op[2:]:
                    self.touch(touch)
                self.arrive(op[1])
                continue
            op = current[i]
            if op[0] == "wait":
                assert self.done.get(op[1], 0) < op[2] + 2, f"aliased wait {op}"
            elif op[0] == "arrive":
                self.arrive(op[1])
            elif op[0] == "async":
                pending.append(op)
            else:
                self.touch(op[1:])
            current[i] = next(roles[i], None)

    def touch(self, t):
        name, op, key = t
        if op == "w":
            self.content[name] = key
        else:
            assert self.content.get(name) == key, (name, "holds", self.content.get(name), "not", key)


WARPS = 2  # per group: enough for the arrival counts to matter


def transform_roles(n, nbuf=4):
    """ntt_tc_kernel: four tile buffers, two column sets."""
    def loader():
        for j in range(min(n, nbuf)):
            yield ("async", f"AFULL{j}", (f"buf{j}", "w", ("input", j)))
        for j in range(n):
            yield ("wait", f"STAGED{j % nbuf}", j // nbuf)
            if j >= 1:  # the store before this one has read its buffer
                yield ("touch", f"buf{(j - 1) % nbuf}", "r", ("result", j - 1))
                if j - 1 + nbuf < n:
                    b = (j - 1) % nbuf
                    yield ("async", f"AFULL{b}", (f"buf{b}", "w", ("input", j - 1 + nbuf)))

    def mma():
        for j in range(n):
            yield ("wait", f"AFULL{j % nbuf}", j // nbuf)
            if j >= 2:
                yield ("wait", f"FREAD{j & 1}", (j >> 1) - 1)
            yield ("async", f"FDONE{j & 1}", (f"buf{j % nbuf}", "r", ("input", j)),
                   (f"col{j & 1}", "w", j))

    def epilogue():
        for j in range(n):
            yield ("wait", f"FDONE{j & 1}", j >> 1)
            yield ("touch", f"col{j & 1}", "r", j)
            yield ("arrive", f"FREAD{j & 1}")
            yield ("touch", f"buf{j % nbuf}", "w", ("result", j))
            yield ("arrive", f"STAGED{j % nbuf}")

    counts = {f"{b}{i}": 2 * WARPS for b in ("FREAD", "STAGED") for i in range(nbuf)}
    return counts, [loader(), mma()] + [epilogue() for _ in range(2 * WARPS)]


def product_roles(n, nxa=3):
    """ntt_mul_tc_kernel: input boxes, b boxes, one S/D operand, two column sets."""
    def loader():
        boxes = 0
        for t in range(n):
            for h in range(2):
                s, use = boxes % nxa, boxes // nxa
                if use:
                    yield ("wait", f"AFREE{s}", use - 1)
                yield ("async", f"AFULL{s}", (f"xa{s}", "w", (t, h)))
                boxes += 1
            for h in range(2):
                if t:
                    yield ("wait", f"BFREE{h}", t - 1)
                yield ("async", f"BFULL{h}", (f"b{h}", "w", t))

    def mma():
        boxes = 0

        def inverse(j):
            yield ("wait", "PREADY", j)
            if j:
                yield ("wait", "EREAD", j - 1)
            yield ("async", "IDONE", ("pp", "r", j), ("icol", "w", j))
        for j in range(n):
            if j:
                yield ("wait", "FREAD", j - 1)
            for kb in range(2):
                s = boxes % nxa
                yield ("wait", f"AFULL{s}", boxes // nxa)
                yield ("async", f"AFREE{s}", (f"xa{s}", "r", (j, kb)))
                boxes += 1
            yield ("async", "FDONE", ("fcol", "w", j))
            if j:
                yield from inverse(j - 1)
        if n:
            yield from inverse(n - 1)

    def forward(h):
        for j in range(n):
            yield ("wait", "FDONE", j)
            for bt in range(2):
                yield ("touch", "fcol", "r", j)
                if bt == 1:
                    yield ("arrive", "FREAD")
                if bt == 0:
                    yield ("wait", f"BFULL{h}", j)
                yield ("touch", f"b{h}", "r", j)
                if bt == 1:
                    yield ("arrive", f"BFREE{h}")
                if bt == 0 and j:
                    yield ("wait", "IDONE", j - 1)
                yield ("touch", "pp", "w", j)
            yield ("arrive", "PREADY")

    def inverse_out():
        for j in range(n):
            yield ("wait", "IDONE", j)
            for bt in range(2):
                yield ("touch", "icol", "r", j)
                if bt == 1:
                    yield ("arrive", "EREAD")

    counts = {"FREAD": 2 * WARPS, "PREADY": 2 * WARPS, "EREAD": 2 * WARPS,
              "BFREE0": WARPS, "BFREE1": WARPS}
    return counts, ([loader(), mma()] + [forward(h) for h in (0, 1) for _ in range(WARPS)]
                    + [inverse_out() for _ in range(2 * WARPS)])


def planes_roles(n, nsx, nsp):
    """emm_pm_kernel: raw slots, plane slots."""
    def loader():
        for c in range(n):
            s = c % nsx
            if c >= nsx:
                yield ("wait", f"RAWFREE{s}", c // nsx - 1)
            yield ("async", f"FULL{s}", (f"raw{s}", "w", c))

    def builder():
        for c in range(n):
            s, p = c % nsx, c % nsp
            yield ("wait", f"FULL{s}", c // nsx)
            if c >= nsp:
                yield ("wait", f"PLFREE{p}", c // nsp - 1)
            yield ("touch", f"raw{s}", "r", c)
            yield ("touch", f"plane{p}", "w", c)
            yield ("arrive", f"BUILT{p}")
            yield ("arrive", f"RAWFREE{s}")

    def mma():
        for c in range(n):
            yield ("wait", f"BUILT{c % nsp}", c // nsp)
            yield ("async", f"PLFREE{c % nsp}", (f"plane{c % nsp}", "r", c))

    counts = {f"{b}{i}": 3 for b in ("BUILT", "RAWFREE") for i in range(2)}
    return counts, [loader(), mma()] + [builder() for _ in range(3)]


def grouped_roles(items, nsa, nsb, nacc):
    """batch_pm_kernel over one CTA's items (chunks each): loader, dead rows, builders, MMA,
    epilogue. A slot's rows are the loaded ones (a) and the cleared ones (z)."""
    chunks = [(it, c) for it, n in enumerate(items) for c in range(n)]

    def loader():
        for g in range(len(chunks)):
            s = g % nsa
            if g >= nsa:
                yield ("wait", f"AFREE{s}", g // nsa - 1)
            yield ("async", f"FULL{s}", (f"a{s}", "w", g))

    def zero(h):
        for g in range(len(chunks)):
            s = g % nsa
            yield ("wait", f"FULL{s}", g // nsa)
            yield ("touch", f"a{s}", "r", g)
            yield ("touch", f"z{h}{s}", "w", g)
            yield ("arrive", f"ZEROED{s}")

    def builder(h):
        for g in range(len(chunks)):
            p = g % nsb
            if g >= nsb:
                yield ("wait", f"BFREE{p}", g // nsb - 1)
            yield ("touch", f"b{h}{p}", "w", g)
            yield ("arrive", f"BUILT{p}")

    def mma():
        for g, (it, c) in enumerate(chunks):
            s, p, acc = g % nsa, g % nsb, it % nacc
            if c == 0 and it >= nacc:
                yield ("wait", f"AEMPTY{acc}", it // nacc - 1)
            yield ("wait", f"FULL{s}", g // nsa)
            yield ("wait", f"ZEROED{s}", g // nsa)
            yield ("wait", f"BUILT{p}", g // nsb)
            yield ("async", f"AFREE{s}", (f"a{s}", "r", g), (f"z0{s}", "r", g), (f"z1{s}", "r", g))
            yield ("async", f"BFREE{p}", (f"b0{p}", "r", g), (f"b1{p}", "r", g))
            if c == items[it] - 1:
                yield ("async", f"ACC{acc}", (f"acc{acc}", "w", it))

    def epilogue():
        for it in range(len(items)):
            acc = it % nacc
            yield ("wait", f"ACC{acc}", it // nacc)
            yield ("touch", f"acc{acc}", "r", it)
            yield ("arrive", f"AEMPTY{acc}")

    counts = {f"{b}{i}": 2 for b in ("ZEROED", "BUILT", "AEMPTY") for i in range(nsa)}
    return counts, ([loader(), mma()] + [zero(h) for h in (0, 1)] + [builder(h) for h in (0, 1)]
                    + [epilogue() for _ in (0, 1)])


def product256_roles(n):
    """ntt256_tc_mulinv_kernel: two groups, each with an operand and a buffer of its own, one
    tile of b between them."""
    def loader():
        for j in range(n):
            g, u = j & 1, j >> 1
            if u:
                yield ("wait", f"XFREE{g}", u - 1)
            yield ("async", f"AFULL{g}", (f"x{g}", "w", ("in", j)))
            if j:
                yield ("wait", f"BFREE{g ^ 1}", (j - 1) >> 1)
            yield ("async", f"BFULL{g}", ("b", "w", j))

    def mma(g):
        for u, j in enumerate(range(g, n, 2)):
            yield ("wait", f"PREP{g}", u)
            yield ("async", f"FDONE{g}", *((f"a{g}{h}", "r", ("fwd", j)) for h in range(WARPS)),
                   (f"col{g}", "w", ("fwd", j)))
            yield ("wait", f"PREADY{g}", u)
            yield ("async", f"IDONE{g}", *((f"a{g}{h}", "r", ("inv", j)) for h in range(WARPS)),
                   (f"col{g}", "w", ("inv", j)))

    def warp(g, h):
        syncs = 0
        for u, j in enumerate(range(g, n, 2)):
            yield ("wait", f"AFULL{g}", u)
            yield ("touch", f"x{g}", "r", ("in", j))
            yield ("touch", f"a{g}{h}", "w", ("fwd", j))
            yield ("arrive", f"PREP{g}")
            yield ("wait", f"FDONE{g}", u)
            yield ("touch", f"col{g}", "r", ("fwd", j))
            yield ("touch", f"x{g}", "w", ("ex", j))
            for phase in ("F", "E", "done"):
                if phase == "E":
                    yield ("wait", f"IDONE{g}", u)
                    yield ("touch", f"col{g}", "r", ("inv", j))
                    yield ("touch", f"a{g}{h}", "w", ("ex", j))
                yield ("arrive", f"SYNC{g}")
                yield ("wait", f"SYNC{g}", syncs)
                syncs += 1
                if phase == "F":
                    yield ("wait", f"BFULL{g}", u)
                    yield ("touch", "b", "r", j)
                    yield ("touch", f"x{g}", "r", ("ex", j))
                    yield ("touch", f"a{g}{h}", "w", ("inv", j))
                    for bar in ("BFREE", "XFREE", "PREADY"):
                        yield ("arrive", f"{bar}{g}")
                elif phase == "E":
                    for o in range(WARPS):
                        yield ("touch", f"a{g}{o}", "r", ("ex", j))

    counts = {f"{b}{g}": WARPS for b in ("XFREE", "BFREE", "PREP", "PREADY", "SYNC") for g in (0, 1)}
    return counts, ([loader(), mma(0), mma(1)]
                    + [warp(g, h) for g in (0, 1) for h in range(WARPS)])


def unit_roles(n, warps=4, group=2):
    """The JL kernels' hand-over: groups of warps share a barrier pair; n units go round
    the warps, a warp without a last unit arrives for its group."""
    def producer(w):
        g, unit, lead, it = w // group, w, w // group * group, 0
        while lead < n:
            if it:
                yield ("wait", f"EMPTY{g}", it - 1)
            if unit >= n:
                yield ("arrive", f"FULL{g}")
                return
            yield ("touch", f"tile{w}", "w", unit)
            yield ("arrive", f"FULL{g}")
            unit, lead, it = unit + warps, lead + warps, it + 1

    def mma():
        base = it = 0
        while base < n:
            for g in range(warps // group):
                if g * group + base >= n:
                    break
                yield ("wait", f"FULL{g}", it)
                reads = [(f"tile{w}", "r", w + base) for w in range(g * group, g * group + group)
                         if w + base < n]
                yield ("async", f"EMPTY{g}", *reads)
            base, it = base + warps, it + 1

    return ({f"FULL{g}": group for g in range(warps // group)},
            [mma()] + [producer(w) for w in range(warps)])


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 9, 13])
@pytest.mark.parametrize("kind", ["transform", "product", "planes11", "planes12", "planes22",
                                  "units", "product256"])
def test_protocol(n, kind):
    rng = random.Random(100 * n + len(kind))
    for _ in range(150):
        if kind == "transform":
            counts, roles = transform_roles(n)
        elif kind == "product":
            counts, roles = product_roles(n)
        elif kind == "product256":
            counts, roles = product256_roles(n)
        elif kind == "units":
            counts, roles = unit_roles(n)
        else:
            counts, roles = planes_roles(n, int(kind[-2]), int(kind[-1]))
        Model(counts, rng).run(roles)


@pytest.mark.parametrize("nsa,nsb,nacc", [(5, 2, 2), (3, 2, 1)])
def test_grouped_protocol(nsa, nsb, nacc):
    rng = random.Random(nsa)
    for _ in range(300):
        items = [rng.randint(1, 7) for _ in range(rng.randint(1, 5))]
        counts, roles = grouped_roles(items, nsa, nsb, nacc)
        Model(counts, rng).run(roles)


def test_model_finds_an_early_refill():
    """Planted in the model: a loader that refills a box one use too early."""
    def bad(n):
        counts, roles = product_roles(n)
        loader = roles[0]

        def skips():
            for op in loader:
                if not (op[0] == "wait" and op[1].startswith("AFREE")):
                    yield op
        return counts, [skips()] + roles[1:]
    rng = random.Random(3)
    with pytest.raises(AssertionError):
        for _ in range(300):
            counts, roles = bad(6)
            Model(counts, rng).run(roles)
