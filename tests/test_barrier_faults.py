"""The CPU models of the kernels' barrier protocols can fail: with any one kind of wait taken
out of a role, random interleavings show a buffer rewritten under a reader, a read of what
is not there yet, an aliased wait or a role that stays stuck. And the protocol of
amortize_tc_kernel, which the other models do not cover."""
import random

import pytest

import test_barrier_models as models
from test_barrier_models import Model

BUILDERS = 3  # warps: the first two write the words, all read them


def amortize_roles(n, na=4, nb=3):
    """amortize_tc_kernel: four tile slots, three matrix slots, the words of a matrix in two
    buffers behind the builders' own barrier."""
    def loader():
        for t in range(n):
            if t >= na:
                yield ("wait", f"AFREE{t % na}", t // na - 1)
            yield ("async", f"FULL{t % na}", (f"a{t % na}", "w", t))

    def mma():
        for t in range(n):
            yield ("wait", f"FULL{t % na}", t // na)
            yield ("wait", f"BUILT{t % nb}", t // nb)
            yield ("async", f"AFREE{t % na}", (f"a{t % na}", "r", t))
            yield ("async", f"BFREE{t % nb}", *((f"m{t % nb}{w}", "r", t) for w in range(BUILDERS)))

    def builder(w):
        for t in range(n):
            if w < 2:
                yield ("touch", f"words{t & 1}{w}", "w", t)
            if t >= nb:
                yield ("wait", f"BFREE{t % nb}", t // nb - 1)
            yield ("arrive", "SYNC")
            yield ("wait", "SYNC", t)
            for o in range(2):
                yield ("touch", f"words{t & 1}{o}", "r", t)
            yield ("touch", f"m{t % nb}{w}", "w", t)
            yield ("arrive", f"BUILT{t % nb}")

    counts = {"SYNC": BUILDERS, **{f"BUILT{i}": BUILDERS for i in range(nb)}}
    return counts, [loader(), mma()] + [builder(w) for w in range(BUILDERS)]


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 9, 13])
def test_amortize_protocol(n):
    rng = random.Random(n)
    for _ in range(150):
        counts, roles = amortize_roles(n)
        Model(counts, rng).run(roles)


def test_amortize_with_one_word_buffer():
    """Planted in the model: the words of every matrix in one buffer."""
    rng = random.Random(5)

    def one(role):
        for op in role:
            yield (op[0], "words0" + op[1][-1], *op[2:]) if op[0] == "touch" \
                and op[1].startswith("words") else op
    with pytest.raises(AssertionError):
        for _ in range(300):
            counts, roles = amortize_roles(7)
            Model(counts, rng).run([one(r) for r in roles])


PROTOCOLS = {
    "transform": lambda: models.transform_roles(9),
    "product": lambda: models.product_roles(6),
    "planes": lambda: models.planes_roles(6, 2, 2),
    "planes11": lambda: models.planes_roles(6, 1, 1),
    "grouped": lambda: models.grouped_roles([3, 2, 4, 1, 5], 3, 2, 1),
    "product256": lambda: models.product256_roles(8),
    "units": lambda: models.unit_roles(13),
    "amortize": lambda: amortize_roles(11),
}


# Waits that others imply: the clearing warps wait for the copies before they arrive, and
# the loader has waited for b's tile, which the same warps release with X.
IMPLIED = {("grouped", "mma", "FULL"), ("product256", "loader", "XFREE")}


class Uneven(random.Random):
    """Interleavings in which copies and MMAs finish late, or one role falls behind."""

    def new_run(self, roles):
        self.late, self.slow = self.random() < 0.5, self.randrange(2 * roles)

    def choice(self, seq):
        if self.random() < 0.9:
            few = [c for c in seq if (c[0] == "role" if self.late else c != ("role", self.slow))]
            seq = few or seq
        return super().choice(seq)


def _waits(name):
    """(role, barrier without its number) of every kind of wait."""
    counts, roles = PROTOCOLS[name]()
    kinds = {(role.__name__, op[1].rstrip("0123456789")) for role in roles for op in role
             if op[0] == "wait"}
    return sorted(k for k in kinds if (name, *k) not in IMPLIED)


@pytest.mark.parametrize("name,role,bar", [(n, r, b) for n in PROTOCOLS for r, b in _waits(n)])
def test_every_wait_is_needed(name, role, bar):
    rng = Uneven(len(bar))

    def without(ops):
        return (op for op in ops if not (op[0] == "wait" and op[1].rstrip("0123456789") == bar))
    with pytest.raises(AssertionError):
        for _ in range(800):
            counts, roles = PROTOCOLS[name]()
            rng.new_run(len(roles))
            Model(counts, rng).run([without(r) if r.__name__ == role else r for r in roles])


@pytest.mark.parametrize("name", PROTOCOLS)
def test_whole_protocols_pass_uneven_runs(name):
    rng = Uneven(1)
    for _ in range(200):
        counts, roles = PROTOCOLS[name]()
        rng.new_run(len(roles))
        Model(counts, rng).run(roles)
