"""The named barriers of the training kernel (kGrad, mlp.cu) as a model on the host.

Row warps, the feature and bias warps and the issuing warp run as coroutines that
arrive at and wait for the kernel's barriers; the waits for a product may give up at any
point, after which a warp no longer waits for products.  However they do, every
warp has to reach the end, each barrier's phases filled by one arrival per warp."""
import random
from collections import Counter

import pytest

ROWS, FEATURES, BIASES, ISSUER = range(16), range(16, 20), range(20, 24), 24


class Barriers:
    def __init__(self):
        self.arrived, self.phase = {}, Counter()

    def arrive(self, name, warp, warps):
        here = self.arrived.setdefault(name, [])
        assert warp not in here, f"warp {warp} twice in a phase of {name}"
        here.append(warp)
        if len(here) == warps:
            self.arrived[name] = []
            self.phase[name] += 1


def run(tiles, seed, give_up, meet):
    """meet: the row warps wait at the operands' barrier (as the kernel does) or only arrive."""
    rng, bar, done = random.Random(seed), Barriers(), Counter()

    def sync(name, warp, warps):
        p = bar.phase[name]
        bar.arrive(name, warp, warps)
        while bar.phase[name] == p:
            yield

    def row(w):
        ok, product = True, 0

        def wait():
            nonlocal ok, product
            product += 1
            while ok and done["products"] < product:
                if rng.random() < give_up:
                    ok = False
                yield

        def ready():
            if meet:
                yield from sync("op", w, 17)
            else:
                bar.arrive("op", w, 17)

        for tile in range(tiles):
            yield from sync(f"x{tile % 2}", w, 21)
            for layer in range(3):
                yield from wait()
                if layer == 0 and 0 < tile < tiles - 1:
                    bar.arrive("xfree", w, 20)
                yield from ready()
            yield from wait()
            if tile:
                yield from sync("free", w, 20)
            for layer in (3, 2, 1, 0):
                if layer < 3:
                    yield from wait()
                bar.arrive(f"dz{layer}", w, 17)
                yield from ready()
        yield from wait()
        yield from sync("rows", w, 16)

    def feature(w):
        for tile in range(tiles):
            if tile >= 2:
                yield from sync("xfree", w, 20)
            bar.arrive(f"x{tile % 2}", w, 21)
            yield

    def biases(w):
        for tile in range(tiles):
            yield from sync(f"dz{w - BIASES[0]}", w, 17)
            if tile + 1 < tiles:
                bar.arrive("free", w, 20)

    def issuer():
        for tile in range(tiles):
            for layer in range(4):
                yield from (sync(f"x{tile % 2}", ISSUER, 21) if layer == 0 else sync("op", ISSUER, 17))
                done["issued"] += 1
            for layer in (3, 2, 1, 0):
                yield from sync("op", ISSUER, 17)
                done["issued"] += layer > 0
        done["issued"] += 1  # the last products

    def tensor_core():
        while True:
            if done["products"] < done["issued"] and rng.random() < 0.2:
                done["products"] += 1
            yield

    live = {w: row(w) for w in ROWS}
    live.update({w: feature(w) for w in FEATURES})
    live.update({w: biases(w) for w in BIASES})
    live[ISSUER] = issuer()
    core = tensor_core()
    for _ in range(400000):
        if not live:
            return True
        next(core)
        w = rng.choice(list(live))
        if next(live[w], "end") == "end":
            del live[w]
    return False


@pytest.mark.parametrize("tiles", [1, 2, 3, 5])
@pytest.mark.parametrize("give_up", [0.0, 0.002, 0.05, 1.0])
def test_every_warp_ends(tiles, give_up):
    for seed in range(4):
        assert run(tiles, seed, give_up, True)


def test_arrivals_alone_fall_out_of_step():
    with pytest.raises(AssertionError, match="twice in a phase of op"):
        for seed in range(20):
            assert run(2, seed, 0.05, False)
