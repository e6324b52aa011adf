"""The GEMM kernels' rings whose faults would depend on timing, model-checked on the CPU.

`fb_gemm_pair` with residual boxes (flint_b200/csrc/gemm.cu, kBoxes) passes an FP32 residual through a ring
of six boxes in shared memory: a warp of its own loads them ahead, in column order; eight epilogue warps,
one per 32 rows of every other box, add the product in place and store their rows by an asynchronous copy; a
warp gives its box back only once its copy has been read, which it learns one box later. The waits carry
only a phase parity. This file restates that protocol (slots, parities, who hands back what and when) as
cooperating generators, runs it under random schedules with random latencies of loads, products and
stores, and checks what every access finds. The generators and barriers are those of
tests/test_attention_protocol.py. A mistake is put into the model to show that the checker finds it.
"""

import random

import pytest

from test_attention_protocol import Barrier, Violation, need, schedule

SLOTS = 6          # kBoxSlots
BOXES = 8          # kPairBN / 32
QUADRANTS = 4


class BoxModel:
    def __init__(self, tiles, seed, variant="kernel"):
        # "kernel"; "early": a box is handed back as its store is issued, not once that has been read;
        # "own": a warp waits for its newest store too (correct, only slower).
        self.tiles, self.variant = tiles, variant
        self.rng = random.Random(seed)
        self.bar = {}
        for s in range(SLOTS):
            self.bar["box_full", s] = Barrier(f"box_full{s}", 1)
            self.bar["box_empty", s] = Barrier(f"box_empty{s}", QUADRANTS)
        for a in range(2):
            self.bar["acc_full", a] = Barrier(f"acc_full{a}", 1)
            self.bar["acc_empty", a] = Barrier(f"acc_empty{a}", 2 * QUADRANTS)
        self.content = [None] * SLOTS          # number of the box whose residual the slot holds
        self.reading = [0] * SLOTS             # stores issued from the slot and not yet read
        self.stored = set()                    # (box number, quadrant) read by its store
        self.accumulator = [None, None]        # tile whose product it holds
        self.loads, self.products, self.stores = [], [], []
        self.unread = {}                       # warp -> stores not yet read, oldest first

    def wait(self, kind, index, parity, phase):
        bar = self.bar[kind, index]
        while not bar.passed(parity & 1):
            yield
        need(bar.completed > phase, f"aliased wait on {bar.name}: meant phase {phase}, {bar.completed} completed")

    def producer(self):
        for sequence in range(self.tiles * BOXES):
            slot, lap = sequence % SLOTS, sequence // SLOTS
            yield from self.wait("box_empty", slot, (lap & 1) ^ 1, lap - 1)
            need(self.reading[slot] == 0, f"slot {slot} refilled while a store still reads it")
            need(lap == 0 or all((sequence - SLOTS, q) in self.stored for q in range(QUADRANTS)),
                 f"slot {slot} refilled before all of box {sequence - SLOTS} was stored")
            self.content[slot] = None
            self.loads.append((slot, sequence))
            yield

    def issuer(self):
        for tile in range(self.tiles):
            acc = tile & 1
            yield from self.wait("acc_empty", acc, ((tile >> 1) & 1) ^ 1, (tile >> 1) - 1)
            self.products.append((acc, tile))
            yield

    def epilogue(self, part, quadrant):
        mine = self.unread[part, quadrant] = []
        held = None
        for tile in range(self.tiles):
            acc = tile & 1
            yield from self.wait("acc_full", acc, (tile >> 1) & 1, tile >> 1)
            for box in range(part, BOXES, 2):
                sequence = tile * BOXES + box
                slot = sequence % SLOTS
                yield from self.wait("box_full", slot, (sequence // SLOTS) & 1, sequence // SLOTS)
                need(self.accumulator[acc] == tile, f"tile {tile} read from an accumulator that holds another")
                if box + 2 >= BOXES:
                    self.bar["acc_empty", acc].arrive()
                yield
                need(self.content[slot] == sequence, f"box {sequence} added to a slot that holds another")
                mine.append((slot, sequence, quadrant))
                self.stores.append(mine)
                self.reading[slot] += 1
                if self.variant == "early":
                    self.bar["box_empty", slot].arrive()
                    continue
                while len(mine) > (0 if self.variant == "own" else 1):     # wait_group.read
                    yield
                if held is not None:
                    self.bar["box_empty", held].arrive()
                held = slot
                yield

    def run_load(self):
        slot, sequence = self.loads.pop(self.rng.randrange(len(self.loads)))
        need(self.reading[slot] == 0, f"box {sequence} lands in a slot that a store still reads")
        self.content[slot] = sequence
        self.bar["box_full", slot].arrive()

    def run_product(self):
        acc, tile = self.products.pop(0)
        self.accumulator[acc] = tile
        self.bar["acc_full", acc].arrive()

    def run_store(self):
        mine = self.stores.pop(self.rng.randrange(len(self.stores)))      # a warp's in order, warps in any
        slot, sequence, quadrant = mine.pop(0)
        need(self.content[slot] == sequence, f"the store of box {sequence} reads another")
        self.reading[slot] -= 1
        self.stored.add((sequence, quadrant))

    def run(self):
        roles = {"producer": self.producer(), "issuer": self.issuer()}
        for part in range(2):
            for quadrant in range(QUADRANTS):
                roles[f"epilogue{part}.{quadrant}"] = self.epilogue(part, quadrant)
        schedule(self.rng, roles, [(self.loads, self.run_load), (self.products, self.run_product),
                                   (self.stores, self.run_store)])
        while self.stores:
            self.run_store()
        need(not self.loads and len(self.stored) == self.tiles * BOXES * QUADRANTS, "work left over at the end")


@pytest.mark.parametrize("tiles", [1, 2, 3, 4, 7])
def test_residual_boxes_hold_under_random_schedules(tiles):
    for seed in range(60):
        BoxModel(tiles, seed).run()


def test_waiting_for_every_store_holds_too():
    for seed in range(20):
        BoxModel(3, seed, variant="own").run()


def test_the_checker_notices_a_box_handed_back_before_its_store_was_read():
    found = 0
    for seed in range(100):
        try:
            BoxModel(3, seed, variant="early").run()
        except Violation as violation:
            found += 1
            assert "still reads" in str(violation) or "before all of box" in str(violation) or "reads another" in str(violation)
    assert found > 0
