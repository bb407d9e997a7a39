"""CPU test of the prefill GEMM's rings: the order that its barriers give, on a model of the kernel's threads (gemm_tc.cu).

Every thread is a list of waits for a barrier's phase and arrivals at one; a phase is over when all that belong to it have arrived.  What
must have happened before what follows from program order and from the waits.  Three things are asked:
  - a wait by parity also returns while the phase before is open: that one must be known to be over;
  - the phase after must not be over before the wait, which would then not return;
  - the scales of an int4 stage have no barrier of their own: they must have been read when a copy fills their slot again.
Ring sizes come from the header (gemm_tile.cuh), compiled on the host.
"""
import json
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
TILES = [(4, 2, 128), (4, 1, 128), (4, 1, 64), (8, 2, 128), (8, 1, 128), (8, 1, 64)]
NAMES = ["kWSlots", "kXSlots", "kABufs", "kUnitBars", "kScaleSlots"]
SEGMENT = 4  # stages of an int8 segment


@pytest.fixture(scope="module")
def sizes(tmp_path_factory):
    d = tmp_path_factory.mktemp("rings")
    values = ", ".join(f"(int)T::{n}" for n in NAMES)
    rows = "\n".join(f'  show<Tile<{b}, {cb}, {nt}>>("{b} {cb} {nt}", "{"{" if i == 0 else ","}");' for i, (b, cb, nt) in enumerate(TILES))
    (d / "rings.cpp").write_text(f"""#include <cstdio>
#include "{ROOT}/ruai_b200/csrc/gemm_tile.cuh"
using namespace gemm_tc;
template <typename T> void show(const char* name, const char* before) {{
  std::printf("%s\\"%s\\": [{", ".join(["%d"] * len(NAMES))}]", before, name, {values});
}}
int main() {{
{rows}
  std::printf("}}\\n");
}}
""")
    subprocess.run(["g++", "-std=c++17", "-o", str(d / "rings"), str(d / "rings.cpp")], check=True)
    out = json.loads(subprocess.run([str(d / "rings")], check=True, capture_output=True, text=True).stdout)
    return {k: dict(zip(NAMES, v)) for k, v in out.items()}


class Model:
    """A CTA of `tiles` tiles with `groups` groups of 32 k each."""

    def __init__(self, bits, cb, ring, groups, tiles):
        self.bits, self.cb, self.ring, self.groups, self.tiles = bits, cb, ring, groups, tiles
        self.nst = (groups + 1) // 2
        self.count = self.nst * tiles
        self.before, self.waits, self.phases, self.last = {}, [], {}, {}
        self.reads, self.copies = {}, {}  # of a stage's scales
        self.copiers()
        for h in range(2):
            self.issuer(h)
        for half in range(2):  # two warps stand for all that do the same
            for block in range(cb):
                if cb == 2:
                    self.drainer(block, half, True)
                else:
                    self.drainer(0, half, False)
                    for it in range(self.count):
                        self.expand(("expand", half), it, 0)

    def op(self, thread, *after):
        node = (thread, len(self.before))
        self.before[node] = [n for n in (self.last.get(thread),) + after if n is not None]
        self.last[thread] = node
        return node

    def wait(self, thread, barrier, phase):
        at = self.last.get(thread)
        self.waits.append((at, self.op(thread, ("over", barrier, phase)), barrier, phase))

    def arrive(self, thread, barrier, phase):
        self.phases.setdefault((barrier, phase), []).append(self.op(thread))

    def copiers(self):
        for name, slots in (("w", self.ring["kWSlots"]), ("x", self.ring["kXSlots"])):
            for it in range(self.count):
                if it >= slots:
                    self.wait(name, (name + "_empty", it % slots), it // slots - 1)
                self.arrive(name, (name + "_full", it % slots), it // slots)
                if name == "w":
                    self.copies[it] = self.last[name]

    def expand(self, thread, it, block):
        ws, ab = self.ring["kWSlots"], self.ring["kABufs"]
        self.wait(thread, ("w_full", it % ws), it // ws)
        if it >= ab:
            self.wait(thread, ("a_free", it % ab), it // ab - 1)
        self.arrive(thread, ("a_ready", it % ab), it // ab)
        self.arrive(thread, ("w_empty", it % ws), it // ws)

    def full(self, u):
        return ("acc_full", u % self.ring["kUnitBars"]), u // self.ring["kUnitBars"]

    def free(self, u):
        return ("acc_free", u % self.ring["kUnitBars"]), u // self.ring["kUnitBars"]

    def units(self, s):
        return min(2, self.groups - 2 * s)

    def issuer(self, h):
        me, cb, nst, ab, xs = ("issue", h), self.cb, self.nst, self.ring["kABufs"], self.ring["kXSlots"]
        unit = 0 if self.bits == 4 and cb == 1 else h

        def sums_free(u):
            if u >= 3:
                self.wait(me, *self.free(u - 3))

        for it in range(self.count):
            s, at = it % nst, it % nst % SEGMENT
            mine = cb == 2 or (s & 1) == h
            if self.bits == 4 and not mine:
                unit += self.units(s)
                continue
            if mine:
                self.wait(me, ("a_ready", it % ab), it // ab)
                self.wait(me, ("x_full", it % xs), it // xs)
                if self.bits == 4:
                    for _ in range(self.units(s)):
                        sums_free(unit)
                        self.arrive(me, *self.full(unit))
                        unit += cb
                else:
                    if at < 3 - cb:
                        sums_free(unit)
                    if at + 3 - cb >= SEGMENT or s + 3 - cb >= nst:
                        self.arrive(me, *self.full(unit))
                        unit += 2
                self.arrive(me, ("x_empty", it % xs), it // xs)
                self.arrive(me, ("a_free", it % ab), it // ab)
            elif h == 1 and at == 0 and s + 1 == nst:
                sums_free(unit)
                self.arrive(me, *self.full(unit))
                unit += 2

    def drainer(self, block, half, both):
        me, cb, nst = ("drain", block, half), self.cb, self.nst
        unit = block
        if both:
            self.expand(me, 0, block)
        for it in range(self.count):
            s = it % nst
            if both and it + 1 < self.count:
                self.expand(me, it + 1, block)
            n = self.units(s) if self.bits == 4 else 3 - cb if s % SEGMENT == SEGMENT - 1 or s + 1 == nst else 0
            for _ in range(n):
                self.wait(me, *self.full(unit))
                self.reads.setdefault(it, []).append(self.op(me))
                self.arrive(me, *self.free(unit))
                unit += cb

    def order(self):
        """For every event the set of those that must have come before it, as a bit mask."""
        edges = {n: list(p) for n, p in self.before.items()}
        for (barrier, phase), arrivals in self.phases.items():
            edges[("over", barrier, phase)] = arrivals
        number, past, todo = {n: i for i, n in enumerate(edges)}, {}, []
        for root in edges:
            todo.append((root, False))
            while todo:
                n, ready = todo.pop()
                if n in past:
                    continue
                if not ready:
                    past_open = [p for p in edges[n] if p not in past]
                    if past_open:
                        todo.append((n, True))
                        todo.extend((p, False) for p in past_open)
                        continue
                mask = 0
                for p in edges[n]:
                    mask |= past[p] | 1 << number[p]
                past[n] = mask
        return lambda a, b: a == b or bool(past[b] >> number[a] & 1)  # a before b

    def faults(self):
        before, out = self.order(), []
        for at, wait, barrier, phase in self.waits:
            if phase >= 1 and (at is None or not all(before(n, at) for n in self.phases[barrier, phase - 1])):
                out.append(("the phase before may be open", wait[0], barrier, phase))
            if (barrier, phase + 1) in self.phases and not before(wait, ("over", barrier, phase + 1)):
                out.append(("the phase after may be over", wait[0], barrier, phase))
        if self.bits == 4:
            n = self.ring["kScaleSlots"]
            out += [("scales overwritten", it) for it in range(self.count - n) if not all(before(r, self.copies[it + n]) for r in self.reads[it])]
        return out


@pytest.mark.parametrize("groups", list(range(1, 13)) + [17, 18])
@pytest.mark.parametrize("bits,cb,nt", TILES)
def test_order_of_the_barriers(sizes, bits, cb, nt, groups):
    ring = sizes[f"{bits} {cb} {nt}"]
    assert Model(bits, cb, ring, groups, max(2, -(-36 // ((groups + 1) // 2)))).faults() == []


def test_the_model_sees_faults():
    ring = {"kWSlots": 6, "kXSlots": 5, "kABufs": 4, "kUnitBars": 6, "kScaleSlots": 13}
    assert {f[0] for f in Model(4, 1, dict(ring, kScaleSlots=12), 1, 36).faults()} == {"scales overwritten"}
    # a barrier per buffer: one column block with an odd number of stages, two with any
    assert any(f[0] == "the phase before may be open" for f in Model(4, 1, dict(ring, kUnitBars=3), 18, 4).faults())
    two = {"kWSlots": 4, "kXSlots": 5, "kABufs": 2, "kUnitBars": 3, "kScaleSlots": 8}
    assert any(f[0] == "the phase before may be open" for f in Model(4, 2, two, 18, 4).faults())
