"""CPU test of the prefill GEMM's shared-memory rings: what a copy overwrites has been read, by the order that the kernel's barriers give.

The scales of an int4 stage have no barrier of their own: their reuse rests on the other rings' (gemm_tile.cuh).  The model below has one
event per copy, expansion, MMA and read-out of a unit, an edge for every barrier wait and for every thread's program order, and asks
whether the read-outs of a stage precede the copy into its slot.  Ring sizes come from the header, compiled on the host.
"""
import json
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
TILES = [(4, 2, 128), (4, 1, 128), (4, 1, 64)]


@pytest.fixture(scope="module")
def sizes(tmp_path_factory):
    d = tmp_path_factory.mktemp("rings")
    rows = "\n".join(f'  show(Tile<{b}, {cb}, {nt}>{{}}, "{b} {cb} {nt}");' for b, cb, nt in TILES)
    (d / "rings.cpp").write_text(f"""#include <cstdio>
#include "{ROOT}/ruai_b200/csrc/gemm_tile.cuh"
using namespace gemm_tc;
template <typename T> void show(T, const char* name) {{
  std::printf("%s\\"%s\\": [%d, %d, %d]", name[2] == '2' ? "{{" : ", ", name, T::kWSlots, T::kABufs, T::kScaleSlots);
}}
int main() {{
{rows}
  std::printf("}}\\n");
}}
""")
    subprocess.run(["g++", "-std=c++17", "-o", str(d / "rings"), str(d / "rings.cpp")], check=True)
    return json.loads(subprocess.run([str(d / "rings")], check=True, capture_output=True, text=True).stdout)


def unread(cb, w_slots, a_bufs, scale_slots, groups, count):
    """Stages whose scales may be overwritten before they are read, among the first `count` of a CTA whose tiles have `groups` groups each."""
    per_tile = (groups + 1) // 2
    units, unit = [], 0  # per stage: its units as (number, issuing thread, draining warps)
    for it in range(count):
        s = it % per_tile
        ng = min(2, groups - 2 * s)
        mine = []
        for _ in range(ng):
            for h in range(cb):
                mine.append((unit, h if cb == 2 else s & 1, h))
                unit += 1
        units.append(mine)
    before = {}  # event -> events that precede it directly

    def after(event, *others):
        before.setdefault(event, []).extend(o for o in others if o is not None)

    last_issue, last_read, last_expand = {}, {}, None
    for it in range(count):
        after(("copy", it), ("copy", it - 1) if it else None, ("expand", it - w_slots) if it >= w_slots else None)
        after(("expand", it), ("copy", it), last_expand)
        if it >= a_bufs:
            after(("expand", it), *[("mma", u) for u, _, _ in units[it - a_bufs]])
        last_expand = ("expand", it)
        for u, thread, block in units[it]:
            after(("mma", u), ("expand", it), last_issue.get(thread), ("read", u - 3) if u >= 3 else None)
            last_issue[thread] = ("mma", u)
            after(("read", u), ("mma", u), last_read.get(block))
            if cb == 2 and it + 1 < count:
                after(("read", u), ("expand", it + 1))  # the draining warps expand the next stage first
            last_read[block] = ("read", u)
    past = {}

    def ancestors(event):
        if event not in past:
            seen, todo = set(), list(before.get(event, ()))
            while todo:
                e = todo.pop()
                if e not in seen:
                    seen.add(e)
                    todo.extend(before.get(e, ()))
            past[event] = seen
        return past[event]

    return [it for it in range(count - scale_slots) if any(("read", u) not in ancestors(("copy", it + scale_slots)) for u, _, _ in units[it])]


@pytest.mark.parametrize("groups", range(1, 9))
@pytest.mark.parametrize("bits,cb,nt", TILES)
def test_scales_are_read_before_their_slot_is_filled_again(sizes, bits, cb, nt, groups):
    w_slots, a_bufs, scale_slots = sizes[f"{bits} {cb} {nt}"]
    assert unread(cb, w_slots, a_bufs, scale_slots, groups, 60) == []


def test_the_model_sees_a_ring_that_is_too_short():
    assert unread(1, 6, 4, 12, 1, 60) and not unread(1, 6, 4, 12, 2, 60)
    assert unread(2, 4, 2, 7, 3, 60)
