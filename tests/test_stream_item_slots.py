"""The item slots of the row-streaming gate/up kernel (csrc/gemv_q4k_stream.cu: produce, Cursor, the s_next wait), replayed as state
machines under random interleavings with warps of very different speed: octet q goes to producer q mod 4 and consumer warp
q mod W, a producer waits only for the octet that had its stage before, the warp that finishes an item's eighth octet writes the
item out, and a warp stores into an item's slot only once the slot's previous item is written out. No slot may ever hold two
items at once, and every item is written out. The words that tell whose turn a slot is start at zero, whatever an earlier launch left."""
import os
import random
import re

import pytest

PRODUCERS, OCTETS = 4, 8


def run(stages, warps, slots, items, rng, guarded, slow, words=None):
    """Returns whether a store ever met another item's unwritten results, and the number of items written out. words: s_next at the start."""
    octets = items * OCTETS
    armed, released = set(), set()
    prod = list(range(PRODUCERS))
    cons = [{"q": w, "state": "wait"} for w in range(warps)]
    holder, done, nxt = [None] * slots, [0] * slots, list(words or [0] * slots)
    clash, written, idle = False, 0, 0
    while written < items and not clash:
        i = rng.randrange(PRODUCERS + warps)
        if i < PRODUCERS:
            q = prod[i]
            if q < octets and (q < stages or q - stages in released):
                armed.add(q)
                prod[i] += PRODUCERS
                idle = 0
        else:
            c = cons[i - PRODUCERS]
            if c["q"] >= octets or (i - PRODUCERS == slow and rng.random() < 0.995):
                continue
            item = c["q"] // OCTETS
            s = item % slots
            if c["state"] == "wait":
                if c["q"] in armed and (not guarded or item < slots or nxt[s] == item):
                    clash |= holder[s] not in (None, item)
                    holder[s] = item
                    c["state"] = "stored"
                    idle = 0
            elif c["state"] == "stored":
                released.add(c["q"])
                done[s] += 1
                c["state"] = "write" if done[s] == OCTETS else "wait"
                if c["state"] == "wait":
                    c["q"] += warps
                else:
                    done[s] = 0
                idle = 0
            else:
                clash |= holder[s] != item
                holder[s], nxt[s] = None, item + slots
                written += 1
                c["q"] += warps
                c["state"] = "wait"
                idle = 0
        idle += 1
        assert idle < 200000, "no progress"
    return clash, written


# stages, consumer warps and item slots that the plan gives for rows of 256 to 2048 weights, few and many entries
@pytest.mark.parametrize("stages,warps,slots", [(40, 16, 16), (31, 16, 8), (20, 16, 8), (13, 10, 8), (4, 2, 4)])
def test_no_slot_holds_two_items(stages, warps, slots):
    rng = random.Random(stages)
    for slow in (None, 0, warps - 1):
        clash, written = run(stages, warps, slots, 60, rng, True, slow)
        assert not clash and written == 60


def test_the_stages_alone_do_not_keep_items_apart():
    """What the wait is for: without it a warp that falls behind meets a slot that a later item has taken."""
    rng = random.Random(3)
    assert any(run(40, 16, 16, 60, rng, False, 0)[0] for _ in range(3))
    assert any(run(31, 16, 8, 60, rng, False, 0)[0] for _ in range(3))


def test_words_of_an_earlier_launch():
    """Shared memory outlives a launch: one of a single lap leaves in s_next the numbers that the next launch's second lap waits for."""
    left = [s + 16 for s in range(16)]
    rng = random.Random(3)
    assert any(run(40, 16, 16, 60, rng, True, 0, left)[0] for _ in range(3))
    src = open(os.path.join(os.path.dirname(__file__), "..", "strix-halo-engine-lab_b200", "csrc", "gemv_q4k_stream.cu")).read()
    assert re.search(r"s_next = s_done \+ plan\.item_slots;", src)
    assert re.search(r"i < 2 \* plan\.item_slots; i \+= blockDim\.x\) s_done\[i\] = 0;\s+ring_init", src), "s_done and s_next start at zero, before the block's barrier"
