"""The order in which the read-out warps of the chunk-parallel backward write and read its partial-sum slots,
taken from the kernel's source: who waits for which barrier and arrives on which, in program order.

`combine` (two warps of the bulk group) reads in item i + 1 what both groups left there for item i.  Every
such read has to come after all writes for item i and before any write for item i + 1, by a chain of program
order and arrivals that lead to waits; how long the parts take does not count.  Nothing is run: a lost wait
is a race on shared memory."""

import itertools
import os
import re

import pytest

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "flashqla_b200", "csrc",
                      "bwd_main_tc.cu")
SLOTS = ("sRowW", "sRowDb", "sRowDg", "sColDg", "sLast")
ITEMS = 3
# the two warps that run combine, and one that stands for the others of the group
WARPS = {"bulk": ("combining", "other"), "chain": ("first", "second"), "issue": ("issue",)}

EVENT = re.compile(r"WAIT\((?P<wait>\w+), ph(?P<before> \^ 1)?\)|signal\((?P<signal>\w+)\)"
                   r"|mbar_arrive\(&bars\[(?P<arrive>\w+)\]\)|umma_commit\(&bars\[(?P<commit>\w+)\]\)"
                   r"|(?P<combine>combine)\(prev|(?P<slot>" + "|".join(SLOTS) + r")\[[^;]*\] = |(?P<take>take_next\(\);)")


def _blocks_without(text, head):
    """`text` without the blocks that `head` opens (and an else behind one)."""
    while (at := text.find(head)) >= 0:
        end = text.index("{", at)
        while True:
            depth = 0
            for end in range(end, len(text)):
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                if depth == 0:
                    break
            more = re.match(r"} else \{", text[end:])
            if not more:
                break
            end += more.end() - 1
        text = text[:at] + text[end + 1:]
    return text


def _events(text):
    text = re.sub(r"//[^\n]*", "", text)
    for m in EVENT.finditer(text):
        if m["wait"]:
            yield "wait", m["wait"], -1 if m["before"] else 0
        elif m["take"]:
            yield "wait", "I_NEXT", 0
        elif m["combine"]:
            yield "read", None, 0
        elif m["slot"]:
            yield "write", m["slot"], 0
        else:
            yield "arrive", m["signal"] or m["arrive"] or m["commit"], 0


def _program():
    """group -> its events of one item, in order"""
    src = open(SOURCE).read()
    cut = lambda a, b: src[src.index(a):src.index(b, src.index(a))]  # noqa: E731
    tail = cut("The chain group goes on to the next item", "prev_first = cur.row0")
    assert "WAIT(R_CH, ph);" in tail and "mbar_arrive(&bars[R_CH]);" in tail
    assert "chain_barrier();" in tail and "bulk_barrier();" in tail
    # which way an item takes here depends on its length: without either, only fewer things are in order
    issue = _blocks_without(_blocks_without(cut("for (bool has_next = true;", "read-out warps ="), "if (partial) {"),
                            "if (!partial) {")
    return {
        "chain": [*_events(cut("= chain group =", "= bulk group =")), ("arrive", "R_CH", 0), ("barrier", None, 0)],
        "bulk": [*_events(cut("= bulk group =", "The chain group goes on")), ("wait", "R_CH", 0), ("barrier", None, 0)],
        "issue": list(_events(issue)),
    }


@pytest.fixture(scope="module")
def order():
    """(nodes by kind, reachable): the events of three items and what comes after each of them"""
    after, seen, arrivals, waits, barriers = {}, {"read": [], "write": []}, {}, [], {}
    for group, events in _program().items():
        for warp in WARPS[group]:
            last = None
            for item, (at, (kind, name, back)) in itertools.product(range(ITEMS), enumerate(events)):
                if kind == "read" and (warp != "combining" or item == 0):
                    continue
                if kind == "wait" and item + back < 0:
                    continue
                node = (group, warp, item, at)
                after.setdefault(node, set())
                if last is not None:
                    after[last].add(node)
                last = node
                if kind == "wait":
                    waits.append((node, name, item + back))
                elif kind == "arrive":
                    arrivals.setdefault((name, item), []).append(node)
                elif kind == "barrier":
                    barriers.setdefault((group, item), []).append(node)
                else:
                    seen[kind].append((node, name))
    for node, name, item in waits:
        for a in arrivals.get((name, item), []):  # (none: the loads arrive on it)
            after[a].add(node)
    followers = {n: set(x) for n, x in after.items()}
    for nodes in barriers.values():
        for a, b in itertools.permutations(nodes, 2):
            after[a] |= followers[b]

    def reachable(a, b):
        todo, done = [a], set()
        while todo:
            n = todo.pop()
            if n == b:
                return True
            if n not in done:
                done.add(n)
                todo += after[n]
        return False

    return seen, reachable


def test_every_slot_is_found(order):
    seen, _ = order
    assert {name for _, name in seen["write"]} == set(SLOTS)
    assert len(seen["read"]) == ITEMS - 1


@pytest.mark.parametrize("slot", SLOTS)
def test_sums_are_read_between_their_writes(order, slot):
    seen, reachable = order
    for read, _ in seen["read"]:
        for write, name in seen["write"]:
            if name != slot:
                continue
            if write[2] < read[2]:
                assert reachable(write, read), (write, read)
            else:
                assert reachable(read, write), (read, write)
