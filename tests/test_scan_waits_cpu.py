"""The waits of the scans' read kernel (``csrc/chunk_scan_tcgen05.cu``): a barrier's phase is awaited by its parity, so that no phase may pass twice
while a warp has not looked at it.  The roles' waits and arrivals are walked through here, with one warp held back at each of its steps in turn
until none of the others can go on; when the parts of the scores may be written anew is read from the source."""

import re
from pathlib import Path

import pytest

SOURCE = (Path(__file__).resolve().parents[1] / "miniserve-llm-nv_b200" / "csrc" / "chunk_scan_tcgen05.cu").read_text()
COUNTS = {"keys": 8, "scores_read": 8, "parts_full": 8, "parts_free": 2, "slot0": 8, "slot1": 8, "result0": 1, "result1": 1}


class Names:
    def __init__(self, **values):
        self.__dict__.update(values)


def rule(pattern, otherwise):
    """A condition or a number of the source as a Python expression."""
    found = re.search(pattern, SOURCE)
    return (found.group(1) if found else otherwise).replace("&&", "and")


WAITED, PARITY = rule(r"if \((.*)\) waits\.wait\(&parts_free", "True"), rule(r"waits\.wait\(&parts_free, (.*), \d+\);", "")
FREED = rule(r"if \((.*)\) umma_commit\(&parts_free\)", "True")


def units_of(first_tile, count, tiles, heads, per_group):
    """(tile, new keys, new head) of a block's units."""
    units, tile, head = [], first_tile, 0
    for i in range(count):
        units.append(Names(tile=tile, new_keys=i == 0 or (tile == 0 and head % per_group == 0), new_head=i == 0 or tile == 0))
        tile += 1
        if tile == tiles:
            tile, head = 0, (head + 1) % heads
    return units


def operand_warp(units, blocks):
    """Steps: ("arrive", barrier), ("wait", barrier, parity), ("meet", place, warps)."""
    keys, results = 0, [0, 0]
    for u in units:
        if u.new_keys:
            yield "arrive", "keys"
            yield "wait", "scores_full", keys & 1
            keys += 1
        for halves in (blocks, 2):                     # the product with S_0, then that of scores and values
            for h in range(halves):
                yield "arrive", f"slot{h}"
            for h in range(halves):
                yield "wait", f"result{h}", results[h] & 1
                results[h] += 1


def score_warp(warp, units, blocks, tiles, seen):
    quarter, half = warp & 3, warp >> 2
    issues, operands, heads, groups = quarter == 0, 0, 0, 0
    run = Names(tiles=tiles, last=len(units))
    for n, u in enumerate(units):
        if u.new_head:
            yield "meet", "all", 8
        start = issues and half < blocks
        if start and u.new_keys:
            yield "wait", "keys", groups & 1
            yield "arrive", "scores_full"
        elif start:
            yield "wait", f"slot{half}", operands & 1
            yield "arrive", f"result{half}"
            operands += 1
        names = dict(u=u, run=run, heads=heads, n=n, at=n)
        if eval(WAITED, {}, names):
            yield "wait", "parts_free", eval(PARITY, {}, names)
        if u.new_head:
            heads += 1
            if u.new_keys:
                yield "wait", "scores_full", groups & 1
                groups += 1
                yield "arrive", "scores_read"
                yield "meet", f"quarter{quarter}", 2
                if start:
                    yield "wait", "scores_read", (groups - 1) & 1
                    yield "wait", f"slot{half}", operands & 1
                    yield "arrive", f"result{half}"
                    operands += 1
            assert all(done >= n for done in seen.values()), "parts written that a product still reads"
            yield "arrive", "parts_full"
        if issues:
            if u.new_head:
                yield "wait", "parts_full", (heads - 1) & 1
            yield "wait", f"slot{half}", operands & 1
            operands += 1
            yield "arrive", f"result{half}"
            seen[half] = n + 1                         # (this half's products of so many units are done)
            if eval(FREED, {}, names):
                yield "arrive", "parts_free"


def finishes(units, blocks, tiles, held, after):
    """Whether all roles come to their end when warp `held` stands still before step `after` until no other can go on."""
    counts = dict(COUNTS, scores_full=blocks)
    phases, arrived, met = {name: 0 for name in counts}, {name: 0 for name in counts}, {}
    seen = {0: 0, 1: 0}
    warps = [operand_warp(units, blocks) for _ in range(8)] + [score_warp(w, units, blocks, tiles, seen) for w in range(8)]
    step, taken, meets, there = [next(w, None) for w in warps], [0] * 16, [{} for _ in warps], [False] * 16

    def advance(w):
        """One step of a warp, if it can take it."""
        if step[w] is None:
            return False
        kind, name, *rest = step[w]
        if kind == "wait" and (phases[name] & 1) == rest[0]:
            return False                               # (the phase under way has the awaited parity)
        if kind == "arrive":
            arrived[name] += 1
            if arrived[name] == counts[name]:
                phases[name], arrived[name] = phases[name] + 1, 0
        if kind == "meet":
            came = not there[w]
            if came:
                met[name], there[w], meets[w][name] = met.get(name, 0) + 1, True, meets[w].get(name, 0) + 1
            if met[name] < meets[w][name] * rest[0]:
                return came
            there[w] = False
        step[w], taken[w] = next(warps[w], None), taken[w] + 1
        return True

    def run(stop):
        going = True
        while going:
            going = False
            for w in range(16):
                while not (stop and w == held and taken[w] == after) and advance(w):
                    going = True

    run(True)
    run(False)
    return all(s is None for s in step), taken[held] if held is not None else 0


@pytest.mark.parametrize("blocks", [1, 2])
@pytest.mark.parametrize("first_tile,count,tiles,heads,per_group", [(0, 12, 5, 8, 1), (3, 9, 5, 8, 1), (0, 9, 1, 8, 4), (1, 10, 2, 6, 3), (0, 7, 3, 2, 2), (0, 1, 1, 1, 1),
                                                                    (0, 8, 8, 1, 1)])
def test_no_wait_is_overtaken(blocks, first_tile, count, tiles, heads, per_group):
    units = units_of(first_tile, count, tiles, heads, per_group)
    done, _ = finishes(units, blocks, tiles, None, None)
    assert done
    for held in (0, 7, 8, 9, 12, 15):                  # an operand warp, the two that issue, others of the scores'
        after = 0
        while True:
            done, steps = finishes(units, blocks, tiles, held, after)
            assert done, f"warp {held} held back before its step {after}"
            after += 1
            if after >= steps:
                break
