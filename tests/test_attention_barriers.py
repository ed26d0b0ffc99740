"""The tcgen05 prompt attention's barriers, every order of events tried on the CPU.

The kernel's parts (a thread that loads keys and issues score products, one that loads values and issues output products,
warps that turn scores into probabilities and zero the unseen rows of a tile's values) are restated as lists of waits and
actions; loads and products complete at any time after they are issued.  The waits before the zeroing are read from the
kernel's source.  An mbarrier knows only its phase's parity: a wait passes where the number of completed phases has the
other parity."""
import os
import re

import pytest

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ghost_infer_b200", "csrc", "attention_prefill_t5.cu")


def waits_before_zeroing(stages):
    """[(condition on j, barrier of j, parity of j)] out of the block that zeroes rows of values."""
    text = open(SOURCE).read()
    block = text[text.index("if (lo > lo_kept || hi < BKV) {"):]
    block = block[:block.index("unsigned char* vt")]

    def python(expr):
        expr = expr.replace("(uint32_t)", "").replace("&&", " and ").replace("/", "//")
        return lambda j: eval(expr, {"j": j, "V_STAGES": stages, "ok": True})

    found = []
    for cond, bar, index, parity in re.findall(r"(?:if \((.*)\) )?ok = mbar_wait\((\w+)0 \+ 8 \* (.+?), (\(uint32_t\).+), 3, &g_attn_status\)", block):
        found.append((python(cond or "True"), lambda j, bar=bar, index=python(index): (bar, index(j)), python(parity)))
    assert len(found) == block.count("mbar_wait(") > 0
    return found


def programs(tiles, stages, warps, waits, edges):
    keys, values, rows = [], [], []
    for t in range(min(2, tiles)):
        keys.append(("issue", ("K", t)))
    for j in range(tiles):
        s = j & 1
        keys.append(("wait", ("k_full", s), j >> 1 & 1))
        if j >= 2:
            keys.append(("wait", ("kv_empty", s), j - 2 >> 1 & 1))
        keys.append(("issue", ("S", j)))
        if j + 2 < tiles:
            keys += [("wait", ("s_full", s), j >> 1 & 1), ("issue", ("K", j + 2))]
    for t in range(min(stages, tiles)):
        values.append(("issue", ("V", t)))
    for j in range(tiles):
        values += [("wait", ("p_full", j & 1), j >> 1 & 1), ("wait", ("v_full", j & stages - 1), j // stages & 1), ("issue", ("O", j))]
        if j + stages < tiles:
            values += [("wait", ("kv_empty", j & 1), j >> 1 & 1), ("issue", ("V", j + stages))]
    for j in range(tiles):
        rows.append(("wait", ("s_full", j & 1), j >> 1 & 1))
        if j in edges:
            rows += [("wait", bar(j), parity(j)) for cond, bar, parity in waits if cond(j)] + [("zero", j)]
        rows.append(("arrive", ("p_full", j & 1)))
    rows.append(("wait", ("kv_empty", tiles - 1 & 1), tiles - 1 >> 1 & 1))
    rows.append(("read output", tiles))
    return [keys, values] + [rows] * warps


def first_fault(tiles, stages, waits, edges, warps=2):
    """What goes wrong in some order of events where the tiles `edges` have rows to zero, or None."""
    progs = programs(tiles, stages, warps, waits, edges)
    # state: places in the programs, loads and products under way, (barrier, arrivals) pairs, per stage of values (tile, has come,
    # warps that zeroed it), output products done
    start = (tuple(0 for _ in progs), frozenset(), (), tuple((None, False, 0) for _ in range(stages)), 0)
    seen, todo = {start}, [start]
    while todo:
        at, flying, arrivals, slots, done = todo.pop()
        count = dict(arrivals)
        phases = lambda bar: count.get(bar, 0) // (warps if bar[0] == "p_full" else 1)
        after = []
        for i, prog in enumerate(progs):
            if at[i] == len(prog):
                continue
            op, moved = prog[at[i]], at[:i] + (at[i] + 1,) + at[i + 1:]
            if op[0] == "wait":
                if phases(op[1]) & 1 != op[2]:
                    after.append((moved, flying, arrivals, slots, done))
            elif op[0] == "issue":
                new = slots
                if op[1][0] == "V":
                    s = op[1][1] % stages
                    new = slots[:s] + ((op[1][1], False, 0),) + slots[s + 1:]
                after.append((moved, flying | {op[1]}, arrivals, new, done))
            elif op[0] == "arrive":
                after.append((moved, flying, tuple(sorted({**count, op[1]: count.get(op[1], 0) + 1}.items())), slots, done))
            elif op[0] == "zero":
                s = op[1] % stages
                tile, come, zeroed = slots[s]
                if tile != op[1] or not come:
                    return f"rows of tile {op[1]} zeroed in a stage that holds or awaits tile {tile}"
                after.append((moved, flying, arrivals, slots[:s] + ((tile, come, zeroed + 1),) + slots[s + 1:], done))
            else:
                if done != op[1]:
                    return "output read before its products are done"
                after.append((moved, flying, arrivals, slots, done))
        for event in flying:                               # something completes
            kind, j = event
            new, ready = slots, done
            bars = {"K": [("k_full", j & 1)], "V": [("v_full", j % stages)], "S": [("s_full", j & 1)], "O": [("o_full", 0), ("kv_empty", j & 1)]}[kind]
            if kind == "V":
                new = slots[:j % stages] + ((j, True, 0),) + slots[j % stages + 1:]
            elif kind == "O":
                if done != j:
                    continue                               # one issuing thread's products run in their order
                if slots[j % stages] != (j, True, warps if j in edges else 0):
                    return f"the product of tile {j} reads {slots[j % stages]}"
                ready = done + 1
            elif kind == "S" and ("S", j - 1) in flying:
                continue
            more = {**count, **{b: count.get(b, 0) + 1 for b in bars}}
            after.append((at, flying - {event}, tuple(sorted(more.items())), new, ready))
        if not after and any(p < len(prog) for p, prog in zip(at, progs)):
            return "all wait for one another"
        for state in after:
            if state not in seen:
                seen.add(state)
                todo.append(state)
    return None


def edge_sets(tiles):
    """A ragged end, a window's edge in the first tile, in the second, every tile."""
    last = tiles - 1
    return {frozenset(e) for e in ((last,), (0,), (0, last), (min(1, last), last), range(tiles))}


@pytest.mark.parametrize("stages", [1, 2])
@pytest.mark.parametrize("tiles", [1, 2, 3, 4, 5])
def test_no_order_of_events_zeroes_or_reads_the_wrong_values(tiles, stages):
    for edges in edge_sets(tiles):
        assert first_fault(tiles, stages, waits_before_zeroing(stages), edges) is None, sorted(edges)


def test_with_one_stage_the_wait_for_a_tiles_own_values_is_not_enough():
    """What the search finds where a tile's own arrival is all that is waited for; with two stages it is enough."""
    own = lambda stages: [(lambda j: True, lambda j: ("v_full", j & stages - 1), lambda j: j // stages & 1)]
    for tiles in (2, 3, 4):
        assert "zeroed" in first_fault(tiles, 1, own(1), {tiles - 1})
        assert first_fault(tiles, 2, own(2), {tiles - 1}) is None
