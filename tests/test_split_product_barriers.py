"""The barriers of the 32-bit product on tensor cores (`csrc/gemm_f32_split.cu`), tried in random orders of events without a GPU.

An mbarrier's wait names a phase by its parity alone, so a role that looks at a barrier only every second phase may pass while the
phase before is still open.  The roles (loads, split rows and tokens, products, draining) are walked here as coroutines over barriers
that know parities only; every piece of data carries its chunk's number, and a stale one is noticed where it is read.  The numbers of
stages, slots and warps, the barriers' counts and the waits' distances are read from the kernel's source; a wait that has another form
there fails the test.
"""
import os
import random
import re

import pytest

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ghost_infer_b200", "csrc", "gemm_f32_split.cu")


def source():
    with open(SOURCE) as f:
        return re.sub(r"\s+", " ", re.sub(r"//[^\n]*", "", f.read()))


def value(expr, names):
    """A C expression of whole numbers, names and `?:`."""
    expr = expr.strip()
    cond = re.fullmatch(r"(\w+) \? (.+?) : (.+)", expr)
    if cond:
        return value(cond.group(2) if names[cond.group(1)] else cond.group(3), names)
    return int(eval(expr.replace("S::", ""), {"__builtins__": {}}, dict(names)))


def kernel(few, cluster):
    """What the walk needs of the kernel, from its source."""
    text, names = source(), {"FEW": few, "CLUSTER": cluster}

    def found(pattern, n=1):
        hits = re.findall(pattern, text)
        assert len(hits) == n, f"the kernel's source has {len(hits)} of {pattern!r}, wanted {n}: bring this walk in line with it"
        return hits[0]

    for name in ("W_STAGES", "X_STAGES", "A_STAGES", "SLOTS", "SETS", "PARTS"):
        names[name] = value(found(rf"\b{name} = ([^,;]+)[,;]"), names)
    names["STRETCHES"] = value(found(r"constexpr int STRETCHES = ([^;]+);"), names)
    k = {n.lower(): names[n] for n in ("W_STAGES", "X_STAGES", "A_STAGES", "SLOTS", "SETS", "PARTS", "STRETCHES")}
    for bar in ("w_full", "w_empty", "full", "done", "large", "small"):
        k["count_" + bar] = value(found(rf"mbar_init\({bar}(?: \+ 8 \* i)?, ([^;]+)\);"), names)
    # the waits: how far behind, and which parity
    k["behind_x"] = value(found(r"wait_done\(it - (S::\w+), 1\)"), names)
    k["behind_a"] = value(found(r"wait_done\(it - (S::\w+), 3\)"), names)
    k["behind_tokens"] = value(found(r"wait_done\(it - (S::\w+), 5\)"), names)
    k["drained_for"] = value(found(r"mbar_arrive\(full \+ 8 \* \(\(it \+ (\d+)\) % S::SLOTS\)\)"), names)
    found(r"mbar_wait\(full \+ 8 \* \(it % S::SLOTS\), \(uint32_t\)\(\(it / S::SLOTS\) & 1\), who\)")
    found(r"it < 0 \|\| mbar_wait\(done \+ 8 \* \(it % S::SLOTS\), \(uint32_t\)\(\(it / S::SLOTS\) & 1\), who\)")
    found(r"mbar_wait\(w_empty \+ 8 \* st, \(uint32_t\)\(\(it / S::W_STAGES\) & 1\) \^ 1, 1\)")
    found(r"mbar_wait\(w_full \+ 8 \* ws, \(uint32_t\)\(\(it / S::W_STAGES\) & 1\), 3\)")
    found(r"if \(fresh && stretches\+\+ > 0\) \{ ok = __all_sync\(0xffffffffu, mbar_wait\(small, \(uint32_t\)\(stretches & 1\), 2\)\)")
    found(r"ok = __all_sync\(0xffffffffu, wait_full\(it, 2\)\)")
    found(r"ok = mbar_wait\(large \+ 8 \* \(it % S::SLOTS\), \(uint32_t\)\(\(it / S::SLOTS\) & 1\), 4\)")
    found(r"ok = wait_done\(it, 4\)")
    found(r"if \(lane == 0\) mbar_arrive\(full\);")
    found(r"it % S::SETS != set")
    found(r"for \(int it = warp - 2; it < total && ok; it \+= 2\)")
    return k


class Bar:
    def __init__(self, count):
        self.count = self.left = count
        self.phase = 0

    def arrive(self):
        assert self.left > 0
        self.left -= 1
        if self.left == 0:
            self.phase += 1
            self.left = self.count

    def ready(self, parity):
        return (self.phase & 1) != parity


def walk(seed, k, few, cluster, w_tma, tiles, chunks):
    """`tiles` tiles of `chunks` chunks (of a cluster's block: its own stretches' chunks of one tile)."""
    rnd = random.Random(seed)
    w_stages, x_stages, a_stages, slots, sets, parts = (k[n] for n in ("w_stages", "x_stages", "a_stages", "slots", "sets", "parts"))
    bars = lambda n, count: [Bar(count) for _ in range(n)]
    w_full, w_empty, full, done = bars(w_stages, k["count_w_full"]), bars(w_stages, k["count_w_empty"]), bars(slots, k["count_full"]), bars(slots, k["count_done"])
    large, small = bars(slots, k["count_large"]), Bar(k["count_small"])
    w, x, a, d, s = [None] * w_stages, [None] * x_stages, [[None] * 4 for _ in range(a_stages)], [None], []
    is_full = lambda it: full[it % slots].ready(it // slots & 1)
    is_done = lambda it: it < 0 or done[it % slots].ready(it // slots & 1)
    per = max(1, (chunks + k["stretches"] - 1) // k["stretches"])
    total = tiles * chunks
    copies, issued, ended = [], [], []

    def loads():
        for it in range(total):
            if w_tma:
                st = it % w_stages
                while not w_empty[st].ready((it // w_stages & 1) ^ 1):
                    yield

                def land(st=st, it=it):
                    w[st] = it
                    w_full[st].arrive()
                copies.append(land)
                yield
            if not few:
                while not is_done(it - k["behind_x"]):
                    yield
                left = [3]

                def plane(it=it, left=left):
                    x[it % x_stages] = it if left[0] == 1 else None
                    left[0] -= 1
                    if left[0] == 0:
                        full[it % slots].arrive()
                copies.extend([plane] * 3)
                yield

    def tokens(first):
        for it in range(first, total, 2):
            while not is_done(it - k["behind_tokens"]):
                yield
            x[it % x_stages] = it
            yield
            full[it % slots].arrive()
            yield

    def split(which, q):
        for it in range(total):
            if it % sets != which:
                continue
            st = it % w_stages
            while w_tma and not w_full[st].ready(it // w_stages & 1):
                yield
            while not is_done(it - k["behind_a"]):
                yield
            for _ in range(2):
                assert not w_tma or w[st] == it, "stale rows"
                a[it % a_stages][q] = it
                yield
            if w_tma:
                w_empty[st].arrive()
                yield
            full[it % slots].arrive()
            yield

    def products():
        stretches = 0
        for it in range(total):
            fresh = it % chunks % per == 0
            while not is_full(it):
                yield

            def first(it=it):
                assert x[it % x_stages] == it and a[it % a_stages] == [it] * 4, "stale operands"
                d[0] = it
            issued.extend([first, large[it % slots].arrive])
            if fresh:
                stretches += 1
                while stretches > 1 and not small.ready(stretches & 1):
                    yield

            def others(it=it, fresh=fresh):
                assert x[it % x_stages] == it and a[it % a_stages] == [it] * 4, "stale operands"
                if fresh:
                    s.clear()
                s.append(it)

            def commit(it=it):
                assert x[it % x_stages] == it and a[it % a_stages] == [it] * 4 and d[0] == it, "operands overwritten"
                done[it % slots].arrive()
            issued.extend([others, commit])
            yield

    def drain(q):
        full[0].arrive()
        yield
        for it in range(total):
            while not large[it % slots].ready(it // slots & 1):
                yield
            for _ in range(2):
                assert d[0] == it, "stale results"
                yield
            full[(it + k["drained_for"]) % slots].arrive()
            yield
            at = it % chunks
            if at % per == per - 1 or at == chunks - 1:
                while not is_done(it):
                    yield
                for _ in range(2):
                    assert s == list(range(it - at % per, it + 1)), "stale small products"
                    yield
                small.arrive()
                yield
        ended.append(1)

    roles = [loads(), products()] + [split(n, q) for n in range(sets) for q in range(4)] + [drain(q) for _ in range(parts) for q in range(4)]
    if few:
        roles += [tokens(0), tokens(1)]
    weights = [rnd.choice([1, 1, 4, 20]) for _ in roles]
    copy_weight, issue_weight = rnd.choice([1, 4, 20]), rnd.choice([1, 4, 20])
    for _ in range(400000):
        if not (roles or copies or issued):
            break
        c = rnd.random() * (sum(weights) + copy_weight + issue_weight)
        if c < copy_weight:
            if copies:
                copies.pop(rnd.randrange(len(copies)))()       # copies land in any order
        elif c < copy_weight + issue_weight:
            if issued:
                issued.pop(0)()
        elif roles:
            i = rnd.choices(range(len(roles)), weights)[0]
            try:
                next(roles[i])
            except StopIteration:
                roles.pop(i)
                weights.pop(i)
    assert len(ended) == 4 * parts and not roles, "not all ended"


@pytest.mark.parametrize("w_tma", [True, False])
@pytest.mark.parametrize("few,cluster", [(True, False), (True, True), (False, False)])
@pytest.mark.parametrize("tiles,chunks", [(1, 1), (1, 2), (1, 37), (3, 17), (2, 24)])
def test_no_order_of_events_shows_stale_data(few, cluster, w_tma, tiles, chunks):
    if cluster and tiles > 1:
        pytest.skip("a cluster's blocks take one tile")
    k = kernel(few, cluster)
    for seed in range(6):
        walk(seed, k, few, cluster, w_tma, tiles, chunks)


@pytest.mark.parametrize("few,cluster", [(True, False), (False, False)])
def test_a_thread_that_gives_up_waits_for_all_its_copies(few, cluster):
    """The loading thread may give up between a chunk's rows of W, which it has asked for by then, and its tokens."""
    text, k = source(), kernel(few, cluster)
    counts = {}
    for kind, stages in (("w", "w_stages"), ("x", "x_stages")):
        # counted behind its own copies, and as many of the last ones waited for as are under way
        assert re.search(rf"tma_load_2d\([^;]*&map_{kind}[^;]*;(?: }})? \+\+{kind}_loaded;", text), kind
        assert re.search(rf"for \(int i = max\(0, {kind}_loaded - S::{kind.upper()}_STAGES\); i < {kind}_loaded; \+\+i\)", text), kind
        counts[kind] = k[stages]
    for given_up_at in range(2 * 12):
        issued, loaded, place = set(), {"w": 0, "x": 0}, 0
        for it in range(12):
            for kind in "wx":
                if kind == "x" and few:
                    continue
                if place == given_up_at:
                    break
                place += 1
                issued = {c for c in issued if c[0] != kind or c[1] > it - counts[kind]} | {(kind, it)}     # the one before in its place has landed
                loaded[kind] += 1
            else:
                continue
            break
        waited = {(kind, i) for kind in "wx" for i in range(max(0, loaded[kind] - counts[kind]), loaded[kind])}
        assert issued <= waited


@pytest.mark.parametrize("change", [dict(w_stages=3), dict(count_small=4), dict(drained_for=2), dict(behind_a=5)])
def test_a_barrier_that_does_not_fit_is_found_out(change):
    """A ring that two sets share unevenly, a barrier that some of its warps do not count for, an accumulator drained for the wrong
    chunk, a place written while it is read."""
    few = "count_small" not in change
    k = dict(kernel(few, False), **change)
    failed = 0
    for seed in range(120):
        try:
            walk(seed, k, few, False, True, 2, 19)
        except AssertionError:
            failed += 1
            break
    assert failed > 0
