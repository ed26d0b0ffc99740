"""The barriers of the 32-bit product on tensor cores (`csrc/gemm_f32_split.cu`), tried in random orders of events without a GPU.

An mbarrier's wait names a phase by its parity alone, so a role that looks at a barrier only every second phase may pass while the
phase before is still open.  The roles (loads, split rows and tokens, products, draining) are walked here as coroutines over barriers
that know parities only; every piece of data carries its chunk's number, and a stale one is noticed where it is read.
"""
import random

import pytest

SLOTS = 8


class Bar:
    def __init__(self, count):
        self.count = self.left = count
        self.phase = 0

    def arrive(self):
        self.left -= 1
        if self.left == 0:
            self.phase += 1
            self.left = self.count

    def ready(self, parity):
        return (self.phase & 1) != parity


def walk(seed, w_stages, x_stages, a_stages, sets, parts, few, chunks):
    rnd = random.Random(seed)
    bars = lambda k, n: [Bar(n) for _ in range(k)]
    w_full, w_empty, full, done = bars(w_stages, 1), bars(w_stages, 4), bars(SLOTS, 5 + 4 * parts), bars(SLOTS, 1)
    w, x, a, d = [None] * w_stages, [None] * x_stages, [[None] * 4 for _ in range(a_stages)], [None] * 2
    fw, fx = [[None] * 4 for _ in range(SLOTS)], [None] * SLOTS
    is_full = lambda it: full[it % SLOTS].ready(it // SLOTS & 1)
    is_done = lambda it: it < 0 or done[it % SLOTS].ready(it // SLOTS & 1)
    copies, commits, ended = [], [], []

    def loads():
        for it in range(chunks):
            st = it % w_stages
            while not w_empty[st].ready((it // w_stages & 1) ^ 1):
                yield

            def land(st=st, it=it):
                w[st] = it
                w_full[st].arrive()
            copies.append(land)
            yield
            if not few:
                while not is_done(it - x_stages):
                    yield
                left = [2]

                def part(which, it=it, left=left):
                    if which:
                        fx[it % SLOTS] = it
                    else:
                        x[it % x_stages] = it
                    left[0] -= 1
                    if left[0] == 0:
                        full[it % SLOTS].arrive()
                copies.extend([lambda part=part: part(0), lambda part=part: part(1)])
                yield

    def tokens(first):
        for it in range(first, chunks, 2):
            while not is_done(it - x_stages):
                yield
            x[it % x_stages] = fx[it % SLOTS] = it
            yield
            full[it % SLOTS].arrive()
            yield

    def split(which, q):
        for it in range(which, chunks, sets):
            st = it % w_stages
            while not w_full[st].ready(it // w_stages & 1):
                yield
            for _ in range(2):
                assert w[st] == it, "stale rows"
                yield
            w_empty[st].arrive()
            while not is_done(it - a_stages):
                yield
            a[it % a_stages][q] = fw[it % SLOTS][q] = it
            yield
            full[it % SLOTS].arrive()
            yield

    def products():
        for it in range(chunks):
            while not is_full(it):
                yield

            def run(it=it):
                assert x[it % x_stages] == it and a[it % a_stages] == [it] * 4, "stale operands"
                d[it & 1] = it

            def commit(it=it):
                assert x[it % x_stages] == it and a[it % a_stages] == [it] * 4 and d[it & 1] == it, "operands overwritten"
                done[it % SLOTS].arrive()
            commits.extend([run, commit])
            yield

    def drain(q):
        full[0].arrive()
        full[1].arrive()
        yield
        for it in range(chunks):
            while not (is_full(it) and is_done(it)):
                yield
            for _ in range(3):
                assert d[it & 1] == it and fw[it % SLOTS][q] == it and fx[it % SLOTS] == it, "stale results"
                yield
            full[(it + 2) % SLOTS].arrive()
            yield
        ended.append(1)

    roles = [loads(), products()] + [split(s, q) for s in range(sets) for q in range(4)] + [drain(q) for _ in range(parts) for q in range(4)]
    if few:
        roles += [tokens(0), tokens(1)]
    weights = [rnd.choice([1, 1, 4, 20]) for _ in roles]
    copy_weight, commit_weight = rnd.choice([1, 4, 20]), rnd.choice([1, 4, 20])
    for _ in range(400000):
        if not (roles or copies or commits):
            break
        c = rnd.random() * (sum(weights) + copy_weight + commit_weight)
        if c < copy_weight:
            if copies:
                copies.pop(rnd.randrange(len(copies)))()       # copies land in any order
        elif c < copy_weight + commit_weight:
            if commits:
                commits.pop(0)()
        elif roles:
            i = rnd.choices(range(len(roles)), weights)[0]
            try:
                next(roles[i])
            except StopIteration:
                roles.pop(i)
                weights.pop(i)
    assert len(ended) == 4 * parts, "not all ended"


@pytest.mark.parametrize("shape", [(6, 4, 4, 2, 1, True), (4, 4, 4, 2, 1, True), (3, 3, 2, 1, 2, False)])
@pytest.mark.parametrize("chunks", [1, 2, 37])
def test_no_order_of_events_shows_stale_data(shape, chunks):
    for seed in range(60):
        walk(seed, *shape, chunks)


def test_a_ring_that_two_sets_share_unevenly_is_found_out():
    failed = 0
    for seed in range(150):
        try:
            walk(seed, 5, 4, 4, 2, 1, True, 37)
        except AssertionError:
            failed += 1
    assert failed > 0
