"""Interleaving models of the union steps of the tile and merge kernels (labeling_b200/csrc).

Hooking before unions (be_common.cuh: shook_pairs, smerge; be_uf3d.cu: ehook3_pairs, eunion3): every
entry of a flat forest stands at its root; warps take their parts of the pairs in turns of a few lanes, drop
pairs of one root, hook the larger root under the smaller with atomicMin and keep the pair as roots; after a
barrier the kept pairs are merged for good, after another the ends of the kept pairs are pointed at their
roots, and then every entry is at most one step from its root.  In 2D entries are parents, in 3D
(slot << 12) | parent, where the smallest slot of a component wins and all entries are flattened at the end.

Jumps beside unions (gunion_keyed, gjump): the nodes' entries are (key, parent); unions climb with halving
and link by CAS while other threads point nodes at their parents' parents.

The table of pairs seen (k_merge_2d, k_merge_3d): a thread that finds its pair in its slot leaves the union
to the one that put it there; pairs that share a slot push one another out.

Each access to shared state is one step of a generator, and a seeded random scheduler interleaves them."""
import random

import pytest

IDX = 0xFFF


def interleave(rng, threads):
    threads = list(threads)
    while threads:
        i = rng.randrange(len(threads))
        try:
            next(threads[i])
        except StopIteration:
            threads[i] = threads[-1]
            threads.pop()


class Sets:
    def __init__(self, n):
        self.p = list(range(n))

    def find(self, x):
        while self.p[x] != x:
            x = self.p[x]
        return x

    def unite(self, a, b):
        a, b = self.find(a), self.find(b)
        self.p[max(a, b)] = min(a, b)


def hook(P, q, lanes, kept_out, index):
    kept = 0
    for k in range(0, len(q), lanes):
        turn = []
        for a, b in q[k:k + lanes]:
            x = P[a]
            yield
            y = P[b]
            yield
            turn.append((x, y))
        for x, y in turn:
            if x == y:
                continue
            hi = index(max(x, y))
            P[hi] = min(P[hi], min(x, y))        # atomicMin, one step
            yield
            q[kept] = (index(x), index(y))
            kept += 1
    kept_out.append(q[:kept])


def sfind(P, a):
    p = P[a]
    yield
    while p != a:
        g = P[p]
        yield
        if g != p:
            P[a] = g
            yield
        a, p = p, g
    return a


def smerge(P, a, b):
    while True:
        a = yield from sfind(P, a)
        b = yield from sfind(P, b)
        if a == b:
            return
        if a < b:
            a, b = b, a
        old = P[a]                               # atomicMin of the larger root, one step
        P[a] = min(old, b)
        yield
        if old == a:
            return
        a = old


def point(P, i):
    x, y = i, P[i]
    yield
    while y != x:
        x = y
        y = P[x]
        yield
    if x != i:
        P[i] = x
        yield


@pytest.mark.parametrize("seed", range(400))
def test_hook_then_unite_2d(seed):
    rng = random.Random(seed)
    n = rng.choice([4, 12, 40])
    P = []
    for i in range(n):                           # a flat forest, roots smaller than what hangs on them
        roots = [j for j in range(i) if P[j] == j]
        P.append(rng.choice(roots) if roots and rng.random() < 0.4 else i)
    sets = Sets(n)
    for i in range(n):
        sets.unite(i, P[i])
    warps = rng.choice([1, 2, 4])
    parts = []
    for _ in range(warps):
        parts.append([tuple(rng.sample(range(n), 2)) for _ in range(rng.randrange(0, n // 2 + 2))])
        for a, b in parts[-1]:
            sets.unite(a, b)
    kept = []
    interleave(rng, [hook(P, q, 3, kept, lambda v: v) for q in parts])
    pairs = [p for part in kept for p in part]
    interleave(rng, [smerge(P, a, b) for a, b in pairs])
    interleave(rng, [point(P, i) for p in pairs for i in p])
    for i in range(n):
        assert P[P[i]] == sets.find(i), (seed, i)


def efind(P, x):
    v = P[x]
    yield
    while (v & IDX) != x:
        y = v & IDX
        vg = P[y]
        yield
        if (vg & IDX) != y:
            P[x] = vg
            yield
        x, v = y, vg
    return x, v


def eunion(P, a, b):
    while True:
        a, ea = yield from efind(P, a)
        b, eb = yield from efind(P, b)
        if a == b:
            return
        hi = b if ea < eb else a
        old = P[hi]
        P[hi] = min(old, min(ea, eb))            # atomicMin, one step
        yield
        if (old & IDX) == hi:
            return
        b = a if ea < eb else b
        a = old & IDX


def eflatten(P, i):
    x = P[i] & IDX
    yield
    if x == i:
        return
    v = P[x]
    yield
    while (v & IDX) != x:
        x = v & IDX
        v = P[x]
        yield
    P[i] = v
    yield


@pytest.mark.parametrize("seed", range(400))
def test_hook_then_unite_3d(seed):
    rng = random.Random(seed)
    n = rng.choice([4, 12, 40])
    slot = rng.sample(range(4096), n)
    P = [0] * n
    roots = []
    for i in sorted(range(n), key=slot.__getitem__):   # a tree's root has its smallest slot
        r = rng.choice(roots) if roots and rng.random() < 0.4 else i
        if r == i:
            roots.append(i)
        P[i] = (slot[r] << 12) | r
    sets = Sets(n)
    for i in range(n):
        sets.unite(i, P[i] & IDX)
    parts = []
    for _ in range(rng.choice([1, 2, 4])):
        parts.append([tuple(rng.sample(range(n), 2)) for _ in range(rng.randrange(0, n // 2 + 2))])
        for a, b in parts[-1]:
            sets.unite(a, b)
    kept = []
    interleave(rng, [hook(P, q, 3, kept, lambda v: v & IDX) for q in parts])
    interleave(rng, [eunion(P, a, b) for part in kept for a, b in part])
    interleave(rng, [eflatten(P, i) for i in range(n)])
    best = {}
    for i in range(n):
        c = sets.find(i)
        if c not in best or slot[i] < slot[best[c]]:
            best[c] = i
    for i in range(n):
        r = best[sets.find(i)]
        assert P[i] == (slot[r] << 12) | r, (seed, i)


def gunion(gp, a, b, on_link):
    ea = gp[a]
    yield
    eb = gp[b]
    yield
    while True:
        if ea[1] == eb[1]:
            return
        if ea[0] < eb[0]:
            a, b, ea, eb = b, a, eb, ea
        pa = ea[1]
        if pa == a:
            old = gp[a]                          # CAS, one step
            if old == ea:
                gp[a] = eb
                on_link(a)
                yield
                return
            yield
            ea = old
            eb = gp[b]
            yield
            continue
        ga = gp[pa]
        yield
        if ga[1] != pa:
            gp[a] = ga
            yield
        a, ea = pa, ga


def gjump(gp, x):
    p = gp[x][1]
    yield
    if p == x:
        return
    ep = gp[p]
    yield
    if ep[1] != p:
        gp[x] = ep
        yield


@pytest.mark.parametrize("seed", range(400))
def test_jumps_beside_unions(seed):
    rng = random.Random(seed)
    n = rng.choice([5, 15, 40])
    key = rng.sample(range(10 * n), n)
    gp = [(key[i], i) for i in range(n)]
    sets, linked = Sets(n), []
    pairs = [tuple(rng.sample(range(n), 2)) for _ in range(rng.randrange(1, 2 * n))]
    if seed % 2:                                 # a path, as a component that winds through many tiles
        order = sorted(range(n), key=key.__getitem__, reverse=rng.random() < 0.5)
        pairs += list(zip(order, order[1:]))
    for a, b in pairs:
        sets.unite(a, b)
    interleave(rng, [gunion(gp, a, b, linked.append) for a, b in pairs] + [gjump(gp, x) for x in range(n) for _ in range(rng.randrange(3))])
    groups = {}
    for i in range(n):
        groups.setdefault(sets.find(i), []).append(i)
    for members in groups.values():
        root = min(members, key=key.__getitem__)
        for i in members:
            x, steps = i, 0
            while gp[x][1] != x:
                assert gp[x][0] == key[gp[x][1]] < key[x]
                x, steps = gp[x][1], steps + 1
                assert steps <= n
            assert x == root, (seed, i)
        assert sorted(x for x in linked if x in members) == sorted(x for x in members if x != root)


def see(table, slot, pair, queue):
    old, table[slot] = table[slot], pair         # atomicExch, one step
    yield
    if old != pair:
        queue.append(pair)
        yield


@pytest.mark.parametrize("seed", range(200))
def test_every_pair_seen_is_united(seed):
    rng = random.Random(seed)
    slots = rng.choice([1, 2, 8])
    table, queue = [None] * slots, []
    pairs = [(rng.randrange(4), rng.randrange(4)) for _ in range(rng.randrange(1, 60))]
    interleave(rng, [see(table, hash(p) % slots, p, queue) for p in pairs])
    assert set(queue) == set(pairs)
