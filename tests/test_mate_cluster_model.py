"""Model check of the mate union's tail (k_pe_cluster) against the reference's in-order loop (metapart.c:2801-2867):
held reservations, pairs asleep behind the pair that holds a root, and singles that commit together.  The model follows
the kernel step by step; reads are also BAD (components of size 0) and the list of pairs comes in any order."""
import random

import pytest


def _find(parent, x):
    while parent[x] != x:
        x = parent[x]
    return x


def sequential(parent, size, limit):
    parent, size = parent[:], size[:]
    for i in range(0, len(parent), 2):
        a, b = _find(parent, i), _find(parent, i + 1)
        if a != b and (size[a] <= limit or size[b] <= limit):
            hi, lo = max(a, b), min(a, b)
            parent[lo] = hi
            size[hi] += size[lo]
            size[lo] = 0
    return [_find(parent, x) for x in range(len(parent))]


def cluster(parent, size, limit, pairs):
    parent, size = parent[:], size[:]
    hold, done = {}, [False] * len(pairs)
    st = [dict(j=j, ha=None, hb=None, live=True, awake=True) for j in pairs]
    n_rounds = 0
    while any(s["live"] for s in st):
        n_rounds += 1
        assert n_rounds <= 2 * len(pairs) + 2
        first, was_done = {}, done[:]

        def stale(v):
            return v is None or was_done[v]
        awake = [t for t, s in enumerate(st)
                 if s["live"] and (s["awake"] or any(h is not None and was_done[h] for h in (s["ha"], s["hb"])))]
        for t in awake:                                    # roots and reservations
            s = st[t]
            a, b = _find(parent, 2 * s["j"]), _find(parent, 2 * s["j"] + 1)
            sa, sb = size[a] <= limit, size[b] <= limit
            s.update(awake=True, a=a, b=b)
            if a == b or not (sa or sb):
                s["live"], done[t] = False, True
                continue
            oa, ob = size[a] <= 1 < size[b] and sb, size[b] <= 1 < size[a] and sa
            s["f"] = sa, sb, oa, ob
            if oa or ob:
                x = b if oa else a
                first[x] = min(first.get(x, s["j"]), s["j"])
                continue
            for x, small in ((a, sa), (b, sb)):
                if small and (stale(hold.get(x)) or st[hold[x]]["j"] > s["j"]):
                    hold[x] = t
        commits = []
        for t in awake:                                    # commits
            s = st[t]
            if not s["live"]:
                continue
            a, b = s["a"], s["b"]
            sa, sb, oa, ob = s["f"]
            ha = hb = None
            ok = True
            if oa or ob:
                v = hold.get(b if oa else a)
                if not stale(v) and st[v]["j"] < s["j"]:
                    ha, ok = v, False
            else:
                if sa:
                    ha = hold[a] if hold[a] != t else None
                    ok = ha is None and first.get(a, s["j"]) >= s["j"]
                if sb:
                    hb = hold[b] if hold[b] != t else None
                    ok = ok and hb is None and first.get(b, s["j"]) >= s["j"]
            if ok:
                s["live"], done[t] = False, True
                commits.append((a, b, s["f"], size[a], size[b]))
            else:
                s.update(ha=ha, hb=hb, awake=ha is None and hb is None)
        groups = {}
        for a, b, (sa, sb, oa, ob), za, zb in commits:
            if sa and sb and not (oa or ob):
                hi, lo = max(a, b), min(a, b)
                assert parent[hi] == hi and parent[lo] == lo
                parent[lo], size[hi], size[lo] = hi, za + zb, 0
            else:
                g, x, z = (b, a, za) if sa and not ob else (a, b, zb)
                groups.setdefault(g, []).append((x, z))
        for g, xs in groups.items():                       # groups of a shared root
            assert parent[g] == g
            r, tot = max([g] + [x for x, _ in xs]), size[g] + sum(z for _, z in xs)
            for y in [g] + [x for x, _ in xs]:
                if y != r:
                    parent[y], size[y] = r, 0
            size[r] = tot
            if r != g:
                hold[r] = hold.get(g)
    return [_find(parent, x) for x in range(len(parent))]


def _forest(rnd, n, limit):
    parent, size, ids, p = list(range(n)), [0] * n, list(range(n)), 0
    rnd.shuffle(ids)
    while p < n:
        grp = ids[p:p + rnd.choice([1, 1, 1, 1, 1, 2, 3, limit // 2 + 1, limit, limit + 1])]
        p += len(grp)
        root = max(grp)
        for x in grp:
            parent[x] = root
        size[root] = 0 if len(grp) == 1 and rnd.random() < 0.3 else len(grp)
    return parent, size


@pytest.mark.parametrize("limit", [2, 3, 20, 100, 1000])
def test_cluster_rounds_equal_sequential(limit):
    rnd = random.Random(limit)
    for n in (2, 4, 20, 20, 80, 80, 400, 400, 2000, 6000):
        parent, size = _forest(rnd, n, limit)
        pairs = list(range(n // 2))
        rnd.shuffle(pairs)
        assert cluster(parent, size, limit, pairs) == sequential(parent, size, limit)
