"""The tile filter of three objectives (lex_items.cuh), on CPU.

A line-by-line Python rendering of one pass over a tile's destinations: the odd-even sort
of unsorted runs and of destinations of many runs, the merge by rank (equal points: the
lower run first), the bit masks inside each 32 positions, the staircase a destination
leaves in a chunk it goes on from, and the later chunks' questions to those staircases
(or, up to the pairwise limit, to the points).  Its keep flags must be the oracle's keep
rule (src/pmdd/enum/gpu/dominance_utils.cuh:10-23) on each destination's merged order:
runs of every kind of length, destinations that start inside a chunk and span many,
ties in every objective, the type's extreme values, and anti-correlated objectives.
"""
import numpy as np
import pytest

import oracle

SORT_RUN, MERGE_RUNS = 32, 16
LOWEST, MOST = -2**31, 2**31 - 1


def before(a, b, tie):
    """Is point a's place before point b's (equal points: if tie)?"""
    return tuple(a) > tuple(b) or (tuple(a) == tuple(b) and tie)


def sort_run(P, lo, n):
    """Batcher's odd-even mergesort with the kernel's indexing (every thread's t in turn)."""
    p = 1
    while p < n:
        k = p
        while k >= 1:
            j0 = k & (p - 1)
            t = 0
            while True:
                a = j0 + (((t & ~(k - 1)) << 1) | (t & (k - 1)))
                if a + k >= n:
                    break
                if ((a ^ (a + k)) & ~(2 * p - 1)) == 0:
                    u, v = lo + a, lo + a + k
                    if tuple(P[u]) < tuple(P[v]):
                        P[u], P[v] = P[v], P[u]
                t += 1
            k >>= 1
        p <<= 1


def stair_covers(s1, s2, q1, q2):
    at = 0
    for step in (16, 8, 4, 2, 1):
        if s1[at + step - 1] >= q1:
            at += step
    if s1[at] >= q1:
        at += 1
    return at > 0 and s2[at - 1] >= q2


def tile_pass(dests, pair_max):
    """dests: per destination its runs, each (points, sorted flag).  Merged points per
    position, keep flags, and the destinations' first positions."""
    P, run_lo, run_item, run_sorted, item_s, item_a = [], [], [], [], [0], [0]
    for k, runs in enumerate(dests):
        for pts, flag in runs:
            run_lo.append(len(P))
            run_item.append(k)
            run_sorted.append(flag)
            P += [tuple(int(x) for x in p) for p in pts]
        item_s.append(len(P))
        item_a.append(len(run_lo))
    total, runs_n = len(P), len(run_lo)
    run_lo.append(total)
    item_of = [k for k in range(len(dests)) for _ in range(item_s[k + 1] - item_s[k])]
    tag = [x for x in range(runs_n) for _ in range(run_lo[x + 1] - run_lo[x])]
    whole = [item_a[k + 1] - item_a[k] > MERGE_RUNS and item_s[k + 1] - item_s[k] > SORT_RUN for k in range(len(dests))]
    for k in range(len(dests)):
        if whole[k]:
            sort_run(P, item_s[k], item_s[k + 1] - item_s[k])
    for x in range(runs_n):
        if not run_sorted[x] and run_lo[x + 1] - run_lo[x] > SORT_RUN and not whole[run_item[x]]:
            run_sorted[x] = True
            sort_run(P, run_lo[x], run_lo[x + 1] - run_lo[x])
    to = [0] * total
    for q in range(total):
        k, x = item_of[q], tag[q]
        rank = q - item_s[k] if whole[k] else 0
        for y in range(item_a[k + 1] if whole[k] else item_a[k], item_a[k + 1]):
            lo, hi = run_lo[y], run_lo[y + 1]
            if not run_sorted[y]:
                rank += sum(before(P[j], P[q], j < q) for j in range(lo, hi))
            elif y == x:
                rank += q - lo
            else:
                a, b = lo, hi
                while a < b:
                    mid = (a + b) >> 1
                    if before(P[mid], P[q], y < x):
                        a = mid + 1
                    else:
                        b = mid
                rank += a - lo
        to[q] = item_s[k] + rank
    assert sorted(to) == list(range(total))
    M = [None] * total
    for q in range(total):
        M[to[q]] = P[q]
    # --- inside the chunks
    chunks = (total + 31) >> 5
    keep = [False] * total
    s1, s2 = [LOWEST] * (32 * chunks), [LOWEST] * (32 * chunks)
    for c in range(chunks):
        c0 = 32 * c
        at = range(c0, min(c0 + 32, total))
        for q in at:
            js = item_s[item_of[q]]
            keep[q] = not any(M[j][1] >= M[q][1] and M[j][2] >= M[q][2] for j in at if max(js, c0) <= j < q)
        if c0 + 32 >= total or item_s[item_of[c0 + 31] + 1] <= c0 + 32:
            continue
        kl = item_of[c0 + 31]
        members = [q for q in at if keep[q] and item_of[q] == kl]
        assert members
        for q in members:
            place = sum(M[m][1] >= M[q][1] and (M[m][1] != M[q][1] or m < q) for m in members)
            assert (s1[c0 + place], s2[c0 + place]) == (LOWEST, LOWEST)
            s1[c0 + place], s2[c0 + place] = M[q][1], M[q][2]
        for i in range(c0 + 1, c0 + 32):
            s2[i] = max(s2[i], s2[i - 1])
        assert all(x >= y for x, y in zip(s1[c0:c0 + 32], s1[c0 + 1:c0 + 32]))
    # --- against the earlier chunks of the destination that reaches into the chunk
    for c in range(chunks - 1, 0, -1):
        c0 = 32 * c
        js, je = item_s[item_of[c0]], item_s[item_of[c0] + 1]
        if js >= c0:
            continue
        for q in range(c0, min(c0 + 32, je)):
            if keep[q] and je - js <= pair_max:
                keep[q] = not any(M[j][1] >= M[q][1] and M[j][2] >= M[q][2] for j in range(js, c0))
            elif keep[q]:
                keep[q] = not any(stair_covers(s1[32 * t:32 * t + 32], s2[32 * t:32 * t + 32], M[q][1], M[q][2])
                                  for t in range(js >> 5, c))
    return M, keep, item_s


def points(rng, n, kind):
    if kind == "anti":
        x, y = rng.integers(0, 1000, size=n), rng.integers(0, 1000, size=n)
        return np.stack([x, y, 2000 - x - y + rng.integers(0, 5, size=n)], 1)
    if kind == "staircase":  # objectives 1 and 2 an antichain
        y = rng.integers(0, 10000, size=n)
        return np.stack([rng.integers(0, 50, size=n), y, 10000 - y], 1)
    if kind == "extremes":
        return rng.choice([LOWEST, LOWEST + 1, 0, MOST - 1, MOST], size=(n, 3))
    return rng.integers(0, kind, size=(n, 3))


def run(rng, n, kind):
    """A run as an arc brings it: a frontier, in order or not."""
    p = np.unique(points(rng, n, kind).astype(np.int64), axis=0)
    p = p[oracle.nd_keep(p.astype(np.int32))]
    flag = bool(rng.integers(0, 4))
    return (p[::-1] if flag else rng.permutation(p)), flag


@pytest.mark.parametrize("pair_max", [0, 48, 1024])
@pytest.mark.parametrize("kind", [3, 30, 100000, "anti", "staircase", "extremes"])
def test_pass_keeps_the_oracle_frontiers(kind, pair_max):
    rng = np.random.default_rng([pair_max, *str(kind).encode()])
    for t in range(12):
        dests = []
        for _ in range(int(rng.integers(1, 9))):
            runs = int(rng.choice([1, 2, 3, 17, 20]))
            most = int(rng.choice([1, 7, 33, 64, 65, 200]))
            dests.append([run(rng, int(rng.integers(1, most + 1)), kind) for _ in range(runs)])
        M, keep, item_s = tile_pass(dests, pair_max)
        for k, runs in enumerate(dests):
            got = np.array(M[item_s[k]:item_s[k + 1]], dtype=np.int64)
            assert sorted(map(tuple, got)) == sorted(tuple(map(int, p)) for r, _ in runs for p in r)
            assert all(tuple(x) >= tuple(y) for x, y in zip(got, got[1:]))
            want = oracle.nd_keep(got.astype(np.int32))
            assert np.array_equal(keep[item_s[k]:item_s[k + 1]], want.astype(bool)), (t, k)


@pytest.mark.parametrize("n", [1, 2, 3, 31, 32, 33, 63, 64, 65, 100, 127, 129, 1000, 1024])
def test_sort_run_orders_any_length(n):
    rng = np.random.default_rng(n)
    for hi in (2, 5, 10000):
        P = [(9, 9, 9)] + [tuple(map(int, p)) for p in rng.integers(0, hi, size=(n, 3))] + [(0, 0, 0)]
        want = [P[0]] + sorted(P[1:-1], reverse=True) + [P[-1]]
        sort_run(P, 1, n)
        assert P == want
