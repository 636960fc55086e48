"""The solver's frontiers, restated on the CPU.

A solver group finds its dependency levels while the updates run: each dynamic
body has a cursor into its own list of updates (pass by pass the contacts it is
the second body of, then its own row), and a contact whose bodies' cursors both
stand on it is ready.  This checks that the frontiers hold exactly the updates
a walk over all updates gives each level to, on random worlds (static bodies,
partial cache hits, no warm start, no sweeps).
"""
import numpy as np
import pytest

from tests.test_level_schedule import walk_levels


def frontiers(contacts, iterations, warm):
    seconds, rows = {}, {}
    for q, (a, b, hit, da, db) in enumerate(contacts):
        if db:
            seconds.setdefault(b, []).append(q)
        if da:
            rows.setdefault(a, []).append(q)
    lists = {s: seconds.get(s, []) + rows.get(s, []) for s in set(seconds) | set(rows)}
    cursor, arrived, out = {}, set(), {}

    def advance(s, p, pos):
        while True:
            if pos >= len(lists[s]):
                p, pos = p + 1, 0
            if p > iterations:
                return None
            q = lists[s][pos]
            if p > 0 or contacts[q][2]:
                break
            pos += 1
        cursor[s] = (p, pos)
        if contacts[q][3] and contacts[q][4]:
            arrived.symmetric_difference_update({q})
            if q in arrived:
                return None
        return p, q

    level = [u for s in lists if (u := advance(s, 0 if warm else 1, 0)) is not None]
    n = 1
    while level:
        after = []
        for p, q in level:
            out[(p, q)] = n
            a, b, _, da, db = contacts[q]
            for s, dynamic in ((a, da), (b, db)):
                if dynamic and (u := advance(s, cursor[s][0], cursor[s][1] + 1)) is not None:
                    after.append(u)
        level, n = after, n + 1
    return out


@pytest.mark.parametrize("seed", range(8))
@pytest.mark.parametrize("iterations,warm", [(8, True), (2, True), (3, False), (0, True), (0, False)])
def test_frontiers_are_the_walks_levels(seed, iterations, warm):
    rng = np.random.default_rng(seed)
    n = int(rng.integers(2, 40))
    static = rng.uniform(size=n) < 0.15
    pairs = {(i, j) for i in range(1, n) for j in range(i)
             if rng.uniform() < 3.0 / n and not (static[i] and static[j])}
    contacts = [(i, j, bool(rng.uniform() < 0.8), not static[i], not static[j])
                for i, j in sorted(pairs, reverse=True) for _ in range(int(rng.integers(1, 3)))]
    assert frontiers(contacts, iterations, warm) == walk_levels(contacts, iterations, warm)
