"""The order in which a world's iteration budget is spent over its islands
(resolve_worlds in cz_resolve.cuh), on sequences of keys: the reference takes
the island with the largest next key, one iteration at a time; the resolver
runs islands side by side until the budget ends, and then goes on from one of
them with the others put back.  Both must spend the same number of iterations
on every island."""
import random

import pytest


def _one_list(seqs, budget):
    """Iterations per island of the reference's order, equal keys to the first island."""
    at = [0] * len(seqs)
    while sum(at) < budget:
        heads = [s[i] if i < len(s) else 0 for s, i in zip(seqs, at)]
        best = max(heads)
        if best == 0:
            break
        at[heads.index(best)] += 1
    return at


class _Runner:
    def __init__(self, seqs):
        self.seqs = seqs
        self.at = [0] * len(seqs)

    def head(self, j):
        s = self.seqs[j]
        return s[self.at[j]] if self.at[j] < len(s) else 0

    def side_by_side(self, islands, budget, stop, groups):
        """resolve_phase: rounds of one iteration for each of up to `groups`
        islands.  (over, U, its key, tie)"""
        queue, live, used, tie = list(islands), [], 0, False
        low = {}
        while True:
            live = [j for j in live if self.head(j) >= stop]
            while len(live) < groups and queue:
                j = queue.pop(0)
                low[j] = 1 << 62
                if self.head(j) >= stop:
                    live.append(j)
            if not live:
                return False, None, 0, tie
            for j in live:
                tie = tie or self.head(j) == stop
                low[j] = min(low[j], self.head(j))
            if used + len(live) > budget:
                u = max(live, key=lambda j: low[j])
                return True, u, low[u], tie
            for j in live:
                self.at[j] += 1
            used += len(live)

    def list(self, islands, budget, stop):
        for _ in range(budget):
            j = max(islands, key=self.head)
            if self.head(j) < stop:
                return False
            self.at[j] += 1
        return max(self.head(j) for j in islands) >= stop


def _resumed(seqs, budget, groups):
    r = _Runner(seqs)
    every = list(range(len(seqs)))
    over, u, c, _ = r.side_by_side(every, budget, 1, groups)
    if not over or len(seqs) == 1:
        return r.at, "islands"
    others = [j for j in every if j != u]
    for j in others:
        r.at[j] = 0
    out, _, _, tie = r.side_by_side(others, budget - r.at[u], c, groups)
    if out or tie:
        return None, "put back"
    if r.list([u], budget - sum(r.at), c):
        return r.at, "resumed"
    r.list(every, budget - sum(r.at), 1)
    return r.at, "to list"


@pytest.mark.parametrize("groups", [1, 4, 16])
@pytest.mark.parametrize("spread", [6, 1000, 1 << 30])
def test_resumed_budget_equals_the_one_list(groups, spread):
    rng = random.Random(groups * 7919 + spread)
    seen = {}
    for _ in range(3000):
        n = rng.randint(1, 9)
        seqs = []
        for _ in range(n):
            scale = rng.choice([1.0, 0.3, 0.02]) * spread
            seqs.append([max(1, int(scale * rng.random() * rng.choice([1.0, 0.98 ** i])))
                         for i in range(rng.randint(1, 40))])
        budget = rng.randint(1, max(1, sum(map(len, seqs)) + 3))
        want = _one_list(seqs, budget)
        got, how = _resumed(seqs, budget, groups)
        seen[how] = seen.get(how, 0) + 1
        if got is not None:
            assert got == want, (seqs, budget, how)
    if spread > 6:  # without ties every way is taken
        assert min(seen.get(k, 0) for k in ("islands", "resumed", "to list")) > 20, seen
