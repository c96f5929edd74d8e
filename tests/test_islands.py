"""The resolver's islands (build_islands, next_record and resolve_phase in
cz_resolve.cuh) on the CPU: the label propagation finds the connected
components of any contact list, the records keep each island's list order,
and the reference's resolver run on each island alone gives the bits and the
iteration counts of its run on the whole list, as long as the islands' counts
stay within the budget."""
import copy

import numpy as np
import pytest

from cubez_gb300 import scenes
from oracle import contact_ref
from oracle.oracle import FP32, FP64, OracleBatch

DT = 1.0 / 60.0


def labels_of(pairs, n):
    """build_islands' rounds: every contact pulls both bodies and the larger
    label down to the smaller label, then labels follow their labels."""
    lab = list(range(n))
    rounds = 0
    while True:
        more = False
        for b0, b1 in pairs:
            if b0 < 0 or b1 < 0 or lab[b0] == lab[b1]:
                continue
            lo, hi = min(lab[b0], lab[b1]), max(lab[b0], lab[b1])
            lab[hi] = min(lab[hi], lo)
            lab[b0] = min(lab[b0], lo)
            lab[b1] = min(lab[b1], lo)
            more = True
        for i in range(n):
            lab[i] = min(lab[i], lab[lab[i]])
        rounds += 1
        if not more:
            return lab, rounds


def islands_of(pairs, n):
    """(records: list index by place, first record of each island)."""
    lab, _ = labels_of(pairs, n)
    label = [lab[b0 if b0 >= 0 else b1] for b0, b1 in pairs]
    cnt = [label.count(r) for r in range(n)]
    size_class = lambda m: 0 if m >= 24 else 1 if m >= 12 else 2 if m >= 6 else 3 if m >= 3 else 4  # noqa: E731
    order = [r for c in range(5) for r in range(n) if cnt[r] > 0 and size_class(cnt[r]) == c]
    first, at = [], 0
    cur = {}
    for r in order:
        first.append(at)
        cur[r] = at
        at += cnt[r]
    first.append(at)
    records = [None] * len(pairs)
    for k, r in enumerate(label):  # next_record, k ascending
        records[cur[r]] = k
        cur[r] += 1
    return records, first


def components(pairs, n):
    f = list(range(n))

    def find(a):
        while f[a] != a:
            a = f[a]
        return a
    for b0, b1 in pairs:
        if b0 >= 0 and b1 >= 0:
            f[find(b0)] = find(b1)
    return [find(i) for i in range(n)]


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 63, 64])
def test_islands_are_the_components_in_list_order(n):
    rng = np.random.default_rng(n)
    for trial in range(60):
        C = int(rng.integers(1, 200))
        b0 = rng.integers(0, n, C)
        b1 = np.where(rng.random(C) < rng.random(), -1, rng.integers(0, n, C))
        if trial % 4 == 0:  # a chain in an unhelpful order
            b0, b1 = np.arange(n - 1, 0, -1) if n > 1 else np.zeros(1, int), np.arange(n - 2, -1, -1) if n > 1 else -np.ones(1, int)
        swap = (rng.random(len(b0)) < 0.2) & (b1 >= 0)  # body 0 nil: prepareContacts swaps it
        pairs = [(-1, int(x)) if s and y < 0 else (int(x), int(y)) for x, y, s in zip(b0, b1, swap)]
        records, first = islands_of(pairs, n)
        comp = components(pairs, n)
        assert sorted(records) == list(range(len(pairs)))
        seen = set()
        for s, e in zip(first[:-1], first[1:]):
            ks = records[s:e]
            assert ks == sorted(ks) and ks
            roots = {comp[b] for k in ks for b in pairs[k] if b >= 0}
            assert len(roots) == 1 and not (roots & seen)
            seen |= roots


@pytest.mark.parametrize("form", [FP64, FP32])
def test_islands_alone_give_the_whole_lists_bits(form, oracle_lib):
    sc = scenes.mixed(num_worlds=6, seed=71, min_bodies=10, max_bodies=24)
    sc.can_sleep[::2] = 1
    o = OracleBatch(sc, form=form)
    o.step(140, DT)
    o.integrate(DT)
    o.narrowphase()
    st = o.bodies()
    real = float if form == FP64 else np.float32
    several = exhausted = 0
    for w in range(sc.num_worlds):
        sl = sc.world_slice(w)
        n = sl.stop - sl.start
        bodies = [{"position": [real(v) for v in st["position"][i]], "orientation": [real(v) for v in st["orientation"][i]],
                   "velocity": [real(v) for v in st["velocity"][i]], "rotation": [real(v) for v in st["rotation"][i]],
                   "iit": [real(v) for v in st["iit_world"][i]], "inverse_mass": real(sc.inverse_mass[i]),
                   "lfa": [real(v) for v in sc.acceleration[i]], "awake": True} for i in range(sl.start, sl.stop)]
        c = o.contacts(w)
        contacts = [contact_ref.Contact(int(b[0]), int(b[1]) if b[1] >= 0 else None, [real(v) for v in p],
                                        [real(v) for v in nn], real(pen))
                    for b, p, nn, pen in zip(c["bodies"], c["point"], c["normal"], c["penetration"])]
        pairs = [(int(b[0]), int(b[1])) for b in c["bodies"]]
        budget = 4 * len(contacts)
        whole_b, whole_c = copy.deepcopy(bodies), copy.deepcopy(contacts)
        pos, vel = contact_ref.resolve_contacts(budget, whole_c, whole_b, DT)
        records, first = islands_of(pairs, n)
        several += len(first) > 3
        pos_sum = vel_sum = 0
        for s, e in zip(first[:-1], first[1:]):
            p, v = contact_ref.resolve_contacts(budget, [contacts[k] for k in records[s:e]], bodies, DT)
            pos_sum, vel_sum = pos_sum + p, vel_sum + v
        if pos_sum > budget or vel_sum > budget:
            assert pos == budget or vel == budget  # the whole list runs out: solved as one list
            exhausted += 1
            continue
        assert (pos_sum, vel_sum) == (pos, vel)
        for k in ("position", "orientation", "velocity", "rotation"):
            assert [list(b[k]) for b in bodies] == [list(b[k]) for b in whole_b], k
        assert [x.penetration for x in contacts] == [x.penetration for x in whole_c]
    assert several >= 3 and exhausted < sc.num_worlds
