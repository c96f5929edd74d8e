"""Islands of contact lists whose half-space contacts name their body second
(body 0 nil, which prepareContacts swaps): the same components, in list order."""
import numpy as np
import pytest

from tests.test_islands import components, islands_of


@pytest.mark.parametrize("n", [1, 2, 31, 64])
def test_body_0_nil(n):
    rng = np.random.default_rng(100 + n)
    for _ in range(40):
        C = int(rng.integers(1, 200))
        b0, b1 = rng.integers(0, n, C), np.where(rng.random(C) < 0.5, -1, rng.integers(0, n, C))
        swap = (b1 < 0) & (rng.random(C) < 0.5)
        pairs = [(int(x), int(y)) for x, y in zip(b0, b1)]
        swapped = [(y, x) if s else (x, y) for (x, y), s in zip(pairs, swap)]
        records, first = islands_of(swapped, n)
        assert (records, first) == islands_of(pairs, n)
        assert components(swapped, n) == components(pairs, n)
        for s, e in zip(first[:-1], first[1:]):
            assert records[s:e] == sorted(records[s:e])
