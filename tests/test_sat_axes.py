"""sat_axes (cz_kernels.cuh) on the CPU: the penetrations of a cube pair's
fifteen axes are the same bits in both orders of the pair, axis by axis under
the lane map `back`, so one set of axes gives the reference's choice for
(one, two) and for (two, one), ties included."""
import numpy as np
import pytest


def _dot(a, b):
    return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]


def _cross(a, b):
    return (a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0])


def penetrations(one, two, real):
    """tryAxis' penetration per axis index, None where the axis is skipped."""
    (x1, c1, h1), (x2, c2, h2) = one, two
    tc = [a - b for a, b in zip(c2, c1)]
    axes = list(x1) + list(x2) + [_cross(a, b) for a in x1 for b in x2]
    out = []
    for a in axes:
        if _dot(a, a) < real(1e-7):
            out.append(None)
            continue
        m = np.sqrt(_dot(a, a))
        if m != 0:
            inv = real(1) / m
            a = [v * inv for v in a]

        def proj(x, h):
            return h[0] * abs(_dot(a, x[0])) + h[1] * abs(_dot(a, x[1])) + h[2] * abs(_dot(a, x[2]))
        out.append(proj(x1, h1) + proj(x2, h2) - abs(_dot(tc, a)))
    return out


def choose(p):
    """The reference's loop: strict <, in index order; (best, best of the first six)."""
    best, single, least = None, None, None
    for i, v in enumerate(p):
        if v is not None and (least is None or v < least):
            best, least = i, v
        if i == 5:
            single = best
    return best, single


BACK = [i + 3 if i < 3 else i - 3 if i < 6 else 6 + 3 * ((i - 6) % 3) + (i - 6) // 3 for i in range(15)]


@pytest.mark.parametrize("real", [np.float64, np.float32])
def test_one_set_of_axes_serves_both_orders(real):
    rng = np.random.default_rng(3)
    ties = 0
    for trial in range(400):
        boxes = []
        for _ in range(2):
            q = rng.normal(size=4)
            if trial % 3 == 0:
                q = np.array([1.0, 0, 0, 0])  # aligned: equal penetrations on several axes
            w, x, y, z = q / np.linalg.norm(q)
            m = np.array([[1 - 2 * y * y - 2 * z * z, 2 * x * y + 2 * w * z, 2 * x * z - 2 * w * y],
                          [2 * x * y - 2 * w * z, 1 - 2 * x * x - 2 * z * z, 2 * y * z + 2 * w * x],
                          [2 * x * z + 2 * w * y, 2 * y * z - 2 * w * x, 1 - 2 * x * x - 2 * y * y]])
            h = np.full(3, 0.5) if trial % 3 == 0 else rng.uniform(0.25, 1.0, 3)
            c = np.round(rng.uniform(-0.5, 0.5, 3), 1) if trial % 3 == 0 else rng.uniform(-0.8, 0.8, 3)
            boxes.append(([[real(v) for v in r] for r in m], [real(v) for v in c], [real(v) for v in h]))
        p, q = penetrations(boxes[0], boxes[1], real), penetrations(boxes[1], boxes[0], real)
        for i in range(15):
            assert (p[i] is None) == (q[BACK[i]] is None)
            assert p[i] is None or p[i] == q[BACK[i]]
        ties += len({v for v in p if v is not None}) < sum(v is not None for v in p)
        # the kernel's selection: the first index of the smallest value, in each order's own index order
        some = [i for i in range(15) if p[i] is not None]
        least = min(p[i] for i in some)
        own = [i for i in some if i < 6]
        least6 = min(p[i] for i in own)
        assert choose(p) == (min(i for i in some if p[i] == least), min(i for i in own if p[i] == least6))
        assert choose(q) == (min(BACK[i] for i in some if p[i] == least), min(BACK[i] for i in own if p[i] == least6))
    assert ties > 50
