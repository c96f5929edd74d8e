"""k_resolve_big's shared iterations: a body with more contacts than one pass
of the world's warps takes (8 each), and worlds whose contact lists are in
shared memory or not: the oracle's bits."""
import numpy as np
import pytest

from cubez_gb300 import scenes
from oracle.oracle import FP32 as ORC_FP32
from oracle.oracle import FP64 as ORC_FP64
from oracle.oracle import OracleBatch

pytestmark = pytest.mark.gpu

DT = 1.0 / 60.0
STATE = ("position", "orientation", "velocity", "rotation", "motion", "is_awake")


def _table(spheres, seed):
    """A wide cube on the plane under `spheres` close-packed spheres: its list
    holds a contact with each, theirs a handful."""
    s = scenes.mixed(num_worlds=2, seed=seed, min_bodies=spheres + 1, max_bodies=spheres + 1)
    n = spheres + 1
    side = int(np.ceil(np.sqrt(spheres)))
    at = np.arange(spheres)
    for w in range(2):
        o = w * n
        s.shape[o] = scenes.CUBE
        s.half_size[o] = (0.5 * side, 0.5, 0.5 * side)
        s.position[o] = (0.0, 0.49, 0.0)
        s.orientation[o] = (1.0, 0.0, 0.0, 0.0)
        ball = slice(o + 1, o + n)
        s.shape[ball] = scenes.SPHERE
        s.radius[ball] = 0.5
        s.half_size[ball] = 0.0
        s.position[ball, 0] = 0.97 * (at % side - 0.5 * (side - 1))
        s.position[ball, 2] = 0.97 * (at // side - 0.5 * (side - 1))
        s.position[ball, 1] = 1.47
        s.can_sleep[ball] = 1 if w else 0
        s.is_awake[ball] = np.arange(spheres) % 3 > 0 if w else 1
    s.velocity[:] = 0.0
    s.rotation[:] = 0.0
    return s


@pytest.mark.parametrize("form", [0, 1])
@pytest.mark.parametrize("spheres,budget", [(64, 0), (100, 0), (100, 57), (170, 400)])
def test_many_contacts_of_one_body_bit_exact(form, spheres, budget, cuda_lib):
    from cubez_gb300.batch import WorldBatch
    orc = ORC_FP64 if form == 0 else ORC_FP32
    scene = _table(spheres, 7)
    gpu = WorldBatch.from_scene(scene, form=form, max_iterations=budget)
    ref = OracleBatch(scene, form=orc)
    for _ in range(4):
        gpu.integrate(DT)
        gpu.narrowphase()
        gpu.resolve(DT)
        ref.integrate(DT)
        ref.narrowphase()
        if budget:
            ref.resolve_fixed(budget, DT)
        else:
            ref.resolve(DT)
        g, r = gpu.download(STATE), ref.bodies()
        for k in STATE:
            assert np.array_equal(g[k], r[k]), k
        gs, rs = gpu.stats(), ref.stats()
        for k in ("pos_iterations", "vel_iterations"):
            assert np.array_equal(gs[k], rs[k]), k
        assert rs["contacts"].min() > spheres
