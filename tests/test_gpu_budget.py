"""Worlds that run out of their iteration budget, solved by a warp each or, the
larger ones, by four (resolve_worlds and wide_phase in cz_resolve.cuh go on from
one island and put the others back): the oracle's bits, for budgets that end in either phase, worlds of many
islands, equal values on different islands, and sleeping bodies."""
import numpy as np
import pytest

from cubez_gb300 import scenes
from oracle.oracle import FP32 as ORC_FP32
from oracle.oracle import FP64 as ORC_FP64
from oracle.oracle import OracleBatch

pytestmark = pytest.mark.gpu

DT = 1.0 / 60.0
STATE = ("position", "orientation", "velocity", "rotation", "motion", "is_awake")
WORLDS = 200  # more than the GPU has SMs


def _alike(seed):
    """Cubes and spheres far apart at whole coordinates, alike and falling
    alike: every island's values equal the others'."""
    s = scenes.precision(num_worlds=WORLDS, bodies=12, seed=seed)
    i = np.arange(s.num_bodies) % 12
    s.position[:, 0], s.position[:, 2] = 8.0 * (i % 4), 8.0 * (i // 4)
    s.position[:, 1] = 1.0
    s.orientation[:] = s.orientation[(i // 6) * 6]
    s.velocity[:] = (0.0, -2.0, 0.0)
    s.rotation[:] = (0.0, 0.5, 0.25)
    for k in ("shape", "half_size", "radius", "inverse_inertia", "inverse_mass"):
        a = getattr(s, k)
        a[:] = a[0]
    return s


def _spread(seed, bodies=20):
    s = scenes.mixed(num_worlds=WORLDS, seed=seed, min_bodies=2, max_bodies=bodies)
    s.position[:, (0, 2)] *= 1.6  # more islands
    s.can_sleep[::4] = 1
    return s


def _spread_large(seed):
    return _spread(seed, 48)


@pytest.mark.parametrize("form", [0, 1])
@pytest.mark.parametrize("make,settle", [(_alike, 0), (_spread, 90), (_spread_large, 90)])
@pytest.mark.parametrize("budget", [0, 3, 12, 40, 90])
def test_out_of_budget_bit_exact(form, make, settle, budget, cuda_lib):
    from cubez_gb300.batch import WorldBatch
    orc = ORC_FP64 if form == 0 else ORC_FP32
    scene = make(60)
    if settle:
        ref = OracleBatch(scene, form=orc)
        ref.step(settle, DT, threads=8)
        st = ref.bodies()
        scene = scene.copy()
        for k in STATE:
            setattr(scene, k, st[k])
    gpu = WorldBatch.from_scene(scene, form=form, max_iterations=budget)
    ref = OracleBatch(scene, form=orc)
    out = 0
    for _ in range(12):
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
        out += int((rs["vel_iterations"] >= (budget or 4 * np.maximum(rs["contacts"], 1))).sum())
    assert out > 0 or make is _alike
