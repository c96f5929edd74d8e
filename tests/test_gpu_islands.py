"""The resolver's islands (build_islands, resolve_phase in cz_resolve.cuh): the
connected components of a world's contacts solved side by side give the
reference's sequence bit for bit, and a world whose islands want more than its
iteration budget is put back and solved as one list."""
import numpy as np
import pytest

from cubez_gb300 import scenes
from oracle.oracle import FP32 as ORC_FP32
from oracle.oracle import FP64 as ORC_FP64
from oracle.oracle import OracleBatch

pytestmark = pytest.mark.gpu

DT = 1.0 / 60.0
STATE = ("position", "orientation", "velocity", "rotation", "motion", "is_awake")


def _settled(form, frames, worlds=24, sleep=False, seed=51):
    """A scene holding the oracle's state after `frames` frames."""
    scene = scenes.mixed(num_worlds=worlds, seed=seed, min_bodies=1, max_bodies=64)
    scene.can_sleep[:] = 1 if sleep else 0
    ref = OracleBatch(scene, form=form)
    ref.step(frames, DT, threads=8)
    st = ref.bodies()
    moved = scene.copy()
    for k in STATE:
        setattr(moved, k, st[k])
    return moved


# budgets from one iteration to more than any world uses: the position phase
# alone runs out, the velocity phase runs out, neither does
@pytest.mark.parametrize("form", [0, 1])
@pytest.mark.parametrize("lanes", [4, 8, 16, 32])
@pytest.mark.parametrize("budget", [1, 2, 7, 33, 150, 4000])
def test_fixed_budget_bit_exact(form, lanes, budget, cuda_lib):
    from cubez_gb300.batch import WorldBatch
    orc = ORC_FP64 if form == 0 else ORC_FP32
    scene = _settled(orc, 130)
    gpu = WorldBatch.from_scene(scene, form=form, max_iterations=budget)
    gpu.set_tuning(resolver_lanes=lanes, resolver_contacts=96)
    ref = OracleBatch(scene, form=orc)
    hit = 0
    for _ in range(3):
        gpu.integrate(DT)
        gpu.narrowphase()
        gpu.resolve(DT)
        ref.integrate(DT)
        ref.narrowphase()
        ref.resolve_fixed(budget, DT)
        g, r = gpu.download(STATE), ref.bodies()
        for k in STATE:
            assert np.array_equal(g[k], r[k]), k
        gs, rs = gpu.stats(), ref.stats()
        assert np.array_equal(gs["pos_iterations"], rs["pos_iterations"])
        assert np.array_equal(gs["vel_iterations"], rs["vel_iterations"])
        hit += int((rs["vel_iterations"] >= budget).sum())
    assert (hit > 0) == (budget < 4000)


@pytest.mark.parametrize("form", [0, 1])
@pytest.mark.parametrize("lanes", [16, 32])
def test_sleeping_islands_and_spilled_tiles_bit_exact(form, lanes, cuda_lib):
    """Bodies asleep and woken inside the solve (a restart puts their awake
    flags and motion back), and worlds whose contacts exceed the shared tile."""
    from cubez_gb300.batch import WorldBatch
    orc = ORC_FP64 if form == 0 else ORC_FP32
    scene = _settled(orc, 150, sleep=True, seed=52)
    for budget in (25, 0):
        gpu = WorldBatch.from_scene(scene, form=form, max_iterations=budget)
        gpu.set_tuning(resolver_lanes=lanes, resolver_contacts=32)
        ref = OracleBatch(scene, form=orc)
        for _ in range(60):
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
        assert ref.stats()["contacts"].max() > 32
