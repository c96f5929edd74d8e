"""cz_step_timed runs what cz_step runs: the same launches, in parts or in one
chain, over one graph or several, and the same bits; its phases' times add up
to the rollout's."""
import numpy as np
import pytest

from cubez_gb300 import scenes

pytestmark = pytest.mark.gpu

DT = 1.0 / 60.0
FIELDS = ("position", "orientation", "velocity", "rotation", "motion", "is_awake")


@pytest.mark.parametrize("form", [0, 1])
@pytest.mark.parametrize("worlds,frames", [(3, 5), (64, 33), (127, 5), (128, 5), (300, 33), (300, 67)])
def test_timed_runs_what_step_runs(form, worlds, frames, cuda_lib):
    from cubez_gb300 import _lib
    from cubez_gb300.batch import WorldBatch
    scene = scenes.mixed(num_worlds=worlds, seed=worlds, min_bodies=1, max_bodies=16)
    a, b = (WorldBatch.from_scene(scene, form=form) for _ in range(2))
    launches = []
    for g in (a, b):
        g.prepare_rollout(frames, DT)
        g.step(50, DT)
        before = _lib.kernel_launches()
        if g is a:
            g.step(frames, DT)
        else:
            total, phases = g.step_timed(frames, DT)
        launches.append(_lib.kernel_launches() - before)
    assert launches[0] == launches[1]
    x, y = a.download(FIELDS), b.download(FIELDS)
    for k in FIELDS:
        assert np.array_equal(x[k], y[k]), k
    assert a.counters() == b.counters()
    # (event nodes lie between the phases of one chain; parts share out the total)
    assert np.all(phases > 0.0) and phases.sum() <= total * 1.0001
    assert phases.sum() >= 0.5 * total
