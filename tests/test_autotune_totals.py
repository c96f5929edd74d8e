"""The autotuner keeps the settings whose whole rollout is fastest, as cz_step
would run it: the parts of a large batch overlap, so a launch that is longer on
its own can make the shorter rollout."""
import numpy as np

from cubez_gb300 import autotune


class OverlappingBatch:
    """The fastest rollout is not the one with the shortest phases."""

    counts = np.full(256, 32, np.int32)

    def __init__(self):
        self.cfg = {"narrowphase_threads": 128, "resolver_contacts": 96, "resolver_lanes": 32, "fused_frame": -1}

    def set_tuning(self, **kw):
        self.cfg.update({k: v for k, v in kw.items() if v})

    def get_tuning(self):
        return dict(self.cfg)

    def restore(self):
        pass

    def step_timed(self, frames, dt):
        c = self.cfg
        if c["fused_frame"] == 1 and c["resolver_lanes"] == 32:
            return 30.0, np.array([0.0, 0.0, 5.0])
        total = 20.0 + abs(c["narrowphase_threads"] - 64) / 32 + abs(c["resolver_lanes"] - 32) / 8
        total += abs(c["resolver_contacts"] - 128) / 32
        return total, np.array([0.5, c["narrowphase_threads"] / 256, (c["resolver_lanes"] + c["resolver_contacts"]) / 10])


def test_whole_rollouts_decide():
    b = OverlappingBatch()
    cfg, _ = autotune.tune(b, frames=2)
    assert cfg == {"narrowphase_threads": 64, "resolver_contacts": 128, "resolver_lanes": 32, "fused_frame": -1}


def test_every_default_setting_runs_other_launches():
    """resolver_lanes 4 runs as 8, and both large_world_lanes settings run the
    same kernel: trying them would let noise pick."""
    assert autotune.DEFAULT_LANES == (8, 16, 32)
    assert len(autotune.DEFAULT_LARGE_LANES) == 1
