"""Autotuner for the batched step's launch shapes.

Searches, on the caller's own batch and scene state, over
  * resolver lanes per world G (worlds per warp = 32 / G),
  * the resolver's shared-memory contact tile (contacts per world kept on chip),
  * the narrowphase CTA size,
  * with worlds of more than 64 bodies in the batch, the caller's list of
    large_world_lanes (by default the one setting: both run the same kernel),
  * with one world per warp, the fused frame (one launch per frame) or the
    three launches,
  * with the learned warm start enabled, optionally the warm-start budget
    threshold (which worlds are warm-started; it changes which of two valid
    solutions a world gets, within the resolver's epsilon, and the speed),
timing a short captured rollout for each candidate with CUDA events (the
whole of it, as cz_step runs it: its parts overlap, so a phase's own time does
not tell), and leaves the batch set to the fastest.  The launch-shape candidates all compute the same
bits (the parity tests run all lanes settings), so they change only speed.

The state is restored from the batch snapshot before every trial, so the
search is reproducible; the snapshot should hold a representative
(settled) state.
"""
import itertools

import numpy as np

DEFAULT_LANES = (8, 16, 32)  # 4 runs as 8
DEFAULT_TILES = (64, 96, 128, 192)
DEFAULT_NP_THREADS = (32, 64, 128, 256)
DEFAULT_LARGE_LANES = (32,)  # both settings run the same kernel
BIG_WORLD = 64  # worlds of more bodies than this go to the large-world resolver


def tune(batch, frames=30, dt=1.0 / 60.0, lanes=DEFAULT_LANES, tiles=DEFAULT_TILES, np_threads=DEFAULT_NP_THREADS,
         warm_shifts=(), large_lanes=DEFAULT_LARGE_LANES, fused=True, repeats=1, log=None):
    """Returns (best_config, trials); the batch is left at best_config."""
    trials = []

    def measure():
        """(ms of the whole rollout, its phases' ms)"""
        runs = []
        for _ in range(repeats):
            batch.restore()
            total, phases = batch.step_timed(frames, dt)
            runs.append((float(total), phases))
        return min(runs, key=lambda r: r[0])

    # narrowphase CTA size first (independent of the resolver settings)
    np_best, np_time = None, None
    for t in np_threads:
        batch.set_tuning(narrowphase_threads=t)
        ms, ph = measure()
        trials.append({"narrowphase_threads": t, "narrowphase_ms": float(ph[1]), "step_ms": ms})
        if np_time is None or ms < np_time:
            np_best, np_time = t, ms
    batch.set_tuning(narrowphase_threads=np_best)
    best, best_ms = None, None
    for g, cs in itertools.product(lanes, tiles):
        try:
            batch.set_tuning(resolver_lanes=g, resolver_contacts=cs)
        except Exception as e:  # a tile that does not fit in shared memory
            trials.append({"resolver_lanes": g, "resolver_contacts": cs, "error": str(e)})
            continue
        ms, ph = measure()
        cfg = batch.get_tuning()
        trials.append({"resolver_lanes": g, "resolver_contacts": cfg["resolver_contacts"],
                       "resolver_ms": float(ph[2]), "step_ms": ms})
        if log:
            log("lanes=%d tile=%d resolve %.3f of %.3f ms" % (g, cfg["resolver_contacts"], ph[2], ms))
        if best_ms is None or ms < best_ms:
            best, best_ms = (g, cfg["resolver_contacts"]), ms
    batch.set_tuning(resolver_lanes=best[0], resolver_contacts=best[1])
    # one launch per frame, where the batch allows it (one world per warp, no
    # world above the slot, the plain resolver): the batch ignores it otherwise
    if (fused and best[0] == 32 and not getattr(batch, "warm_start", False)
            and not (np.asarray(batch.counts) > BIG_WORLD).any()):
        best_f, f_ms = None, None
        for f in (-1, 1):
            batch.set_tuning(fused_frame=f)
            ms, ph = measure()
            trials.append({"fused_frame": f, "step_ms": ms})
            if f_ms is None or ms < f_ms:
                best_f, f_ms = f, ms
        batch.set_tuning(fused_frame=best_f)
    if large_lanes and (np.asarray(batch.counts) > BIG_WORLD).any():
        best_ll, ll_ms = None, None
        for g in large_lanes:
            batch.set_tuning(large_world_lanes=g)
            ms, ph = measure()
            trials.append({"large_world_lanes": g, "resolver_ms": float(ph[2]), "step_ms": ms})
            if ll_ms is None or ms < ll_ms:
                best_ll, ll_ms = g, ms
        batch.set_tuning(large_world_lanes=best_ll)
    if warm_shifts:
        best_shift, shift_ms = None, None
        for sh in warm_shifts:
            batch.set_tuning(warm_start_budget_shift=sh)
            ms, ph = measure()
            trials.append({"warm_start_budget_shift": sh, "resolver_ms": float(ph[2]), "step_ms": ms})
            if shift_ms is None or ms < shift_ms:
                best_shift, shift_ms = sh, ms
        batch.set_tuning(warm_start_budget_shift=best_shift)
    batch.restore()
    cfg = batch.get_tuning()
    return cfg, trials
