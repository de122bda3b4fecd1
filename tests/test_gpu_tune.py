"""The autotuner times only knobs that act on the scene (pfm/tune.py)."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import pfm  # noqa: E402
from pfm import _lib, tune  # noqa: E402

KEYS = {"mg_tail_cells": _lib.TUNE_MG_TAIL_CELLS, "smooth_tma": _lib.TUNE_SMOOTH_TMA,
        "p2g2_column": _lib.TUNE_P2G2_COLUMN}


def _sim(res, opts):
    dx = 1.0 / res[1]
    if len(res) == 2:
        return pfm.Sim2D(pfm.vortex_blobs2(res, dx, seed=1), pfm.jittered(res, dx, 4, seed=1), res, dx,
                         poisson_opts=opts)
    import __graft_entry__ as G
    return pfm.Sim3D(G._ring_velocity(res, dx), pfm.jittered(res, dx, 8, seed=1), res, dx, poisson_opts=opts)


# solves that are one cluster launch, and one that is not: of 16-bit levels with the residual replaced
@pytest.mark.parametrize("res,opts,cluster,timed", [
    ((64, 48), {}, 1, set()), ((64, 48), {}, 0, {"mg_tail_cells"}),
    ((32, 32, 32), dict(precision=1), 1, set()),
    ((32, 32, 32), dict(precision=1, true_residual_every=2, true_residual_replace=True), 1,
     {"mg_tail_cells", "smooth_tma"})])
def test_idle_knobs_keep_their_value(res, opts, cluster, timed):
    sim = _sim(res, dict(tol=1e-6, tol_mode=1, max_iters=50, **opts))
    sim.scene.set_tuning(_lib.TUNE_MG_CLUSTER, cluster)
    assert sim.scene.solve_on_cluster(**sim.poisson_opts) == (not timed)
    before = {name: sim.scene.get_tuning(key) for name, key in KEYS.items()}
    chosen = tune.autotune(sim, reps=1)
    for name, (value, times) in chosen.items():
        assert bool(times) == (name in timed), name
        assert value == (sim.scene.get_tuning(KEYS[name]) if times else before[name])
    tune.apply(sim, chosen)
    assert all(sim.scene.get_tuning(KEYS[n]) == v for n, (v, _) in chosen.items())
