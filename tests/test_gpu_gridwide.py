"""The grid-wide MGPCG kernels on grids that a thread-block cluster solves whole by default: with that switched off,
the knobs of the grid-wide form give bitwise the same solves, and a work-list batch may hold scenes of either form."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import pfm  # noqa: E402
from pfm import _lib  # noqa: E402
from __graft_entry__ import _ring_velocity  # noqa: E402


def _solve(sc, r, key, value, **kw):
    """(x, iterations, r.r, kernels) of a solve with knob `key` at `value`."""
    sc.set_tuning(key, value)
    kw = dict(tol=1e-6, tol_mode=1, max_iters=200, **kw)
    assert not sc.solve_on_cluster(**kw)
    x = torch.zeros_like(r)
    before = sc.launches
    info = sc.mgpcg_solve(r, x, k=-1.0, **kw)
    torch.cuda.synchronize()
    return x, info.iterations, info.rTr, sc.launches - before


def _scene(res, seed, **kw):
    sc = pfm.Scene(len(res), res, 1.0 / res[1], 0, **kw)
    assert sc.solve_on_cluster()
    sc.set_tuning(_lib.TUNE_MG_CLUSTER, 0)
    return sc, torch.as_tensor(np.random.default_rng(seed).standard_normal(res).astype(np.float32)).cuda()


@pytest.mark.parametrize("res,base,cells", [((48, 32, 32), 2, (0, 4096, 8192)), ((64, 48), 3, (0, 256, 4096)),
                                            ((96, 160), 3, (0, 1024, 4096))])
def test_tail_thresholds(res, base, cells):
    """FP32 levels: without a tail, with a tail of levels that fit its registers, and of larger ones; the tail's
    levels take one kernel instead of theirs."""
    sc, r = _scene(res, 8, base_level=base)
    out = [_solve(sc, r, _lib.TUNE_MG_TAIL_CELLS, c) for c in cells]
    for x, it, rtr, kernels in out[1:]:
        assert torch.equal(out[0][0], x) and (it, rtr) == out[0][1:3] and kernels < out[0][3]


@pytest.mark.parametrize("precision", [1, 2])
@pytest.mark.parametrize("res", [(64, 64, 64), (40, 24, 48)])
def test_tma_smoother(res, precision):
    sc, r = _scene(res, 21)
    out = [_solve(sc, r, _lib.TUNE_SMOOTH_TMA, v, precision=precision) for v in (0, 1)]
    assert torch.equal(out[0][0], out[1][0]) and out[0][1:3] == out[1][1:3]
    assert min(o[3] for o in out) > 20  # half-sweeps, not one launch


def _sim(spec, opts, cluster, graph):
    dx = 1.0 / spec[1]
    if len(spec) == 2:
        sim = pfm.Sim2D(pfm.vortex_blobs2(spec, dx, seed=sum(spec)), pfm.jittered(spec, dx, 4, seed=1), spec, dx,
                        reinit_every=5, reinit_every_grad_m=2, poisson_opts=opts, graph=graph)
    else:
        sim = pfm.Sim3D(_ring_velocity(spec, dx), pfm.jittered(spec, dx, 8, seed=1), spec, dx, reinit_every=4,
                        poisson_opts=opts, graph=graph)
    sim.scene.set_tuning(_lib.TUNE_MG_CLUSTER, cluster)
    return sim


def test_tail_threshold_in_a_step():
    opts = dict(tol=1e-6, tol_mode=1, max_iters=400)
    a, b = (_sim((64, 48), opts, 0, True) for _ in range(2))
    b.scene.set_tuning(_lib.TUNE_MG_TAIL_CELLS, 0)
    for _ in range(5):
        a.step()
        b.step()
    torch.cuda.synchronize()
    assert all(torch.equal(x, y) for x, y in zip(a.u, b.u))
    assert torch.equal(a.p, b.p) and torch.equal(a.pos, b.pos)


@pytest.mark.parametrize("form", ["none", "mixed", "all"])
@pytest.mark.parametrize("precision", ["fp32", "fp16"])
@pytest.mark.parametrize("dim", [2, 3])
def test_worklist_forms(dim, precision, form):
    """A work-list batch whose scenes solve grid-wide, on a cluster, or some of each: bitwise the scenes stepped alone
    in the same form, with their iterations; one scene without a V-cycle tail."""
    opts = dict(tol=1e-6, tol_mode=1, max_iters=400)
    if precision == "fp16":
        opts = dict(tol=1e-6, tol_mode=2, max_iters=400, precision="fp16", warm_start=dim == 3, true_residual_every=5)
    specs = ([(32, 32), (128, 128), (48, 48), (256, 64), (96, 80)] if dim == 2 else
             [(16, 16, 16), (32, 16, 24), (24, 24, 24), (32, 32, 32)])
    cluster = {"none": [0] * 5, "all": [1] * 5, "mixed": [0, 1, 0, 1, 0]}[form]
    alone = [_sim(s, opts, c, False) for s, c in zip(specs, cluster)]
    together = [_sim(s, opts, c, True) for s, c in zip(specs, cluster)]
    for sims in (alone, together):
        sims[0].scene.set_tuning(_lib.TUNE_MG_TAIL_CELLS, 0)
    solver = {k: v for k, v in opts.items() if k != "warm_start"}
    on = [s.scene.solve_on_cluster(**solver) for s in together]
    assert any(on) == (form != "none") and (form != "mixed" or not all(on))
    batch = pfm.Batch(together, worklist=True)
    for _ in range(6):
        for sim in alone:
            sim.step()
        batch.step()
    torch.cuda.synchronize()
    for a, b in zip(alone, together):
        assert all(torch.equal(x, y) for x, y in zip(a.u, b.u))
        assert torch.equal(a.pos, b.pos) and torch.equal(a.p, b.p)
        info = b.step_info()
        assert info.step == a.i == 5 and info.dt == a.last_dt
        assert [info.iterations[0], info.iterations[1]] == [a.infos[-2].iterations, a.infos[-1].iterations]
    # a solve on a cluster is one of its scene's kernels, a grid-wide one many
    kernels = [b.scene.launches for b in together]
    assert len({k for k, o in zip(kernels, on) if o}) <= 1
    assert all(k > 1.2 * max((c for c, o in zip(kernels, on) if o), default=0) for k, o in zip(kernels, on) if not o)
