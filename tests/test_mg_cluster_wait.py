"""A solve on a thread-block cluster whose waits run out (csrc/pfm_mgcluster.cu): the limit is set to zero, so every
wait between its blocks gives up at once; the call returns PFM_ERR_CUDA and the handle solves as before once the
limit is back."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import pfm  # noqa: E402
from pfm import _lib  # noqa: E402


# one block and sixteen, with and without levels on one block alone, levels distributed to the bottom, and the
# coarse levels of larger grids
# (a 16-bit solve of at most 4,096 cells is the one-block kernels')
@pytest.mark.parametrize("precision", ["fp32", "fp16"])
@pytest.mark.parametrize("res,kw", [((16, 60), {}), ((128, 128), {}), ((512, 512), {}), ((64, 64, 64), {}),
                                    ((48, 32, 32), dict(true_residual_every=1)),
                                    ((128, 128), dict(max_iters=0, true_residual_every=2)),
                                    ((160, 96, 72), {}), ((1024, 512), {})])
def test_wait_limit_is_reported(res, kw, precision):
    if precision == "fp16" and res == (16, 60):
        res = (80, 60)
    kw = {**dict(tol=1e-6, tol_mode=1, max_iters=100, precision=precision), **kw}
    g = torch.Generator(device="cuda").manual_seed(sum(res))
    r = torch.randn(res, device="cuda", generator=g)
    sc, fresh = (pfm.Scene(len(res), res, 1.0 / res[1], 0) for _ in range(2))
    want, x = torch.zeros_like(r), torch.zeros_like(r)
    info = fresh.mgpcg_solve(r, want, **kw)
    limit = sc.get_tuning(_lib.TUNE_MG_CLUSTER_WAIT)
    sc.set_tuning(_lib.TUNE_MG_CLUSTER_WAIT, 0)
    for _ in range(2):
        with pytest.raises(pfm.PfmError, match="bounded wait gave up"):
            sc.mgpcg_solve(r, x, **kw)
    sc.set_tuning(_lib.TUNE_MG_CLUSTER_WAIT, limit)
    again = sc.mgpcg_solve(r, x, **kw)
    assert (again.iterations, again.rTr, again.rTr_true) == (info.iterations, info.rTr, info.rTr_true)
    assert torch.equal(want, x)


def test_wait_limit_ends_a_step_graph():
    """The whole-step graph goes on behind such a solve, whose status the step's record holds; the next run of the
    graph's scene with the limit back is a fresh scene's."""
    res, dx = (64, 64), 1.0 / 64
    opts = dict(tol=1e-6, tol_mode=1, max_iters=100)

    def make():
        return pfm.Sim2D(pfm.vortex_blobs2(res, dx, seed=5), pfm.jittered(res, dx, 4, seed=1), res, dx, reinit_every=5,
                         reinit_every_grad_m=2, poisson_opts=opts, graph=True)

    a = make()
    a.scene.set_tuning(_lib.TUNE_MG_CLUSTER_WAIT, 0)
    a.step()
    torch.cuda.synchronize()
    assert not a.step_info().converged[1]
    b, c = make(), make()
    b.step()
    c.step()
    torch.cuda.synchronize()
    assert b.step_info().converged[1] and torch.equal(b.p, c.p)


def test_wait_limit_range():
    sc = pfm.Scene(2, (32, 32), 1 / 32, 0)
    for bad in (-1, 4000001):
        with pytest.raises(pfm.PfmError):
            sc.set_tuning(_lib.TUNE_MG_CLUSTER_WAIT, bad)
    assert sc.get_tuning(_lib.TUNE_MG_CLUSTER_WAIT) == 2000000
