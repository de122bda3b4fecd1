"""The sums of a pressure solve, on a thread-block cluster (csrc/pfm_mgcluster.cu) and grid-wide (csrc/pfm_mgpcg.cu)."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import pfm  # noqa: E402
from pfm import _lib  # noqa: E402


def _smooth_divergence(res, seed):
    """The divergence of the f32 gradient of a few Gaussian blobs: its sum is the rounding of its terms."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    phi = torch.zeros(res, device="cuda", dtype=torch.float64)
    for _ in range(6):
        e = torch.ones([1] * len(res), device="cuda", dtype=torch.float64) * float(torch.randn(1, generator=g, device="cuda"))
        for a, n in enumerate(res):
            shape = [1] * len(res)
            shape[a] = n
            at = torch.arange(n, device="cuda", dtype=torch.float64) / n
            e = e * torch.exp(-((at - float(torch.rand(1, generator=g, device="cuda")) * 0.6 - 0.2) / 0.06) ** 2).view(shape)
        phi += e
    d = torch.zeros_like(phi)
    for a, n in enumerate(res):
        q = (phi.narrow(a, 1, n - 1) - phi.narrow(a, 0, n - 1)).float().double()
        d.narrow(a, 0, n - 1).add_(q)
        d.narrow(a, 1, n - 1).sub_(q)
    return d.float()


@pytest.mark.parametrize("res,seed", [((448, 512), 67), ((448, 512), 12), ((512, 512), 48), ((64, 64, 64), 45)])
def test_mean_of_the_residual(res, seed):
    """All walls Neumann: the residual's mean is what its own rounding leaves, and an error in it moves the pressure's
    constant through the singular coarsest level.  After eight iterations the pressure is the grid-wide solve's
    to the rounding of its FP32 storage, 2^-24 of its norm."""
    r = _smooth_divergence(res, seed)
    sc = pfm.Scene(len(res), res, 1.0 / res[1], 0)
    x = []
    for cluster in (1, 0):
        sc.set_tuning(_lib.TUNE_MG_CLUSTER, cluster)
        x.append(torch.zeros_like(r))
        sc.mgpcg_solve(r, x[-1], tol=0.0, max_iters=8)
    a, b = (t.double() for t in x)
    assert (a - b).norm() <= 2.0 ** -24 * b.norm()


# tolerances an f32 cannot hold, beside ordinary ones
@pytest.mark.parametrize("mode,tol", [(0, 1e-60), (0, 0.0), (0, -1.0), (0, 1e-6), (0, 1e300), (0, float("inf")),
                                      (0, float("nan")), (1, 1e-60), (1, 0.0), (1, 1e-6), (1, 1e200), (1, float("inf")),
                                      (2, 1e-5), (2, 1e-40), (2, float("inf"))])
def test_stopping_rule(mode, tol):
    """Every tolerance ends a solve where it ends the grid-wide one, for a right-hand side and for a fluid at rest."""
    res = (64, 48)
    sc = pfm.Scene(2, res, 1 / 48, 0)
    g = torch.Generator(device="cuda").manual_seed(3)
    for r in (torch.randn(res, device="cuda", generator=g), torch.zeros(res, device="cuda")):
        got = []
        for cluster in (1, 0):
            sc.set_tuning(_lib.TUNE_MG_CLUSTER, cluster)
            info = sc.mgpcg_solve(r, torch.zeros_like(r), tol=tol, tol_mode=mode, max_iters=12)
            got.append((info.iterations, info.converged, info.status))
        assert got[0] == got[1]


@pytest.mark.parametrize("precision", ["fp32", "fp16"])
@pytest.mark.parametrize("res,cluster", [((512, 512), 1), ((64, 64, 64), 1), ((64, 64, 64), 0), ((512, 512), 0)])
def test_large_residuals(res, cluster, precision):
    """A right-hand side whose products are f32 numbers and whose sum of squares is not: the solve is that of the
    same numbers a power of two smaller.  Beside eps = 1e-12 and the FP16 scale (one rounding), every operation
    scales exactly; each of the few iterations may round alpha and beta otherwise, 2^-24 of the pressure each."""
    g = torch.Generator(device="cuda").manual_seed(7)
    r = torch.randn(res, device="cuda", generator=g)
    sc = pfm.Scene(len(res), res, 1.0 / res[1], 0)
    sc.set_tuning(_lib.TUNE_MG_CLUSTER, cluster)
    kw = dict(tol=1e-5, tol_mode=2, max_iters=40, precision=precision, true_residual_every=3)
    a, b = torch.zeros_like(r), torch.zeros_like(r)
    small = sc.mgpcg_solve(r, a, **kw)
    f = 2.0 ** 56
    assert float((r.double() * f).square().sum()) > 3.5e38 > float((r * f).square().max())
    large = sc.mgpcg_solve(r * f, b, **kw)
    assert small.converged and (small.iterations, small.converged) == (large.iterations, large.converged)
    assert (a.double() - b.double() / f).norm() <= 2.0 ** -20 * a.double().norm()
    for x, y in ((small.rTr0, large.rTr0), (small.bTb, large.bTb)):
        assert abs(x - y / f / f) <= 1e-12 * x
