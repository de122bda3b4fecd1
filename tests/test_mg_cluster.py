"""The MGPCG solves and coarse levels that run on one thread-block cluster (csrc/pfm_mgcluster.cu)."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "particle-flow-maps_gb300"))


@pytest.mark.parametrize("m", [1, 2, 3, 4, 5, 6])
def test_two_operation_division_is_the_ieee_quotient(m):
    """fma(x, zh, RN(x zl)) with zh = RN(1/m), zl = RN(1/m - zh) rounds to x / m for every f32
    significand (three binades: the quotient's binade changes within one)."""
    f = np.float32
    zh = f(1) / f(m)
    zl = f((1 - m * np.float64(zh)) / m)
    for e in (126, 127, 128):
        x = (np.arange(1 << 23, dtype=np.uint32) | np.uint32(e << 23)).view(f)
        t = (x * zl).astype(f)
        # x zh is exact in f64 (48 bits); its sum with t rounds to 53 bits first, then to 24: a double
        # rounding could only hide a tie, which a quotient by 3, 5 or 6 never is
        q = (x.astype(np.float64) * np.float64(zh) + t.astype(np.float64)).astype(f)
        assert np.array_equal(q, x / f(m))


def _laplacian_neg(x):
    """A x (mult x - neighbour sum, all-Neumann) in f64."""
    out = np.zeros_like(x)
    for a in range(x.ndim):
        d = np.diff(x, axis=a)
        lo = [slice(None)] * x.ndim
        hi = [slice(None)] * x.ndim
        lo[a], hi[a] = slice(0, -1), slice(1, None)
        out[tuple(lo)] -= d
        out[tuple(hi)] += d
    return out


def _solve(res, cluster, precision, **kw):
    import torch
    import pfm
    from pfm import _lib
    sc = pfm.Scene(len(res), res, 1.0 / res[1], 0)
    sc.set_tuning(_lib.TUNE_MG_CLUSTER, cluster)
    rng = np.random.default_rng(sum(res))
    b = rng.standard_normal(res)
    r = torch.as_tensor((b - b.mean()).astype(np.float32)).cuda()
    x = torch.as_tensor((0.1 * rng.standard_normal(res)).astype(np.float32)).cuda()
    info = sc.mgpcg_solve(r, x, k=1.0, precision=precision, max_iters=100, **kw)
    torch.cuda.synchronize()
    return info, r.cpu().numpy().astype(np.float64), x


# sizes at the edges of the shares, vectors and levels: one CTA to sixteen, bottoms of odd and even
# extents that are no multiple of four, two levels and many, solo levels of more than one vector per thread
WHOLE = [(16, 16), (64, 64), (40, 72), (72, 40), (120, 456), (512, 512), (16, 16, 16), (64, 64, 64), (48, 32, 32),
         (24, 40, 36), (44, 52, 60), (96, 48, 56), (64, 104, 40)]


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp32", "fp16", "bf16"])
@pytest.mark.parametrize("res", WHOLE)
def test_cluster_solve_meets_the_rule(res, precision):
    """From a random warm start to |r| < 1e-6 |b|: the residual of the returned x, formed in f64, is the
    rule's plus what FP32 storage of x leaves (each of the 2 D + 1 terms of A x carries x's rounding, 2^-24
    of it, once per update), and the iterations are those of the grid-wide kernels to within one."""
    kw = dict(tol=1e-6, tol_mode=2, warm_start=True, true_residual_every=2)
    info, b, x = _solve(res, 1, precision, **kw)
    grid, _, _ = _solve(res, 0, precision, **kw)
    assert info.converged and abs(info.iterations - grid.iterations) <= 1
    x = x.cpu().numpy().astype(np.float64)
    left = np.linalg.norm(b - _laplacian_neg(x))
    floor = 4 * len(res) * 2.0 ** -24 * np.linalg.norm(x) * (info.iterations + 2)
    assert left <= 1e-6 * np.linalg.norm(b) + floor
    assert info.rTr_true ** 0.5 <= left + floor
    assert info.bTb == pytest.approx(grid.bTb, rel=1e-6)


@pytest.mark.gpu
@pytest.mark.parametrize("res", [(1024, 512), (160, 96, 72), (104, 112, 88), (72, 48, 96)])
def test_cluster_tail_is_bitwise_the_grid_kernels(res):
    """Grids too large for one cluster: the coarse levels of their V-cycles on a cluster give the grid-wide
    kernels' solve bit for bit (FP32), with and without levels small enough for one CTA."""
    kw = dict(tol=1e-6, tol_mode=1)
    a, _, xa = _solve(res, 1, "fp32", **kw)
    b, _, xb = _solve(res, 0, "fp32", **kw)
    assert (a.iterations, a.rTr) == (b.iterations, b.rTr)
    assert bool((xa == xb).all())


@pytest.mark.gpu
def test_cluster_solve_limits_and_statuses():
    """max_iters 0 and 1, a zero right-hand side, a wall that is not Neumann and a non-finite right-hand
    side end as the grid-wide solve ends."""
    import torch
    import pfm
    from pfm import _lib
    res = (64, 48)
    r = torch.randn(res, device="cuda", generator=torch.Generator(device="cuda").manual_seed(1))
    for bc in ([[2, 2], [2, 2]], [[2, 2], [1, 2]]):
        got = []
        for cluster in (1, 0):
            sc = pfm.Scene(2, res, 1 / 48, 0, boundary=bc)
            sc.set_tuning(_lib.TUNE_MG_CLUSTER, cluster)
            out = []
            for it in (0, 1, 200):
                x = torch.zeros_like(r)
                i = sc.mgpcg_solve(r, x, tol=1e-6, tol_mode=1, max_iters=it)
                out.append((i.iterations, i.converged, float(x.abs().max()) > 0))
            x = torch.zeros_like(r)
            i = sc.mgpcg_solve(torch.zeros_like(r), x, tol=1e-6, tol_mode=1)
            out.append((i.iterations, i.converged, float(x.abs().max())))
            bad = r.clone()
            bad[3, 5] = float("nan")
            with pytest.raises(pfm.PfmError, match="NONFINITE"):
                sc.mgpcg_solve(bad, x, tol=1e-6, tol_mode=1)
            got.append(out)
        assert got[0] == got[1]
