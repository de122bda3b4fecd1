"""Hierarchies with levels of odd extents: the prolongation over the last cells finds no coarse one behind the level's
end, and a solve does not depend on what the workspace held."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import pfm  # noqa: E402
from pfm import _lib  # noqa: E402


# odd first, middle and last axes on the second level; rows of a multiple of eight and of none; 2D
@pytest.mark.parametrize("precision", ["fp32", "fp16"])
@pytest.mark.parametrize("res,levels", [((48, 40, 42), 3), ((50, 40, 48), 3), ((100, 100, 100), 4), ((70, 64), 3),
                                        ((66, 130), 4), ((300, 260), 5)])
@pytest.mark.parametrize("tail", [0, 4096])
def test_solve_ignores_the_workspace(res, levels, precision, tail):
    g = torch.Generator(device="cuda").manual_seed(sum(res))
    r = torch.randn(res, device="cuda", generator=g)
    r -= r.mean()
    sc = pfm.Scene(len(res), res, 1.0 / res[1], 0, mg_levels=levels)
    sc.set_tuning(_lib.TUNE_MG_TAIL_CELLS, tail)
    out = []
    for byte in (0, 255, 0x7B):  # zeros, NaN in every float type, large numbers
        sc.workspace.fill_(byte)
        assert sc.lib.pfm_set_workspace(sc.h, sc.workspace.data_ptr(), sc.workspace.numel()) == 0
        x = torch.zeros_like(r)
        info = sc.mgpcg_solve(r, x, tol=1e-5, tol_mode=1, max_iters=60, precision=precision)
        assert torch.isfinite(x).all() and info.rTr < 1e-6 * info.rTr0
        out.append((x, info.iterations, info.rTr))
    for x, *rest in out[1:]:
        assert torch.equal(x, out[0][0]) and tuple(rest) == out[0][1:]
