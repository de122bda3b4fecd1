"""3D P2G where a face's sum comes from one to eight cell tiles (4 x 4 x 16 cells): grids of one tile, of tiles cut
short on every axis and of odd and even tile counts, particles over the whole box and beyond it, against the oracle
(f32 sums of the reference's taps; the bar of the other P2G tests)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import oracle as O  # noqa: E402
import pfm  # noqa: E402


@pytest.mark.parametrize("res", [(4, 4, 4), (4, 8, 16), (5, 9, 17), (12, 4, 33), (7, 13, 31), (9, 16, 48)])
def test_p2g3_tiles(res):
    rng = np.random.default_rng(sum(res))
    dx = 1.0 / res[1]
    P = 6 * res[0] * res[1] * res[2]
    pos = (rng.uniform(-0.03, 1.03, (P, 3)) * np.array(res) * dx).astype(np.float32)
    T = (np.eye(3)[None] + 0.1 * rng.standard_normal((P, 3, 3))).astype(np.float32)
    Ti = (np.eye(3)[None] + 0.1 * rng.standard_normal((P, 3, 3))).astype(np.float32)
    C = rng.standard_normal((P, 3, 3)).astype(np.float32)
    m0 = rng.standard_normal((P, 3)).astype(np.float32)
    sc = pfm.Scene(3, res, dx, P, mg_levels=1)
    u, w = sc.alloc_faces(), sc.alloc_faces()
    for t in u + w:
        t.fill_(float("nan"))  # every face is written
    sc.p2g3(pfm.soa(m0), pfm.soa(pos), pfm.soa_T(T), pfm.soa_T(Ti), pfm.soa_T(C), u, w)
    ou, ow = O.p2g3(m0, pos, T, Ti, C, res, dx)
    for got, ref in zip(u + w, list(ou) + list(ow)):
        got, ref = got.cpu().numpy().astype(np.float64), np.asarray(ref, np.float64)
        assert np.linalg.norm(got - ref) < 1e-5 * np.linalg.norm(ref)
