"""2D P2G by face: grids whose rows end inside a warp and whose columns end inside a block, cells of zero to many
particles, and both forms of the kernel (one face per thread below 160,000 cells, two from there), against the oracle
(f32 sums of the reference's taps; the bar of the other P2G tests)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import oracle as O  # noqa: E402
import pfm  # noqa: E402


@pytest.mark.parametrize("res,ppc", [((4, 4), 5), ((5, 33), 4), ((31, 64), 2.5), ((8, 97), 9), ((401, 400), 2)])
@pytest.mark.parametrize("apic", [True, False])
def test_p2g2_faces(res, ppc, apic):
    rng = np.random.default_rng(res[0] + res[1])
    dx = 1.0 / res[1]
    P = int(ppc * res[0] * res[1])
    pos = (rng.uniform(-0.01, 1.01, (P, 2)) * np.array(res) * dx).astype(np.float32)
    imp = rng.standard_normal((P, 2)).astype(np.float32)
    C = (0.3 * rng.standard_normal((P, 2, 2))).astype(np.float32)
    psi = (pos + 0.01 * rng.standard_normal((P, 2))).astype(np.float32)
    sc = pfm.Scene(2, res, dx, P, mg_levels=1, use_apic=apic)
    u, w = sc.alloc_faces(), sc.alloc_faces()
    psi_g = [torch.full(s + (2,), float("nan"), device="cuda") for s in sc.face_shapes]
    for t in u + w:
        t.fill_(float("nan"))  # every face is written
    sc.p2g2(pfm.soa(imp), pfm.soa(pos), pfm.soa_T(C), pfm.soa(psi), u, w, psi_out=psi_g)
    refs = O.p2g2(imp, pos, C if apic else 0 * C, psi, res, dx)
    for got, ref in zip(u + w + psi_g, [r for pair in refs for r in pair]):
        got, ref = got.cpu().numpy().astype(np.float64), np.asarray(ref, np.float64)
        assert np.linalg.norm(got - ref) < 1e-5 * np.linalg.norm(ref)
