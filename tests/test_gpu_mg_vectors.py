"""The solver's vector passes over grids just above the size from which they use 16-byte vectors: a scene stepped
alone (vectors; sums over lanes in FP32, runs of eight in the mixed solve) against the same scene in a work-list
batch, whose FP32 passes take one element per thread -- bitwise, as the sums keep their order -- with rows of a
multiple of 8, of 4 and of neither."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("opts", [dict(tol=1e-6, tol_mode=1, max_iters=60),
                                  dict(tol=1e-6, tol_mode=2, max_iters=60, precision="fp16", warm_start=3,
                                       true_residual_every=2)])
def test_vector_passes_equal_worklist(opts):
    import pfm
    from pfm import _lib

    def make(res, graph):
        levels = 2 if res[2] % 4 else 0  # every level halves exactly
        dx = 1.0 / res[1]
        g = torch.Generator(device="cuda").manual_seed(sum(res))
        u = [torch.randn([n + (a == f) for a, n in enumerate(res)], device="cuda", generator=g) for f in range(3)]
        for f in range(3):
            u[f].select(f, 0).zero_()
            u[f].select(f, res[f]).zero_()
        sim = pfm.Sim3D(u, pfm.jittered(res, dx, 8, seed=2), res, dx, reinit_every=4, poisson_opts=opts, graph=graph,
                        mg_levels=levels)
        sim.scene.set_tuning(_lib.TUNE_MG_CLUSTER, 0)
        return sim

    specs = [(48, 40, 40), (48, 48, 36), (48, 40, 42)]
    alone = [make(s, False) for s in specs]
    together = [make(s, True) for s in specs]
    batch = pfm.Batch(together, worklist=True)
    for _ in range(2):
        for sim in alone:
            sim.step()
        batch.step()
    torch.cuda.synchronize()
    for a, b in zip(alone, together):
        assert torch.equal(a.p, b.p)
        for f in range(3):
            assert torch.equal(a.u[f], b.u[f])


@pytest.mark.parametrize("res,precision,walls", [((141, 200, 184), "fp16", [[2, 2]] * 3),
                                                 ((143, 250, 144), "bf16", [[1, 2], [2, 1], [2, 1]]),
                                                 ((142, 196, 184), "fp16", [[2, 1], [1, 2], [1, 2]])])
def test_plane_march_equals_tma_tiles(res, precision, walls):
    """16-bit levels large enough for the half-sweep that goes up several planes, with 1 to 3 planes left at the
    end: bitwise the tiled kernel, whose update is the per-cell one's."""
    import pfm
    from pfm import _lib

    sc = pfm.Scene(3, res, 1.0 / res[1], 0, mg_levels=1, boundary=walls, bottom_smoothing=3)
    g = torch.Generator(device="cuda").manual_seed(11)
    u0 = [torch.randn(s, device="cuda", generator=g) for s in sc.face_shapes]
    out = []
    for tma in (0, 1):
        sc.set_tuning(_lib.TUNE_SMOOTH_TMA, tma)
        p = torch.zeros(sc.cell_shape, device="cuda")
        sc.poisson([x.clone() for x in u0], p, precision=precision, tol=1e-6, tol_mode=1, max_iters=3)
        out.append(p)
    assert torch.isfinite(out[0]).all() and out[0].abs().max() > 0
    assert torch.equal(out[0], out[1])


@pytest.mark.parametrize("nz", [31, 32, 63, 64, 127, 128, 160])
@pytest.mark.parametrize("walls", [[2, 2], [1, 2], [2, 1]])
def test_z_faces_lose_the_pressure_gradient(nz, walls):
    """The last axis' faces after a projection: bitwise u - (p above - p below), zero on the walls."""
    import pfm

    res = (9, 7, nz)
    sc = pfm.Scene(3, res, 1.0 / 8, 0, mg_levels=1, boundary=[[2, 2], [2, 2], walls])
    g = torch.Generator(device="cuda").manual_seed(nz)
    u = [torch.randn(s, device="cuda", generator=g) for s in sc.face_shapes]
    if walls[0] == 2:
        u[2][..., 0] = 0
    if walls[1] == 2:
        u[2][..., nz] = 0
    before, p = u[2].clone(), torch.zeros(sc.cell_shape, device="cuda")
    sc.poisson(u, p, tol=1e-6, tol_mode=1, max_iters=20)
    pad = torch.zeros(res[0], res[1], 1, device="cuda")
    want = before - (torch.cat([p, pad], 2) - torch.cat([pad, p], 2))
    if walls[0] == 2:
        want[..., 0] = 0
    if walls[1] == 2:
        want[..., nz] = 0
    assert torch.equal(u[2], want)
