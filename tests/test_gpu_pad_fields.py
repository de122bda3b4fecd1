"""The padded copies of velocity fields that the midpoint and RK4 kernels read on grids without an instance of their
extent, one grid per pitch (128, 256, 512): bitwise the kernels with run-time strides, also from two streams at once
and in a captured graph (which takes the run-time strides)."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import pfm  # noqa: E402
from pfm import _lib  # noqa: E402


def _fields(sc, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return [0.3 * torch.randn(s, device="cuda", generator=g) for s in sc.face_shapes]


@pytest.mark.parametrize("res", [(70, 61, 75), (41, 130, 140), (20, 300, 260)])
def test_padded_equal_runtime_strides(res):
    dx = 1.0 / res[1]
    P = 2 * res[0] * res[1] * res[2]
    sc = pfm.Scene(3, res, dx, P, mg_levels=1)
    g = torch.Generator(device="cuda").manual_seed(3)
    u, ua = _fields(sc, 1), _fields(sc, 2)
    eye = torch.eye(3, device="cuda").reshape(3, 3, 1)
    pos = torch.rand(3, P, device="cuda", generator=g) * 1.02 - 0.01
    for a in range(3):
        pos[a] *= res[a] * dx
    T, Ti = (eye + 0.05 * torch.randn(3, 3, P, device="cuda", generator=g) for _ in range(2))
    imp = torch.randn(3, P, device="cuda", generator=g)
    dt = 0.4 * dx
    outs = []
    for cube in (1, 0):
        sc.set_tuning(_lib.TUNE_CUBE_KERNELS, cube)
        p0, T0, Ti0, C0 = pos.clone(), T.clone(), Ti.clone(), torch.zeros(3, 3, P, device="cuda")
        sc.gradm_rk4_records3(p0, T0, Ti0, C0, imp, u, ua, dt)
        p1, T1 = pos.clone(), T.clone()
        sc.rk4_T_forward(p1, T1, ua, dt)
        mid = sc.alloc_faces()
        sc.midpoint(u, mid, 0.5 * dt)
        outs.append([p0, T0, Ti0, C0, p1, T1] + list(mid))
    for x, y in zip(*outs):
        assert torch.equal(x, y)


def test_padded_streams_and_capture():
    res = (70, 61, 75)
    sc = pfm.Scene(3, res, 1.0 / 61, 0, mg_levels=1)
    fields = [_fields(sc, 4 + k) for k in range(4)]
    want = []
    for u in fields:
        mid = sc.alloc_faces()
        sc.midpoint(u, mid, 0.003)
        want.append(mid)
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in fields]
    got = [sc.alloc_faces() for _ in fields]
    torch.cuda.synchronize()
    for _ in range(5):
        for s, u, mid in zip(streams, fields, got):
            with torch.cuda.stream(s):
                sc.midpoint(u, mid, 0.003)
    torch.cuda.synchronize()
    cap = sc.alloc_faces()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        sc.midpoint(fields[1], cap, 0.003)
    graph.replay()
    torch.cuda.synchronize()
    for a, b in zip(want + [want[1]], got + [cap]):
        for x, y in zip(a, b):
            assert torch.equal(x, y)


def test_padded_beside_a_step_graph():
    """Midpoint calls on another stream while step graphs of the same handle run: both as when run alone."""
    res = (72, 64, 80)
    dx = 1.0 / 64

    def sim():
        g = torch.Generator(device="cuda").manual_seed(7)
        u = [torch.randn([n + (a == f) for a, n in enumerate(res)], device="cuda", generator=g) for f in range(3)]
        for f in range(3):
            u[f].select(f, 0).zero_()
            u[f].select(f, res[f]).zero_()
        return pfm.Sim3D(u, pfm.jittered(res, dx, 8, seed=2), res, dx, reinit_every=4,
                         poisson_opts=dict(tol=1e-6, tol_mode=1, max_iters=60), graph=True)

    alone = sim()
    for _ in range(4):
        alone.step()
    other = _fields(alone.scene, 9)
    want = alone.scene.alloc_faces()
    alone.scene.midpoint(other, want, 0.003)
    torch.cuda.synchronize()
    both, side = sim(), torch.cuda.Stream()
    got = [both.scene.alloc_faces() for _ in range(8)]
    torch.cuda.synchronize()
    for k in range(4):
        both.step()
        with torch.cuda.stream(side):
            for mid in got[2 * k:2 * k + 2]:
                both.scene.midpoint(other, mid, 0.003)
    torch.cuda.synchronize()
    for mid in got:
        for x, y in zip(want, mid):
            assert torch.equal(x, y)
    for x, y in zip(alone.u + [alone.pos], both.u + [both.pos]):
        assert torch.equal(x, y)
