"""The framework's work as a user's program calls it, as measurable cases.

``listed()`` names twelve cases and ``draw(rng)`` gives more of the same ranges; ``prepare`` builds what a
program holds before the call (scene, fields, network), ``run`` is one pass through the public entry
points, ``work`` the bytes and operations the pass cannot do without, and ``exact`` the same outputs
in 64-bit torch arithmetic without this package.

Kinds:
  solve2d / solve3d   one pressure projection (Scene.poisson): what the drop-in MGPCG.Poisson does
  step2d / step3d     one whole step of the simulation loop as a graph launch (Sim2D / Sim3D)
  batch2d             one step of many uneven 2D scenes (Batch)
  transport3d         the particle half of a 3D step: reinitialisation, RK4, P2G (fused as Sim3D
                      runs it, or phase by phase as the drop-in run_3D does)
  midpoint3d          the midpoint velocity and the CFL speed of a 3D step
  unet_predict        the learned warm start's inference on one divergence field
  unet_grad           its forward and backward on one (divergence, pressure) pair
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "particle-flow-maps_gb300"))

FACE3 = ((1, 0, 0), (0, 1, 0), (0, 0, 1))


def listed():
    return [
        # the smallest call: the drop-in's 2D projection with the reference's absolute rule (launch latency)
        {"name": "solve2d_128", "kind": "solve2d", "nx": 128, "ny": 128, "precision": "fp32", "relative": False},
        # the 2D leapfrog workload's step: 256 x 256, 262,144 particles
        {"name": "step2d_256", "kind": "step2d", "nx": 256, "ny": 256},
        # the batched workload in small: scenes of four sizes advanced by one launch, solver as a work list
        {"name": "batch2d_16", "kind": "batch2d", "n128": 8, "n256": 4, "n512": 2, "worklist": True},
        # a small 3D step in plain FP32, as a user tries the solver out
        {"name": "step3d_64_fp32", "kind": "step3d", "nx": 64, "ny": 64, "nz": 64, "precision": "fp32"},
        # the 128^3 two-ring workload's step with the mixed-precision, warm-started solves of the benchmark
        {"name": "step3d_128_fp16", "kind": "step3d", "nx": 128, "ny": 128, "nz": 128, "precision": "fp16"},
        # the drop-in's 3D projection on an elongated grid, plain FP32
        {"name": "solve3d_fp32", "kind": "solve3d", "nx": 160, "ny": 96, "nz": 72, "precision": "fp32",
         "relative": False},
        # the precision study's projection: 256^3, FP16 multigrid levels, to 1e-6 relative
        {"name": "solve3d_256_fp16", "kind": "solve3d", "nx": 256, "ny": 256, "nz": 256, "precision": "fp16",
         "relative": True},
        # the particle half of a step on a ragged grid (no extent a multiple of a tile), 6.0M particles
        {"name": "transport3d_ragged", "kind": "transport3d", "nx": 101, "ny": 75, "nz": 99, "fused": True},
        # the same phase by phase, as the drop-in step loop calls it, 7.1M particles
        {"name": "transport3d_dropin", "kind": "transport3d", "nx": 96, "ny": 96, "nz": 96, "fused": False},
        # the plume workload's midpoint phase at its own 192^3
        {"name": "midpoint3d_192", "kind": "midpoint3d", "nx": 192, "ny": 192, "nz": 192},
        # the learned warm start at the plume workload's 192^3 (inference) and 96^3 (training)
        {"name": "unet_predict_192", "kind": "unet_predict", "nx": 192, "ny": 192, "nz": 192},
        {"name": "unet_grad_96", "kind": "unet_grad", "nx": 96, "ny": 96, "nz": 96},
    ]


def _size(rng, lo, hi, step):
    """A size spread over the logarithm of [lo, hi], a multiple of step."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step)) * step))


def _grid(rng, dim, lo, hi):
    """Extents a multigrid hierarchy can halve down to its base level: with the shortest in [2^m, 2^(m+1)) the
    hierarchy has m - 2 levels, so every extent is a multiple of 2^(m-3)."""
    short = _size(rng, lo, hi, 4)
    step = max(4, 1 << (int(math.log2(short)) - 3))
    n = [short // step * step] + [_size(rng, short // step * step, hi, step) for _ in range(dim - 1)]
    rng.shuffle(n)
    return dict(zip(("nx", "ny", "nz"), n))


def draw(rng):
    kind = rng.choice(["solve2d", "step2d", "batch2d", "step3d", "step3d", "solve3d", "solve3d", "transport3d",
                       "transport3d", "midpoint3d", "unet_predict", "unet_grad"])
    if kind == "solve2d":
        return {"kind": kind, **_grid(rng, 2, 64, 1024), "precision": rng.choice(["fp32", "fp32", "fp16"]),
                "relative": True}
    if kind == "step2d":
        return {"kind": kind, **_grid(rng, 2, 96, 512)}
    if kind == "batch2d":
        return {"kind": kind, "n128": rng.randint(2, 12), "n256": rng.randint(1, 6), "n512": rng.randint(0, 2),
                "worklist": rng.random() < 0.5}
    if kind == "step3d":
        return {"kind": kind, **_grid(rng, 3, 40, 128), "precision": rng.choice(["fp32", "fp16", "bf16"])}
    if kind == "solve3d":
        return {"kind": kind, **_grid(rng, 3, 48, 256), "precision": rng.choice(["fp32", "fp32", "fp16", "bf16"]),
                "relative": rng.random() < 0.5}
    if kind == "transport3d":
        return {"kind": kind, "nx": _size(rng, 33, 128, 1), "ny": _size(rng, 33, 128, 1),
                "nz": _size(rng, 33, 128, 1), "fused": rng.random() < 0.6}
    if kind == "midpoint3d":
        return {"kind": kind, "nx": _size(rng, 33, 256, 1), "ny": _size(rng, 33, 256, 1),
                "nz": _size(rng, 33, 256, 1)}
    hi = 192 if kind == "unet_predict" else 96
    return {"kind": kind, "nx": _size(rng, 32, hi, 4), "ny": _size(rng, 32, hi, 4), "nz": _size(rng, 32, hi, 4)}


# ------------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------------
def _res(case):
    return tuple(case[k] for k in ("nx", "ny", "nz") if k in case)


def _dx(case):
    return 1.0 / case["ny"]  # the reference's dx = 1 / res_y


def _rng(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 17)


def _centres(n, dx, half, dim, axis):
    shape = [1] * dim
    shape[axis] = n
    return ((torch.arange(n, device="cuda", dtype=torch.float64) + half) * dx).view(shape)


def _blobs(res, dx, seed, count=6):
    """A smooth random cell field: a sum of Gaussian blobs, f64."""
    r = np.random.default_rng(seed)
    out = torch.zeros(res, device="cuda", dtype=torch.float64)
    for _ in range(count):
        s = r.uniform(0.04, 0.12)
        f = torch.ones([1] * len(res), device="cuda", dtype=torch.float64) * r.uniform(-1.0, 1.0)
        for a, n in enumerate(res):
            c = r.uniform(0.2, 0.8) * n * dx
            f = f * torch.exp(-((_centres(n, dx, 0.5, len(res), a) - c) / s) ** 2)
        out += f
    return out


def _swirl3(res, dx, seed):
    """Face velocities of a few smooth vortices (u = curl of Gaussian blobs), f32: of order one, as the
    rings of the workloads, smooth on the scale of ten cells, zero on the walls' normal faces."""
    r = np.random.default_rng(seed)
    u = [torch.zeros([n + d for n, d in zip(res, FACE3[f])], device="cuda", dtype=torch.float64) for f in range(3)]
    for _ in range(4):
        s = r.uniform(0.06, 0.12)
        w = r.uniform(-1.0, 1.0, 3)
        w *= 1.0 / (np.linalg.norm(w) + 1e-9)
        c = [r.uniform(0.3, 0.7) * n * dx for n in res]
        for f in range(3):
            d = [_centres(n + FACE3[f][a], dx, 0.0 if a == f else 0.5, 3, a) - c[a] for a, n in enumerate(res)]
            e = torch.exp(-(d[0] / s) ** 2) * torch.exp(-(d[1] / s) ** 2) * torch.exp(-(d[2] / s) ** 2)
            a, b = (f + 1) % 3, (f + 2) % 3
            u[f] += e * (w[a] * d[b] - w[b] * d[a]) * (2.3 / s)
    for f in range(3):
        u[f].select(f, 0).zero_()
        u[f].select(f, res[f]).zero_()
    return [a.float().contiguous() for a in u]


def _add_grad(u, phi, dx):
    """u += dx grad(phi) on interior faces: the divergence a transported velocity has before projection."""
    for f, a in enumerate(u):
        n = phi.shape[f]
        a.narrow(f, 1, n - 1).add_((phi.narrow(f, 1, n - 1) - phi.narrow(f, 0, n - 1)).float())


def _velocity(case, seed):
    res, dx = _res(case), _dx(case)
    if len(res) == 3:
        u = _swirl3(res, dx, seed)
    else:
        import pfm
        u = [torch.as_tensor(a).cuda() for a in pfm.vortex_blobs2(res, dx, seed)]
    return u


def _solver_opts(case):
    if case.get("relative", True):
        o = dict(tol=1e-6, tol_mode=2, max_iters=400)
    else:
        o = dict(tol=1e-12, tol_mode=0, max_iters=400)  # MGPCG.Poisson's own rule
    if case.get("precision", "fp32") != "fp32":
        o["precision"] = case["precision"]
        o["true_residual_every"] = 5
    return o


def _scene(case, particles):
    import pfm
    return pfm.Scene(len(_res(case)), _res(case), _dx(case), particles)


def _solve_state(case, seed):
    u0 = _velocity(case, seed)
    _add_grad(u0, _blobs(_res(case), _dx(case), seed + 1), _dx(case))
    sc = _scene(case, 0)
    return {"scene": sc, "u0": u0, "u": [torch.empty_like(a) for a in u0], "opts": _solver_opts(case),
            "p": torch.zeros(_res(case), device="cuda")}


def _step2d_sim(res, seed, graph=True):
    import pfm
    dx = 1.0 / res[1]
    opts = dict(tol=1e-6, tol_mode=1, max_iters=400)
    sim = pfm.Sim2D(pfm.vortex_blobs2(res, dx, seed), pfm.jittered(res, dx, 4, seed=seed), res, dx, visualize_dt=1e3,
                    reinit_every=12, reinit_every_grad_m=8, poisson_opts=opts)
    sim.scene.poisson(sim.u, sim.p, **opts)  # the projection of the initial velocity
    sim.set_graph(graph)
    return sim


def _step3d_sim(case, seed):
    import pfm
    res, dx = _res(case), _dx(case)
    opts = dict(tol=1e-6, tol_mode=2, max_iters=400)
    if case["precision"] != "fp32":
        opts.update(precision=case["precision"], warm_start=3, true_residual_every=5)
    seeds = torch.empty(3, res[0] * res[1] * res[2] * 8, device="cuda")
    sim = pfm.Sim3D(_swirl3(res, dx, seed), seeds, res, dx, visualize_dt=1e3, reinit_every=20, reinit_every_grad_m=1,
                    poisson_opts=opts)
    sim.scene.seed_jittered(sim.seeds, seed, 2)
    sim.scene.poisson(sim.u, sim.p, tol=1e-6, tol_mode=2, max_iters=400)
    sim.set_graph(True)
    return sim


def _batch_sizes(case):
    return [128] * case["n128"] + [256] * case["n256"] + [512] * case["n512"]


def _transport_state(case, seed):
    res, dx = _res(case), _dx(case)
    P = res[0] * res[1] * res[2] * 8
    sc = _scene(case, P)
    seeds = torch.empty(3, P, device="cuda")
    sc.seed_jittered(seeds, seed, 2)
    u = _swirl3(res, dx, seed)
    z = lambda *s: torch.zeros(*s, device="cuda")  # noqa: E731
    # u_adv: the projected midpoint velocity, a small change of u
    v = _swirl3(res, dx, seed + 1)
    s = {"scene": sc, "case": dict(case), "seeds": seeds, "u": u, "u_adv": [a + 0.05 * b for a, b in zip(u, v)],
         "pos": z(3, P), "T_gm": z(3, 3, P), "T_init": z(3, 3, P), "init_C": z(3, 3, P), "init_imp": z(3, P),
         "u_out": sc.alloc_faces(), "w_out": sc.alloc_faces(), "i": 0, "dt": _transport_dt(u, dx)}
    return s


def _transport_dt(u, dx):
    return float(np.float32(0.5 * dx / max(float(a.abs().max()) for a in u)))


def _unet_state(case, seed):
    import pfm
    from pfm import nn
    res, dx = _res(case), _dx(case)
    g = _rng(seed)
    p = _blobs(res, dx, seed, 8)
    div = _laplacian(p) + 1e-3 * p.abs().max() * torch.randn(res, device="cuda", dtype=torch.float64, generator=g) * dx
    assert pfm.Scene is not None
    return {"net": nn.UNet3D(seed=seed % 1000), "div": div.float(), "p": p.float(), "out": torch.empty(res, device="cuda")}


def _laplacian(p):
    out = torch.zeros_like(p)
    for a in range(p.dim()):
        n = p.shape[a]
        d = p.narrow(a, 1, n - 1) - p.narrow(a, 0, n - 1)
        out.narrow(a, 0, n - 1).add_(d)
        out.narrow(a, 1, n - 1).sub_(d)
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("solve2d", "solve3d"):
        return kind, _solve_state(case, seed)
    if kind == "step2d":
        return kind, _step2d_sim(_res(case), seed)
    if kind == "step3d":
        return kind, _step3d_sim(case, seed)
    if kind == "batch2d":
        import pfm
        sims = [_step2d_sim((n, n), seed * 100 + k, graph=False) for k, n in enumerate(_batch_sizes(case))]
        return kind, (pfm.Batch(sims, worklist=case["worklist"]), sims)
    if kind == "transport3d":
        return kind, _transport_state(case, seed)
    if kind == "midpoint3d":
        u = _swirl3(_res(case), _dx(case), seed)
        sc = _scene(case, 0)
        return kind, {"scene": sc, "u": u, "u_mid": sc.alloc_faces(), "dt_half": 0.5 * _transport_dt(u, _dx(case))}
    return kind, _unet_state(case, seed)


# ------------------------------------------------------------------------------------------------
# one pass
# ------------------------------------------------------------------------------------------------
def run(state):
    kind, s = state
    if kind in ("solve2d", "solve3d"):
        for a, b in zip(s["u"], s["u0"]):  # the velocity the transport has just written
            a.copy_(b)
        s["scene"].poisson(s["u"], s["p"], **s["opts"])
        return {"u": s["u"], "p": s["p"]}
    if kind == "step2d":
        s.step()
        return {"u": s.u, "p": s.p, "pos": s.pos, "imp": s.imp, "T": s.T, "C": s.C}
    if kind == "step3d":
        s.step()
        return {"u": s.u, "p": s.p, "pos": s.pos, "init_imp": s.init_imp, "T_gm": s.T_gm, "T_init": s.T_init,
                "init_C": s.init_C}
    if kind == "batch2d":
        batch, sims = s
        batch.step()
        return {"u": [q for x in sims for q in x.u][:30], "p": [x.p for x in sims][:16], "pos": [x.pos for x in sims][:16]}
    if kind == "transport3d":
        sc = s["scene"]
        if s["i"] % 20 == 0:  # the step loop's particle reinitialisation
            s["pos"].copy_(s["seeds"])
            sc.g2p(s["pos"], s["u"], imp_out=s["init_imp"])
            sc.reset_T(s["T_init"])
            sc.reset_T(s["T_gm"])
        s["i"] += 1
        if s["case"]["fused"]:
            sc.gradm_rk4_records3(s["pos"], s["T_gm"], s["T_init"], s["init_C"], s["init_imp"], s["u"], s["u_adv"],
                                  s["dt"])
            sc.p2g_from_records3(s["u_out"], s["w_out"])
        else:
            sc.g2p(s["pos"], s["u"], C_out=s["init_C"])
            sc.update_T(s["T_init"], s["T_gm"])
            sc.rk4_T_forward(s["pos"], s["T_gm"], s["u_adv"], s["dt"])
            sc.p2g3(s["init_imp"], s["pos"], s["T_gm"], s["T_init"], s["init_C"], s["u_out"], s["w_out"])
        return {k: s[k] for k in ("u_out", "w_out", "pos", "T_gm", "T_init", "init_C", "init_imp")}
    if kind == "midpoint3d":
        m = s["scene"].calc_max_speed_async(s["u"])
        s["scene"].midpoint(s["u"], s["u_mid"], s["dt_half"])
        return {"u_mid": s["u_mid"], "max_speed": m}
    if kind == "unet_predict":
        return {"p": s["net"].predict(s["div"], out=s["out"])}
    stats = s["net"].loss_and_grad(s["div"], s["p"])
    return {"loss": stats[:1], "grads": s["net"].grads}


# ------------------------------------------------------------------------------------------------
# compulsory work
# ------------------------------------------------------------------------------------------------
INTERP3 = 558  # 3 components x (9 rows x 6 + 9 x 3 + 3 x 4) FMAs: value and gradient of a 27-tap sample
INTERP2 = 90   # 2 components x (3 rows x 6 + 3 x 3) FMAs less the shared ones


def work(case):
    kind, res = case["kind"], _res(case)
    C = float(np.prod(res)) if res else 0.0
    if kind in ("solve2d", "solve3d"):
        d = len(res)
        # velocity read and written, pressure written; one V-cycle's stencils
        return {"bytes": C * 4 * (2 * d + 1), "flops": C * 60.0}
    if kind == "step2d":
        return _work_step2d(C)
    if kind == "batch2d":
        w = [_work_step2d(float(n * n)) for n in _batch_sizes(case)]
        return {"bytes": sum(x["bytes"] for x in w), "flops": sum(x["flops"] for x in w)}
    P = 8 * C
    if kind == "step3d":
        # pos, T_gm, T_init read and written, init_imp read, init_C written; velocity and pressure
        return {"bytes": P * (24 + 72 + 72 + 12 + 36) + C * (24 + 8),
                "flops": P * (5 * INTERP3 + 600) + 3 * C * 5 * INTERP3 + 2 * C * 60}
    if kind == "transport3d":
        return {"bytes": P * (24 + 72 + 72 + 12 + 36) + C * (24 + 24), "flops": P * (5 * INTERP3 + 600)}
    if kind == "midpoint3d":
        return {"bytes": C * 24, "flops": 3 * C * (5 * INTERP3)}
    # convolutions: 2 x 27 x cin x cout per voxel (the first layer has one input channel)
    f = 27 * 2 * (C * (1 * 16 + 16 * 16 + 48 * 16 + 16 * 16 + 16) + C / 8 * (16 * 32 + 32 * 32 + 96 * 32 + 32 * 32)
                  + C / 64 * (32 * 64 + 64 * 64))
    return {"bytes": C * 8, "flops": f if kind == "unet_predict" else 3 * f}


def _work_step2d(C):
    P = 4 * C
    # pos, T, T_gm read and written, T_init, init_C, init_imp, psi read, imp and C written
    return {"bytes": P * (16 + 32 + 32 + 16 + 16 + 8 + 8 + 8 + 16) + C * (16 + 8),
            "flops": P * (4 * INTERP2 + 150) + 2 * C * 5 * INTERP2 + 2 * C * 60}


# ------------------------------------------------------------------------------------------------
# the same outputs in 64-bit torch
# ------------------------------------------------------------------------------------------------
def exact(case, seed):
    kind = case["kind"]
    if kind in ("solve2d", "solve3d"):
        return _exact_solve(case, seed)
    if kind == "transport3d":
        return _exact_transport(case, seed)
    if kind == "midpoint3d":
        return _exact_midpoint(case, seed)
    if kind in ("unet_predict", "unet_grad"):
        return _exact_unet(case, seed)
    return None  # whole steps: their phases and solves are the other cases


def _dct(x, a, inverse):
    """DCT-II along axis a (or its inverse), f64, by the FFT of the even extension."""
    n = x.shape[a]
    x = x.movedim(a, -1)
    k = torch.arange(n, device=x.device, dtype=torch.float64)
    ph = torch.exp(-1j * math.pi * k / (2 * n))
    if not inverse:
        y = (torch.fft.fft(torch.cat([x, x.flip(-1)], -1), dim=-1)[..., :n] * ph).real * 0.5
    else:
        z = torch.zeros(x.shape[:-1] + (2 * n,), device=x.device, dtype=torch.complex128)
        z[..., :n] = x * ph.conj() * 2
        z[..., n + 1:] = z[..., 1:n].flip(-1).conj()
        y = torch.fft.ifft(z, dim=-1)[..., :n].real
    return y.movedim(-1, a)


def _exact_solve(case, seed):
    res = _res(case)
    _, s = prepare(case, seed)
    u = [a.double() for a in s["u0"]]
    del s
    for f, a in enumerate(u):
        a.select(f, 0).zero_()
        a.select(f, res[f]).zero_()
    div = sum(a.narrow(f, 1, res[f]) - a.narrow(f, 0, res[f]) for f, a in enumerate(u))
    b = div - div.mean()
    lam = torch.zeros(res, device="cuda", dtype=torch.float64)
    for a, n in enumerate(res):
        shape = [1] * len(res)
        shape[a] = n
        k = torch.arange(n, device="cuda", dtype=torch.float64)
        lam = lam + (2 * torch.cos(math.pi * k / n) - 2).view(shape)
        b = _dct(b, a, False)
    lam.view(-1)[0] = 1.0
    b /= lam
    b.view(-1)[0] = 0.0
    for a in range(len(res)):
        b = _dct(b, a, True)
    for f, a in enumerate(u):
        a.narrow(f, 1, res[f] - 1).sub_(b.narrow(f, 1, res[f] - 1) - b.narrow(f, 0, res[f] - 1))
    return {"u": u, "p": None}  # the all-Neumann pressure is defined up to a constant


def _taps(s, n=None):
    """Middle tap and the three N_2 weights and derivatives at s (grid units); clamped to [1, n - 2] with n."""
    if n is not None:
        s = s.clamp(1.0, n - 2 - 1e-6)
    m = torch.floor(s + 0.5)
    t = s - m
    w = (0.5 * (0.5 - t) ** 2, 0.75 - t * t, 0.5 * (0.5 + t) ** 2)
    d = (t - 0.5, -2 * t, t + 0.5)
    return m.long() - 1, w, d


def _interp(u, x, dx, grad=True):
    """Velocity and gradient G[c][r] at positions x [3, n], f64."""
    X = x / dx
    val, G = [], []
    for c in range(3):
        n = u[c].shape
        t = [_taps(X[a] - (0.0 if a == c else 0.5), n[a]) for a in range(3)]
        flat = u[c].reshape(-1)
        v = torch.zeros_like(X[0])
        g = [torch.zeros_like(v) for _ in range(3)]
        for i in range(3):
            for j in range(3):
                for k in range(3):
                    f = flat[((t[0][0] + i) * n[1] + t[1][0] + j) * n[2] + t[2][0] + k]
                    wx, wy, wz = t[0][1][i], t[1][1][j], t[2][1][k]
                    v += wx * wy * wz * f
                    if grad:
                        g[0] += t[0][2][i] * wy * wz * f
                        g[1] += wx * t[1][2][j] * wz * f
                        g[2] += wx * wy * t[2][2][k] * f
        val.append(v)
        G.append(torch.stack(g) / dx)
    return torch.stack(val), torch.stack(G) if grad else None


def _exact_transport(case, seed):
    res, dx = _res(case), _dx(case)
    _, s = prepare(case, seed)
    u, ua = [[a.double() for a in s[k]] for k in ("u", "u_adv")]
    seeds, dt = s["seeds"], s["dt"]
    del s
    P = seeds.shape[1]
    out = {k: [] for k in ("pos", "T_gm", "T_init", "init_C", "init_imp")}
    num = [torch.zeros(a.numel(), device="cuda", dtype=torch.float64) for a in u]
    den = [torch.zeros_like(a) for a in num]
    eye = torch.eye(3, device="cuda", dtype=torch.float64)[:, :, None]
    for c0 in range(0, P, 1 << 21):
        p0 = seeds[:, c0:c0 + (1 << 21)].double()
        n = p0.shape[1]
        imp, C = _interp(u, p0, dx)
        T0 = eye.expand(3, 3, n)
        # RK4 of x' = u, T_v' = -grad(u)^T T_v
        pk, Tk, su, sT = p0, T0, 0, 0
        for k in range(4):
            v, G = _interp(ua, pk, dx)
            dT = torch.einsum("crn,vcn->vrn", G, Tk)
            w = 1.0 if k in (0, 3) else 2.0
            su, sT = su + w * v, sT + w * dT
            if k < 3:
                h = 0.5 * dt if k < 2 else dt
                pk, Tk = p0 + h * v, T0 - h * dT
        pos, T = p0 + dt / 6 * su, T0 - dt / 6 * sT
        # P2G: m = T^T (T_init = I) imp, affine rows T^T C T, quadratic weights, APIC
        m = torch.einsum("arn,an->rn", T, imp)
        A = torch.einsum("arn,abn,bcn->rcn", T, C, T)
        X = pos / dx
        for f in range(3):
            shape = u[f].shape
            t = [_taps(X[a] - (0.0 if a == f else 0.5)) for a in range(3)]
            for i in range(3):
                for j in range(3):
                    for k in range(3):
                        e = [t[0][0] + i, t[1][0] + j, t[2][0] + k]
                        ok = torch.ones(n, device="cuda", dtype=torch.bool)
                        off = 0
                        for a in range(3):
                            ok &= (e[a] >= 0) & (e[a] < shape[a])
                            off = off + A[f, a] * ((e[a].double() + (0.0 if a == f else 0.5)) * dx - pos[a])
                        w = t[0][1][i] * t[1][1][j] * t[2][1][k]
                        idx = ((e[0] * shape[1] + e[1]) * shape[2] + e[2])[ok]
                        num[f].index_add_(0, idx, ((m[f] + off) * w)[ok])
                        den[f].index_add_(0, idx, w[ok])
        for k, v in (("pos", pos), ("T_gm", T), ("T_init", T0.expand(3, 3, n)), ("init_C", C), ("init_imp", imp)):
            out[k].append(v)
    out = {k: torch.cat(v, -1) for k, v in out.items()}
    out["u_out"] = [torch.where(d > 0, a / d.clamp_min(1e-300), a).view(g.shape) for a, d, g in zip(num, den, u)]
    out["w_out"] = [d.view(g.shape) for d, g in zip(den, u)]
    return out


def _exact_midpoint(case, seed):
    res, dx = _res(case), _dx(case)
    _, s = prepare(case, seed)
    u = [a.double() for a in s["u"]]
    dt = -float(np.float32(s["dt_half"]))
    del s
    speed2 = sum((0.5 * (a.narrow(f, 1, res[f]) + a.narrow(f, 0, res[f]))) ** 2 for f, a in enumerate(u))
    out = []
    for f in range(3):
        nf = u[f].shape
        total = u[f].numel()
        got = torch.empty(total, device="cuda", dtype=torch.float64)
        for c0 in range(0, total, 1 << 21):
            e = torch.arange(c0, min(total, c0 + (1 << 21)), device="cuda")
            idx = [e // (nf[1] * nf[2]), e // nf[2] % nf[1], e % nf[2]]
            p0 = torch.stack([(idx[a].double() + (0.0 if a == f else 0.5)) * dx for a in range(3)])
            T0 = torch.zeros_like(p0)
            T0[f] = 1.0
            pk, Tk, su, sT = p0, T0, 0, 0
            for k in range(4):
                v, G = _interp(u, pk, dx)
                dT = torch.einsum("crn,rn->cn", G, Tk)
                w = 1.0 if k in (0, 3) else 2.0
                su, sT = su + w * v, sT + w * dT
                if k < 3:
                    h = 0.5 * dt if k < 2 else dt
                    pk, Tk = p0 + h * v, T0 + h * dT
            ua, _ = _interp(u, p0 + dt / 6 * su, dx, grad=False)
            got[c0:c0 + e.numel()] = ((T0 + dt / 6 * sT) * ua).sum(0)
        out.append(got.view(nf))
    return {"u_mid": out, "max_speed": speed2.max().sqrt().view(1)}


def _exact_unet(case, seed):
    res = _res(case)
    if case["kind"] == "unet_predict" and np.prod(res) > 2 ** 21 or np.prod(res) > 2 ** 20:
        return None  # too long in 64 bits
    _, s = prepare(case, seed)
    F = torch.nn.functional
    net, div, p = s["net"], s["div"].double(), s["p"].double()
    flat = net.params.double().requires_grad_(case["kind"] == "unet_grad")
    W, off = {}, 0
    for name, cin, cout in (("enc0a", 16, 16), ("enc0b", 16, 16), ("enc1a", 16, 32), ("enc1b", 32, 32),
                            ("bot_a", 32, 64), ("bot_b", 64, 64), ("dec1a", 96, 32), ("dec1b", 32, 32),
                            ("dec0a", 48, 16), ("dec0b", 16, 16), ("out", 16, 1)):
        w = flat[off:off + cout * cin * 27].view(cout, cin, 3, 3, 3)
        off += cout * cin * 27
        W[name] = (w, flat[off:off + cout])
        off += cout
    conv = lambda n, x, relu=True: (F.relu if relu else (lambda y: y))(F.conv3d(x, *W[n], padding=1))  # noqa: E731
    up = lambda x: F.interpolate(x, scale_factor=2, mode="nearest")  # noqa: E731
    rms = div.square().mean().sqrt()
    x = torch.zeros((1, 16) + res, device="cuda", dtype=torch.float64)
    x[0, 0] = div / rms
    e0 = conv("enc0b", conv("enc0a", x))
    e1 = conv("enc1b", conv("enc1a", F.avg_pool3d(e0, 2)))
    b = conv("bot_b", conv("bot_a", F.avg_pool3d(e1, 2)))
    d1 = conv("dec1b", conv("dec1a", torch.cat([e1, up(b)], 1)))
    d0 = conv("dec0b", conv("dec0a", torch.cat([e0, up(d1)], 1)))
    y = conv("out", d0, False)[0, 0]
    if case["kind"] == "unet_predict":
        return {"p": y.detach() * rms}
    e = y - p / rms
    loss = e.square().mean() - e.mean() ** 2
    loss.backward()
    return {"loss": loss.detach().view(1), "grads": flat.grad}
