"""The convolution's sweep along d0 and the weight gradient at the sizes where their bookkeeping can go wrong,
against the float64 oracle: segments longer than the ring of accumulators (a plane's columns straddle the ring's
end) with a shorter last segment, weights streamed from L2 with two tiles per CTA and an odd count of tiles, three
planes of more than 256 columns, and the largest channel counts (one stage for the streamed taps)."""
import ctypes

import numpy as np
import pytest
import torch

import nn_oracle as O

pytestmark = pytest.mark.gpu

SWEEPS = [  # c1, c2, cout, dims
    (16, 0, 16, (23, 250, 121)),
    (16, 32, 16, (19, 250, 121)),
    (64, 32, 32, (21, 136, 92)),
    (32, 0, 96, (11, 90, 70)),
    (128, 0, 128, (24, 100, 96)),
]


def blocked(x):
    t = torch.as_tensor(x).reshape(x.shape[0] // 8, 8, *x.shape[1:]).permute(0, 2, 3, 4, 1).contiguous()
    return t.to(torch.bfloat16).reshape(-1).cuda()


def ptr(t):
    return None if t is None else ctypes.c_void_p(t.data_ptr())


@pytest.mark.parametrize("c1,c2,cout,dims", SWEEPS)
def test_conv_sweep(c1, c2, cout, dims):
    from pfm import _lib
    lib = _lib.load()
    rng = np.random.default_rng(c1 + 3 * c2 + cout)
    cin = c1 + c2
    x = O.bf16(rng.standard_normal((cin,) + dims).astype(np.float32))
    W = O.bf16((rng.standard_normal((cout, cin, 27)) * 0.1).astype(np.float32))
    b = rng.standard_normal(cout).astype(np.float32)
    Wt, bias = torch.as_tensor(W, dtype=torch.float32).cuda().contiguous(), torch.as_tensor(b).cuda()
    wp = torch.empty(27 * cin * cout, dtype=torch.bfloat16, device="cuda")
    assert lib.pfm_nn_pack_weights(ptr(Wt), cout, cin, 0, cin, cout, ptr(wp), None) == 0
    x1, x2 = blocked(x[:c1]), blocked(x[c1:]) if c2 else None
    yf = torch.full((cout,) + dims, float("nan"), device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    a = _lib.Conv3Args(*dims, ptr(x1), c1, ptr(x2), c2, ptr(wp), ptr(bias), cout, 0, None, cout, None, ptr(yf), None,
                       ptr(err))
    assert lib.pfm_nn_conv3(ctypes.byref(a), None) == 0
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    got = yf.cpu().numpy()
    assert np.all(np.isfinite(got))
    # the first and the last rows of d1 against the oracle on slabs with their halo row
    for rows, keep in ((slice(0, 20), slice(0, 19)), (slice(dims[1] - 20, dims[1]), slice(1, 20))):
        xs = x[:, :, rows]
        ref, bound = O.conv3(xs, W, b)[:, :, keep], O.conv3(np.abs(xs), np.abs(W), np.abs(b))[:, :, keep]
        out = got[:, :, rows][:, :, keep]
        # 27 cin / 16 accumulations of 2^-23 each stay below 2.6e-5 of the absolute sum
        assert np.all(np.abs(out - ref) <= 1e-4 * bound + 1e-6), np.max(np.abs(out - ref) / (bound + 1e-6))


GRADS = [  # c1, c2, cout, cdy, dims
    (16, 0, 16, 16, (23, 250, 121)),   # two planes in M, a last odd plane, sums moved to the second accumulator
    (16, 32, 16, 16, (18, 130, 90)),   # three input groups, x1 and x2
    (32, 64, 32, 32, (11, 90, 70)),    # an input group across x1 and x2, no room for a second accumulator
    (16, 0, 5, 8, (9, 33, 20)),        # four planes in M, fewer real channels
    (16, 0, 24, 24, (6, 20, 12)),      # M rows that do not fill a tile
    (128, 0, 128, 128, (5, 24, 16)),   # three M tiles, most shared memory per stage
]


@pytest.mark.parametrize("c1,c2,cout,cdy,dims", GRADS)
def test_weight_gradient_groups(c1, c2, cout, cdy, dims):
    from pfm import _lib
    lib = _lib.load()
    rng = np.random.default_rng(7 + c1 + 3 * c2 + cout)
    cin = c1 + c2
    x = O.bf16(rng.standard_normal((cin,) + dims).astype(np.float32))
    dy = np.zeros((cdy,) + dims, np.float32)
    dy[:cout] = O.bf16(rng.standard_normal((cout,) + dims).astype(np.float32))
    x1, x2, dyt = blocked(x[:c1]), blocked(x[c1:]) if c2 else None, blocked(dy)
    dw = torch.full((cout, cin, 27), float("nan"), device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    a = _lib.Conv3WgradArgs(*dims, ptr(x1), c1, ptr(x2), c2, ptr(dyt), cdy, cout, ptr(dw), None, 0, ptr(err))
    nb = ctypes.c_size_t()
    assert lib.pfm_nn_wgrad_workspace(ctypes.byref(a), ctypes.byref(nb)) == 0
    part = torch.full((nb.value // 4 + 1,), float("nan"), device="cuda")
    a.partial, a.partial_bytes = ptr(part), nb.value - 1
    assert lib.pfm_nn_conv3_wgrad(ctypes.byref(a), None) == 3  # PFM_ERR_WORKSPACE
    a.partial_bytes = nb.value
    assert lib.pfm_nn_conv3_wgrad(ctypes.byref(a), None) == 0
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    ref, bound = O.conv3_wgrad(x, dy[:cout]), O.conv3_wgrad(np.abs(x), np.abs(dy[:cout]))
    db, scratch = torch.full((cout,), float("nan"), device="cuda"), torch.empty(296 * max(cdy, 2), device="cuda")
    dw2 = torch.full_like(dw, float("nan"))
    a.dw = ptr(dw2)
    assert lib.pfm_nn_conv3_wgrad_bias(ctypes.byref(a), ptr(db), ptr(scratch), None) == 0
    torch.cuda.synchronize()
    assert int(err.item()) == 0 and torch.equal(dw, dw2)
    flat = dy[:cout].reshape(cout, -1).astype(np.float64)
    # partial sums of a few hundred f32 additions each, compensated from there
    assert np.all(np.abs(db.cpu().numpy() - flat.sum(1)) <= 2e-5 * np.abs(flat).sum(1))
    # a sum of at most V / 16 / 45 + 48 truncated steps of 2^-23 each stays below 1e-4 of the absolute sum
    got = dw.cpu().numpy()
    assert np.all(np.abs(got - ref) <= 1e-4 * bound + 1e-6), np.nanmax(np.abs(got - ref) / (bound + 1e-6))
