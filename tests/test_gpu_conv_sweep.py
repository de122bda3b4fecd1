"""The convolution's sweep along d0 at the sizes where its bookkeeping can go wrong, against the float64 oracle:
segments longer than the ring of accumulators (a plane's columns straddle the ring's end) with a shorter last
segment, weights streamed from L2 with two tiles per CTA and an odd count of tiles, three planes of more than 256
columns, and the largest channel counts (one stage for the streamed taps)."""
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
