"""The bias gradient that the weight gradient's kernel sums beside it (csrc/pfm_nn.cu, k_conv3_wgrad)."""
import ctypes

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from pfm import _lib  # noqa: E402


def _gradients(dims, cin, cdy, dy):
    """(dw, db) of a zero input and the output gradient dy [cdy/8][d0][d1][d2][8] (bf16)."""
    lib = _lib.load()
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    x = torch.zeros(cin * dims[0] * dims[1] * dims[2], dtype=torch.bfloat16, device="cuda")
    dw, db = torch.zeros(cdy, cin, 27, device="cuda"), torch.zeros(cdy, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    a = _lib.Conv3WgradArgs(*dims, p(x), cin, None, 0, p(dy), cdy, cdy, p(dw), None, 0, p(err))
    nb = ctypes.c_size_t()
    assert lib.pfm_nn_wgrad_workspace(ctypes.byref(a), ctypes.byref(nb)) == 0
    part, scratch = torch.empty(nb.value // 4, device="cuda"), torch.empty(296 * cdy, device="cuda")
    a.partial, a.partial_bytes = p(part), nb.value
    assert lib.pfm_nn_conv3_wgrad_bias(ctypes.byref(a), p(db), p(scratch), None) == 0
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    return dw, db


# runs of many steps per CTA: of 16, 32 and 128 channels (rows per thread and step: 8, 8 and 32 at most)
@pytest.mark.parametrize("cdy,dims", [(16, (192, 192, 192)), (8, (192, 192, 96)), (32, (128, 192, 128)),
                                      (128, (64, 128, 64))])
def test_small_terms_beside_large_ones(cdy, dims):
    """One voxel in 512 is 1, the others 2^-25, half of what a plain f32 sum that has reached 1 still takes: a chain of
    n terms loses up to n 2^-25.  At most 32 terms are summed plainly, then compensated: 40 roundings of 2^-24 of the
    sum (the plain chain over a CTA's steps lost 7e-6 of it at 192^3)."""
    g = torch.Generator(device="cuda").manual_seed(cdy)
    dy = torch.full((cdy // 8, *dims, 8), 2.0 ** -25, dtype=torch.bfloat16, device="cuda")
    dy[torch.rand(dy.shape, device="cuda", generator=g) < 1 / 512] = 1.0
    want = dy.double().sum((1, 2, 3)).reshape(-1)
    _, db = _gradients(dims, 16, cdy, dy)
    assert ((db.double() - want).abs() <= 40 * 2.0 ** -24 * want).all(), ((db.double() - want) / want).abs().max()


@pytest.mark.parametrize("cdy", [16, 24])
def test_infinite_sums(cdy):
    """Gradients that overflow come out as the infinities of a plain f32 sum, in db (both of its paths) and in dW: an
    infinite term in channel 0, a sum beyond f32 in channel 1; the other channels keep their sums."""
    dims = (12, 40, 24)
    V = dims[0] * dims[1] * dims[2]
    dy = torch.zeros((cdy // 8, *dims, 8), dtype=torch.bfloat16, device="cuda")
    dy[0, 5, 7, 9, 0] = float("-inf")
    dy[0, ..., 1] = 3e38
    dy[0, ..., 2] = 0.5
    dw, db = _gradients(dims, 16, cdy, dy)
    assert db[0] == float("-inf") and db[1] == float("inf") and db[2] == 0.5 * V
    assert (dw[1:] == 0).all()
    # dW: the sum of 2 x 3e38 over the grid's inner voxels
    lib = _lib.load()
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    x = torch.full((2, *dims, 8), 2.0, dtype=torch.bfloat16, device="cuda")
    dy[0, 5, 7, 9, 0] = 0
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    a = _lib.Conv3WgradArgs(*dims, p(x), 16, None, 0, p(dy), cdy, cdy, p(dw), None, 0, p(err))
    nb = ctypes.c_size_t()
    assert lib.pfm_nn_wgrad_workspace(ctypes.byref(a), ctypes.byref(nb)) == 0
    part = torch.empty(nb.value // 4, device="cuda")
    a.partial, a.partial_bytes = p(part), nb.value
    assert lib.pfm_nn_conv3_wgrad(ctypes.byref(a), None) == 0
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    assert (dw[1] == float("inf")).all() and (dw[0] == 0).all() and torch.isfinite(dw[2]).all()
