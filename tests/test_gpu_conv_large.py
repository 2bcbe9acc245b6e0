"""Warm-start convolutions on single slices with more voxels than 32-bit offsets reach, in their last rows,
against the float64 oracle of those rows."""

import numpy as np
import pytest

from _fixtures import pkg
from oracle import conv as oconv

pytestmark = pytest.mark.gpu


def _torch(gigabytes):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    if torch.cuda.mem_get_info()[0] < gigabytes << 30:
        pytest.skip(f"needs {gigabytes} GB of device memory")
    return torch


def _rnd(rng, *shape):
    """Random values that bf16 holds exactly."""
    return (rng.integers(-64, 65, shape) / 64.0).astype(np.float32)


@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
def test_forward_of_a_large_slice(dtype):
    torch = _torch(24)
    ws = pkg("warmstart")
    n = 16400                                                   # n * n > 2^31 / 8
    rng = np.random.default_rng(1)
    x = torch.zeros((1, 1, n, n, 2), dtype=getattr(torch, dtype), device="cuda")
    tail, w = _rnd(rng, 1, 1, 12, 20, 2), _rnd(rng, 8, 27, 2)
    x[:, :, -12:, -20:] = torch.from_numpy(tail).cuda().to(x.dtype)
    packed = ws.pack_weights(torch.from_numpy(w).cuda(), 2, 8)
    y = ws.conv3d_fwd_packed(x, packed, 8)
    ref = oconv.conv3d(np.pad(tail, ((0, 0), (0, 0), (1, 0), (1, 0), (0, 0))), w)
    # 54 products of multiples of 2^-12 below 4: exact sums
    assert np.array_equal(y[:, :, -13:, -21:].cpu().numpy(), ref.astype(np.float32))
    assert int(torch.count_nonzero(y)) == int(np.count_nonzero(ref))
    del x, y
    torch.cuda.empty_cache()


def test_weight_gradient_of_a_large_slice():
    torch = _torch(72)
    ws = pkg("warmstart")
    n = 46400                                                   # n * n > 2^31
    rng = np.random.default_rng(2)
    x = torch.zeros((1, 1, n, n, 2), dtype=torch.bfloat16, device="cuda")
    gy = torch.zeros((1, 1, n, n, 8), dtype=torch.bfloat16, device="cuda")
    xt, gt = _rnd(rng, 1, 1, 12, 20, 2), _rnd(rng, 1, 1, 12, 20, 8)
    x[:, :, -12:, -20:] = torch.from_numpy(xt).cuda().bfloat16()
    gy[:, :, -12:, -20:] = torch.from_numpy(gt).cuda().bfloat16()
    dw = ws.conv3d_wgrad_bf16(x, gy).cpu().numpy()
    assert np.array_equal(dw, oconv.conv3d_wgrad(xt, gt).astype(np.float32))
    del x, gy
    torch.cuda.empty_cache()
