"""Warm-start convolution kernels at the edges of their tiles (8 x 16 voxels of one to four z slices,
16-channel steps, 64-channel weight-gradient chunks) against the float64 CPU oracle."""

import numpy as np
import pytest

from _fixtures import pkg
from oracle import conv as oconv

pytestmark = pytest.mark.gpu

# (N, D, H, W), Cin, Cout: one voxel; one tile and one voxel more per axis; tails of every channel step;
# several tiles per CTA (persistent walk), several voxel columns per weight-gradient CTA
CASES = [((1, 1, 1, 1), 2, 8), ((1, 4, 16, 8), 16, 16), ((1, 5, 17, 9), 18, 24), ((2, 3, 15, 7), 48, 40),
         ((1, 2, 33, 10), 66, 72), ((1, 9, 20, 12), 128, 128), ((3, 24, 40, 72), 8, 8), ((1, 3, 16, 16), 130, 56)]


def _problem(shape, cin, cout):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    rng = np.random.default_rng(cin * 131 + cout)
    rnd = lambda a: torch.from_numpy(a.astype(np.float32)).bfloat16().float().numpy()
    x, w = rnd(rng.standard_normal(shape + (cin,))), rnd(rng.standard_normal((cout, 27, cin)) * 0.2)
    return torch, x, w, rng.standard_normal(cout).astype(np.float32), rnd(rng.standard_normal(shape + (cout,)))


@pytest.mark.parametrize("shape,cin,cout", CASES)
def test_tile_edges(shape, cin, cout):
    torch, x, w, b, gy = _problem(shape, cin, cout)
    ws = pkg("warmstart")
    dev = lambda a: torch.from_numpy(a).cuda()
    xb, wb, gb = dev(x).bfloat16(), dev(w).bfloat16(), dev(gy).bfloat16()
    # products are exact and summed in float32: every 16-product step and the final adds lose at most
    # 2^-23 of the sum of magnitudes
    step = lambda k: (k / 16 + 20) * 2.0 ** -23
    y = ws.conv3d_fwd_bf16(xb, wb, dev(b))
    bound = step(27 * (cin + 16)) * (oconv.conv3d(np.abs(x), np.abs(w), np.abs(b)))
    assert np.all(np.abs(y.cpu().numpy() - oconv.conv3d(x, w, b)) <= bound)
    # float input rounds to the same bf16 operands: the same bits
    pk = ws.pack_weights(dev(w), cin, cout)
    assert torch.equal(ws.conv3d_fwd_packed(dev(x), pk, cout, dev(b)), y)
    if cin <= 128:
        dx = ws.conv3d_dgrad_bf16(gb, wb).cpu().numpy()
        bound = step(27 * (cout + 16)) * oconv.conv3d_dgrad(np.abs(gy), np.abs(w))
        assert dx.shape == shape + (cin,) and np.all(np.abs(dx - oconv.conv3d_dgrad(gy, w)) <= bound)
    else:                                  # the data gradient's output channels stay limited to 128
        with pytest.raises(ValueError):
            ws.conv3d_dgrad_bf16(gb, wb)
    dw = ws.conv3d_wgrad_bf16(xb, gb)
    bound = step(int(np.prod(shape)) + 4096) * oconv.conv3d_wgrad(np.abs(x), np.abs(gy))
    assert np.all(np.abs(dw.cpu().numpy() - oconv.conv3d_wgrad(x, gy)) <= bound)
    assert torch.equal(dw, ws.conv3d_wgrad_bf16(xb, gb))


def test_autograd_layer_without_gradients_gives_the_same_values():
    torch, x, w, b, _ = _problem((2, 5, 9, 11), 24, 16)
    ws = pkg("warmstart")
    t = [torch.from_numpy(a).cuda() for a in (x, w, b)]
    with torch.no_grad():
        y0 = ws.conv3d(*t)
    t[1].requires_grad_(True)
    y1 = ws.conv3d(*t)
    assert y1.requires_grad and torch.equal(y0, y1.detach())
    with torch.no_grad():
        assert torch.equal(ws.conv3d(*t), y0)
