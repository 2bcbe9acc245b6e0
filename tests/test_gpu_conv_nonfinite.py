"""Weight gradient with an infinite or NaN activation: only the taps that pair it with a voxel of the volume
see it, also where tiles of 8 x 16 voxels reach past the volume; against float64."""

import pytest

from _fixtures import pkg
from test_gpu_conv_sums import _wgrad64

pytestmark = pytest.mark.gpu

# (N, D, H, W), Cin, Cout, place of the value (n, z, y, x): last column, last row, corner, their
# neighbours in other tiles, one tile wide and high, several runs and images, and whole tiles without tails
CASES = [((1, 5, 17, 9), 24, 40, (0, 2, 5, 8)), ((1, 5, 17, 9), 24, 40, (0, 4, 16, 3)),
         ((1, 5, 17, 9), 40, 24, (0, 0, 16, 8)), ((1, 5, 17, 9), 24, 40, (0, 2, 15, 8)),
         ((1, 5, 17, 9), 24, 40, (0, 2, 16, 7)), ((2, 3, 33, 12), 66, 72, (1, 1, 15, 11)),
         ((2, 3, 33, 12), 18, 8, (1, 1, 32, 7)), ((1, 3, 5, 3), 16, 16, (0, 1, 4, 1)),
         ((3, 40, 24, 20), 32, 64, (2, 39, 23, 19)), ((3, 40, 24, 20), 128, 128, (1, 17, 23, 8)),
         ((1, 2, 16, 16), 16, 16, (0, 1, 15, 15))]


@pytest.mark.parametrize("shape,cin,cout,at", CASES)
@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan")])
def test_one_value(shape, cin, cout, at, value):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    ws = pkg("warmstart")
    g = torch.Generator("cuda").manual_seed(cin)
    x = torch.rand(shape + (cin,), generator=g, device="cuda").bfloat16()
    gy = torch.rand(shape + (cout,), generator=g, device="cuda").bfloat16() + 1.0
    gy[..., ::2] *= -1.0                                        # no zero: products with the value are infinite
    ci = cin - 1
    x[at + (ci,)] = value
    dw = ws.conv3d_wgrad_bf16(x, gy).double()
    x[at + (ci,)] = 0.0
    rest = _wgrad64(torch, x, gy)
    # taps t with the voxel at - offset(t) inside the volume take value * gy there, the others nothing
    ref = rest.clone()
    for t in range(27):
        k = (at[0],) + tuple(a - d for a, d in zip(at[1:], (t // 9 - 1, t // 3 % 3 - 1, t % 3 - 1)))
        if all(0 <= i < n for i, n in zip(k, shape)):
            ref[:, t, ci] += value * gy[k].double()
    hit = ~torch.isfinite(ref)
    assert hit.any()
    assert torch.equal(torch.nan_to_num(dw[hit], nan=7.0, posinf=1.0, neginf=-1.0),
                       torch.nan_to_num(ref[hit], nan=7.0, posinf=1.0, neginf=-1.0))
    # every step of 16 products and every addition loses at most 2^-23 of the sum of magnitudes
    steps = 2.0 ** -23 * (128 + 64)
    assert torch.all((dw - rest).abs()[~hit] <= steps * _wgrad64(torch, x.abs(), gy.abs())[~hit])
