"""Length of the weight gradient's tensor-core sums: sums of same-signed products, whose error adds up, over
voxel counts that give a thread block many times the 2,048 voxels of one sum; against float64."""

import pytest

from _fixtures import pkg

pytestmark = pytest.mark.gpu


def _wgrad64(torch, x, gy):
    N, D, H, W, C = x.shape
    xp = torch.zeros((N, D + 2, H + 2, W + 2, C), dtype=torch.float64, device=x.device)
    xp[:, 1:-1, 1:-1, 1:-1] = x.double()
    g = gy.double().reshape(-1, gy.shape[-1])
    taps = [xp[:, t // 9:t // 9 + D, (t // 3) % 3:(t // 3) % 3 + H, t % 3:t % 3 + W] for t in range(27)]
    return torch.stack([g.T @ s.reshape(-1, C) for s in taps], 1)


# whole tiles and tails; one and several units a run; volumes deeper than a run; two rounds of 13 slices
@pytest.mark.parametrize("shape,cin,cout", [((8, 32, 32, 32), 128, 128), ((8, 32, 32, 32), 64, 64),
                                            ((2, 40, 45, 77), 64, 128), ((8, 24, 24, 24), 128, 128),
                                            ((1, 96, 96, 96), 48, 24), ((64, 5, 16, 24), 128, 128),
                                            ((1, 300, 32, 32), 128, 64)])
def test_error_does_not_grow_with_the_volume(shape, cin, cout):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    ws = pkg("warmstart")
    g = torch.Generator("cuda").manual_seed(cin + cout)
    x = torch.rand(shape + (cin,), generator=g, device="cuda").bfloat16()
    gy = torch.rand(shape + (cout,), generator=g, device="cuda").bfloat16()
    dw, ref = ws.conv3d_wgrad_bf16(x, gy), _wgrad64(torch, x, gy)
    # a sum of 2,048 voxels takes 128 steps, each of which may drop 2^-23 of what is summed so far, half of
    # the sum on average; then at most 64 float32 additions of 2^-24 of partial sums, half of them on average
    bound = (64 * 2.0 ** -23 + 32 * 2.0 ** -24) * ref
    assert torch.all((dw.double() - ref).abs() <= bound), float(((dw.double() - ref).abs() / ref).max())
    assert torch.equal(dw, ws.conv3d_wgrad_bf16(x, gy))
