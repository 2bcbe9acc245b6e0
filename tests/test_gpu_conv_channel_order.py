"""Order of the forward convolution's channel steps: a partial step of fewer than 16 input channels comes first, where
it rounds least.  The same channels padded with zeros to full steps put it last and must round more."""

import pytest

from _fixtures import pkg

pytestmark = pytest.mark.gpu


def _conv64(torch, x, w):
    N, D, H, W, C = x.shape
    xp = torch.zeros((N, D + 2, H + 2, W + 2, C), dtype=torch.float64, device=x.device)
    xp[:, 1:-1, 1:-1, 1:-1] = x.double()
    return sum(xp[:, t // 9:t // 9 + D, (t // 3) % 3:(t // 3) % 3 + H, t % 3:t % 3 + W] @ w[:, t].double().T
               for t in range(27))


@pytest.mark.parametrize("cin,cout", [(24, 48), (20, 16), (40, 24)])
def test_partial_step_first(cin, cout):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    ws = pkg("warmstart")
    pad = (-cin) % 16
    first = last = 0.0
    for seed in range(4):
        g = torch.Generator("cuda").manual_seed(seed)
        x = torch.randn((1, 12, 32, 32, cin), generator=g, device="cuda").relu_().bfloat16()
        w = torch.randn((cout, 27, cin), generator=g, device="cuda").bfloat16()
        ref = _conv64(torch, x, w)
        y = ws.conv3d_fwd_bf16(x, w)
        z = ws.conv3d_fwd_bf16(torch.nn.functional.pad(x, (0, pad)), torch.nn.functional.pad(w, (0, pad)))
        first += float((y - ref).norm() / ref.norm())
        last += float((z - ref).norm() / ref.norm())
    # steps lose a share of the partial sum: mean of sqrt(t) over the steps, small ones first against last
    assert first < 0.97 * last, (first / 4, last / 4)
