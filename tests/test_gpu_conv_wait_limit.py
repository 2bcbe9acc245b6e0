"""Convolution kernels whose bounded device waits run out: the call returns, the outputs carry the NaN mark, and
the next call at the default limit gives the same bits as ever."""

import threading

import pytest

from _fixtures import pkg

pytestmark = pytest.mark.gpu


# one tile; several tiles a block, two runs of weight-gradient sums; 128 channels on both sides
CASES = [((1, 4, 16, 8), 16, 16), ((1, 48, 96, 96), 64, 64), ((2, 20, 33, 40), 128, 128)]


@pytest.mark.parametrize("shape,cin,cout", CASES)
def test_waits_that_give_up_at_once(shape, cin, cout):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    ws, lib = pkg("warmstart"), pkg("_lib")
    set_limit = lambda n: lib.check(lib.load().tr_conv3d_set_wait_limit(n))
    g = torch.Generator("cuda").manual_seed(cin)
    x = torch.randn(shape + (cin,), generator=g, device="cuda")
    w = torch.randn((cout, 27, cin), generator=g, device="cuda")
    gy = torch.randn(shape + (cout,), generator=g, device="cuda").bfloat16()
    xb, packed = x.bfloat16(), ws.pack_weights(w, cin, cout)
    run = lambda: (ws.conv3d_fwd_packed(x, packed, cout), ws.conv3d_fwd_packed(xb, packed, cout),
                   ws.conv3d_wgrad_bf16(xb, gy))
    ref = run()
    assert all(torch.isfinite(t).all() for t in ref)
    try:
        set_limit(0)
        bad = run()
        torch.cuda.synchronize()
        other = []
        t = threading.Thread(target=lambda: other.extend(run()))       # the limit is the calling thread's
        t.start()
        t.join()
    finally:
        set_limit(lib.DEFAULT_WAIT_POLLS)
    assert all(torch.isnan(t).all() for t in bad)
    for again in (tuple(other), run()):
        assert all(torch.equal(a, b) for a, b in zip(again, ref))


def test_limit_is_checked():
    lib = pkg("_lib")
    with pytest.raises(ValueError):
        lib.check(lib.load().tr_conv3d_set_wait_limit(-1))
