"""Warm-start convolutions on buffers that are only aligned to their element type: views at odd offsets
of a caller's allocation give the same bits as aligned ones."""

import ctypes

import pytest

from _fixtures import pkg

pytestmark = pytest.mark.gpu

SHAPE, CIN, COUT = (1, 5, 17, 9), 24, 40


def _torch():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _at(torch, t, offset):
    """A contiguous copy of t that starts `offset` elements into its allocation."""
    buf = torch.empty(t.numel() + offset + 8, dtype=t.dtype, device=t.device)
    v = buf[offset:offset + t.numel()].view(t.shape)
    v.copy_(t)
    return v


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


@pytest.mark.parametrize("offset", [1, 2, 3])
def test_forward_into_unaligned_output(offset):
    torch = _torch()
    ws, lib = pkg("warmstart"), pkg("_lib")
    x = torch.randn(SHAPE + (CIN,), device="cuda").bfloat16()
    w = torch.randn(COUT, 27, CIN, device="cuda").bfloat16()
    ref = ws.conv3d_fwd_bf16(x, w)
    packed = ws.pack_weights(w, CIN, COUT)
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    for call, weights in (("tr_conv3d_fwd", w), ("tr_conv3d_fwd_packed", packed)):
        buf = torch.full((ref.numel() + 8,), -7.0, device="cuda")
        y = buf[offset:offset + ref.numel()]
        assert y.data_ptr() % 16 == 4 * offset
        head = (_ptr(x),) if call == "tr_conv3d_fwd" else (_ptr(x), 0)
        lib.check(getattr(lib.load(), call)(*head, _ptr(weights), None, _ptr(y), *SHAPE, CIN, COUT, stream))
        assert torch.equal(y.view(ref.shape), ref)
        assert torch.all(buf[:offset] == -7.0) and torch.all(buf[offset + ref.numel():] == -7.0)


@pytest.mark.parametrize("cin,cout", [(24, 40), (18, 24)])
@pytest.mark.parametrize("offset", [1, 2, 3])
def test_inputs_at_odd_offsets(offset, cin, cout):
    torch = _torch()
    ws = pkg("warmstart")
    x = torch.randn(SHAPE + (cin,), device="cuda").bfloat16()
    gy = torch.randn(SHAPE + (cout,), device="cuda").bfloat16()
    w = torch.randn(cout, 27, cin, device="cuda").bfloat16()
    xo, go = _at(torch, x, offset), _at(torch, gy, offset)
    assert xo.data_ptr() % 16 == 2 * offset and xo.is_contiguous()
    dw = ws.conv3d_wgrad_bf16(x, gy)
    for a, b in ((xo, gy), (x, go), (xo, go)):
        assert torch.equal(ws.conv3d_wgrad_bf16(a, b), dw)
    assert torch.equal(ws.conv3d_fwd_bf16(xo, w), ws.conv3d_fwd_bf16(x, w))


@pytest.mark.parametrize("cin,cout", [(24, 40), (18, 24)])
def test_strided_weights(cin, cout):
    torch = _torch()
    ws = pkg("warmstart")
    w = torch.randn(cout, 27, cin, device="cuda").bfloat16()
    gy = torch.randn(SHAPE + (cout,), device="cuda").bfloat16()
    x = torch.randn(SHAPE + (cin,), device="cuda").bfloat16()
    views = [w.permute(2, 1, 0).contiguous().permute(2, 1, 0), w.repeat_interleave(2, dim=2)[:, :, ::2]]
    assert not any(v.is_contiguous() for v in views)
    for v in views + [w[:1].expand(cout, 27, cin)]:
        c = v.contiguous()
        assert torch.equal(ws.conv3d_dgrad_bf16(gy, v), ws.conv3d_dgrad_bf16(gy, c))
        assert torch.equal(ws.conv3d_fwd_bf16(x, v), ws.conv3d_fwd_bf16(x, c))


def test_weight_gradient_with_unaligned_scratch():
    torch = _torch()
    ws, lib = pkg("warmstart"), pkg("_lib")
    shape, cin, cout = (1, 300, 32, 32), 64, 64                 # several runs a thread block
    x = torch.randn(shape + (cin,), device="cuda").bfloat16()
    gy = torch.randn(shape + (cout,), device="cuda").bfloat16()
    ref = ws.conv3d_wgrad_bf16(x, gy)
    nbytes = ctypes.c_size_t(0)
    lib.check(lib.load().tr_conv3d_wgrad_workspace(*shape, cin, cout, ctypes.byref(nbytes)))
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    for offset in (0, 1, 2):
        scratch = torch.empty(nbytes.value // 4 + 8, device="cuda")[offset:]
        buf = torch.zeros(ref.numel() + 4, device="cuda")
        dw = buf[offset:offset + ref.numel()]
        lib.check(lib.load().tr_conv3d_wgrad(_ptr(x), _ptr(gy), _ptr(dw), *shape, cin, cout, _ptr(scratch),
                                             nbytes, stream))
        assert torch.equal(dw.view(ref.shape), ref)
