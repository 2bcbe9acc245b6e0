"""Rounding of the db6 synthesis: its error against 64 bits is no larger than with six (low, high) pairs added
in emulated float32, and so smaller than with twelve products added one after another from the first tap on."""

import numpy as np
import pytest

from _fixtures import pkg
from oracle import wavelets as ow

pytestmark = pytest.mark.gpu


def _fma(a, b, c):
    """Float32 fused multiply-add of (real) arrays."""
    return (a.astype(np.float64) * b.astype(np.float64) + c.astype(np.float64)).astype(np.float32)


def _synthesis(lo, hi, axis, n, mode):
    """n outputs along axis: y[o] = sum_j g_lo[2j + o%2] lo[i - j] + g_hi[2j + o%2] hi[i - j], i = o//2 + 5."""
    g_lo = ow.daubechies_rec_lo(6)
    g_hi = np.array([(-1.0) ** (12 - j) * g_lo[11 - j] for j in range(12)])
    real = np.float64 if mode == "exact" else np.float32
    pad = [(0, 0)] * lo.ndim
    pad[axis] = (0, 6)
    lo, hi = (np.moveaxis(np.pad(a.astype(real), pad), axis, 0) for a in (lo, hi))
    out = []
    for o in range(n):
        acc = np.zeros(lo.shape[1:], real)
        for j in range(6):
            i = o // 2 + 5 - j
            u, v, a, b = lo[i], hi[i], real(g_lo[2 * j + o % 2]), real(g_hi[2 * j + o % 2])
            if mode == "exact":
                acc = acc + a * u + b * v
            elif mode == "pairs":
                acc = acc + _fma(b, v, a * u)
            else:
                acc = _fma(b, v, _fma(a, u, acc))
        out.append(acc)
    return np.moveaxis(np.stack(out), 0, axis)


def _inverse(bands, shape, mode):
    """One level, along y, x, z in turn, of bands (2, 2, 2, Z, Y, X, real and imaginary part)."""
    a = _synthesis(bands[:, 0], bands[:, 1], 3, shape[1], mode)               # (bz, bx, Z, y, X, 2)
    a = _synthesis(a[:, 0], a[:, 1], 3, shape[2], mode)                       # (bz, Z, y, x, 2)
    return _synthesis(a[0], a[1], 0, shape[0], mode)


@pytest.mark.parametrize("shape", [(28, 25, 36), (24, 40, 32)])               # one level
def test_synthesis_rounds_no_more_than_pairs(shape):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    rng = np.random.default_rng(6)
    half = tuple((n + 11) // 2 for n in shape)
    bands = rng.standard_normal((2, 2, 2) + half + (2,)).astype(np.float32)
    be = pkg("nufft_backend").B200NufftBackend(shape, [np.zeros((1, 3), np.float32)], 0, n_coils=1, n_echoes=1)
    tree = torch.view_as_complex(torch.from_numpy(bands.reshape(1, -1, 2).copy())).cuda()
    assert tree.shape[1] == be.wavelet_coeffs
    got = torch.view_as_real(be.wavelet_adjoint(tree)).cpu().numpy().reshape(shape + (2,))
    be.close()
    exact = _inverse(bands, shape, "exact")
    err = lambda a: np.linalg.norm(a - exact) / np.linalg.norm(exact)
    pairs, chain = err(_inverse(bands, shape, "pairs")), err(_inverse(bands, shape, "chain"))
    assert pairs < chain
    assert err(got) < 0.5 * (pairs + chain), (err(got), pairs, chain)
