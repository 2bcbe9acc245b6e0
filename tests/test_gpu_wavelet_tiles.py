"""db6 analysis and synthesis at odd sizes, partial runs and tiles, one to three levels, against the oracle."""

import numpy as np
import pytest

from _fixtures import pkg
from oracle import nufft as onf
from oracle import wavelets as ow
from test_gpu_wavelet import _flatten, _unflatten

pytestmark = pytest.mark.gpu


# odd and even lines (single and double loads along z), several and partial runs, slices and row tiles
@pytest.mark.parametrize("shape", [(24, 25, 28), (25, 51, 57), (57, 67, 89), (100, 112, 89), (28, 36, 256)])
def test_odd_shapes_match_oracle(shape):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    rng = np.random.default_rng(sum(shape))
    be = pkg("nufft_backend").B200NufftBackend(shape, [np.zeros((1, 3), np.float32)] * 3, 0, n_coils=1, n_echoes=1)
    cplx = lambda *s: (rng.standard_normal(s) + 1j * rng.standard_normal(s)).astype(np.complex64)
    x, c = cplx(3, *shape), cplx(3, be.wavelet_coeffs)
    out = torch.full((3, be.wavelet_coeffs), float("nan"), dtype=torch.complex64, device="cuda")
    f = be.wavelet_forward(torch.from_numpy(x).cuda(), out=out).cpu().numpy()
    a = be.wavelet_adjoint(torch.from_numpy(c).cuda()).cpu().numpy().reshape((3,) + shape)
    for i in range(3):
        # twelve (six pairs of) float32 products per axis and level: a few 1e-7
        assert onf.rel_l2(f[i], _flatten(ow.wavedec3(x[i].astype(np.complex128), "db6"))) < 2e-6
        rec = ow.waverec3(_unflatten(c[i].astype(np.complex128), shape), "db6")
        assert onf.rel_l2(a[i], rec[tuple(slice(0, s) for s in shape)]) < 2e-6
    be.close()
