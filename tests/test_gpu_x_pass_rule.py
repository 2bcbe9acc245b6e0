"""x passes on both sides of the lines of their kernel choice (coil groups of 8 and 4, one to four images, the
lengths with TMA kernels) against the oracle and against a plan without TMA."""

import numpy as np
import pytest

from _fixtures import pkg
from oracle import nufft as onf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("x", [48, 64, 80, 96, 112, 128, 160, 192, 256])
@pytest.mark.parametrize("coils,images", [(8, 2), (8, 3), (4, 2), (4, 3), (12, 1), (12, 2), (20, 1)])
def test_matches_oracle(x, coils, images):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    rng = np.random.default_rng(x + coils)
    shape, M = (12, 16, x), 200
    k = np.stack([rng.uniform(-n / 2, n / 2, M) for n in shape], -1).astype(np.float32)
    cplx = lambda *s: (rng.standard_normal(s) + 1j * rng.standard_normal(s)).astype(np.complex64)
    img, maps, ksp = cplx(images, *shape), cplx(coils, *shape), cplx(images * coils, M)
    out = []
    for tma in (True, False):
        be = pkg("nufft_backend").B200NufftBackend(shape, [k], 0, n_coils=coils, n_echoes=images, tma=tma)
        be.set_maps(torch.from_numpy(maps))
        out.append((be.unsort_kspace(be.forward_bin(torch.from_numpy(img).cuda(), 0), 0).cpu().numpy(),
                    be.adjoint_bin(be.sort_kspace(torch.from_numpy(ksp), 0), 0, use_dcf=False).cpu().numpy()))
        be.close()
    # float32 transforms of the same values: about 1e-6
    assert onf.rel_l2(out[0][0], out[1][0]) < 1e-5 and onf.rel_l2(out[0][1], out[1][1]) < 1e-5
    e = images - 1
    for c in (0, coils - 1):
        assert onf.rel_l2(out[0][0][e * coils + c], onf.nufft(img[e] * maps[c], k)) < 1e-5
    ao = sum(np.conj(maps[c]) * onf.nufft_adjoint(ksp[e * coils + c], k, shape) for c in range(coils))
    assert onf.rel_l2(out[0][1][e], ao) < 1e-5
