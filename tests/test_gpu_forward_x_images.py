"""Forward x pass of several images of one coil at long lengths: a row's images beside one another, tails of the last
block, images that do not divide its 16 columns; against the oracle."""

import numpy as np
import pytest

from _fixtures import pkg
from oracle import nufft as onf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("x", [192, 196, 224, 240, 256])
@pytest.mark.parametrize("images,zy", [(2, (12, 16)), (3, (12, 16)), (6, (14, 19)), (16, (12, 16)), (19, (14, 19))])
def test_matches_oracle(x, images, zy):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    rng = np.random.default_rng(x + images)
    shape, M = zy + (x,), 150
    k = np.stack([rng.uniform(-n / 2, n / 2, M) for n in shape], -1).astype(np.float32)
    cplx = lambda *s: (rng.standard_normal(s) + 1j * rng.standard_normal(s)).astype(np.complex64)
    maps, img = cplx(1, *shape), cplx(images, *shape)
    be = pkg("nufft_backend").B200NufftBackend(shape, [k], 0, n_coils=1, n_echoes=images)
    be.set_maps(torch.from_numpy(maps))
    y = be.unsort_kspace(be.forward_bin(torch.from_numpy(img).cuda(), 0), 0).cpu().numpy()
    be.close()
    for e in {0, images // 2, images - 1}:
        assert onf.rel_l2(y[e], onf.nufft(img[e] * maps[0], k)) < 1e-5           # float32 transforms: about 1e-6
