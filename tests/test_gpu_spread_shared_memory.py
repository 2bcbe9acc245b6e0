"""Gridding of 82 to 96 columns, around the column counts from which a block's values and weights together
pass 48 KB of shared memory; against the oracle."""

import numpy as np
import pytest

from _fixtures import pkg
from oracle import nufft as onf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ncoil,necho", [(41, 2), (85, 1), (43, 2), (29, 3), (11, 8), (15, 6), (31, 3), (47, 2), (95, 1)])
def test_column_counts_match_oracle(ncoil, necho):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    rng = np.random.default_rng(ncoil * 100 + necho)
    shape, M = (12, 16, 20), 301
    k = np.stack([rng.uniform(-n / 2, n / 2, M) for n in shape], -1).astype(np.float32)
    dcf = rng.uniform(0.1, 1.0, M).astype(np.float32)
    cplx = lambda *s: (rng.standard_normal(s) + 1j * rng.standard_normal(s)).astype(np.complex64)
    maps, ksp = cplx(ncoil, *shape), cplx(necho * ncoil, M)
    be = pkg("nufft_backend").B200NufftBackend(shape, [k], 0, dcf=[dcf], n_coils=ncoil, n_echoes=necho)
    be.set_maps(torch.from_numpy(maps))
    a = be.adjoint_bin(be.sort_kspace(torch.from_numpy(ksp), 0), 0).cpu().numpy()
    be.close()
    ao = np.stack([sum(np.conj(maps[c]) * onf.nufft_adjoint(ksp[e * ncoil + c] * dcf, k, shape) for c in range(ncoil))
                   for e in range(necho)])
    assert onf.rel_l2(a, ao) < 1e-5                            # float32 sums; about 1e-6 at other sizes
