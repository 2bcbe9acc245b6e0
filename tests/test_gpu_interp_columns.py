"""Interpolation lanes: pairs of columns where the count is even, single ones where it is odd, one to
eight pieces a lane, last lanes partly past the end; few columns with many samples; against the oracle."""

import numpy as np
import pytest

from _fixtures import pkg
from oracle import nufft as onf

pytestmark = pytest.mark.gpu


# one to eight pieces a lane, as far as few samples reach them
@pytest.mark.parametrize("ncoil,necho", [(3, 3), (5, 2), (7, 2), (6, 2), (5, 3), (19, 1), (11, 6), (13, 10), (11, 9),
                                         (25, 5), (30, 8), (31, 7)])
def test_column_counts_match_oracle(ncoil, necho):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    rng = np.random.default_rng(ncoil * 100 + necho)
    shape, M = (16, 20, 12), 301
    k = np.stack([rng.uniform(-n / 2, n / 2, M) for n in shape], -1).astype(np.float32)
    k[0] = 0.0                                                 # five taps per axis
    k[1] = [-shape[0] / 2, -shape[1] / 2, -shape[2] / 2]       # wraps
    cplx = lambda *s: (rng.standard_normal(s) + 1j * rng.standard_normal(s)).astype(np.complex64)
    maps, img = cplx(ncoil, *shape), cplx(necho, *shape)
    be = pkg("nufft_backend").B200NufftBackend(shape, [k], 0, n_coils=ncoil, n_echoes=necho)
    be.set_maps(torch.from_numpy(maps))
    y = be.unsort_kspace(be.forward_bin(torch.from_numpy(img).cuda(), 0), 0).cpu().numpy()
    be.close()
    yo = np.stack([onf.nufft(img[e] * maps[c], k) for e in range(necho) for c in range(ncoil)])
    assert onf.rel_l2(y, yo) < 1e-5                            # float32 sums; about 1e-6 at other sizes


# 1 to 8 columns: the largest bin of the row kernel and one sample more; 12 to 26: of one piece a lane; a sample's value does not
# depend on the others, so that the oracle takes the first 300 and the last 20
@pytest.mark.parametrize("ncol,limit", [(1, 65536), (2, 98304), (3, 65536), (4, 131072), (5, 49152), (6, 81920),
                                        (7, 20480), (8, 196608), (12, 50517), (15, 80827), (26, 23315)])
def test_few_columns_with_many_samples(ncol, limit):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    rng = np.random.default_rng(ncol)
    shape = (16, 20, 12)
    k = np.stack([rng.uniform(-n / 2, n / 2, limit + 1) for n in shape], -1).astype(np.float32)
    k[0] = 0.0
    cplx = lambda *s: (rng.standard_normal(s) + 1j * rng.standard_normal(s)).astype(np.complex64)
    maps, img = cplx(ncol, *shape), cplx(1, *shape)
    for M in (limit, limit + 1):
        at = np.r_[0:300, M - 20:M]
        be = pkg("nufft_backend").B200NufftBackend(shape, [k[:M]], 0, n_coils=ncol)
        be.set_maps(torch.from_numpy(maps))
        y = be.unsort_kspace(be.forward_bin(torch.from_numpy(img).cuda(), 0), 0).cpu().numpy()
        yo = np.stack([onf.nufft(img[0] * maps[c], k[at]) for c in range(ncol)])
        assert onf.rel_l2(y[:, at], yo) < 1e-5
        if ncol == 1:                                          # the drop-in call: acquisition order
            y1 = be.forward(torch.from_numpy(img[0]).cuda(), 0).cpu().numpy()
            assert onf.rel_l2(y1[at], onf.nufft(img[0], k[at])) < 1e-5
        be.close()
