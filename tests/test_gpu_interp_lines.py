"""Interpolation on both sides of the lines of its kernel choice: the largest bin of the row kernel and one sample
more, and the last bin of one piece a lane and one sample more; against the oracle for the first 300 samples and
the last 20 (a sample's value does not depend on the others)."""

import numpy as np
import pytest

from _fixtures import pkg
from oracle import nufft as onf

pytestmark = pytest.mark.gpu

WAVE = 148 * 2048


@pytest.mark.parametrize("ncol,line", [(2, 131072), (5, 196608 // 5), (6, 131072), (7, 196608 // 7), (8, 131072),
                                       (10, WAVE // 5), (14, WAVE // 7)])
def test_both_sides(ncol, line):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    rng = np.random.default_rng(ncol)
    shape = (16, 20, 12)
    maps = (rng.standard_normal((ncol,) + shape) + 1j * rng.standard_normal((ncol,) + shape)).astype(np.complex64)
    img = (rng.standard_normal((1,) + shape) + 1j * rng.standard_normal((1,) + shape)).astype(np.complex64)
    for M in (line, line + 1):
        k = np.stack([rng.uniform(-n / 2, n / 2, M) for n in shape], -1).astype(np.float32)
        be = pkg("nufft_backend").B200NufftBackend(shape, [k], 0, n_coils=ncol, n_echoes=1)
        be.set_maps(torch.from_numpy(maps))
        y = be.unsort_kspace(be.forward_bin(torch.from_numpy(img).cuda(), 0), 0).cpu().numpy()
        be.close()
        part = np.r_[0:300, M - 20:M]
        yo = np.stack([onf.nufft(img[0] * maps[c], k[part]) for c in range(ncol)])
        assert onf.rel_l2(y[:, part], yo) < 1e-5               # float32 sums; about 1e-6 at other sizes
