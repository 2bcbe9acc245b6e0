"""NUFFT parity at every compiled FFT length, on each axis, for odd coil counts, several rows and
several column chunks per x-pass CTA (the kernels of tr_lines_part.cuh and the TMA kernels)."""

import math

import numpy as np
import pytest

from _fixtures import pkg
from oracle import nufft as onf

pytestmark = pytest.mark.gpu


def _smooth(n):
    for r in (2, 3, 5, 7):
        while n % r == 0:
            n //= r
    return n == 1


SIZES = [n for n in range(10, 257) if _smooth(math.ceil(1.25 * n))]
# coils, echoes: 1-5 columns (several rows per CTA), 16 exactly, 15 / 18 / 21 (a tail; images across chunks)
COLUMNS = [(1, 1), (5, 1), (16, 1), (5, 3), (18, 1), (7, 3), (3, 1), (8, 2), (20, 2), (12, 2), (4, 1)]


@pytest.mark.parametrize("index", range(len(SIZES)))
def test_each_length_on_each_axis(index):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    nb = pkg("nufft_backend")
    n = SIZES[index]
    rng = np.random.default_rng(n)
    for axis in range(3):
        shape = [12, 16, 14]
        shape[axis] = n
        shape = tuple(shape)
        C, E = COLUMNS[(3 * index + axis) % len(COLUMNS)]
        M = 600
        k = np.stack([rng.uniform(-s / 2, s / 2, M) for s in shape], -1).astype(np.float32)
        k[0] = 0.0
        cplx = lambda *s: (rng.standard_normal(s) + 1j * rng.standard_normal(s)).astype(np.complex64)
        img, maps, ksp = cplx(E, *shape), cplx(C, *shape), cplx(E * C, M)
        be = nb.B200NufftBackend(shape, [k], 0, n_coils=C, n_echoes=E)
        be.set_maps(torch.from_numpy(maps))
        y = be.unsort_kspace(be.forward_bin(torch.from_numpy(img).cuda(), 0), 0).cpu().numpy()
        a = be.adjoint_bin(be.sort_kspace(torch.from_numpy(ksp), 0), 0, use_dcf=False).cpu().numpy()
        a1 = be.adjoint(ksp[0], 0)
        be.close()
        # float32 transforms: about 1e-6; every column of the first and the last image
        for e in {0, E - 1}:
            yo = np.stack([onf.nufft(img[e] * maps[c], k) for c in range(C)])
            assert onf.rel_l2(y[e * C:(e + 1) * C], yo) < 1e-5, (shape, C, E)
            ao = sum(np.conj(maps[c]) * onf.nufft_adjoint(ksp[e * C + c], k, shape) for c in range(C))
            assert onf.rel_l2(a[e], ao) < 1e-5, (shape, C, E)
        assert onf.rel_l2(a1, onf.nufft_adjoint(ksp[0], k, shape)) < 1e-5, shape
