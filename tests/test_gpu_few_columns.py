"""Interpolation and gridding with few k-space columns (1-8: kernels of their own, 9: the general
ones) against the oracle: partial tiles, wrapped and integer coordinates, split lists."""

import numpy as np
import pytest

from _fixtures import pkg
from oracle import nufft as onf

pytestmark = pytest.mark.gpu


def _setup(ncoil, necho, seed, shape=(20, 28, 36), M=2600):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    rng = np.random.default_rng(seed)
    k = np.stack([rng.uniform(-n / 2, n / 2, M) for n in shape], -1).astype(np.float32)
    k[:700] *= 0.02                                            # lists longer than one work item
    k[700] = 0.0                                               # five taps per axis
    k[701] = [-shape[0] / 2, -shape[1] / 2, -shape[2] / 2]     # wraps
    k[702] = [1.0, -2.25, 3.0]                                 # five taps along z and x only
    dcf = rng.uniform(0.1, 1.0, M).astype(np.float32)
    cplx = lambda *s: (rng.standard_normal(s) + 1j * rng.standard_normal(s)).astype(np.complex64)
    maps = cplx(ncoil, *shape)
    be = pkg("nufft_backend").B200NufftBackend(shape, [k], 0, dcf=[dcf], n_coils=ncoil, n_echoes=necho)
    be.set_maps(torch.from_numpy(maps))
    return torch, be, k, dcf, maps, cplx(necho, *shape), cplx(necho * ncoil, M)


@pytest.mark.parametrize("ncoil,necho", [(1, 1), (2, 1), (1, 3), (4, 1), (5, 1), (3, 2), (7, 1), (2, 4), (3, 3)])
def test_batched_bin_matches_oracle(ncoil, necho):
    torch, be, k, dcf, maps, img, ksp = _setup(ncoil, necho, ncoil * 10 + necho)
    y = be.unsort_kspace(be.forward_bin(torch.from_numpy(img).cuda(), 0), 0).cpu().numpy()
    yo = np.stack([onf.nufft(img[e] * maps[c], k) for e in range(necho) for c in range(ncoil)])
    assert onf.rel_l2(y, yo) < 1e-5                            # float32 sums; about 1e-6 at other sizes
    v = be.sort_kspace(torch.from_numpy(ksp), 0)
    a = be.adjoint_bin(v, 0)
    ao = np.stack([sum(np.conj(maps[c]) * onf.nufft_adjoint(ksp[e * ncoil + c] * dcf, k, be.img_shape)
                       for c in range(ncoil)) for e in range(necho)])
    assert onf.rel_l2(a.cpu().numpy(), ao) < 1e-5
    assert torch.equal(a, be.adjoint_bin(v, 0))                # list order: the same bits
    be.close()


@pytest.mark.parametrize("ncoil", [1, 2, 8])
def test_zero_weight_ignores_an_infinite_sample(ncoil):
    torch, be, k, dcf, maps, img, ksp = _setup(ncoil, 1, 5)
    be.close()
    dcf[11] = 0.0
    be = pkg("nufft_backend").B200NufftBackend(be.img_shape, [k], 0, dcf=[dcf], n_coils=ncoil)
    be.set_maps(torch.from_numpy(maps))
    good = be.adjoint_bin(be.sort_kspace(torch.from_numpy(ksp), 0), 0)
    ksp[:, 11] = np.inf
    bad = be.adjoint_bin(be.sort_kspace(torch.from_numpy(ksp), 0), 0)
    assert torch.equal(good, bad)
    be.close()


def test_drop_in_calls_take_samples_in_acquisition_order():
    torch, be, k, dcf, maps, img, ksp = _setup(1, 1, 9)
    y = be.forward(torch.from_numpy(img[0]).cuda(), 0).cpu().numpy()
    assert onf.rel_l2(y, onf.nufft(img[0], k)) < 1e-5
    a = be.adjoint(torch.from_numpy(ksp[0]).cuda(), 0).cpu().numpy()
    assert onf.rel_l2(a, onf.nufft_adjoint(ksp[0], k, be.img_shape)) < 1e-5
    be.close()
