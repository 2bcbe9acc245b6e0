"""Adjoint x pass of one image at long lengths: coil counts that fill a tile of 16 columns, leave some idle or take
several, few rows (a row a tile), with and without maps, against the oracle; many rows (whole tiles over several
rows, a tail of rows) against the kernel of several images."""

import numpy as np
import pytest

from _fixtures import pkg
from oracle import nufft as onf

pytestmark = pytest.mark.gpu


def _adjoint(shape, coils):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    rng = np.random.default_rng(coils + shape[2])
    M = 150
    k = np.stack([rng.uniform(-n / 2, n / 2, M) for n in shape], -1).astype(np.float32)
    cplx = lambda *s: (rng.standard_normal(s) + 1j * rng.standard_normal(s)).astype(np.complex64)
    maps, ksp = cplx(coils, *shape), cplx(coils, M)
    be = pkg("nufft_backend").B200NufftBackend(shape, [k], 0, n_coils=coils, n_echoes=1, tma=False)
    be.set_maps(torch.from_numpy(maps))
    a = be.adjoint_bin(be.sort_kspace(torch.from_numpy(ksp), 0), 0, use_dcf=False).cpu().numpy()[0]
    single = be.adjoint(ksp[0], 0)
    be.close()
    parts = [onf.nufft_adjoint(ksp[c], k, shape) for c in range(coils)]
    # float32 transforms and sums: about 1e-6
    assert onf.rel_l2(a, sum(np.conj(maps[c]) * parts[c] for c in range(coils))) < 1e-5
    assert onf.rel_l2(single, parts[0]) < 1e-5


@pytest.mark.parametrize("x", [192, 196, 224, 240, 256])
@pytest.mark.parametrize("coils", [1, 3, 6, 9, 16, 17, 20])
def test_few_rows(x, coils):
    _adjoint((12, 16, x), coils)


@pytest.mark.parametrize("rows,coils", [((78, 67), 6), ((89, 108), 9), ((78, 67), 10), ((89, 108), 11)])
def test_rows_that_fill_tiles(rows, coils):
    """Against the same image as the first of two, which the kernel of several images takes (one row a tile)."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    rng = np.random.default_rng(coils)
    shape, M = rows + (192,), 400
    k = np.stack([rng.uniform(-n / 2, n / 2, M) for n in shape], -1).astype(np.float32)
    maps = torch.randn((coils,) + shape, dtype=torch.complex64, device="cuda")
    ksp = torch.randn((2 * coils, M), dtype=torch.complex64, device="cuda")
    images = []
    for echoes in (1, 2):
        be = pkg("nufft_backend").B200NufftBackend(shape, [k], 0, n_coils=coils, n_echoes=echoes, tma=False)
        be.set_maps(maps)
        images.append(be.adjoint_bin(be.sort_kspace(ksp[:echoes * coils], 0), 0, use_dcf=False)[0])
        be.close()
    # the same transforms; sums of at most 11 coils in another order, and gridding of other column counts
    assert float((images[0] - images[1]).norm() / images[1].norm()) < 1e-6
