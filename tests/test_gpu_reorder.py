"""K-space reordering between acquisition and tile order: column and sample tails, both directions."""

import numpy as np
import pytest

from _fixtures import pkg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("samples,ncol", [(1, 1), (63, 1), (64, 5), (65, 32), (700, 33), (129, 96), (2000, 12)])
def test_round_trip_and_rows(samples, ncol):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    rng = np.random.default_rng(samples + ncol)
    shape = (16, 20, 24)
    k = [np.stack([rng.uniform(-n / 2, n / 2, m) for n in shape], -1).astype(np.float32) for m in (40, samples)]
    be = pkg("nufft_backend").B200NufftBackend(shape, k, 0)
    ext = torch.randn((ncol, samples), dtype=torch.complex64, device="cuda")
    index = torch.arange(samples, device="cuda").to(torch.complex64)[None]
    order = be.sort_kspace(index, 1)[:, 0].real.long()         # acquisition index of each tile-ordered sample
    assert torch.equal(order.sort().values, torch.arange(samples, device="cuda"))
    inner = be.sort_kspace(ext, 1)
    assert torch.equal(inner, ext[:, order].T)
    assert torch.equal(be.unsort_kspace(inner, 1), ext)
    be.close()
