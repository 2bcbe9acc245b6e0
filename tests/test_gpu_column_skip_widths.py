"""Empty-column skip of the z passes at 240 and 320 points with column counts that are multiples of 8 but not
of the 16 lines of a block: the same bits as with every line transformed, and fewer bytes."""

import numpy as np
import pytest

from _fixtures import pkg

pytestmark = pytest.mark.gpu


# odd and even grid widths: a block's 16 lines lie in one to three (y, x) columns, across rows as well
@pytest.mark.parametrize("z,y,x", [(192, 20, 36), (192, 28, 24), (256, 20, 36), (256, 28, 24)])
@pytest.mark.parametrize("coils,echoes", [(8, 1), (8, 3), (10, 4)])
@pytest.mark.parametrize("tma", [True, False])
def test_same_bits(z, y, x, coils, echoes, tma):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    nb, shape = pkg("nufft_backend"), (z, y, x)
    rng = np.random.default_rng(z + x)
    # samples in a few (ky, kx) columns: most tile columns stay empty
    k = np.stack([rng.uniform(-z / 2, z / 2, 900)] + [rng.choice(rng.uniform(-n / 2.2, n / 2.2, 6), 900) for n in (y, x)],
                 -1).astype(np.float32)
    images = torch.randn((echoes,) + shape, dtype=torch.complex64, device="cuda")
    ksp = torch.randn((900, coils * echoes), dtype=torch.complex64, device="cuda")
    maps = torch.randn((coils,) + shape, dtype=torch.complex64, device="cuda")
    outs, moved = [], []
    for skip in (True, False):
        be = nb.B200NufftBackend(shape, [k], 0, n_coils=coils, n_echoes=echoes, column_skip=skip, tma=tma)
        be.set_maps(maps)
        prof = be.profile(0, reps=1)
        be.adjoint_bin(torch.full_like(ksp, float("nan")), 0)          # what unwritten tiles hold from an earlier call
        outs.append((be.forward_bin(images, 0), be.adjoint_bin(ksp, 0)))
        moved.append(prof["fwd_z"]["bytes"] + prof["adj_z"]["bytes"] + prof["spread"]["bytes"])
        be.close()
    assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])
    assert torch.isfinite(torch.view_as_real(outs[0][1])).all()
    assert moved[0] < 0.9 * moved[1]
