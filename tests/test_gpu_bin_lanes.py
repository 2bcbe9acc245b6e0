"""PDHG with bins side by side (small workspaces): more bins than lanes, uneven and empty-ish bins,
two solvers on threads of their own, against the FP64 oracle."""

import threading

import numpy as np
import pytest

from _fixtures import pkg
from oracle import nufft as onf
from oracle import pdhg as op

pytestmark = pytest.mark.gpu


def _problem(bins, seed):
    rng = np.random.default_rng(seed)
    shape, C, E = (12, 16, 20), 2, 2
    counts = [1 + 37 * b * b for b in range(bins)]
    coords = [np.stack([rng.uniform(-n / 2, n / 2, m) for n in shape], -1).astype(np.float32) for m in counts]
    dcf = [rng.uniform(0.1, 1.0, m).astype(np.float32) for m in counts]
    cplx = lambda *s: (rng.standard_normal(s) + 1j * rng.standard_normal(s)).astype(np.complex64)
    mps = cplx(C, *shape)
    mps /= np.sqrt(np.sum(np.abs(mps) ** 2, axis=0))
    return shape, coords, dcf, mps, [cplx(E, C, m) for m in counts]


def _solve(problem):
    s = pkg("solver").PdhgSolver("tvme", *problem, lam_m=1e-3, lam_e=1e-3)
    image = s.run(max_iter=5, tol=0.0).image.cpu().numpy()
    again = s.run(max_iter=5, tol=0.0).image.cpu().numpy()
    s.close()
    assert np.array_equal(image, again)
    return image


@pytest.mark.parametrize("bins", [2, 9])
def test_bins_on_lanes_match_oracle(bins):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    p = _problem(bins, bins)
    shape, coords, dcf, mps, ksp = p
    ref = op.run("tvme", op.Problem(op.OracleNufft(shape, coords), [k.astype(np.complex128) for k in ksp], dcf, mps),
                 max_iter=5, tol=0.0, lam_m=1e-3, lam_e=1e-3)
    assert onf.rel_l2(_solve(p), ref.image) < 1e-5            # float32 iterations, about 1e-6


def test_two_solvers_on_two_threads():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    problems = [_problem(4, 11), _problem(5, 12)]
    alone = [_solve(p) for p in problems]
    got = [None, None]

    def work(i):
        got[i] = _solve(problems[i])
    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert all(np.array_equal(a, g) for a, g in zip(alone, got))
