"""Plans of different sizes on threads of their own: kernels whose shared memory depends on the level, the
column count or the coil count keep valid limits while another thread launches them with other sizes."""

import threading

import numpy as np
import pytest

from _fixtures import pkg

pytestmark = pytest.mark.gpu


def _torch():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _on_threads(torch, jobs):
    """Each job on a thread and stream of its own, all started together; their results."""
    out, errors, gate = [None] * len(jobs), [], threading.Barrier(len(jobs))

    def work(i):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                gate.wait()
                out[i] = jobs[i]()
                torch.cuda.current_stream().synchronize()
        except Exception as e:
            errors.append(e)
    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    return out


def test_wavelets_of_two_plans():
    torch = _torch()
    nb = pkg("nufft_backend")
    jobs, ref = [], []
    for n, shape in enumerate([(24, 28, 256), (48, 48, 224)]):             # one and two levels
        be = nb.B200NufftBackend(shape, [np.zeros((1, 3), np.float32)], 0, n_coils=1, n_echoes=1)
        x = torch.randn((1, 1) + shape, dtype=torch.complex64, device="cuda")
        tree = torch.randn((1, be.wavelet_coeffs), dtype=torch.complex64, device="cuda")
        ref.append((be.wavelet_forward(x), be.wavelet_adjoint(tree)))

        def job(be=be, x=x, tree=tree):
            f, a = torch.empty_like(tree), torch.empty_like(x)
            for _ in range(2000):
                be.wavelet_forward(x, out=f)
                be.wavelet_adjoint(tree, out=a)
            return f, a
        jobs.append(job)
    torch.cuda.synchronize()
    for got, want in zip(_on_threads(torch, jobs), ref):
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


def test_x_passes_of_two_plans():
    torch = _torch()
    nb = pkg("nufft_backend")
    rng = np.random.default_rng(3)
    jobs, ref = [], []
    for coils, echoes in ((1, 2), (3, 1)):                                 # 16 and 6 image rows a block
        shape = (12, 16, 252)
        k = np.stack([rng.uniform(-n / 2, n / 2, 500) for n in shape], -1).astype(np.float32)
        be = nb.B200NufftBackend(shape, [k], 0, n_coils=coils, n_echoes=echoes)
        be.set_maps(torch.randn((coils,) + shape, dtype=torch.complex64, device="cuda"))
        x = torch.randn((echoes,) + shape, dtype=torch.complex64, device="cuda")
        ref.append(be.forward_bin(x, 0))

        def job(be=be, x=x, out=torch.empty_like(ref[-1])):
            for _ in range(2000):
                be.forward_bin(x, 0, out=out)
            return out
        jobs.append(job)
    torch.cuda.synchronize()
    for got, want in zip(_on_threads(torch, jobs), ref):
        assert torch.equal(got, want)


def test_two_tvmw_solvers():
    torch = _torch()
    solver = pkg("solver")
    rng = np.random.default_rng(4)
    cplx = lambda *s: (rng.standard_normal(s) + 1j * rng.standard_normal(s)).astype(np.complex64)
    problems, alone = [], []
    for shape in ((24, 28, 256), (48, 48, 224)):
        coords = [np.stack([rng.uniform(-n / 2, n / 2, 300) for n in shape], -1).astype(np.float32) for _ in range(2)]
        mps = cplx(2, *shape)
        mps /= np.sqrt(np.sum(np.abs(mps) ** 2, axis=0))
        problems.append((shape, coords, [np.full(300, 0.5, np.float32)] * 2, mps, [cplx(2, 2, 300) for _ in coords]))

    def solve(p):
        s = solver.PdhgSolver("tvmw", *p)
        images = [s.run(max_iter=6, tol=0.0).image.cpu() for _ in range(6)]
        s.close()
        return images
    alone = [solve(p) for p in problems]
    got = _on_threads(torch, [lambda p=p: solve(p) for p in problems])
    for a, g in zip(alone, got):
        assert all(torch.equal(x, a[0]) for x in a + g)
