"""PDHG with bins side by side on lanes of the plan against the same bins one after another
(TR_PLAN_SERIAL_BINS): the same bits, for every algorithm, eagerly, by graph replay, in the split phases of a
sharded solve, and in a capture of the caller's with and without lanes that exist already."""

import ctypes

import numpy as np
import pytest

from _fixtures import pkg

pytestmark = pytest.mark.gpu

SHAPE, C = (24, 28, 32), 2                             # one db6 level
ALGORITHMS = [("tvm", False, 1), ("tvme", False, 3), ("tvme", True, 2), ("tvmw", False, 2)]


def _torch():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _solver(alg, l2, echoes, bins, lanes, graph=True, autotune=True):
    """The same random problem for every call with the same arguments; bins of uneven counts, one of a single sample."""
    rng = np.random.default_rng(100 * bins + echoes)
    counts = [1 + 61 * b * b % 997 for b in range(bins)]
    coords = [np.stack([rng.uniform(-n / 2, n / 2, m) for n in SHAPE], -1).astype(np.float32) for m in counts]
    dcf = [rng.uniform(0.1, 1.0, m).astype(np.float32) for m in counts]
    cplx = lambda *s: (rng.standard_normal(s) + 1j * rng.standard_normal(s)).astype(np.complex64)
    mps = cplx(C, *SHAPE)
    mps /= np.sqrt(np.sum(np.abs(mps) ** 2, axis=0))
    ksp = [cplx(echoes, C, m) for m in counts]
    be = pkg("nufft_backend").B200NufftBackend(SHAPE, coords, 0, dcf=dcf, n_coils=C, n_echoes=echoes,
                                               autotune=autotune, bin_lanes=lanes)
    return pkg("solver").PdhgSolver(alg, SHAPE, coords, dcf, mps, ksp, l2_coupling=l2, lam_m=1e-3, lam_e=1e-3,
                                    lam_w1=1e-3, lam_w2=1e-3, use_graph=graph, backend=be)


def _workspace(s):
    info, lib = pkg("_lib").PlanInfo(), pkg("_lib")
    lib.check(lib.load().tr_plan_info(s.backend.plan, ctypes.byref(info)))
    return int(info.workspace_bytes)


def _state(s):
    names = ("u", "u_bar", "p_m", "p_ex", "p_ey", "p_ez", "p_w1", "p_w2", "q")
    return {n: getattr(s, n).clone() for n in names if getattr(s, n) is not None}


def _same(torch, a, b):
    assert a.keys() == b.keys()
    for n in a:
        assert torch.equal(a[n], b[n]), n


@pytest.mark.parametrize("bins", [2, 5, 9])            # fewer bins than lanes, and more
@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("alg,l2,echoes", ALGORITHMS)
def test_solve(alg, l2, echoes, graph, bins):
    torch = _torch()
    got = []
    for lanes in (True, False):
        s = _solver(alg, l2, echoes, bins, lanes, graph)
        if alg == "tvmw":
            s.backend.wavelet_adjoint(s.p_w2)          # the wavelets' workspace
        before = _workspace(s)
        res = s.run(max_iter=6, tol=0.0)
        os_ = s.backend.os_shape
        one = 8 * echoes * C * (os_[0] + SHAPE[0]) * os_[1] * os_[2]           # one bin's workspace
        assert _workspace(s) - before == one * (min(bins, 8) if lanes else 1)
        got.append((_state(s), res.tols))
        s.close()
    _same(torch, got[0][0], got[1][0])
    assert got[0][1] == got[1][1]


@pytest.mark.parametrize("alg,l2,echoes", ALGORITHMS)
def test_split_phases(alg, l2, echoes):
    torch = _torch()
    got = []
    for lanes in (True, False):
        s = _solver(alg, l2, echoes, 5, lanes)
        e = pkg("parallel").B200ShardEngine(s, 0, 5)
        e.reset(None)
        sums = []
        for _ in range(4):
            e.phase1a(1 / 6, 1 / 6)
            e.phase1b(1 / 6, 1 / 6)
            sums.append(e.phase2(1 / 6, 1 / 6).clone())
        torch.cuda.synchronize()
        got.append({**_state(s), "sums": torch.stack(sums)})
        s.close()
    _same(torch, *got)


@pytest.mark.parametrize("made", [True, False])        # lanes exist before the capture, or cannot be made in it
@pytest.mark.parametrize("alg,l2,echoes", ALGORITHMS)
def test_phases_in_a_capture(alg, l2, echoes, made):
    torch = _torch()
    ref = _solver(alg, l2, echoes, 5, False)
    ref.run(max_iter=4, tol=0.0)
    s = _solver(alg, l2, echoes, 5, True, autotune=False)
    e = pkg("parallel").B200ShardEngine(s, 0, 5)
    if made:
        s.run(max_iter=1, tol=0.0)
    else:                                              # the workspaces of one bin, the wavelets and the sums only
        s.backend.adjoint_bin(s.backend.forward_bin(s.u_bar[0], 0), 0)
        if alg == "tvmw":
            s.backend.wavelet_adjoint(s.p_w2)
        e.phase2(1 / 6, 1 / 6)
    s.reset()
    torch.cuda.synchronize()
    lib = pkg("_lib")
    st, pr = s._state_struct(), s._params(1 / 6, 1 / 6)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s.stream):
        for phase in (1, 2):
            lib.check(lib.load().tr_pdhg_phase(s.backend.plan, ctypes.byref(st), ctypes.byref(pr), ctypes.byref(e.shard),
                                               phase, ctypes.c_void_p(e.sums.data_ptr()),
                                               ctypes.c_void_p(s.stream.cuda_stream)), "tr_pdhg_phase")
    for _ in range(4):
        graph.replay()
    torch.cuda.synchronize()
    _same(torch, _state(s), _state(ref))
    del graph
    s.close()
    ref.close()
