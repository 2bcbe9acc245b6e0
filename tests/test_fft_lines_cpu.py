"""Host check of the FFT line passes' radix plans and further register butterflies (no GPU).

``tests/native/line_plan_host.cu`` prints the plan of every compiled length and runs the
butterflies of radices 6, 9, 12, 14, 15, 18 and 21; a NumPy restatement of the pass indexing of
``lp_pass`` (in place, sixteen columns side by side are independent) must give the DFT.
"""

import math
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def printed(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        pytest.skip("nvcc not available")
    exe = tmp_path_factory.mktemp("plan") / "line_plan_host"
    subprocess.run([nvcc, "-std=c++17", "-x", "cu", "-Wno-deprecated-gpu-targets", "-I", str(ROOT / "include"),
                    "-I", str(ROOT / "multinodemri-miccai26_b200" / "csrc"), str(ROOT / "tests/native/line_plan_host.cu"),
                    "-o", str(exe)], check=True, capture_output=True)
    lines = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split("\n")
    plans, dfts, i = {}, {}, 0
    while i < len(lines) and lines[i]:
        f = lines[i].split()
        i += 1
        if f[0] == "L":
            plans[int(f[1])] = (int(f[2]), [int(v) for v in f[3:]])
        else:
            r, inv = int(f[1]), int(f[2])
            v = np.array([complex(*map(float, ln.split())) for ln in lines[i:i + 2 * r]])
            dfts[r, inv] = (v[:r], v[r:])
            i += 2 * r
    return plans, dfts


def _smooth(n):
    for r in (2, 3, 5, 7):
        while n % r == 0:
            n //= r
    return n == 1


def test_every_plan_length_up_to_320_is_compiled(printed):
    plans, _ = printed
    wanted = {math.ceil(1.25 * n) for n in range(10, 257)}
    assert set(plans) == {L for L in wanted if _smooth(L)}
    for L, (threads, radices) in plans.items():
        assert math.prod(radices) == L and 2 <= len(radices) <= 3
        assert threads % 32 == 0 and threads <= 416
        # a CTA's tile, twiddles and the adjoint x pass's maps fit its shared memory
        assert 8 * L * (2 * 16 + 1) <= 227 * 1024


def test_pass_indexing_gives_the_dft(printed):
    plans, _ = printed
    rng = np.random.default_rng(0)
    for L, (_, radices) in plans.items():
        x = rng.standard_normal(L) + 1j * rng.standard_normal(L)
        buf, Ns = x.copy(), 1
        for R in radices:
            nb, out, written = L // R, np.empty(L, complex), np.zeros(L, int)
            for j in range(nb):
                k = j % Ns
                v = buf[j + nb * np.arange(R)] * np.exp(-2j * np.pi * k * np.arange(R) / (Ns * R))
                at = (j // Ns) * Ns * R + k + Ns * np.arange(R)
                out[at] = np.fft.fft(v)
                written[at] += 1
            assert np.all(written == 1)
            buf, Ns = out, Ns * R
        assert np.allclose(buf, np.fft.fft(x), rtol=0, atol=1e-10 * L), L


@pytest.mark.parametrize("radix", (6, 9, 12, 14, 15, 18, 21))
@pytest.mark.parametrize("inv", (0, 1))
def test_register_butterflies(printed, radix, inv):
    x, y = printed[1][radix, inv]
    ref = np.fft.ifft(x) * radix if inv else np.fft.fft(x)
    # a handful of float32 roundings (6e-8 each) per output
    assert np.linalg.norm(y - ref) / np.linalg.norm(ref) < 5e-7
