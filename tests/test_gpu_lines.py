"""The register-FFT row, column and energy passes at every supported line length
and at their ragged edges (last tiles of fewer rows or columns, row lengths that
break the 128-byte alignment, one state), against numpy's FFT and the oracle."""
import os
import re

import numpy as np
import pytest

from oracle import itp_oracle as O

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
LENGTHS = [int(n) for n in re.findall(r"ITP2D_LINE\((\d+),", open(
    os.path.join(HERE, "..", "itp2d_b200", "csrc", "lines.cuh")).read())]
# relative to the largest element: rounding of a transform is about eps log2(N)
TOL = {"fp64": 2e-15 * 10, "fp32": 1.2e-7 * 20}


@pytest.fixture(scope="module")
def capi():
    import torch
    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for gpu tests")
    from itp2d_b200 import capi as C
    C.lib()
    return C


def _rel(a, b):
    return np.max(np.abs(a - b)) / np.max(np.abs(b))


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("n", LENGTHS)
def test_transforms_match_numpy(capi, n, precision):
    rng = np.random.default_rng(n)
    prec = capi.FP64 if precision == "fp64" else capi.FP32
    for sx, sy, k, kinds in [(n, 7, 3, ("FFTx", "iFFTx")), (21, n, 3, ("FFTy", "iFFTy"))]:
        psi = rng.standard_normal((k, sy, sx)) + 1j * rng.standard_normal((k, sy, sx))
        c = capi.Context(sx, sy, 0.1, k, precision=prec)
        for kind in kinds:
            c.upload(psi)
            c.transform(kind)
            assert _rel(c.download(), O.transform(psi, kind)) < TOL[precision], (sx, sy, kind)
        c.close()


# lengths with a beta item for every thread, with two per thread, with idle
# threads in the first stage, and lines that straddle warps; odd partner sizes
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("B", [0.0, 0.8])
@pytest.mark.parametrize("shape", [(36, 35), (35, 40), (96, 108), (192, 160), (200, 21), (21, 320), (384, 64),
                                   (32, 500), (512, 9), (9, 1024), (90, 100)])
def test_step_hamiltonian_and_energies_match_oracle(capi, shape, B, precision):
    sx, sy = shape
    g = O.Grid(sx, sy, 0.15)
    V = O.harmonic(g)
    for k in (1, 5):
        psi = O.gaussian_states(g, k, 3)
        c = capi.Context(sx, sy, g.dx, k, capi.PERIODIC, B, 2, capi.FP64 if precision == "fp64" else capi.FP32)
        c.set_potential(V)
        c.set_time_step(0.05)
        c.upload(psi)
        E, sigma, _, _ = c.energies()
        mean, sd = O.energies(O.Hamiltonian(g, V, O.PERIODIC, B), psi)
        c.propagate()
        step = c.download()
        c.upload(psi)
        c.apply_hamiltonian()
        h = c.download()
        c.close()
        # the bounds of the other sizes: 1e-12 FP64; 2e-5 and 2e-6 FP32
        tol, etol = (1e-12, 1e-12) if precision == "fp64" else (2e-5, 2e-6)
        assert _rel(step, O.MultiProductSplit(g, V, O.PERIODIC, B, 2, 0.05).apply(psi)) < tol
        assert _rel(h, O.Hamiltonian(g, V, O.PERIODIC, B).apply(psi)) < tol
        assert np.max(np.abs(E - mean.real)) < etol * np.max(np.abs(mean))
        assert np.max(np.abs(sigma - sd.real)) < etol * np.max(np.abs(sd))


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("n", LENGTHS)
def test_sine_transforms_match_oracle(capi, n, precision):
    rng = np.random.default_rng(n)
    prec = capi.FP64 if precision == "fp64" else capi.FP32
    for sx, sy, kinds in [(n, 7, ("DSTx", "iDSTx")), (21, n, ("DSTy", "iDSTy"))]:
        psi = rng.standard_normal((3, sy, sx)) + 1j * rng.standard_normal((3, sy, sx))
        c = capi.Context(sx, sy, 0.1, 3, capi.DIRICHLET, precision=prec)
        for kind in kinds:
            c.upload(psi)
            c.transform(kind)
            assert _rel(c.download(), O.transform(psi, kind)) < TOL[precision], (sx, sy, kind)
        c.close()


# even and odd factors (item A / 2 exists or not, N / 2 in item 0 or A / 2), both
# accumulating and in-place members
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("shape", [(64, 90), (90, 40), (150, 100), (36, 225), (240, 72), (512, 9)])
def test_dirichlet_step_matches_oracle(capi, shape, precision):
    sx, sy = shape
    g = O.Grid(sx, sy, 0.15)
    V = O.harmonic(g)
    for k, m in [(1, 1), (4, 3)]:
        psi = O.gaussian_states(g, k, 3)
        c = capi.Context(sx, sy, g.dx, k, capi.DIRICHLET, 0.0, m, capi.FP64 if precision == "fp64" else capi.FP32)
        c.set_potential(V)
        c.set_time_step(0.05)
        c.upload(psi)
        c.propagate()
        step = c.download()
        c.upload(psi)
        c.apply_hamiltonian()
        h = c.download()
        c.close()
        tol = 1e-12 if precision == "fp64" else 2e-5
        assert _rel(step, O.MultiProductSplit(g, V, O.DIRICHLET, 0.0, m, 0.05).apply(psi)) < tol
        assert _rel(h, O.Hamiltonian(g, V, O.DIRICHLET, 0.0).apply(psi)) < tol
