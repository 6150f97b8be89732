"""Eigensolves of one to six indices (sweeps pair after pair up to four, of the
whole 32-index subproblem beyond) against LAPACK: close and equal eigenvalues,
diagonal matrices, elements far apart in size, and k states of a context."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def capi():
    import torch
    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for gpu tests")
    from itp2d_b200 import capi as C
    C.lib()
    return C


def _cases(n):
    rng = np.random.default_rng(n)
    X = np.linalg.qr(rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)))[0]
    for lam in (np.linspace(-1, 1, n), np.ones(n), 1 + 1e-9 * np.arange(n), 10.0 ** -np.arange(0, 2 * n, 2)):
        M = (X * lam) @ X.conj().T
        yield 0.5 * (M + M.conj().T)
    yield np.diag(np.arange(n, 0, -1)).astype(complex)
    D = 2.0 ** (-300.0 * np.arange(n) / max(1, n - 1))
    H = (X * np.linspace(1, 2, n)) @ X.conj().T
    yield D[:, None] * (0.5 * (H + H.conj().T)) * D[None, :]


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 6])
def test_matches_lapack(capi, n):
    for M in _cases(n):
        ev, U = capi.hermitian_eigensolve(M)
        ref = np.linalg.eigvalsh(M)
        # backward errors of a few roundings of the largest eigenvalue
        top = np.max(np.abs(ref))
        assert np.max(np.abs(ev - ref)) < 1e-14 * top
        assert np.max(np.abs(U.conj().T @ U - np.eye(n))) < 1e-14
        assert np.max(np.abs(M @ U - U * ev[None, :])) < 1e-14 * top


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("k", [2, 3, 4, 5])
def test_orthonormalises_few_states(capi, k, precision):
    n, dx = 32, 0.25
    rng = np.random.default_rng(k)
    psi = rng.standard_normal((k, n, n)) + 1j * rng.standard_normal((k, n, n))
    c = capi.Context(n, n, dx, k, precision=capi.FP64 if precision == "fp64" else capi.FP32)
    c.upload(psi)
    c.orthonormalize()
    out = c.download().reshape(k, -1)
    c.close()
    assert np.max(np.abs(out.conj() @ out.T * dx * dx - np.eye(k))) < (1e-13 if precision == "fp64" else 1e-4)
