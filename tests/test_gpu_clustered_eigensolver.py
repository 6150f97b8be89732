"""Eigensolves with clusters of equal eigenvalues (the shells of a harmonic dot):
pairs inside a cluster are turned by any angle for an element of rounding size, and
must not bring back elements that the sweep has taken away."""
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


@pytest.mark.parametrize("size", [2, 3, 5])
@pytest.mark.parametrize("n", [4, 6, 18, 33, 63, 128, 260])
def test_clusters(capi, n, size):
    for seed in range(24 if n < 100 else 8):
        rng = np.random.default_rng([n, size, seed])
        X = np.linalg.qr(rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)))[0]
        lam = np.repeat(rng.uniform(0, 1, (n + size - 1) // size), size)[:n]
        M = (X * lam) @ X.conj().T
        M = 0.5 * (M + M.conj().T)
        ev, U = capi.hermitian_eigensolve(M)
        # the bounds of the solver without clusters, eigenvalues up to one
        assert np.max(np.abs(ev - np.sort(lam))) < 1e-13
        assert np.max(np.abs(U.conj().T @ U - np.eye(n))) < 2e-14
        assert np.max(np.abs(M @ U - U * ev[None, :])) < 1e-13
