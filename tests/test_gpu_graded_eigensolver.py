"""Eigensolves of graded matrices D H D (H well conditioned, D over up to thirty
decades): states of very different norms. Every tangent of such a solve can be
tiny while elements are as large as the geometric mean of their diagonals."""
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


# one warp (2, 3, 4), one subproblem (8, 20), several blocks (33, 70)
@pytest.mark.parametrize("decades", [6, 9, 15, 30])
@pytest.mark.parametrize("n", [2, 3, 4, 8, 20, 33, 70])
def test_small_eigenvalues_to_their_own_size(capi, n, decades):
    for seed in range(4):
        rng = np.random.default_rng([n, decades, seed])
        X = np.linalg.qr(rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)))[0]
        H = (X * rng.uniform(0.5, 2, n)) @ X.conj().T
        H = 0.5 * (H + H.conj().T)
        D = 10.0 ** -np.linspace(0, decades, n)
        if seed % 2:
            D = rng.permutation(D)
        ev, U = capi.hermitian_eigensolve(D[:, None] * H * D[None, :])
        # W = U l^{-1/2} orthonormalises: D H D in the scale of H. The last sweep's
        # elements are below 3e-8 of their diagonals' mean and leave 1e-7 of that;
        # beside it the rounding of the products and of the matrix's entries
        Y = D[:, None] * U / np.sqrt(ev)[None, :]
        assert np.max(np.abs(Y.conj().T @ H @ Y - np.eye(n))) < 1e-13


@pytest.mark.parametrize("k", [2, 5, 40])
def test_states_of_different_norms(capi, k):
    n, dx = 32, 0.25
    rng = np.random.default_rng(k)
    psi = rng.standard_normal((k, n, n)) + 1j * rng.standard_normal((k, n, n))
    psi *= (10.0 ** -np.linspace(0, 12, k))[:, None, None]
    c = capi.Context(n, n, dx, k)
    c.upload(psi)
    c.orthonormalize()
    out = c.download().reshape(k, -1)
    c.close()
    assert np.max(np.abs(out.conj() @ out.T * dx * dx - np.eye(k))) < 1e-12
