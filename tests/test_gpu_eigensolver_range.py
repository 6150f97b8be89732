"""The eigensolver over the exponent range of double precision, against LAPACK on
the same matrix scaled by a power of two: elements whose squares underflow or
overflow, alone and beside a block of ordinary size."""
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


def _matrix(n, seed):
    """Eigenvalues 0.3 .. 1, random eigenvectors."""
    rng = np.random.default_rng([n, seed])
    X = np.linalg.qr(rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)))[0]
    M = (X * np.linspace(0.3, 1.0, n)) @ X.conj().T
    return 0.5 * (M + M.conj().T)


# one pair, one subproblem, several block pairs (odd and even), the first sizes
# above 256. 2^-500 and 2^500: products of two diagonals leave the range; 2^-560:
# squares of elements vanish; the last ones are near the ends of the range
@pytest.mark.parametrize("exponent", [-1000, -560, -500, 500, 560, 1000])
@pytest.mark.parametrize("n", [2, 3, 33, 129, 257])
def test_scaled_matrices(capi, n, exponent):
    M = _matrix(n, 1)
    ev, U = capi.hermitian_eigensolve(np.ldexp(M.real, exponent) + 1j * np.ldexp(M.imag, exponent))
    ev = np.ldexp(ev, -exponent)
    # the bounds of the solver at ordinary scale, top eigenvalue 1
    assert np.max(np.abs(ev - np.linalg.eigvalsh(M))) < 1e-13
    assert np.max(np.abs(U.conj().T @ U - np.eye(n))) < 2e-14
    assert np.max(np.abs(M @ U - U * ev[None, :])) < 1e-13


@pytest.mark.parametrize("n", [2, 40, 150])
def test_small_block_beside_an_ordinary_one(capi, n):
    """diag(A, 2^-560 B): each block's eigenvalues to its own scale."""
    A, B = _matrix(n, 2), _matrix(n, 3)
    M = np.zeros((2 * n, 2 * n), dtype=complex)
    M[:n, :n] = A
    M[n:, n:] = np.ldexp(B.real, -560) + 1j * np.ldexp(B.imag, -560)
    ev, U = capi.hermitian_eigensolve(M)
    assert np.max(np.abs(np.ldexp(ev[:n], 560) - np.linalg.eigvalsh(B))) < 1e-13
    assert np.max(np.abs(ev[n:] - np.linalg.eigvalsh(A))) < 1e-13
    assert np.max(np.abs(B @ U[n:, :n] - U[n:, :n] * np.ldexp(ev[:n], 560)[None, :])) < 1e-13


def test_orthonormalisation_of_decayed_states(capi):
    """States of norm 2^-285 (overlaps of 2^-570), as an imaginary time step under
    a large constant potential leaves them."""
    k, n, dx = 24, 32, 0.25
    rng = np.random.default_rng(4)
    psi = (rng.standard_normal((k, n, n)) + 1j * rng.standard_normal((k, n, n))) * 0.125 * 2.0 ** -285
    c = capi.Context(n, n, dx, k)
    c.upload(psi)
    c.orthonormalize()
    out = c.download().reshape(k, -1)
    c.close()
    assert np.max(np.abs(out.conj() @ out.T * dx * dx - np.eye(k))) < 1e-13


# null eigenvalues whose rounding would be subnormal, sums of products beside the
# largest number
@pytest.mark.parametrize("exponent", [-1000, -560, 560, 1015])
@pytest.mark.parametrize("n,rank", [(5, 3), (20, 7), (40, 20), (130, 50), (260, 100)])
def test_scaled_rank_deficient_matrices(capi, n, rank, exponent):
    rng = np.random.default_rng([n, rank])
    B = (rng.standard_normal((n, rank)) + 1j * rng.standard_normal((n, rank))) / np.sqrt(2 * n)
    M = B @ B.conj().T
    ev, U = capi.hermitian_eigensolve(np.ldexp(M.real, exponent) + 1j * np.ldexp(M.imag, exponent))
    ev = np.ldexp(ev, -exponent)
    top = np.max(np.abs(ev))
    assert np.max(np.abs(ev - np.linalg.eigvalsh(M))) < 1e-13 * top
    assert np.max(np.abs(U.conj().T @ U - np.eye(n))) < 2e-14
    assert np.max(np.abs(M @ U - U * ev[None, :])) < 1e-13 * top
