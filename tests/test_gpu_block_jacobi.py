"""The block Jacobi eigensolver at the edges of its 32-index padding and block
pairs, against LAPACK: one subproblem (n <= 32), the first sizes with 2, 3 and 4
block pairs, and matrices whose off-diagonal elements leave the range in which
the rotation angles come from single precision."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps


@pytest.fixture(scope="module")
def capi():
    import torch
    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for gpu tests")
    from itp2d_b200 import capi as C
    C.lib()
    return C


def _overlap_like(n, seed):
    """Eigenvalues exp(-0.1 E) over three decades with near-degenerate pairs."""
    rng = np.random.default_rng(seed)
    E = np.sort(rng.uniform(1, 70, n))
    E[1::5] = E[0::5][: len(E[1::5])] + 1e-9
    X = np.linalg.qr(rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)))[0]
    M = (X * np.exp(-0.1 * E)[None, :]) @ X.conj().T
    return 0.5 * (M + M.conj().T)


# scale 1e-25 and 1e25: every rotation of the solve takes the double-precision set-up
@pytest.mark.parametrize("scale", [1.0, 1e-25, 1e25])
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 64, 65, 96, 129, 257])
def test_edges_match_lapack(capi, n, scale):
    M = _overlap_like(n, n) * scale
    ev, U = capi.hermitian_eigensolve(M)
    ref = np.linalg.eigvalsh(M)
    top = np.max(np.abs(ref))
    # the bounds of the solver at other sizes: eps-scale eigenvalues, rounding
    # of the accumulated rotations growing like sqrt(n) eps
    assert np.max(np.abs(ev - ref)) < 1e-13 * top
    assert np.max(np.abs(U.conj().T @ U - np.eye(n))) < max(2e-14, 1e-15 * math.sqrt(n))
    assert np.max(np.abs(M @ U - U * ev[None, :])) < 1e-13 * top


def test_indefinite_and_rank_deficient(capi):
    """A null space of dimension 20 and eigenvalues of both signs."""
    n = 70
    rng = np.random.default_rng(5)
    X = np.linalg.qr(rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)))[0]
    lam = np.concatenate([np.linspace(-2, -1, 25), np.zeros(20), np.linspace(0.5, 3, 25)])
    M = (X * lam[None, :]) @ X.conj().T
    M = 0.5 * (M + M.conj().T)
    ev, U = capi.hermitian_eigensolve(M)
    assert np.max(np.abs(ev - lam)) < 1e-13 * 3
    assert np.max(np.abs(U.conj().T @ U - np.eye(n))) < 2e-14
    assert np.max(np.abs(M @ U - U * ev[None, :])) < 1e-13 * 3


def test_tiny_coupling_is_resolved(capi):
    """A degenerate pair coupled by 1e-20: the exact eigenvectors mix it evenly
    when the coupling is above the rounding of the diagonal, and stay put when
    it is below (1e-15 of the diagonal); both leave M U = U diag(l)."""
    M = np.diag([1.0, 1.0, 2.0]).astype(complex)
    M[0, 1], M[1, 0] = 1e-20j, -1e-20j
    M[0, 2], M[2, 0] = 1e-3, 1e-3
    ev, U = capi.hermitian_eigensolve(M)
    ref = np.linalg.eigvalsh(M)
    assert np.max(np.abs(ev - ref)) < 8 * EPS
    assert np.max(np.abs(M @ U - U * ev[None, :])) < 8 * EPS


# first size on the single-precision solver, odd sizes, the last of a padding block
@pytest.mark.parametrize("k", [256, 257, 289, 352])
def test_single_precision_orthonormalisation(capi, k):
    n = 64
    rng = np.random.default_rng(k)
    dx = 0.2
    # overlap X diag(l) X^H with eigenvalues in [0.5, 1], one pair 1e-5 apart
    lam = np.linspace(0.5, 1.0, k)
    lam[1] = lam[0] + 1e-5
    X = np.linalg.qr(rng.standard_normal((k, k)) + 1j * rng.standard_normal((k, k)))[0]
    Y = np.linalg.qr(rng.standard_normal((n * n, k)) + 1j * rng.standard_normal((n * n, k)))[0]
    psi = ((Y * np.sqrt(lam)) @ X.conj().T).T.reshape(k, n, n) / dx
    c = capi.Context(n, n, dx, k, precision=capi.FP32)
    c.upload(psi)
    c.orthonormalize()
    out = c.download().reshape(k, -1)
    c.close()
    S = out.conj() @ out.T * dx * dx
    # an element of the overlap and of the rotation is good to about 1e-5; the
    # rotations left out after the last sweep are below 1e-6, over 0.5
    assert np.max(np.abs(S - np.eye(k))) < 1e-4
