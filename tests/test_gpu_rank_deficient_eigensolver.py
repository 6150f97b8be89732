"""Rank-deficient matrices: null eigenvalues at the rounding of the others. The
sweeps have to end on them (a solve that does not converge raises)."""
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


def _cases(n, rank):
    for seed in range(4):
        rng = np.random.default_rng([n, rank, seed])
        B = rng.standard_normal((n, rank)) + 1j * rng.standard_normal((n, rank))
        if seed == 1:
            B[n // 2:] = B[:n - n // 2]  # equal states
        if seed == 2:
            B[1::2] = 0.0  # zero states
        if seed == 3:
            B *= 10.0 ** -rng.uniform(0, 12, n)[:, None]  # states of different norms
        yield B @ B.conj().T


# one warp, one subproblem (5 to 32 indices), two and more block pairs
@pytest.mark.parametrize("n,rank", [(2, 1), (4, 2), (5, 1), (8, 4), (16, 5), (20, 7), (24, 20), (31, 12), (32, 16),
                                    (33, 12), (40, 20), (40, 40), (96, 50), (200, 3), (300, 120)])
def test_sweeps_end(capi, n, rank):
    for M in _cases(n, rank):
        ev, U = capi.hermitian_eigensolve(M)
        # the bounds of the solver at full rank
        top = np.max(np.abs(ev))
        assert np.max(np.abs(ev - np.linalg.eigvalsh(M))) < 1e-13 * top
        assert np.max(np.abs(U.conj().T @ U - np.eye(n))) < 2e-14
        assert np.max(np.abs(M @ U - U * ev[None, :])) < 1e-13 * top
