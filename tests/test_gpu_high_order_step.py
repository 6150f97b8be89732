"""Time steps of 12th to 16th order against the oracle, whose coefficients are
exact: the denominators of the 16th order pass 2^31."""
import numpy as np
import pytest

from oracle import itp_oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def capi():
    import torch
    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for gpu tests")
    from itp2d_b200 import capi as C
    C.lib()
    return C


# one launch (40 x 40), also with a field, line passes (40 x 48), sine passes (40 x 48, hard walls)
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("sy,boundary,B", [(40, O.PERIODIC, 0.0), (40, O.PERIODIC, 0.8), (48, O.PERIODIC, 0.0),
                                           (48, O.DIRICHLET, 0.0)])
@pytest.mark.parametrize("m", [6, 7, 8])
def test_step_matches_oracle(capi, m, sy, boundary, B, precision):
    g = O.Grid(40, sy, 0.2)
    V = O.harmonic(g)
    psi = O.gaussian_states(g, 3, m)
    ref = O.MultiProductSplit(g, V, boundary, B, m, 0.05)
    c = capi.Context(40, sy, g.dx, 3, boundary, B, m, capi.FP64 if precision == "fp64" else capi.FP32)
    c.set_potential(V)
    c.set_time_step(0.05)
    c.upload(psi)
    c.propagate()
    out = c.download()
    c.close()
    exact = ref.apply(psi)
    # a member alone is good to 1e-12 and 2e-5; the sum grows that by the sum of
    # the coefficients' sizes (115 at m = 8)
    tol = (1e-12 if precision == "fp64" else 2e-5) * sum(abs(x) for x in ref.coeffs)
    assert np.max(np.abs(out - exact)) < tol * np.max(np.abs(exact))
