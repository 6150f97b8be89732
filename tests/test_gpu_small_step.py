"""Steps of small square grids in one launch (lines_small.cuh): every way the
members share a cluster's CTAs (1 to 8 members), factors with A = B and A != B,
the largest grids that fit in shared memory, and grids on the other side of the
rule, against the oracle's split step."""
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


def _rel(a, b):
    return np.max(np.abs(a - b)) / np.max(np.abs(b))


def _split(g, V, B, m, eps):
    """The oracle's step with the library's 32-bit coefficient denominators
    (their product passes 2^31 at m = 8)."""
    ref = O.MultiProductSplit(g, V, O.PERIODIC, B, m, eps)
    ref.coeffs = []
    for t in range(1, m + 1):
        denom = 1
        for n in range(1, m + 1):
            if n != t:
                denom = (denom * (t * t - n * n) + 2 ** 31) % 2 ** 32 - 2 ** 31
        ref.coeffs.append(float(t) ** (2 * (m - 1)) / denom)
    ref.set_time_step(eps)
    return ref


# precision, n, states, members, field, one launch
CASES = [
    ("fp64", 32, 1, 1, 0.0, True), ("fp64", 36, 3, 2, 0.8, True), ("fp64", 32, 3, 3, 0.0, True),
    ("fp64", 40, 2, 4, 0.8, True), ("fp64", 64, 5, 5, 0.0, True), ("fp64", 64, 5, 5, 0.8, True),
    ("fp64", 60, 2, 6, 0.8, True), ("fp64", 72, 2, 7, 0.0, True), ("fp64", 80, 3, 8, 0.8, True),
    ("fp64", 108, 60, 2, 0.8, True), ("fp64", 108, 3, 2, 0.8, False), ("fp64", 90, 2, 3, 0.0, False),
    ("fp64", 35, 3, 2, 0.8, False),
    ("fp32", 32, 80, 3, 0.0, True), ("fp32", 48, 3, 8, 0.8, True), ("fp32", 108, 2, 5, 0.8, True),
    ("fp32", 128, 60, 2, 0.8, True), ("fp32", 160, 2, 2, 0.0, False),
]


@pytest.mark.parametrize("precision,n,k,m,B,one", CASES)
def test_small_step_matches_oracle(capi, precision, n, k, m, B, one):
    g = O.Grid(n, n, 0.15)
    V = O.harmonic(g)
    psi = O.gaussian_states(g, k, 3)
    c = capi.Context(n, n, g.dx, k, capi.PERIODIC, B, m, capi.FP64 if precision == "fp64" else capi.FP32)
    c.set_potential(V)
    c.set_time_step(0.05)
    c.upload(psi)
    before = capi.lib().itp2d_launch_count(c.h)
    c.propagate()
    launched = capi.lib().itp2d_launch_count(c.h) - before
    step = c.download()
    c.close()
    assert (launched == 1) == one
    # the coefficients of the members cancel in part: their absolute sum grows
    # the rounding of one member's step (bounds 1e-12 and 2e-5 for up to 3)
    ref = _split(g, V, B, m, 0.05)
    grow = sum(abs(x) for x in ref.coeffs) if m > 3 else 1.0
    assert _rel(step, ref.apply(psi)) < (1e-12 if precision == "fp64" else 2e-5) * max(grow, 1.0)
