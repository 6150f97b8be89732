"""Edges of the int8 FP64 contractions (csrc/oz.cu): digits at extreme scales and
signs, grid ranges of one step, of an odd number of steps and just past a chunk
of 512 steps, and state counts around the 16, 64 and 128 of the tiles."""
import numpy as np
import pytest

from itp2d_b200 import capi

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    import torch
    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for gpu tests")


def _overlap(psi, engine):
    k, sy, sx = psi.shape
    c = capi.Context(sx, sy, 1.0, k)
    c.set_fp64_engine(engine)
    c.upload(psi)
    S = c.overlap_matrix()
    n = c.int8_contractions()
    c.close()
    assert n == (1 if engine == capi.FP64_INT8 else 0)
    return S


@pytest.mark.parametrize("sx,sy", [(5, 3), (35, 3), (128, 64), (120, 70)])
@pytest.mark.parametrize("k", [2, 17, 64, 65, 129])
def test_overlap_at_step_and_tile_edges(sx, sy, k):
    rng = np.random.default_rng(k * sx)
    psi = rng.standard_normal((k, sy, sx)) + 1j * rng.standard_normal((k, sy, sx))
    S = _overlap(psi, capi.FP64_INT8)
    P = psi.reshape(k, -1)
    # the split's bound: 2 G real products of values below 2^e, each off by about
    # 9.1 x 2^-56 x 2^(e_x + e_y)
    e = np.frexp(np.maximum(np.abs(P.real), np.abs(P.imag)).max(axis=1))[1].astype(float)
    bound = 10.0 * 2.0 ** -56 * 2 * P.shape[1] * 2.0 ** (e[:, None] + e[None, :])
    assert np.all(np.abs(S - P.conj() @ P.T) <= bound)


def test_power_of_two_scales_and_signs_are_exact():
    """Scaling a state by a power of two scales its row and column of the overlap
    exactly (the digits do not change), negating and conjugating it changes signs
    only."""
    rng = np.random.default_rng(3)
    k, sy, sx = 20, 12, 16
    psi = rng.standard_normal((k, sy, sx)) + 1j * rng.standard_normal((k, sy, sx))
    psi[3, 2] = 0.0
    psi[4] *= 10.0 ** rng.uniform(-30, 0, (sy, sx))
    S = _overlap(psi, capi.FP64_INT8)
    p = rng.integers(-480, 400, k).astype(float)
    f = 2.0 ** p
    assert np.array_equal(_overlap(psi * f[:, None, None], capi.FP64_INT8), (S * f[:, None]) * f[None, :])
    sign = rng.choice([-1.0, 1.0], k)
    assert np.array_equal(_overlap(psi * sign[:, None, None], capi.FP64_INT8), S * sign[:, None] * sign[None, :])
    assert np.array_equal(_overlap(psi.conj(), capi.FP64_INT8), S.conj())


@pytest.mark.parametrize("sx,sy", [(5, 3), (21, 3), (64, 45)])
@pytest.mark.parametrize("k", [2, 16, 17, 127, 129])
def test_rotation_at_step_and_tile_edges(sx, sy, k):
    """Cholesky orthonormalisation of nearly orthonormal states on both engines:
    W is close to the identity, the rotated states agree to rounding."""
    if k > sx * sy // 2:
        pytest.skip("more states than the grid holds")
    rng = np.random.default_rng(k + sx)
    G = sx * sy
    Q = np.linalg.qr(rng.standard_normal((G, k)) + 1j * rng.standard_normal((G, k)))[0]
    psi = (Q @ (np.eye(k) + 0.01 * rng.standard_normal((k, k)))).T.reshape(k, sy, sx)
    out = {}
    for engine in (capi.FP64_DMMA, capi.FP64_INT8):
        c = capi.Context(sx, sy, 1.0, k)
        c.set_fp64_engine(engine)
        c.upload(psi)
        c.orthonormalize(capi.ORTHO_CHOLESKY)
        out[engine] = c.download()
        c.close()
    d = np.max(np.abs(out[capi.FP64_INT8] - out[capi.FP64_DMMA])) / np.max(np.abs(out[capi.FP64_DMMA]))
    assert d < 1e-13
