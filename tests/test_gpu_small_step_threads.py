"""One-launch steps (lines_small.cuh) of contexts in several host threads: the
kernel of a grid size is shared by every number of members, whose launches need
different amounts of shared memory."""
import threading

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


def _context(capi, m, precision):
    g = O.Grid(64, 64, 0.2)
    c = capi.Context(64, 64, g.dx, 3, capi.PERIODIC, 0.0, m, precision)
    # zero point energy taken off: the states keep their size over the steps
    c.set_potential(O.harmonic(g) - 1.0)
    c.set_time_step(0.02)
    c.upload(O.gaussian_states(g, 3, m))
    return c


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_threads_with_different_members(capi, precision):
    """m = 2 needs half the shared memory of m = 5; each thread's states are those
    of the same steps taken alone, bit for bit."""
    prec = capi.FP64 if precision == "fp64" else capi.FP32
    steps, members = 4000, (2, 5, 2, 5)
    alone = {}
    for m in set(members):
        c = _context(capi, m, prec)
        for _ in range(steps):
            c.propagate()
        alone[m] = c.download()
        c.close()
    contexts = [_context(capi, m, prec) for m in members]
    failed = []

    def run(c):
        try:
            for _ in range(steps):
                c.propagate()
        except capi.ITP2DError as e:
            failed.append(str(e))

    threads = [threading.Thread(target=run, args=(c,)) for c in contexts]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    out = [c.download() for c in contexts]
    for c in contexts:
        c.close()
    assert not failed
    for m, x in zip(members, out):
        assert np.array_equal(x, alone[m])
