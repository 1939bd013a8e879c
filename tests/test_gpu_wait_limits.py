"""Bounded waits that run out: a limit too short for the work ends the call with DFM_WAIT_TIMEOUT, and the context
and its objects go on to work with the usual limit."""
import numpy as np
import pytest

from tests import cases

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

LIMIT_NS = 2_000_000_000  # the default


def _make(S):
    from delfem_b200 import lib
    ctx = lib.Context(0)
    A = lib.Matrix(ctx, S.rowptr, S.colind, S.b, lib.COMPLEX if S.cplx else lib.REAL)
    A.set_values(S.diag, S.off)
    return ctx, A, lib.ILU(A)


@pytest.mark.parametrize("kind", ["poisson", "solid2d", "solid3d", "helmholtz"])
def test_factor(kind):
    """A limit of 1 ns ends a wait after 64 looks (~17 us).  On the box, rows 12 levels of ~5 us ahead are waiting
    for longer; the others may get through.  A factorisation after that is the oracle's to the bit."""
    from delfem_b200 import lib
    S = {"poisson": lambda: cases.poisson(70), "solid2d": lambda: cases.solid2d(40),
         "solid3d": lambda: cases.solid3d(24, 7, 6), "helmholtz": lambda: cases.helmholtz(20, "bands")}[kind]()[1]
    ctx, A, M = _make(S)
    _, fd, fo = S.ilu0()
    for _ in range(3):
        ctx.set_wait_limit(1)
        rc, _ = M.factor(allow=(lib.OK, lib.WAIT_TIMEOUT))
        assert rc == lib.WAIT_TIMEOUT or kind != "solid3d"
        ctx.set_wait_limit(LIMIT_NS)
        M.factor()
        gd, go = M.get_values()
        assert np.array_equal(gd, fd) and np.array_equal(go, fo)
