"""Bounded waits that run out: a limit too short for the work ends the call with DFM_WAIT_TIMEOUT, and the context
and its objects go on to work with the usual limit."""
import numpy as np
import pytest

from oracle import port as P
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


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a, np.float64)).cuda()


def _chain(N, b, cplx=False):
    """Row i coupled with rows i - 1 and i + 1."""
    cols = [[j for j in (i - 1, i + 1) if 0 <= j < N] for i in range(N)]
    rp = np.concatenate([[0], np.cumsum([len(c) for c in cols])]).astype(np.uint32)
    S = P.System(rp, np.concatenate(cols).astype(np.uint32), b, cplx=cplx)
    S.off[:] = np.random.default_rng(b).uniform(-1.0, 1.0, S.off.size) / (4 * b)
    S.diag[:] = np.tile([1.0, 0.5] if cplx else np.eye(b).ravel(), N)
    return S


@pytest.mark.parametrize("b,cplx", [(1, False), (2, False), (3, False), (1, True)])
@pytest.mark.parametrize("warps", [(1, 2, 1), (4, 4, 8)])
@pytest.mark.parametrize("mode", [9, 10])
def test_halo_sweep(b, cplx, warps, mode):
    """Eight CTAs with 2,500 rows of a chain each: a CTA waits for its predecessor's last row, 100 ns a row at the
    least, past the limit."""
    from delfem_b200 import lib
    S = _chain(20000, b, cplx)
    ctx, A, M = _make(S)
    M.factor()
    lib.check(lib.lib().dfm_ilu_set_sweep_tuning(M.h, 8, 0))
    M.sweep = mode
    M.sweep_warps = warps
    _, fd, fo = S.ilu0()
    rng = np.random.default_rng(3)
    z = torch.zeros(S.N * S.xw, dtype=torch.float64, device="cuda")
    for limit in (100_000, 50_000):
        r = rng.standard_normal(S.N * S.xw)
        ctx.set_wait_limit(limit)
        with pytest.raises(lib.DfmError) as e:
            M.apply(_dev(r), z)
        assert e.value.code == lib.WAIT_TIMEOUT
        ctx.set_wait_limit(LIMIT_NS)
        M.apply(_dev(r), z)
        ref = S.precond(fd, fo, r)
        assert np.allclose(z.cpu().numpy(), ref, rtol=1e-11, atol=1e-12 * np.abs(ref).max())


@pytest.mark.parametrize("b,cplx", [(1, False), (3, False), (1, True)])
@pytest.mark.parametrize("mode", [3, 9, 10])
def test_copies_land_before_the_exit(b, cplx, mode):
    """With a limit of 1 ns the waits for the chunks themselves may run out while copies are in flight; the CTAs wait
    for those with a limit of their own before they exit, and do so at once (a thousand chunks a CTA)."""
    import time
    from delfem_b200 import lib
    S = _chain(20000, b, cplx)
    ctx, A, M = _make(S)
    M.factor()
    lib.check(lib.lib().dfm_ilu_set_sweep_tuning(M.h, 8, 0))
    M.sweep = mode
    _, fd, fo = S.ilu0()
    r = np.random.default_rng(4).standard_normal(S.N * S.xw)
    ref = S.precond(fd, fo, r)
    z = torch.zeros(S.N * S.xw, dtype=torch.float64, device="cuda")
    M.apply(_dev(r), z)
    for _ in range(10):
        ctx.set_wait_limit(1)
        t0 = time.perf_counter()
        with pytest.raises(lib.DfmError) as e:
            M.apply(_dev(r), z)
        assert e.value.code == lib.WAIT_TIMEOUT and time.perf_counter() - t0 < 1.0
        ctx.set_wait_limit(LIMIT_NS)
        M.apply(_dev(r), z)
        assert np.allclose(z.cpu().numpy(), ref, rtol=1e-11, atol=1e-12 * np.abs(ref).max())


def test_an_autotuner_that_times_out_gives_its_memory_back():
    """60 applications whose tuning runs into the limit: two vectors of 1.6 MB each would be 190 MB."""
    from delfem_b200 import lib
    S = _chain(200000, 1)
    ctx, A, M = _make(S)
    M.factor()
    r = _dev(np.random.default_rng(5).standard_normal(S.N))
    z = torch.zeros_like(r)
    free = []
    for _ in range(60):
        ctx.set_wait_limit(1)
        with pytest.raises(lib.DfmError) as e:
            M.apply(r, z)
        assert e.value.code == lib.WAIT_TIMEOUT
        torch.cuda.synchronize()
        free.append(torch.cuda.mem_get_info()[0])
    assert free[4] - free[-1] < 64 << 20, free
    ctx.set_wait_limit(LIMIT_NS)
    M.apply(r, z)
