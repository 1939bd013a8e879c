"""Schedules 9 and 10 at the edges of their packing: rows longer than a lane's
registers, slices and halo areas kept as rings, a fused dot without room for
its vector, and partitions by chains.  The preconditioner to 1e-11 of the
oracle, solves to 1e-8, as in the tests of the other schedules."""
import numpy as np
import pytest

from tests import cases
from oracle import port as P

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a, np.float64)).cuda()


def _make(ctx, S):
    from delfem_b200 import lib
    A = lib.Matrix(ctx, S.rowptr, S.colind, S.b, lib.COMPLEX if S.cplx else lib.REAL)
    A.set_values(S.diag, S.off)
    M = lib.ILU(A)
    M.factor()
    return A, M


def _apply(M, S, fd, fo, seed=5):
    r = np.random.default_rng(seed).standard_normal(S.N * S.xw)
    ref = S.precond(fd, fo, r)
    z = torch.zeros(S.N * S.xw, dtype=torch.float64, device="cuda")
    M.apply(_dev(r), z)
    assert np.allclose(z.cpu().numpy(), ref, rtol=1e-11, atol=1e-12 * np.abs(ref).max())


def _pattern(N, rows, b, seed):
    """A diagonally dominant system from each row's set of lower columns, made symmetric in pattern."""
    full = [set() for _ in range(N)]
    for i, cols in enumerate(rows):
        for j in cols:
            full[i].add(j)
            full[j].add(i)
    rp = np.concatenate([[0], np.cumsum([len(s) for s in full])]).astype(np.uint32)
    ci = np.concatenate([np.array(sorted(s), np.uint32) for s in full])
    S = P.System(rp, ci, b)
    rng = np.random.default_rng(seed)
    S.off[:] = rng.uniform(-1.0, 1.0, S.off.size) / (2 * b * max(len(s) for s in full))
    S.diag[:] = np.tile(np.eye(b).ravel(), N)
    S.rhs[:] = rng.standard_normal(N * b)
    return S


@pytest.mark.parametrize("b", [1, 2, 3])
@pytest.mark.parametrize("warps", [(1, 2, 1), (2, 4, 4), (4, 8, 8)])
@pytest.mark.parametrize("mode", [9, 10])
@pytest.mark.parametrize("ctas", [1, 5])
def test_rows_longer_than_the_registers(ctx, b, warps, mode, ctas):
    """Blocks per lane below, at and far past what a lane holds."""
    from delfem_b200 import lib
    S = cases.random_spd_like(220, b, seed=31, density=14)
    A, M = _make(ctx, S)
    lib.check(lib.lib().dfm_ilu_set_sweep_tuning(M.h, ctas, 0))
    M.sweep = mode
    M.sweep_warps = warps
    _, fd, fo = S.ilu0()
    _apply(M, S, fd, fo)
    lib.check(lib.lib().dfm_ilu_set_sweep_tuning(M.h, 0, 0))


@pytest.mark.parametrize("kind", ["poisson", "solid2d", "solid3d", "helmholtz"])
@pytest.mark.parametrize("ctas", [1, 6])
def test_slice_ring_wraps(ctx, kind, ctas):
    """Parts many times as long as the slice, so its places are taken over; the fused dot follows the ring."""
    from delfem_b200 import lib
    S = {"poisson": lambda: cases.poisson(90), "solid2d": lambda: cases.solid2d(60),
         "solid3d": lambda: cases.solid3d(60, 5, 5), "helmholtz": lambda: cases.helmholtz(30, "bands")}[kind]()[1]
    A, M = _make(ctx, S)
    lib.check(lib.lib().dfm_ilu_set_sweep_tuning(M.h, ctas, 0))
    M.sweep = 9
    _, fd, fo = S.ilu0()
    _apply(M, S, fd, fo)
    if kind != "helmholtz":
        ref = S.solve(fd, fo, tol=1e-10, maxit=2000)
        x = torch.zeros(S.N * S.xw, dtype=torch.float64, device="cuda")
        rc, it, _ = lib.solve_pcg(A, M, _dev(S.rhs), x, tol=1e-10, maxit=2000)
        assert rc == lib.OK and abs(int(it) - int(ref["iters"])) <= 2
        assert np.linalg.norm(x.cpu().numpy() - ref["x"]) <= 1e-8 * np.linalg.norm(ref["x"])
    lib.check(lib.lib().dfm_ilu_set_sweep_tuning(M.h, 0, 0))


@pytest.mark.parametrize("b", [1, 3])
def test_early_rows_read_to_the_end(ctx, b):
    """The first 64 rows are read by every later row: the slice holds a whole part (12,000 doubles of a
    part of one CTA leave no room for the dot's vector) and the halo of the other CTAs spans everything."""
    from delfem_b200 import lib
    N = 12000 if b == 1 else 4000
    S = _pattern(N, [{i - 64, i % 64} if i >= 128 else {i - 64} if i >= 64 else set() for i in range(N)], b, 7)
    A, M = _make(ctx, S)
    _, fd, fo = S.ilu0()
    ref = S.solve(fd, fo, tol=1e-10, maxit=500)
    for ctas in (1, 9):
        lib.check(lib.lib().dfm_ilu_set_sweep_tuning(M.h, ctas, 0))
        M.sweep = 9
        _apply(M, S, fd, fo)
        x = torch.zeros(S.N * b, dtype=torch.float64, device="cuda")
        rc, it, _ = lib.solve_pcg(A, M, _dev(S.rhs), x, tol=1e-10, maxit=500)
        assert rc == lib.OK and abs(int(it) - int(ref["iters"])) <= 1
        assert np.linalg.norm(x.cpu().numpy() - ref["x"]) <= 1e-8 * np.linalg.norm(ref["x"])
    lib.check(lib.lib().dfm_ilu_set_sweep_tuning(M.h, 0, 0))


def test_halo_ring(ctx):
    """Every part reads most rows of the others: the halo area (6,000 rows of 24 bytes) is a ring."""
    from delfem_b200 import lib
    rng = np.random.default_rng(2)
    N = 6000
    S = _pattern(N, [set(rng.integers(0, i, 6).tolist()) if i else set() for i in range(N)], 3, 9)
    A, M = _make(ctx, S)
    lib.check(lib.lib().dfm_ilu_set_sweep_tuning(M.h, 8, 0))
    M.sweep = 9
    _, fd, fo = S.ilu0()
    _apply(M, S, fd, fo)
    lib.check(lib.lib().dfm_ilu_set_sweep_tuning(M.h, 0, 0))


@pytest.mark.parametrize("fill", [0, 1])
def test_partition_by_chains(ctx, fill):
    """The autotuner's own partitions (chains of a box and of a plane grid) and their PCG."""
    from delfem_b200 import lib
    for S in (cases.solid3d(24, 7, 6)[1], cases.poisson(70)[1]):
        A = lib.Matrix(ctx, S.rowptr, S.colind, S.b)
        A.set_values(S.diag, S.off)
        M = lib.ILU(A, fill)
        M.factor()
        if fill == 0:
            _, fd, fo = S.ilu0()
            _apply(M, S, fd, fo)
            ref = S.solve(fd, fo, tol=1e-10, maxit=2000)["x"]
        else:
            M0 = lib.ILU(A)
            M0.factor()
            _, fd, fo = S.ilu0()
            ref = S.solve(fd, fo, tol=1e-12, maxit=4000)["x"]
        x = torch.zeros(S.N * S.xw, dtype=torch.float64, device="cuda")
        rc, _, _ = lib.solve_pcg(A, M, _dev(S.rhs), x, tol=1e-10, maxit=2000)
        assert rc == lib.OK
        assert np.linalg.norm(x.cpu().numpy() - ref) <= 1e-8 * np.linalg.norm(ref)


@pytest.mark.parametrize("name", ["poisson", "solid3d", "helmholtz"])
@pytest.mark.parametrize("mode", [1, 2, 3, 4, 5, 8, 9, 10])
def test_factor_values_set_by_the_caller(ctx, name, mode):
    """Applications and solves after dfm_ilu_set_values use the new factor: the schedules' packed values follow it."""
    from delfem_b200 import lib
    S = {"poisson": lambda: cases.poisson(30), "solid3d": lambda: cases.solid3d(12, 4, 4),
         "helmholtz": lambda: cases.helmholtz(12, "bands")}[name]()[1]
    A, M = _make(ctx, S)
    M.sweep = mode
    _, fd, fo = S.ilu0()
    _apply(M, S, fd, fo)
    rng = np.random.default_rng(8)
    gd, go = fd * 0.5, fo * rng.uniform(0.2, 0.4, fo.size)
    M.set_values(gd, go)
    _apply(M, S, gd, go)
    if not S.cplx:  # a solve whose preconditioner is the same factor as before: the iterations tell
        M.set_values(fd, fo)
        x = torch.zeros(S.N * S.xw, dtype=torch.float64, device="cuda")
        ref = S.solve(fd, fo, tol=1e-10, maxit=2000)
        rc, it, _ = lib.solve_pcg(A, M, _dev(S.rhs), x, tol=1e-10, maxit=2000)
        assert rc == lib.OK and abs(int(it) - int(ref["iters"])) <= 2


@pytest.mark.parametrize("b", [1, 2, 3])
@pytest.mark.parametrize("mode", [0, 9, 10])
def test_the_shape_in_use_can_be_pinned(ctx, b, mode):
    """What sweep_warps reports is accepted and gives the same bits: after the autotuner (mode 0), and for the shape
    that a schedule starts with."""
    S = {1: lambda: cases.poisson(60), 2: lambda: cases.solid2d(30), 3: lambda: cases.solid3d(20, 5, 5)}[b]()[1]
    _, M = _make(ctx, S)
    r = _dev(np.random.default_rng(6).standard_normal(S.N * S.xw))
    z, y = torch.zeros_like(r), torch.zeros_like(r)
    M.sweep = mode
    M.apply(r, z)
    if M.sweep not in (9, 10):
        pytest.skip("the autotuner picked another schedule")
    shape = M.sweep_warps
    M.sweep_warps = shape
    assert M.sweep_warps == shape
    M.apply(r, y)
    assert torch.equal(z, y)


@pytest.mark.parametrize("b", [1, 3])
@pytest.mark.parametrize("cw", [1, 2, 4])
def test_one_lane_per_component(ctx, b, cw):
    S = cases.poisson(40)[1] if b == 1 else cases.solid3d(14, 5, 4)[1]
    _, M = _make(ctx, S)
    _, fd, fo = S.ilu0()
    for mode in (9, 10):
        M.sweep = mode
        M.sweep_warps = (cw, 1, 4)
        assert M.sweep_warps == (cw, 1, 4)
        _apply(M, S, fd, fo)


@pytest.mark.parametrize("b", [1, 2, 3])
@pytest.mark.parametrize("mode", [9, 10])
@pytest.mark.parametrize("ctas", [1, 2])
def test_lanes_set_are_the_lanes_that_run(ctx, b, mode, ctas):
    """A row of 16 blocks whose sum tells how many lanes shared it: lane h adds blocks h, h + lanes, ..., and 1 is lost
    beside 1e16 unless another lane has it.  Blocks 0, 4 and 8 are 1e16, 1 and -1e16: one of 8 lanes has 0 and 8,
    another has 4; one of 4 lanes, of 2 and of 1 has all three in this order."""
    from delfem_b200 import lib
    S = _pattern(17, [set()] * 16 + [set(range(16))], b, 3)
    _, M = _make(ctx, S)
    lib.check(lib.lib().dfm_ilu_set_sweep_tuning(M.h, ctas, 0))
    off = np.zeros((int(S.rowptr[-1]), b, b))
    for k, v in ((0, 1e16), (4, 1.0), (8, -1e16)):
        off[S.rowptr[16] + k] = v * np.eye(b)
    M.set_values(np.tile(np.eye(b).ravel(), 17), off.ravel())
    M.sweep = mode
    for lanes, want in ((1, 1.0), (2, 1.0), (4, 1.0), (8, 0.0)):
        for cw in (1, 2, 4):
            M.sweep_warps = (cw, lanes, 4)
            z = torch.zeros(17 * b, dtype=torch.float64, device="cuda")
            M.apply(torch.ones_like(z), z)
            assert z.cpu().numpy().tolist() == [1.0] * (16 * b) + [want] * b, (lanes, cw)
    lib.check(lib.lib().dfm_ilu_set_sweep_tuning(M.h, 0, 0))


def test_fp32_plans_follow_the_partition(ctx):
    """An autotuned partition by chains, a mixed solve, then ranges of the natural order with as many CTAs and the
    same warps: the next mixed solve's plans are of those ranges."""
    from delfem_b200 import lib
    S = cases.solid3d(40, 12, 12)[1]
    A, M = _make(ctx, S)
    _, fd, fo = S.ilu0()
    _apply(M, S, fd, fo)
    if M.sweep not in (9, 10) or M.sweep_info().partition != 2:
        pytest.skip("the autotuner picked no partition by chains")
    M.sweep_warps = (2, 2, 4)
    x = torch.zeros(S.N * 3, dtype=torch.float64, device="cuda")

    def mixed():
        rc, it, _ = lib.solve_pcg_mixed(A, M, _dev(S.rhs), x, tol=1e-8, maxit=2000)
        assert rc == lib.OK
        for back in (False, True):
            d, f = M.sweep_info(back), M.sweep_info(back, fp32=True)
            assert (f.ctas, f.partition, f.merged, f.part_rows) == (d.ctas, d.partition, d.merged, d.part_rows)

    mixed()
    mode, ctas = M.sweep, M.sweep_info().ctas
    lib.check(lib.lib().dfm_ilu_set_sweep_tuning(M.h, ctas, 0))
    M.sweep = mode
    M.sweep_warps = (2, 2, 4)
    assert M.sweep_info().partition == 0 and M.sweep_info().ctas == ctas
    mixed()
    lib.check(lib.lib().dfm_ilu_set_sweep_tuning(M.h, 0, 0))


@pytest.mark.parametrize("N,k", [(5000, 30), (2000, 60)])
def test_the_autotuner_finds_the_fast_schedules(ctx, N, k):
    """Rows with k random neighbours on either side (no mesh): the pick is no more than a quarter slower than any
    schedule set by hand on all SMs."""
    from delfem_b200 import lib
    rng = np.random.default_rng(0)
    i, j = np.repeat(np.arange(N), k), rng.integers(0, N, N * k)
    i, j = i[i != j], j[i != j]
    e = np.unique(np.concatenate([i * N + j, j * N + i]))
    rp = np.concatenate([[0], np.cumsum(np.bincount(e // N, minlength=N))]).astype(np.uint32)
    A = lib.Matrix(ctx, rp, (e % N).astype(np.uint32), 3)
    A.set_values(np.tile(np.eye(3).ravel(), N), rng.uniform(-1.0, 1.0, e.size * 9) / (6 * np.diff(rp.astype(int)).max()))
    M = lib.ILU(A)
    M.factor()
    r = torch.randn(3 * N, dtype=torch.float64, device="cuda")
    z = torch.zeros_like(r)

    def ms():
        M.apply(r, z)
        return 1e3 * min(M.time_apply(r, z, 10) for _ in range(3))

    auto, pick = ms(), M.sweep
    by_hand = {}
    for mode in (1, 2, 3, 7, 9):
        M.sweep = mode
        by_hand[mode] = ms()
    assert auto <= 1.25 * min(by_hand.values()), (auto, pick, by_hand)


def _read_first_rows(b):
    """The first 64 rows are read by every later row."""
    N = 12000 if b == 1 else 4000
    return _pattern(N, [{i - 64, i % 64} if i >= 128 else {i - 64} if i >= 64 else set() for i in range(N)], b, 7)


@pytest.mark.parametrize("b", [1, 2, 3])
def test_fp32_plan_where_there_is_an_fp64_plan(ctx, b):
    """Rows of hundreds of blocks beside a slice that holds the whole part: the mixed solve takes the schedule that
    the FP64 one takes."""
    from delfem_b200 import lib
    S = _read_first_rows(b)
    A, M = _make(ctx, S)
    _, fd, fo = S.ilu0()
    ref = S.solve(fd, fo, tol=1e-10, maxit=500)["x"]
    for ctas in (1, 3):
        lib.check(lib.lib().dfm_ilu_set_sweep_tuning(M.h, ctas, 0))
        M.sweep = 9
        for solve in (lib.solve_pcg, lib.solve_pcg_mixed):
            x = torch.zeros(S.N * b, dtype=torch.float64, device="cuda")
            rc, _, _ = solve(A, M, _dev(S.rhs), x, tol=1e-10, maxit=500)
            assert rc == lib.OK
            assert np.linalg.norm(x.cpu().numpy() - ref) <= 1e-8 * np.linalg.norm(ref)
        assert M.sweep_info(fp32=True).ctas == M.sweep_info(backward=True, fp32=True).ctas == ctas
    lib.check(lib.lib().dfm_ilu_set_sweep_tuning(M.h, 0, 0))


def _read_random_rows():
    rng = np.random.default_rng(2)
    return _pattern(6000, [set(rng.integers(0, i, 6).tolist()) if i else set() for i in range(6000)], 3, 9)


# system, CTAs, what the plans must have come out as: (forward and backward, backward only)
FORMS = {
    "long rows 1": (lambda: cases.random_spd_like(220, 1, seed=31, density=14), 5, {"long_rows": 1}, {}),
    "long rows 3": (lambda: cases.random_spd_like(220, 3, seed=31, density=14), 5, {"long_rows": 1}, {}),
    "slice ring 1": (lambda: cases.poisson(90)[1], 1, {"slice ring": 1}, {}),
    "slice ring 2": (lambda: cases.solid2d(100)[1], 2, {"slice ring": 1}, {}),
    "slice ring 3": (lambda: cases.solid3d(100, 5, 5)[1], 8, {"slice ring": 1}, {}),
    "fused dot over a ring": (lambda: cases.solid3d(100, 5, 5)[1], 6, {"slice ring": 1}, {"dot_fused": 1}),
    "whole slice, separate dot": (lambda: _read_first_rows(1), 1, {"slice ring": 0}, {"dot_fused": 0}),
    "smaller rounds": (lambda: _read_first_rows(3), 1, {}, {"dot_fused": 0, "long_rows": 1}),
    "halo ring": (_read_random_rows, 8, {"halo_ring": 1}, {}),
}


@pytest.mark.parametrize("name", sorted(FORMS))
@pytest.mark.parametrize("fp32", [False, True])
def test_forms_of_a_plan(ctx, name, fp32):
    """Each form of the plans, known to be the one that runs, in the application and in a PCG with FP64 or FP32
    factor values; x to 1e-8 of the oracle's."""
    from delfem_b200 import lib
    make, ctas, both, backward = FORMS[name]
    S = make()
    A, M = _make(ctx, S)
    lib.check(lib.lib().dfm_ilu_set_sweep_tuning(M.h, ctas, 0))
    M.sweep = 9
    _, fd, fo = S.ilu0()
    _apply(M, S, fd, fo)
    x = torch.zeros(S.N * S.xw, dtype=torch.float64, device="cuda")
    solve = lib.solve_pcg_mixed if fp32 else lib.solve_pcg
    rc, _, _ = solve(A, M, _dev(S.rhs), x, tol=1e-10, maxit=4000)
    assert rc == lib.OK
    for back in (False, True):
        info = M.sweep_info(back, fp32)
        seen = {n: getattr(info, n) for n, _ in info._fields_} | {"slice ring": int(info.slice_rows < info.part_rows)}
        want = both | (backward if back else {})
        assert {k: seen[k] for k in want} == want and seen["ctas"] == ctas, seen
    if name.startswith("long rows"):  # values without symmetry, which PCG takes in its stride: A x = rhs tells
        res = S.spmv(-1.0, x.cpu().numpy(), 1.0, S.rhs.copy())
        assert np.linalg.norm(res) <= 1e-8 * np.linalg.norm(S.rhs)
    else:
        ref = S.solve(fd, fo, tol=1e-10, maxit=4000)["x"]
        assert np.linalg.norm(x.cpu().numpy() - ref) <= 1e-8 * np.linalg.norm(ref)
    lib.check(lib.lib().dfm_ilu_set_sweep_tuning(M.h, 0, 0))



@pytest.mark.parametrize("fill", [0, 1])
def test_the_partition_by_chains_ran(ctx, fill):
    """Boxes on which the autotuner picks the partition by chains: both directions' plans are of that partition, and
    the application is the oracle's (ILU(0)) or that of the one-CTA schedule (ILU(1))."""
    from delfem_b200 import lib
    S = cases.solid3d(40, 12, 12)[1]
    A = lib.Matrix(ctx, S.rowptr, S.colind, 3)
    A.set_values(S.diag, S.off)
    M = lib.ILU(A, fill)
    M.factor()
    r = np.random.default_rng(5).standard_normal(S.N * 3)
    z, y = (torch.zeros(S.N * 3, dtype=torch.float64, device="cuda") for _ in range(2))
    M.apply(_dev(r), z)
    if M.sweep not in (9, 10) or M.sweep_info().partition != 2:
        pytest.skip("the autotuner picked no partition by chains")
    assert M.sweep_info(backward=True).partition == 2
    if fill == 0:
        _, fd, fo = S.ilu0()
        ref = S.precond(fd, fo, r)
    else:
        M.sweep = 2
        M.apply(_dev(r), y)
        ref = y.cpu().numpy()
    assert np.allclose(z.cpu().numpy(), ref, rtol=1e-11, atol=1e-12 * np.abs(ref).max())
