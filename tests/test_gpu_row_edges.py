"""The numeric factorisation and the element assembly at the edges of their
work split, bit-identical to the oracle: rows whose lower rows' blocks fill one
batch, need several, or leave shared memory; nodes with fewer, as many and more
elements than lanes, and a node without any."""
import numpy as np
import pytest

from delfem_b200 import meshes
from oracle import port as P
from tests import cases

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _system(N, reach, b, cplx):
    """Row i coupled with the rows within reach: every update has a target."""
    cols = [[j for j in range(max(0, i - reach), min(N, i + reach + 1)) if j != i] for i in range(N)]
    rp = np.concatenate([[0], np.cumsum([len(c) for c in cols])]).astype(np.uint32)
    S = P.System(rp, np.concatenate(cols).astype(np.uint32), b, cplx=cplx)
    rng = np.random.default_rng(N + reach)
    S.off[:] = rng.uniform(-1.0, 1.0, S.off.size) / (4 * b * reach)
    S.diag[:] = np.tile([1.0, 0.5] if cplx else np.eye(b).ravel(), N)
    return S


# reach 10/11: 45-55 and 55-66 blocks against a batch of 64; 63-65: one row's blocks
# against a batch; 190: rows beyond 24 KB of shared memory for 3 x 3 blocks
@pytest.mark.parametrize("b,cplx", [(1, False), (2, False), (3, False), (1, True)])
@pytest.mark.parametrize("N,reach", [(40, 1), (90, 10), (90, 11), (70, 33), (150, 63), (150, 65), (200, 190)])
def test_factor(ctx, b, cplx, N, reach):
    from delfem_b200 import lib
    S = _system(N, reach, b, cplx)
    A = lib.Matrix(ctx, S.rowptr, S.colind, b, lib.COMPLEX if cplx else lib.REAL)
    A.set_values(S.diag, S.off)
    M = lib.ILU(A)
    rc, ns = M.factor()
    ons, fd, fo = S.ilu0()
    gd, go = M.get_values()
    assert rc == lib.OK and ns == ons == 0
    assert np.array_equal(gd, fd) and np.array_equal(go, fo)


def _fan(k, dim):
    """k triangles around a node, or k tetrahedra around an edge, numbered among their neighbours; one node is in
    no element."""
    n = k + dim  # the hub's dim - 1 nodes, k + 1 - (closed) ring nodes, a loose one
    ring = np.arange(k, dtype=np.float64) * (2 * np.pi / k)
    xy = np.stack([np.cos(ring), np.sin(ring)], axis=1)
    pts = np.zeros((n, dim))
    hub = [k // 2 + q for q in range(dim - 1)]
    rest = [q for q in range(n) if q not in hub]
    loose, nodes = rest[-1], rest[:k]
    pts[nodes, :2] = xy
    pts[loose] = 3.0
    if dim == 3:
        pts[hub[0], 2], pts[hub[1], 2] = -0.5, 0.5
    elem = np.array([hub + [nodes[q], nodes[(q + 1) % k]] for q in range(k)], np.int32)
    return meshes.Mesh(pts, elem, np.zeros((0, 2), np.int32))


@pytest.mark.parametrize("k", [3, 7, 8, 9, 31, 32, 33, 62, 70])
@pytest.mark.parametrize("dim", [2, 3])
def test_assembly(ctx, k, dim):
    from delfem_b200 import lib
    m = _fan(k, dim)
    rp, ci = P.pattern(m.nnode, m.elem)
    S = P.System(rp, ci, dim)
    A = lib.Matrix(ctx, rp, ci, dim)
    G = lib.Mesh(ctx, m.coord, m.elem)
    rng = np.random.default_rng(k)
    u = rng.standard_normal(dim * m.nnode)
    rhs = torch.full((dim * m.nnode,), float("nan"), dtype=torch.float64, device="cuda")
    A.set_values(np.full(S.diag.size, np.nan), np.full(S.off.size, np.nan))
    ud = torch.from_numpy(u).cuda()
    if np.diff(rp.astype(np.int64)).max() + 1 > 64:  # more blocks in a row than assembly takes
        with pytest.raises(lib.DfmError):
            (G.assemble_solid2d if dim == 2 else G.assemble_solid3d)(A, 1.0, 1.0, *[0.0] * (dim + 1), rhs)
        return
    if dim == 2:
        theta = rng.lognormal(0, 0.5, k)
        S.asm_solid2d(m, cases.LAM2_PS, cases.MYU2, 0.8, 0.1, -1.0, theta, u)
        G.assemble_solid2d(A, cases.LAM2_PS, cases.MYU2, 0.8, 0.1, -1.0, rhs, torch.from_numpy(theta).cuda(), ud)
    else:
        S.asm_solid3d(m, cases.LAM3, cases.MYU3, 1.0, 0.0, 0.0, -1.0, u)
        G.assemble_solid3d(A, cases.LAM3, cases.MYU3, 1.0, 0.0, 0.0, -1.0, rhs, ud)
    d, o = A.get_values()
    assert np.array_equal(d, S.diag) and np.array_equal(o, S.off)
    assert np.array_equal(rhs.cpu().numpy(), S.rhs)
    flags = (rng.random(dim * m.nnode) < 0.3).astype(np.int32)
    S.apply_bc(flags)
    lib.apply_dirichlet(A, torch.from_numpy(flags).cuda(), rhs)
    d, o = A.get_values()
    assert np.array_equal(d, S.diag) and np.array_equal(o, S.off)
    assert np.array_equal(rhs.cpu().numpy(), S.rhs)


@pytest.mark.parametrize("b,cplx", [(1, False), (3, False), (1, True)])
@pytest.mark.parametrize("W,k,tail", [(4000, 3, 300), (3000, 12, 40), (300, 40, 700)])
def test_factor_of_a_wide_level_and_a_chain(ctx, b, cplx, W, k, tail):
    """W rows of one level, k lower blocks each, then a chain: the grid is sized by the widest level, and by the blocks
    of a row, not by the average level."""
    from delfem_b200 import lib
    rng = np.random.default_rng(W)
    first = max(4 * k, W // 8)
    N = first + W + tail
    rows = [set() for _ in range(N)]
    for i in range(first, N):
        lower = rng.choice(first, size=k, replace=False).tolist() if i < first + W else [i - 1]
        for j in lower:
            rows[i].add(j)
            rows[j].add(i)
    rp = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.uint32)
    S = P.System(rp, np.concatenate([np.array(sorted(r), np.uint32) for r in rows]), b, cplx=cplx)
    S.off[:] = rng.uniform(-1.0, 1.0, S.off.size) / (4 * b * max(len(r) for r in rows))
    S.diag[:] = np.tile([1.0, 0.5] if cplx else np.eye(b).ravel(), N)
    A = lib.Matrix(ctx, S.rowptr, S.colind, b, lib.COMPLEX if cplx else lib.REAL)
    A.set_values(S.diag, S.off)
    M = lib.ILU(A)
    rc, ns = M.factor()
    ons, fd, fo = S.ilu0()
    gd, go = M.get_values()
    assert rc == lib.OK and ns == ons == 0
    assert np.array_equal(gd, fd) and np.array_equal(go, fo)
