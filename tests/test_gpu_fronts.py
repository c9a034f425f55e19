"""The multifrontal LU of Shell_1 structures (through the C ABI) where its
schedule has edges: single elements and single fronts, fronts on either side
of the shared-memory limit, meshes of several components, strips, nodes with
load stiffness, and structures of different heights in one batch.  Each
structure as the oracle's banded LU with partial pivoting solves it: the same
step counts and 1e-10 of the coordinate scale (the plain path's stated
tolerance)."""
import numpy as np
import pytest

from giraffe_gb300 import configs, gpu
from giraffe_gb300.model import NodalLoad, Table
from oracle import oracle

pytestmark = pytest.mark.gpu


def strip(nx, ny, steps=3):
    """nx x ny squares of the plate family, clamped along every edge but one long one."""
    s = configs.square_plate(max(nx, ny), steps=steps)
    m = 2 * max(nx, ny) + 1
    keep = [i for i in range(m * m) if i % m <= 2 * nx and i // m <= 2 * ny]
    new = {old: k for k, old in enumerate(keep)}
    shells = [tuple(new[q] for q in row[:6]) + tuple(row[6:]) for row in s.shells if all(q in new for q in row[:6])]
    s.shells = shells
    s.nodes = s.nodes[keep]
    s.constraints = np.zeros((len(keep), 6), dtype=np.int32)
    for k, old in enumerate(keep):
        if old % m in (0, 2 * nx) or old // m == 0:
            s.constraints[k] = 1
    s.loads[0].shells = list(range(len(shells)))
    return s


def two_plates(n1, n2):
    """Two plates apart in one structure: the graph has two components."""
    a, b = configs.square_plate(n1, steps=3), configs.square_plate(n2, steps=3)
    k = a.n_nodes
    a.nodes = np.concatenate([a.nodes, b.nodes + [3.0, 0.0, 0.0]])
    a.shells.extend([tuple(q + k for q in row[:6]) + tuple(row[6:]) for row in b.shells])
    a.constraints = np.concatenate([a.constraints, b.constraints])
    a.loads[0].shells = list(range(len(a.shells)))
    return a


def loaded(n):
    """A plate with a moment on a midside node: load stiffness in K_AA."""
    s = configs.square_plate(n, steps=3)
    m = 2 * n + 1
    node = 2 * (n // 2) * m + 2 * (n // 2) + 1
    s.loads.append(NodalLoad([node], 0, Table(np.array([0.0, 1.0]), np.array([[0.0] * 6, [0, 0, -200.0, 15.0, 5.0, 0]]))))
    return s


@pytest.mark.parametrize("make", [
    lambda: configs.square_plate(1, steps=2), lambda: configs.square_plate(2, steps=2),
    lambda: configs.square_plate(3, steps=2), lambda: configs.square_plate(5, steps=2),
    lambda: configs.square_plate(13, steps=2), lambda: strip(1, 1), lambda: strip(9, 1), lambda: strip(12, 3),
    lambda: two_plates(2, 5), lambda: loaded(4), lambda: loaded(9),
], ids=["plate1", "plate2", "plate3", "plate5", "plate13", "strip1x1", "strip9x1", "strip12x3", "two", "loaded4", "loaded9"])
def test_solves_as_the_oracle(gpu_ctx, make):
    s = make()
    b = gpu.BatchSolver(gpu_ctx, [s, configs.square_plate(4, steps=2), make()])
    b.reset()
    b.run()
    finals, stats = b.results()
    b.close()
    fo, so, _ = oracle.solve(s, 0)
    assert tuple(stats[0]) == tuple(so)
    scale = np.abs(fo[:, :3]).max()
    assert np.abs(finals[0][:, :3] - fo[:, :3]).max() <= 1e-10 * scale
    assert np.abs(finals[0][:, 6:] - fo[:, 6:]).max() <= 1e-9
    # the same structure elsewhere in the batch, and alone: the same bits
    assert np.array_equal(finals[0], finals[2])
    alone, _ = gpu.solve([make()])
    assert np.array_equal(finals[0], alone[0])


def solve_dense(A, b):
    return np.linalg.solve(A, b)


def to_csr(A):
    rows, cols = np.nonzero(A)
    rp = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=len(A)))]).astype(np.int32)
    return rp, cols.astype(np.int32), A[rows, cols]


def pattern(kind, seed):
    """Diagonally dominant matrices (row sums 1.5 times the off-diagonal's, so
    no pivoting is needed) whose graphs the ordering meets in earnest or not."""
    rng = np.random.default_rng(seed)
    if kind == "dense":
        n = 150
        M = np.ones((n, n), dtype=bool)
    elif kind == "grid":
        g, d = 13, 3
        n = g * g * d
        x = np.arange(n) // d
        M = (np.abs(x[:, None] % g - x[None, :] % g) <= 1) & (np.abs(x[:, None] // g - x[None, :] // g) <= 1)
    elif kind == "unsymmetric":
        n = 400
        M = rng.random((n, n)) < 4.0 / n
    elif kind == "arrow":
        n = 300
        M = np.eye(n, dtype=bool)
        M[-40:] = M[:, -40:] = True
    elif kind == "blocks":  # three components and rows without off-diagonals
        n = 330
        c = np.arange(n) // 110
        M = (c[:, None] == c[None, :]) & (rng.random((n, n)) < 0.05)
    elif kind == "scrambled":
        n = 500
        p = rng.permutation(n)
        M = np.abs(p[:, None] - p[None, :]) <= 5
    else:  # one row past the narrow band
        n = 100
        M = np.abs(np.arange(n)[:, None] - np.arange(n)[None, :]) <= 18
    A = np.where(M, rng.uniform(-1.0, 1.0, (n, n)), 0.0)
    np.fill_diagonal(A, 0.0)
    np.fill_diagonal(A, 1.5 * np.abs(A).sum(axis=1) + 0.1)
    return A


@pytest.mark.parametrize("kind", ["dense", "grid", "unsymmetric", "arrow", "blocks", "scrambled", "past17"])
def test_sparse_patterns_match_dense(gpu_ctx, kind):
    # forward error bound n eps cond with cond <= 5 for these row sums: 1e-13
    A = pattern(kind, 3)
    b = np.random.default_rng(4).normal(size=len(A))
    x, info = gpu_ctx.sparse_solve(*to_csr(A), b)
    assert info == 0
    ref = solve_dense(A, b)
    assert np.abs(x - ref).max() <= 1e-13 * np.abs(ref).max()


def test_sparse_rows_in_any_order_and_repeated(gpu_ctx):
    A = pattern("grid", 5)
    rp, ci, v = to_csr(A)
    rng = np.random.default_rng(6)
    ci2, v2 = np.repeat(ci, 2), np.repeat(v, 2) * np.tile([0.25, 0.75], len(v))
    rp2 = 2 * rp
    for i in range(len(A)):
        p = rp2[i] + rng.permutation(rp2[i + 1] - rp2[i])
        ci2[rp2[i]:rp2[i + 1]], v2[rp2[i]:rp2[i + 1]] = ci2[p], v2[p]
    b = rng.normal(size=len(A))
    x, info = gpu_ctx.sparse_solve(rp2, ci2, v2, b)
    ref = solve_dense(A, b)
    assert info == 0 and np.abs(x - ref).max() <= 1e-13 * np.abs(ref).max()


@pytest.mark.parametrize("n,kl,ku", [(2000, 17, 17), (2001, 3, 9), (1500, 0, 1), (800, 1, 0), (3000, 40, 33),
                                     (2600, 97, 96), (1501, 300, 2), (700, 12, 13)])
def test_bands_match_a_banded_lu(gpu_ctx, n, kl, ku):
    from scipy.linalg import solve_banded

    rng = np.random.default_rng(n + kl)
    ab = np.full((n, 2 * kl + ku + 1), np.nan)  # unreferenced entries may hold anything
    for j in range(n):
        i = np.arange(max(0, j - ku), min(n, j + kl + 1))
        ab[j, kl + ku + i - j] = rng.uniform(-1.0, 1.0, len(i))
        ab[j, kl + ku] = 1.5 * (kl + ku + 1)
    b = rng.normal(size=n)
    x, info = gpu_ctx.band_solve(ab, kl, ku, b)
    ref = solve_banded((kl, ku), np.nan_to_num(np.ascontiguousarray(ab[:, kl:].T)), b)
    assert info == 0 and np.abs(x - ref).max() <= 1e-13 * np.abs(ref).max()


@pytest.mark.parametrize("at", [0, 777, 1999])
def test_a_zero_pivot_is_reported(gpu_ctx, at):
    n, kl = 2000, 17
    ab = np.zeros((n, 3 * kl + 1))
    ab[:, 2 * kl] = 1.0
    ab[at, 2 * kl] = 0.0
    _, info = gpu_ctx.band_solve(ab, kl, kl, np.ones(n))
    assert info == 1


@pytest.mark.parametrize("make", [
    lambda: configs.square_plate(1, steps=2), lambda: strip(12, 3), lambda: two_plates(2, 5), lambda: loaded(9),
    lambda: configs.square_plate(13, steps=2),
], ids=["plate1", "strip12x3", "two", "loaded9", "plate13"])
def test_mixed_fronts_refine_to_the_fp64_solve(gpu_ctx, make):
    """The FP32 fronts' forward and backward sweeps against the element
    matrices' residual (and the nodal load stiffness'): the FP64 path's counts
    and, refined to the FP64 floor, its states to 1e-10 of the displacement
    scale, every solve without the FP64 fallback."""
    run = {}
    for p in (gpu.GF_PREC_MIXED, gpu.GF_PREC_FP64):
        b = gpu.BatchSolver(gpu_ctx, [make()], gpu_ctx.opts(precision=p))
        b.reset()
        b.run()
        run[p] = b.results() + (b.solve_stats(),)
        b.close()
    (fm, sm, em), (ff, sf, _) = run[gpu.GF_PREC_MIXED], run[gpu.GF_PREC_FP64]
    assert np.array_equal(sm, sf)
    scale = np.abs(ff[0][:, :3] - make().nodes).max()
    assert np.abs(fm[0][:, :3] - ff[0][:, :3]).max() <= 1e-10 * scale
    assert em[0][2] == 0 and em[0][1] >= em[0][0] > 0


@pytest.mark.parametrize("n", [28, 36])
def test_tensor_core_fronts(gpu_ctx, n):
    """Plates whose larger fronts take the tensor cores, beside a small one: the FP64 fronts' counts and states to 1e-10
    of the displacement scale (the plain path's stated tolerance), the same bits
    alone, and the mixed path's fallback still the FP64 path exactly."""
    def run(structs, **kw):
        b = gpu.BatchSolver(gpu_ctx, structs, gpu_ctx.opts(**kw))
        b.reset()
        b.run()
        out = b.results()
        b.close()
        return out

    make = lambda: configs.square_plate(n, steps=2)
    ft, st = run([configs.square_plate(5, steps=2), make()], wide_update=gpu.GF_WIDE_TENSOR)
    ff, sf = run([make()], wide_update=gpu.GF_WIDE_FP64)
    fa, _ = run([make()])
    fb, _ = run([make()], precision=gpu.GF_PREC_MIXED, max_refine=1)
    assert np.array_equal(st[1], sf[0])
    scale = np.abs(ff[0][:, :3] - make().nodes).max()
    assert np.abs(ft[1][:, :3] - ff[0][:, :3]).max() <= 1e-10 * scale
    assert np.array_equal(ft[1], fa[0]) and np.array_equal(fa[0], fb[0])


def test_tensor_core_fronts_of_a_sparse_system(gpu_ctx):
    # rows scaled over eight decades; forward error bound n eps cond with cond <= 5
    # for these row sums once the scaling is taken out: 1e-12
    g, d = 40, 3
    n = g * g * d
    x = np.arange(n) // d
    rng = np.random.default_rng(9)
    rows, cols = [], []
    for v in range(g * g):
        for a in (-1, 0, 1):
            for b in (-1, 0, 1):
                if 0 <= v % g + a < g and 0 <= v // g + b < g:
                    w = v + a + g * b
                    for i in range(d):
                        rows += [v * d + i] * d
                        cols += list(range(w * d, w * d + d))
    rows, cols = np.array(rows), np.array(cols)
    val = rng.uniform(-1.0, 1.0, len(rows))
    val[rows == cols] = 0.0
    sums = np.bincount(rows, np.abs(val), n)
    val[rows == cols] = 1.5 * sums[rows[rows == cols]] + 0.1
    val = val * 10.0 ** rng.integers(-4, 5, n)[rows]
    order = np.lexsort((cols, rows))
    rp = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))]).astype(np.int32)
    ref = rng.normal(size=n)
    b = np.zeros(n)
    np.add.at(b, rows, val * ref[cols])
    sol, info = gpu_ctx.sparse_solve(rp, cols[order].astype(np.int32), val[order], b)
    assert info == 0
    assert np.abs(sol - ref).max() <= 1e-12 * np.abs(ref).max()


@pytest.mark.parametrize("n", [1, 31, 32, 33, 64, 65, 97, 257, 600])
def test_substitution_of_one_front(gpu_ctx, n):
    # a full matrix is one front of n own DOFs: clusters of one to eight CTAs, blocks
    # of 32 with and without a remainder; diagonally dominant, forward error n eps cond
    # with cond <= 5: 1e-12
    rng = np.random.default_rng(n)
    A = rng.uniform(-1.0, 1.0, (n, n))
    A[np.arange(n), np.arange(n)] = 1.5 * np.abs(A).sum(1) + 0.1
    ref = rng.normal(size=n)
    rp = np.arange(0, n * n + 1, n, dtype=np.int32)
    sol, info = gpu_ctx.sparse_solve(rp, np.tile(np.arange(n, dtype=np.int32), n), A.ravel(), A @ ref)
    assert info == 0
    assert np.abs(sol - ref).max() <= 1e-12 * np.abs(ref).max()


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("n,copies", [(3, 160), (9, 30), (13, 12)])
def test_substitution_does_not_depend_on_the_batch(gpu_ctx, n, copies, mixed):
    # a front's CTAs follow from the fronts of its height, its bits do not
    opts = gpu_ctx.opts(precision=gpu.GF_PREC_MIXED if mixed else gpu.GF_PREC_FP64)
    out = []
    for k in (1, copies):
        b = gpu.BatchSolver(gpu_ctx, [configs.square_plate(n, steps=2)] * k, opts)
        b.reset()
        b.run()
        out.append(b.results())
        b.close()
    for q in range(copies):
        assert np.array_equal(out[0][0][0], out[1][0][q]) and np.array_equal(out[0][1][0], out[1][1][q])


def junction():
    """A plate of 2x2 squares and one of half its size beside it: a midside node of the
    coarse one's edge is a corner of the fine one's elements."""
    a, b = configs.square_plate(2, steps=2, pressure=1e3), configs.square_plate(2, side=0.5, steps=2)
    xy = [tuple(p) for p in a.nodes]
    new = []
    for p in b.nodes + [1.0, 0.0, 0.0]:
        if p[1] in (0.0, 0.25, 0.5) and p[0] == 1.0:
            new.append(xy.index(tuple(p)))
        else:
            new.append(len(xy))
            xy.append(tuple(p))
    a.nodes = np.array(xy)
    a.shells.extend([tuple(new[q] for q in row[:6]) + tuple(row[6:]) for row in b.shells])
    a.constraints = np.zeros((len(xy), 6), dtype=np.int32)
    a.constraints[(a.nodes[:, 0] == 0.0) | (a.nodes[:, 0] == 1.5) | (a.nodes[:, 1] == 0.0)] = 1
    a.loads[0].shells = list(range(len(a.shells)))
    return a


@pytest.mark.parametrize("precision", [gpu.GF_PREC_FP64, gpu.GF_PREC_MIXED])
def test_a_node_that_is_corner_and_midside(gpu_ctx, precision):
    # forces and matrices are gathered per node: a node with rotations in some of its
    # elements only
    fo, so, _ = oracle.solve(junction(), 0)
    b = gpu.BatchSolver(gpu_ctx, [junction()], gpu_ctx.opts(precision=precision))
    b.reset()
    b.run()
    finals, stats = b.results()
    b.close()
    assert tuple(stats[0]) == tuple(so)
    scale = np.abs(fo[:, :3]).max()
    assert np.abs(finals[0][:, :3] - fo[:, :3]).max() <= 1e-10 * scale
    assert np.abs(finals[0][:, 6:] - fo[:, 6:]).max() <= 1e-9


def test_more_fronts_of_a_height_than_a_grid_has_rows(gpu_ctx):
    # a band of 200,000 blocks of 33: 65,535 fronts of 99 rows and more at the lowest
    # heights, beyond the y of a grid; unit sums, so x is a sum of the row's terms exactly
    n, kl = 33 * 200000, 33
    ab = np.zeros((n, 2 * kl + 1))
    ab[:, kl] = 2.0
    ab[:, 2 * kl] = -0.5
    b = np.full(n, 1.5)
    b[:kl] = 2.0
    x, info = gpu_ctx.band_solve(ab, kl, 0, b)
    assert info == 0 and np.array_equal(x, np.ones(n))


def test_slices_hold_an_exponent_per_64_pivots(gpu_ctx):
    # two blocks of 128 pivots coupled to 128 rows: L21 is 1 over the first 64 pivots and
    # 1e-8 over the others, half of U12's columns 0 and 1e-8, so their Schur complement of
    # 1e-16 comes from the small entries alone.  An emulated product errs by 2^-52 64 max|L|
    # max|U| over 64 pivots each: 64 x 128 of it against a diagonal of 200e-16 and sums
    # below half of that, 2^-52 x 82; under one exponent for all 128 pivots 1e8 times that
    rng = np.random.default_rng(11)
    m, e = 128, 1e-8
    n = 3 * m
    A = np.eye(n)
    S, half = slice(2 * m, n), 2 * m + m // 2
    for q in range(2):
        first, last = slice(q * m, q * m + m // 2), slice(q * m + m // 2, q * m + m)
        A[S, first] = rng.uniform(-1.0, 1.0, (m, m // 2))
        A[S, last] = e * rng.uniform(-1.0, 1.0, (m, m // 2))
        A[first, 2 * m:half] = rng.uniform(-1.0, 1.0, (m // 2, m // 2))
        A[last, half:] = e * rng.uniform(-1.0, 1.0, (m // 2, m // 2))
    A[S, S] = np.diag(np.where(np.arange(m) < m // 2, 200.0, 200.0 * e * e))
    # the same system with columns and rows of like size, for the reference
    r = np.ones(n)
    c = np.ones(n)
    c[half:] = 1.0 / (e * e)
    for q in range(2):
        last = slice(q * m + m // 2, q * m + m)
        r[last], c[last] = e, 1.0 / e
    b = rng.normal(size=n)
    b /= r
    ref = np.linalg.solve(r[:, None] * A * c, r * b) * c
    rows, cols = np.nonzero(np.kron(np.array([[1, 0, 1], [0, 1, 1], [1, 1, 1]]), np.ones((m, m))))
    rp = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))]).astype(np.int32)
    x, info = gpu_ctx.sparse_solve(rp, cols.astype(np.int32), A[rows, cols], b)
    assert info == 0 and (np.abs(x - ref) / c).max() <= 1e-12 * (np.abs(ref) / c).max()


def test_a_large_system_of_wide_fronts(gpu_ctx):
    # a hundred full blocks of 530 DOFs, each coupled to the same six: fronts of more own
    # DOFs than the substitution's partial sums hold at once, with a boundary; a matrix
    # beyond the pinned staging and a workspace beyond the 512 MB that a context keeps.
    # Rows dominant by 1.5: forward error n eps cond with cond <= 5, 1e-12
    rng = np.random.default_rng(3)
    k, m, h = 100, 530, 6
    n = k * m + h
    block = rng.uniform(-1.0, 1.0, (k * m, m + h))
    own = np.arange(k * m) % m
    block[np.arange(k * m), own] = 0.0
    block[np.arange(k * m), own] = 1.5 * np.abs(block).sum(1) + 0.1
    cols = np.concatenate([np.arange(m)[None] + m * np.arange(k)[:, None], np.full((k, h), k * m) + np.arange(h)], axis=1)
    hub = rng.uniform(-1.0, 1.0, (h, n))
    hub[np.arange(h), k * m + np.arange(h)] = 0.0
    hub[np.arange(h), k * m + np.arange(h)] = 1.5 * np.abs(hub).sum(1) + 0.1
    ref = rng.normal(size=n)
    b = np.concatenate([np.einsum("kij,kj->ki", block.reshape(k, m, m + h), ref[cols]).ravel(), hub @ ref])
    ci = np.concatenate([np.repeat(cols, m, axis=0).ravel(), np.tile(np.arange(n), h)]).astype(np.int32)
    rp = np.concatenate([np.arange(k * m) * (m + h), k * m * (m + h) + np.arange(h + 1) * n]).astype(np.int32)
    A = pattern("grid", 5)
    small = (*to_csr(A), np.ones(len(A)))
    before, _ = gpu_ctx.sparse_solve(*small)
    x, info = gpu_ctx.sparse_solve(rp, ci, np.concatenate([block.ravel(), hub.ravel()]), b)
    assert info == 0 and np.abs(x - ref).max() <= 1e-12 * np.abs(ref).max()
    after, _ = gpu_ctx.sparse_solve(*small)
    assert np.array_equal(before, after)
