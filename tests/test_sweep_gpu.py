"""Pair plans of a whole grid run as a tree of 1D passes: every form such a
list can come in, and lists that are not quite a grid's, against the oracle.

FP64 within 1e-13 relative (L2), FP32 within 1e-5, the bars of the pair
kernels (test_kronmult_gpu.py).  Where only the tree or its chains run, FP32
within TREE_FP32: a value meets the rounding of x, of d factors and of at most
2 d - 1 stored passes and their sums, some 4 d roundings of u = 2^-24, and
independent roundings add up like a random walk, to sqrt(4 d) u <= 5 u (seen:
1.5e-7 to 2.6e-7); the bar is 12 u."""
import numpy as np
import pytest

import oracle
from conftest import rel_err

pytestmark = pytest.mark.gpu

TREE_FP32 = 12 * 2.0 ** -24

# (d, level, terms): pairs x terms on both sides of each dimension's line
# (400 thousand for d <= 3, 262144 for d = 4, 65536 for d = 5, 163840 above;
# half as much again in FP32), pencils of 1 to 128 cells
LEAST = {2: 400000, 3: 400000, 4: 262144, 5: 65536, 6: 163840}
CASES = [(2, 7, 2), (2, 7, 3), (2, 7, 5), (3, 6, 1), (3, 6, 2), (4, 4, 7), (4, 5, 1), (4, 5, 2),
         (5, 3, 7), (5, 4, 1), (6, 3, 3), (6, 3, 6), (6, 4, 1)]


def _dev(a, dtype=None):
    import torch
    t = torch.from_numpy(np.ascontiguousarray(a))
    return (t if dtype is None else t.to(dtype)).cuda()


def _apply(mat, alpha, x, beta, y, precision="fp64", dtype=None):
    import torch
    xd, yd = _dev(x, dtype), _dev(y, dtype)
    mat.apply(alpha, xd, beta, yd, precision=precision)
    torch.cuda.synchronize()
    return yd.double().cpu().numpy()


def _expect(op, row_ptr, col, conn, alpha, x, beta, y):
    import asgard_b200 as ab
    return oracle.kronmult(op.d, 3, row_ptr.astype(np.int32), col, op.terms,
                           ab.expand_iA(conn, op.d, 3, op.terms), op.vA, alpha, x, beta, y.copy())


@pytest.mark.parametrize("d,L,T", CASES)
def test_forms_of_a_whole_grid(cuda, d, L, T):
    import asgard_b200 as ab
    import torch
    op = ab.SparseGridOperator(d, L, T, kind="random", seed=d)
    rng = np.random.default_rng(L)
    x, y0 = rng.uniform(-1, 1, op.N), rng.uniform(-1, 1, op.N)
    expect = _expect(op, op.row_ptr, op.col, op.conn, 0.7, x, -1.3, y0)
    conn = op.kronmult_matrix()
    got = _apply(conn, 0.7, x, -1.3, y0)
    assert rel_err(got, expect) < 1e-13
    low = TREE_FP32 if op.nnz * T >= LEAST[d] * 3 // 2 else 1e-5
    assert rel_err(_apply(conn, 0.7, x, -1.3, y0, "fp32"), expect) < low
    assert rel_err(_apply(conn, 0.7, x, -1.3, y0, "fp32", torch.float32), expect) < low
    assert conn.num_pairs() == op.nnz and conn.kind() == "sparse"
    # the same grid found on the device and behind the reference's offsets
    assert np.array_equal(_apply(ab.kronmult_matrix.from_grid(d, 3, L, T, op.vA), 0.7, x, -1.3, y0), got)
    csr = op.kronmult_matrix(expanded=True)
    assert np.array_equal(_apply(csr, 0.7, x, -1.3, y0), got)
    # beta = 0 overwrites y, an x that is only 8-byte aligned, the Euler form
    buf = torch.zeros(op.N + 1, dtype=torch.float64, device="cuda")
    buf[1:] = _dev(x)
    yd = torch.full((op.N,), float("nan"), dtype=torch.float64, device="cuda")
    conn.apply_euler(1e-3, -1.0, buf[1:], 0.0, yd)
    kx = _expect(op, op.row_ptr, op.col, op.conn, 1.0, x, 0.0, np.zeros(op.N))
    assert rel_err(yd.cpu().numpy(), -(x - 1e-3 * kx)) < 1e-13
    # new values
    v2 = op.vA[::-1].copy()
    for mat in (conn, csr):
        mat.update_stored_coefficients(v2)
    op.vA = v2
    assert rel_err(_apply(conn, 1.0, x, 0.0, y0),
                   _expect(op, op.row_ptr, op.col, op.conn, 1.0, x, 0.0, y0)) < 1e-13
    assert np.array_equal(_apply(csr, 1.0, x, 0.0, y0), _apply(conn, 1.0, x, 0.0, y0))


def _relabel(op, perm):
    """The pair list with cell i renamed perm[i], rows in the new order, the
    columns of a row shuffled."""
    rows = np.repeat(np.arange(op.rows), np.diff(op.row_ptr))
    r, c = perm[rows], perm[op.col]
    order = np.lexsort((np.random.default_rng(1).permutation(len(r)), r))
    ptr = np.concatenate([[0], np.cumsum(np.bincount(r, minlength=op.rows))]).astype(np.int64)
    return ptr, c[order].astype(np.int32), op.conn[order]


@pytest.mark.parametrize("change", ["relabelled", "pair dropped", "pair twice", "pair moved",
                                    "cells dropped", "other connection"])
@pytest.mark.parametrize("d,L,T", [(3, 6, 2), (4, 5, 2)])
def test_lists_beside_a_whole_grid(cuda, d, L, T, change):
    """A grid in any cell order is still a grid; a list with a pair or coarse
    cells missing, a pair twice, or a pair that uses other factors than its
    cells' is computed as it is given."""
    import asgard_b200 as ab
    op = ab.SparseGridOperator(d, L, T, kind="random", seed=1)
    ptr, col, conn = op.row_ptr, op.col, op.conn
    cells = op.rows
    if change == "relabelled":
        ptr, col, conn = _relabel(op, np.random.default_rng(0).permutation(op.rows))
    elif change == "cells dropped":
        # without the cells of level 0 in dimension 0 but the finest others
        keep = ~((op.table[:, 0] == 0) & (op.table[:, 1:d].sum(axis=1) > 1))
        new = np.cumsum(keep) - 1
        rows = np.repeat(np.arange(op.rows), np.diff(ptr))
        on = keep[rows] & keep[col]
        cells = int(keep.sum())
        ptr = np.concatenate([[0], np.cumsum(np.bincount(new[rows[on]], minlength=cells))]).astype(np.int64)
        col, conn = new[col[on]].astype(np.int32), conn[on]
    else:
        at = int(ptr[5]) + 3
        ptr, col, conn = ptr.copy(), col.copy(), conn.copy()
        if change == "pair dropped":
            col, conn = np.delete(col, at), np.delete(conn, at, axis=0)
            ptr[6:] -= 1
        elif change == "pair twice":
            col[at], conn[at] = col[at + 1], conn[at + 1]
        elif change == "pair moved":
            col[at] = (col[at] + 1) % cells
        else:
            conn[at, d - 1] = (conn[at, d - 1] + 1) % len(ab.connect_1d(L)[1])
    rng = np.random.default_rng(2)
    N = cells * 3 ** d
    x, y0 = rng.uniform(-1, 1, N), rng.uniform(-1, 1, N)
    mat = ab.kronmult_matrix.from_conn(d, 3, cells, cells, T, ptr, col, conn, op.vA)
    expect = _expect(op, ptr, col, conn, -0.5, x, 2.0, y0)
    assert rel_err(_apply(mat, -0.5, x, 2.0, y0), expect) < 1e-13
    assert rel_err(_apply(mat, -0.5, x, 2.0, y0, "fp32"), expect) < 1e-5
    csr = ab.kronmult_matrix.from_csr(d, 3, cells, cells, T, ptr, col,
                                      ab.expand_iA(conn, d, 3, T), op.vA)
    assert rel_err(_apply(csr, -0.5, x, 2.0, y0), expect) < 1e-13


def test_not_finite_input_reaches_connected_cells_only(cuda):
    """An infinity or NaN in x shows in the rows of the cells connected to its
    cell and in no other, as over the pair list."""
    import asgard_b200 as ab
    op = ab.SparseGridOperator(4, 5, 2, kind="random", seed=4)
    mat = op.kronmult_matrix()
    rows = np.repeat(np.arange(op.rows), np.diff(op.row_ptr))
    rng = np.random.default_rng(3)
    base = rng.uniform(-1, 1, op.N)
    clean = _apply(mat, 1.0, base, 0.0, np.zeros(op.N))
    for bad in (np.inf, np.nan):
        for cell in (0, op.rows // 2, op.rows - 1):
            x = base.copy()
            x[cell * 81 + 40] = bad
            y = _apply(mat, 1.0, x, 0.0, np.zeros(op.N)).reshape(op.rows, 81)
            hit = np.zeros(op.rows, bool)
            hit[rows[op.col == cell]] = True
            assert not np.isfinite(y[hit]).any()
            assert np.array_equal(y[~hit].ravel(), clean.reshape(op.rows, 81)[~hit].ravel())


def test_dense_form_and_capture(cuda):
    """The dense form of a grid, and an apply inside a captured graph."""
    import asgard_b200 as ab
    import torch
    op = ab.SparseGridOperator(3, 6, 1, kind="random", seed=2)
    dense = op.kronmult_matrix(mode="dense")
    x = np.random.default_rng(5).uniform(-1, 1, op.N)
    expect = _expect(op, op.row_ptr, op.col, op.conn, 1.0, x, 0.0, np.zeros(op.N))
    assert dense.is_dense() and dense.num_pairs() == op.rows ** 2
    assert rel_err(_apply(dense, 1.0, x, 0.0, np.zeros(op.N)), expect) < 1e-13
    xd, yd = _dev(x), torch.zeros(op.N, dtype=torch.float64, device="cuda")
    dense.apply(1.0, xd, 0.0, yd)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        dense.apply(1.0, xd, 0.0, yd)
    x2 = np.random.default_rng(6).uniform(-1, 1, op.N)
    xd.copy_(_dev(x2))
    g.replay()
    torch.cuda.synchronize()
    assert np.array_equal(yd.cpu().numpy(), _apply(dense, 1.0, x2, 0.0, np.zeros(op.N)))


@pytest.mark.parametrize("d,L,T,precision,tree", [
    (2, 7, 2, "fp64", False), (2, 7, 3, "fp64", True), (2, 7, 3, "fp32", False), (2, 7, 4, "fp32", True),
    (4, 4, 6, "fp64", False), (4, 5, 1, "fp64", True), (4, 5, 1, "fp32", False), (5, 3, 6, "fp64", False),
    (5, 4, 1, "fp64", True), (5, 4, 1, "fp32", True), (6, 3, 6, "fp64", False), (6, 3, 6, "fp32", False),
    (6, 4, 1, "fp64", True), (6, 4, 1, "fp32", True)])
def test_lists_that_take_the_tree(cuda, d, L, T, precision, tree):
    """The grids on either side of each line: a launch per pass with the tree,
    the pair kernel (and the copy of x at d = 4) below it."""
    import asgard_b200 as ab
    import torch
    mat = ab.kronmult_matrix.from_grid(d, 3, L, T, ab.factor_values(d, L, T, "random"))
    x = torch.zeros(mat.output_size(), dtype=torch.float64, device="cuda")
    y = torch.empty_like(x)
    before = ab.launch_count()
    mat.apply(1.0, x, 0.0, y, precision=precision)
    launches = ab.launch_count() - before
    assert launches > d if tree else launches <= (2 if d == 4 else 1)


@pytest.mark.parametrize("d,L,T", [(2, 2, 1), (2, 4, 3), (2, 5, 1), (2, 9, 1), (2, 9, 2), (3, 3, 1), (3, 4, 1),
                                   (3, 5, 2), (4, 3, 2), (5, 3, 1), (5, 4, 1), (6, 3, 1), (6, 4, 1)])
def test_pair_kernels_beside_a_whole_grid(cuda, d, L, T):
    """Lists with one pair dropped, from a few cells to several thousand: the
    pair kernels with every number of warps per cell, FP64, FP32 and FP32
    vectors, against the oracle."""
    import asgard_b200 as ab
    import torch
    op = ab.SparseGridOperator(d, L, T, kind="random", seed=1)
    at = int(op.row_ptr[1]) - 1
    ptr = op.row_ptr.copy()
    ptr[1:] -= 1
    col, conn = np.delete(op.col, at), np.delete(op.conn, at, axis=0)
    mat = ab.kronmult_matrix.from_conn(d, 3, op.rows, op.rows, T, ptr, col, conn, op.vA)
    rng = np.random.default_rng(L)
    x, y0 = rng.uniform(-1, 1, op.N), rng.uniform(-1, 1, op.N)
    expect = _expect(op, ptr, col, conn, 0.7, x, -1.3, y0)
    assert rel_err(_apply(mat, 0.7, x, -1.3, y0), expect) < 1e-13
    assert rel_err(_apply(mat, 0.7, x, -1.3, y0, "fp32"), expect) < 1e-5
    assert rel_err(_apply(mat, 0.7, x, -1.3, y0, "fp32", torch.float32), expect) < 1e-5


def test_expanded_list_without_a_tree_holds_no_factor_copies(cuda):
    """The whole connectivity of a grid that is not closed below runs on the
    pair kernels; as an expanded list it holds what a list with a pair missing
    holds, but for that pair."""
    import asgard_b200 as ab
    d, L, T = 4, 6, 1
    op = ab.SparseGridOperator(d, L, T, kind="random", seed=1)
    keep = ~((op.table[:, 0] == 0) & (op.table[:, 1:d].sum(axis=1) > 1))
    new = np.cumsum(keep) - 1
    rows = np.repeat(np.arange(op.rows), np.diff(op.row_ptr))
    on = keep[rows] & keep[op.col]
    cells = int(keep.sum())
    ptr = np.concatenate([[0], np.cumsum(np.bincount(new[rows[on]], minlength=cells))]).astype(np.int64)
    col, conn = new[op.col[on]].astype(np.int32), op.conn[on]
    assert len(col) * T >= 262144       # enough pairs for the tree

    def plan(ptr, col, conn):
        return ab.kronmult_matrix.from_csr(d, 3, cells, cells, T, ptr, col, ab.expand_iA(conn, d, 3, T), op.vA)
    less = ptr.copy()
    less[1:] -= 1
    at = int(ptr[1]) - 1
    mat = plan(ptr, col, conn)
    missing = plan(less, np.delete(col, at), np.delete(conn, at, axis=0))
    assert mat.device_bytes() == missing.device_bytes() + 4 * (1 + T * d)
    rng = np.random.default_rng(2)
    x, y0 = rng.uniform(-1, 1, cells * 81), rng.uniform(-1, 1, cells * 81)
    expect = _expect(op, ptr, col, conn, -0.5, x, 2.0, y0)
    assert rel_err(_apply(mat, -0.5, x, 2.0, y0), expect) < 1e-13


@pytest.mark.parametrize("d,L,T", [(6, 6, 1), (6, 4, 6)])
def test_tree_that_goes_depth_first(cuda, d, L, T):
    """Terms acting in every dimension on grids whose vectors of a whole tree
    would not fit the tree's memory: one term's branches one after the other
    (64 vectors of 31 MB), and one term after the other (384 of 2.9 MB).
    Rows of every level against the oracle, FP64 and FP32."""
    import asgard_b200 as ab
    import torch
    op = ab.SparseGridOperator(d, L, T, kind="random", seed=d)
    mat = ab.kronmult_matrix.from_grid(d, 3, L, T, op.vA)
    rows = np.unique(np.concatenate([[0, op.rows - 1], np.random.default_rng(0).integers(0, op.rows, 30)]))
    at = np.concatenate([np.arange(op.row_ptr[r], op.row_ptr[r + 1]) for r in rows])
    ptr = np.concatenate([[0], np.cumsum(np.diff(op.row_ptr)[rows])])
    x = np.random.default_rng(1).uniform(-1, 1, op.N)
    expect = _expect(op, ptr, op.col[at], op.conn[at], 1.0, x, 0.0, np.zeros(len(rows) * 3 ** d))
    xd, yd = _dev(x), torch.empty(op.N, dtype=torch.float64, device="cuda")
    for precision, bar in (("fp64", 1e-13), ("fp32", TREE_FP32)):
        before = ab.launch_count()
        mat.apply(1.0, xd, 0.0, yd, precision=precision)
        # a tree whose levels are one launch each takes 2 d - 1, and the sum
        assert ab.launch_count() - before > 2 * d
        assert rel_err(yd.reshape(op.rows, -1)[_dev(rows)].cpu().numpy().ravel(), expect) < bar
