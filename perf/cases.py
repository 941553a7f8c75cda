"""Performance cases of the framework: the calls its users make, over the
sizes the tests, the benchmark and the documented workloads use.

Five families, each through a public entry point:

* ``apply``: ``kronmult_matrix.apply`` / ``apply_euler`` of an operator in
  the connected-pair form (built from the per-1D-connection indices, on the
  device, or from the reference's expanded offsets) or in the global
  Kronecker form, FP64 and FP32 arithmetic, FP64 and FP32 vectors;
* ``line``: one application of the line preconditioner;
* ``cgs``: one classical Gram-Schmidt step over a Krylov basis;
* ``solve``: one backward-Euler solve to a 1e-10 relative residual by the
  benchmark's method (global operator, line preconditioner, FP32 operator
  inside FP64 refinement, restart 50);
* ``steps``: a few implicit time steps by plain FP64 GMRES, the reference's
  own configuration.

The operators are the two of ``SparseGridOperator``: "advdiff" (term t acts
in dimension t mod d, advection and diffusion in turn) and "random" (every
factor uniform in [-1, 1], every term acting in every dimension).
"""
import functools
import math

import numpy as np
import torch

import asgard_b200 as ab

N1 = 3          # polynomials per dimension
NU = 0.1        # diffusion coefficient of the advection/diffusion operators


def listed():
    return [
        # the smallest documented workload: a two-dimensional operator with
        # random factors, one FP64 apply (launch latency)
        {"name": "pairs_d2_l6", "call": "apply", "form": "pairs", "d": 2, "level": 6, "terms": 3,
         "kind": "random", "vectors": "f64", "precision": "fp64", "euler": False, "alpha": 1.0, "beta": 0.0},
        # reference callers that hand over the expanded offsets (iA), FP32
        # vectors as kronmult_matrix<float>, accumulating into y
        {"name": "csr_d3_l5_f32", "call": "apply", "form": "csr", "d": 3, "level": 5, "terms": 3,
         "kind": "random", "vectors": "f32", "precision": "fp32", "euler": False, "alpha": 0.7, "beta": -1.3},
        # the d=4 level-7 implicit workload's operator as the plain FP64
        # GMRES applies it, the pairs found on the device
        {"name": "grid_d4_l7", "call": "apply", "form": "grid", "d": 4, "level": 7, "terms": 4,
         "kind": "advdiff", "vectors": "f64", "precision": "fp64", "euler": True, "alpha": 1.0, "beta": 0.0},
        # six dimensions, all six terms of the largest workload
        {"name": "grid_d6_l5", "call": "apply", "form": "grid", "d": 6, "level": 5, "terms": 6,
         "kind": "advdiff", "vectors": "f64", "precision": "fp64", "euler": False, "alpha": 1.0, "beta": 0.0},
        # the global form with terms acting in every dimension
        {"name": "global_d3_l6_random", "call": "apply", "form": "global", "d": 3, "level": 6, "terms": 2,
         "kind": "random", "vectors": "f64", "precision": "fp64", "euler": False, "alpha": 1.0, "beta": 0.0},
        # the global form's FP64 residual of an implicit solve: y = b - A x
        {"name": "global_d4_l7", "call": "apply", "form": "global", "d": 4, "level": 7, "terms": 4,
         "kind": "advdiff", "vectors": "f64", "precision": "fp64", "euler": True, "alpha": -1.0, "beta": 1.0},
        # the largest workload's operator as the FP32 inner solve applies it
        {"name": "global_d6_l7_fp32", "call": "apply", "form": "global", "d": 6, "level": 7, "terms": 6,
         "kind": "advdiff", "vectors": "f64", "precision": "fp32", "euler": True, "alpha": 1.0, "beta": 0.0},
        # its preconditioner in the arithmetic of the inner solve
        {"name": "line_d6_l7_fp32", "call": "line", "d": 6, "level": 7, "terms": 6, "precision": "fp32"},
        # a Gram-Schmidt step half-way through a restart cycle of that size
        {"name": "cgs_d6_k25", "call": "cgs", "n": 11789388, "k": 25},
        # reference users' time loop: plain FP64 GMRES, two dimensions
        {"name": "steps_d2_l6", "call": "steps", "form": "pairs", "d": 2, "level": 6, "terms": 2, "steps": 4},
        # the implicit solve at the ordinary and the largest workload
        {"name": "solve_d4_l7", "call": "solve", "d": 4, "level": 7, "terms": 4, "iterations": 36},
        {"name": "solve_d6_l7", "call": "solve", "d": 6, "level": 7, "terms": 6, "iterations": 25},
    ]


def draw(rng):
    call = rng.choice(["apply"] * 7 + ["line", "cgs", "solve", "steps"])
    if call == "cgs":
        return {"call": "cgs", "n": int(math.exp(rng.uniform(math.log(2000), math.log(11789388)))),
                "k": rng.randint(1, 25)}
    if call == "steps":
        d = rng.choice([2, 3])
        return {"call": "steps", "form": "pairs", "d": d, "level": rng.randint(3, 6 if d == 2 else 5),
                "terms": d, "steps": rng.randint(1, 4)}
    if call in ("line", "solve"):
        d = rng.randint(2, 6)
        c = {"call": call, "d": d, "level": rng.randint(3, 6), "terms": d}
        if call == "line":
            c["precision"] = rng.choice(["fp64", "fp32"])
        else:
            c["iterations"] = 30
        return c
    form = rng.choice(["pairs", "pairs", "grid", "csr", "global", "global"])
    kind = rng.choice(["advdiff", "random"])
    precision = rng.choice(["fp64", "fp64", "fp32"])
    vectors = "f64" if form == "global" or precision == "fp64" else rng.choice(["f64", "f32"])
    while True:
        d, level, terms = rng.randint(2, 6), rng.randint(3, 7), rng.randint(1, 6)
        nnz = num_pairs(d, level)
        cost = nnz * terms * d * N1 ** (d + 1)      # the pair form's multiply-adds
        if form == "global" and kind == "advdiff":
            break
        # lists made on the host: what their building stays quick for
        host = {"pairs": nnz * d < 1e7, "csr": nnz * terms * d < 3e7}.get(form, True)
        if cost <= 2.2e11 and host:
            break
    return {"call": "apply", "form": form, "d": d, "level": level, "terms": terms, "kind": kind,
            "vectors": vectors, "precision": precision, "euler": vectors == "f64" and rng.random() < 0.5,
            "alpha": rng.choice([1.0, -1.0, 0.7]), "beta": rng.choice([0.0, 0.0, 1.0, -1.3])}


# ------------------------------------------------------------- preparation

@functools.lru_cache(maxsize=None)
def operator_data(d, level, terms, kind):
    """Element table and factor values, the arrays an operator is built from."""
    return ab.sparse_grid(d, level), ab.factor_values(d, level, terms, kind, NU, 1, N1)


def build(case):
    """The operator as a user's program holds it."""
    form = case.get("form", "global")
    kind = case.get("kind", "advdiff")
    d, level, terms = case["d"], case["level"], case["terms"]
    table, vA = operator_data(d, level, terms, kind)
    if form == "global":
        return ab.kronmult_matrix.from_global(d, N1, level, table, terms, vA)
    if form == "grid":
        return ab.kronmult_matrix.from_grid(d, N1, level, terms, vA)
    cells = table.shape[0]
    row_ptr, col, conn = ab.build_pairs(d, level, table)
    if form == "csr":
        return ab.kronmult_matrix.from_csr(d, N1, cells, cells, terms, row_ptr, col,
                                           ab.expand_iA(conn, d, N1, terms), vA)
    return ab.kronmult_matrix.from_conn(d, N1, cells, cells, terms, row_ptr, col, conn, vA)


def step_size(case):
    return 5e-4 if case["d"] == 6 else 1e-3


def uniform(seed, n, dtype=torch.float64, count=1):
    g = torch.Generator(device="cuda").manual_seed(seed)
    out = [torch.rand(n, dtype=torch.float64, device="cuda", generator=g) * 2 - 1 for _ in range(count)]
    return [v.to(dtype) for v in out]


def basis(case, seed):
    """k orthonormal columns (as rows) and the vector to orthogonalise."""
    n, k = case["n"], case["k"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    V = torch.zeros((k, n), dtype=torch.float64, device="cuda")
    for j in range(k):
        v = torch.rand(n, dtype=torch.float64, device="cuda", generator=g) * 2 - 1
        for _ in range(2 if j else 0):
            v -= V[:j].T @ (V[:j] @ v)
        V[j] = v / torch.linalg.vector_norm(v)
    w = torch.rand(n, dtype=torch.float64, device="cuda", generator=g) * 2 - 1
    return V, w


def size(case):
    if "n" in case:
        return case["n"]
    return operator_data(case["d"], case["level"], case["terms"],
                         case.get("kind", "advdiff"))[0].shape[0] * N1 ** case["d"]


def prepare(case, seed):
    call = case["call"]
    if call == "cgs":
        V, w = basis(case, seed)
        return {"case": case, "V": V, "w": w, "out": torch.empty_like(w), "h": torch.empty(
            case["k"], dtype=torch.float64, device="cuda")}
    mat = build(case)
    n = size(case)
    s = {"case": case, "mat": mat}
    if call == "apply":
        dtype = torch.float32 if case["vectors"] == "f32" else torch.float64
        s["x"], s["y0"] = uniform(seed, n, dtype, 2)
        s["y"] = torch.empty_like(s["x"])
    elif call == "line":
        s["pc"] = ab.JacobiPreconditioner(mat, step_size(case), kind="line")
        s["v"], = uniform(seed, n)
        s["z"] = torch.empty_like(s["v"])
    elif call == "solve":
        s["pc"] = ab.JacobiPreconditioner(mat, step_size(case), kind="line")
        s["b"], = uniform(seed, n)
        s["x"] = torch.empty_like(s["b"])
    else:
        s["x0"], s["f"] = uniform(seed, n, count=2)
        s["x"] = torch.empty_like(s["x0"])
    return s


# ------------------------------------------------------------- one pass

def run(s):
    case = s["case"]
    call = case["call"]
    if call == "apply":
        if case["beta"] != 0.0:
            s["y"].copy_(s["y0"])
        if case["euler"]:
            s["mat"].apply_euler(step_size(case), case["alpha"], s["x"], case["beta"], s["y"],
                                 precision=case["precision"])
        else:
            s["mat"].apply(case["alpha"], s["x"], case["beta"], s["y"], precision=case["precision"])
        return s["y"]
    if call == "line":
        return s["pc"].apply(s["v"], s["z"], precision=case["precision"])
    if call == "cgs":
        s["out"].copy_(s["w"])
        h, norm = ab.cgs_step(s["V"], case["k"], s["out"], s["h"])
        return {"h": h, "w": s["out"], "norm": norm}
    if call == "solve":
        s["x"].zero_()
        info = ab.simple_gmres_euler(step_size(case), s["mat"], s["x"], s["b"], restart=50, max_iter=400,
                                     tol=1e-10, tol_mode="rel", precision="fp32", precond=s["pc"])
        if info.status != 0:
            raise RuntimeError(f"the solve did not converge: {info}")
        return s["x"]
    s["x"].copy_(s["x0"])
    for info in ab.implicit_advance(step_size(case), s["mat"], s["x"], case["steps"], s["f"], restart=50,
                                    max_iter=400, tol=1e-10, tol_mode="rel"):
        if info.status != 0:
            raise RuntimeError(f"a step did not converge: {info}")
    return s["x"]


# ------------------------------------------------------------- floors

@functools.lru_cache(maxsize=None)
def connections(level):
    """connect_1d as a (cells x cells) table of connection indices, -1 where
    two 1D cells are not connected."""
    pntr, indx = ab.connect_1d(level)
    lut = np.full((len(pntr) - 1,) * 2, -1, np.int64)
    lut[np.repeat(np.arange(len(pntr) - 1), np.diff(pntr)), indx] = np.arange(len(indx))
    return lut


def level_pairs(level):
    """Connected 1D pairs by the levels of the two cells."""
    lev = np.array([0] + [int(i).bit_length() for i in range(1, 1 << level)])
    out = np.zeros((level + 1, level + 1))
    np.add.at(out, (lev[:, None].repeat(len(lev), 1), lev[None, :].repeat(len(lev), 0)), connections(level) >= 0)
    return out


def num_pairs(d, level):
    """Connected cell pairs of the sparse grid."""
    one, acc = level_pairs(level), np.ones((1, 1))
    for _ in range(d):
        new = np.zeros((level + 1, level + 1))
        for a in range(acc.shape[0]):
            for b in range(acc.shape[1]):
                new[a:, b:] += acc[a, b] * one[:level + 1 - a, :level + 1 - b]
        acc = new
    return int(acc.sum())


def line_pairs(d, level):
    """Connected cell pairs that agree outside one given dimension."""
    one = level_pairs(level)
    cells = np.array([1.0] + [2.0 ** max(l - 1, 0) for l in range(1, level + 1)])
    rest = np.ones(1)
    for _ in range(d - 1):
        rest = np.convolve(rest, cells)[:level + 1]
    return int(sum(rest[s] * one[:level + 1 - s, :level + 1 - s].sum() for s in range(len(rest))))


def work(case):
    """Inputs read once and outputs written once; a multiply-add of every 1D
    block along its own dimension once (an operator cannot do with less)."""
    call = case["call"]
    if call == "cgs":
        n, k = case["n"], case["k"]
        return {"bytes": 8 * n * (k + 2), "flops": 4 * n * k}
    d, level, terms, n = case["d"], case["level"], case["terms"], size(case)
    fibres = 2 * N1 ** (d + 1)
    single = min(terms, d) * line_pairs(d, level) * fibres    # one dimension per term, shared operators summed
    every = terms * d * line_pairs(d, level) * fibres         # every term in every dimension
    factors = 8 * terms * d * N1 * N1 * int((connections(level) >= 0).sum())
    if call == "apply":
        eb = 4 if case["vectors"] == "f32" else 8
        acts_once = case["form"] == "global" and case["kind"] == "advdiff"
        return {"bytes": eb * n * (2 + (case["beta"] != 0.0)) + factors, "flops": single if acts_once else every}
    if call == "line":
        return {"bytes": 16 * n, "flops": min(terms, d) // 2 * line_pairs(d, level) * fibres}
    if call == "solve":
        # each iteration reads and writes a vector in the operator, the
        # preconditioner and the basis, FP32 where the method holds FP32
        it = case["iterations"]
        return {"bytes": 16 * n + it * n * (8 + 8 + 4 * 2 * (it + 1) / 2), "flops": it * single}
    its = 12 * case["steps"]
    return {"bytes": 8 * n * 3 * case["steps"], "flops": its * every}


# ------------------------------------------------------------- accuracy

def tolerance(case):
    # About four times the largest difference seen against exact() and between
    # the pair and the global form (the same sums in another order) over the
    # declared ranges: FP64 applies 2e-15, FP32 9e-7, line preconditioner
    # 2.6e-14 and 2.8e-7, Gram-Schmidt 2.4e-15.  Two solutions of 1e-10
    # relative residual: 7e-11 per solve, 2.7e-10 after four time steps.
    call = case["call"]
    if call == "apply":
        return {"rel": 1e-14, "max": 1e-13} if case["precision"] == "fp64" else {"rel": 4e-6, "max": 6e-5}
    if call == "line":
        return {"rel": 1e-13} if case["precision"] == "fp64" else {"rel": 1.2e-6}
    if call == "cgs":
        return {"rel": 1e-14}
    return {"rel": 3e-10} if call == "solve" else {"rel": 1.2e-9}


class Reference:
    """The operator in plain torch, FP64, from the element table, the 1D
    connectivity and the factor values."""

    def __init__(self, case):
        self.d, self.level, self.terms = case["d"], case["level"], case["terms"]
        self.kind = case.get("kind", "advdiff")
        self.dt = step_size(case)
        table, vA = operator_data(self.d, self.level, self.terms, self.kind)
        lev, pos = table[:, :self.d].astype(np.int64), table[:, self.d:].astype(np.int64)
        self.c1 = np.where(lev == 0, 0, (1 << np.maximum(lev - 1, 0)) + pos)
        self.cells = table.shape[0]
        # (connection, term, dimension, row, column)
        self.vA = torch.from_numpy(vA.reshape(-1, self.terms, self.d, N1, N1).swapaxes(-1, -2).copy()).cuda()
        self.lut = torch.from_numpy(connections(self.level)).cuda()
        self.groups = {}

    def dims(self, t):
        return [t % self.d] if self.kind == "advdiff" else list(range(self.d))

    def operator_1d(self, k):
        """The terms acting in dimension k alone, summed: (R, R, 3, 3)."""
        R = self.lut.shape[0]
        B = torch.zeros((R, R, N1, N1), dtype=torch.float64, device="cuda")
        on = self.lut >= 0
        for t in range(self.terms):
            if self.dims(t) == [k]:
                B[on] += self.vA[self.lut[on], t, k]
        return B

    def pencils(self, k):
        """Cells that agree outside k, grouped by the 1D cells they hold:
        [(1D cells, cell table (pencils x members))]."""
        if k not in self.groups:
            others = np.delete(self.c1, k, axis=1)
            order = np.lexsort([self.c1[:, k]] + [others[:, j] for j in range(others.shape[1])])
            key = others[order]
            new = np.ones(self.cells, bool)
            new[1:] = (key[1:] != key[:-1]).any(axis=1)
            first = np.flatnonzero(new)
            sizes = np.diff(np.append(first, self.cells))
            by = {}
            for f, m in zip(first, sizes):
                mem = order[f:f + m]
                by.setdefault(tuple(self.c1[mem, k]), []).append(mem)
            self.groups[k] = [(torch.tensor(ids, device="cuda"), torch.from_numpy(np.array(c)).cuda())
                              for ids, c in by.items()]
        return self.groups[k]

    def along(self, x, k, matrix):
        """matrix(1D cells) (3m x 3m) applied along the pencils of dimension k."""
        x = x.reshape(self.cells, N1 ** k, N1, -1)
        y = torch.zeros_like(x)
        for ids, cells in self.pencils(k):
            M = matrix(ids)
            g = x[cells].permute(0, 1, 3, 2, 4)            # pencil, member, k, before, after
            p, m, _, a, b = g.shape
            out = torch.matmul(M, g.reshape(p, m * N1, a * b)).reshape(p, m, N1, a, b)
            y[cells] = out.permute(0, 1, 3, 2, 4)
        return y.reshape(-1)

    def apply(self, x):
        if self.kind == "advdiff":
            y = torch.zeros_like(x)
            for k in range(min(self.d, self.terms)):
                B = self.operator_1d(k)

                def matrix(ids):
                    m = len(ids)
                    return B[ids][:, ids].permute(0, 2, 1, 3).reshape(m * N1, m * N1)
                y += self.along(x, k, matrix)
            return y
        return self.apply_pairs(x)

    def apply_pairs(self, x):
        """Every connected pair of cells and every term, one after the other."""
        d, ts = self.d, N1 ** self.d
        c1 = torch.from_numpy(self.c1).cuda()
        xs, y = x.reshape(self.cells, ts), torch.zeros((self.cells, ts), dtype=torch.float64, device="cuda")
        step = max(1, (200_000_000 // ts) // self.cells)
        for r0 in range(0, self.cells, step):
            rows = c1[r0:r0 + step]
            on = torch.ones((len(rows), self.cells), dtype=torch.bool, device="cuda")
            for k in range(d):
                on &= self.lut[rows[:, k]][:, c1[:, k]] >= 0
            r, c = on.nonzero(as_tuple=True)
            conn = torch.stack([self.lut[rows[r, k], c1[c, k]] for k in range(d)])
            total = torch.zeros((len(r), ts), dtype=torch.float64, device="cuda")
            for t in range(self.terms):
                v = xs[c]
                for k in range(d):
                    A = self.vA[conn[k], t, k]
                    w = v.reshape(len(r), N1 ** k, N1, -1)
                    v = sum(A[:, None, :, j, None] * w[:, :, j, None, :] for j in range(N1)).reshape(len(r), ts)
                total += v
            y.index_add_(0, r + r0, total)
        return y.reshape(-1)

    def euler(self, x):
        return x - self.dt * self.apply(x)

    def solve(self, b, x, tol=1e-14, most=2000):
        """BiCGStab to a relative residual of tol (or where it stops falling)."""
        x = x.clone()
        bn = torch.linalg.vector_norm(b)
        best, at = None, math.inf
        for _ in range(4):
            r = b - self.euler(x)
            res = float(torch.linalg.vector_norm(r) / bn)
            if res < at:
                best, at = x.clone(), res
            if res < tol:
                break
            r0, p, rho = r.clone(), r.clone(), torch.dot(r, r)
            e = torch.zeros_like(x)
            stop = max(0.05 * tol / max(res, 1e-300), 1e-12) * torch.linalg.vector_norm(r)
            for _ in range(most):
                v = self.euler(p)
                alpha = rho / torch.dot(r0, v)
                s = r - alpha * v
                t = self.euler(s)
                omega = torch.dot(t, s) / torch.dot(t, t)
                e += alpha * p + omega * s
                r = s - omega * t
                if torch.linalg.vector_norm(r) <= stop:
                    break
                new = torch.dot(r0, r)
                p = r + (new / rho) * (alpha / omega) * (p - omega * v)
                rho = new
            x = x + e
        return best

    def line(self, v):
        """z = M_km^-1 B ... B M_k1^-1 v over the dimensions with a symmetric
        operator: M_k = I - dt (K_k + sum of the other ones' cell-diagonal
        parts), B = I - dt (all their cell-diagonal parts)."""
        d, dt = self.d, self.dt
        ops, eig = {}, {}
        for k in range(min(d, self.terms)):
            B = self.operator_1d(k)
            full = B.permute(0, 2, 1, 3).reshape(B.shape[0] * N1, -1)
            if torch.allclose(full, full.T, rtol=1e-10, atol=1e-10 * float(full.abs().max())):
                ops[k] = B
                lam, P = torch.linalg.eigh(B[torch.arange(B.shape[0]), torch.arange(B.shape[0])])
                eig[k] = (lam, P)

        def cellwise(x, k, M):
            c = torch.from_numpy(self.c1[:, k]).cuda()
            w = x.reshape(self.cells, N1 ** k, N1, -1)
            return torch.einsum("cij,cajb->caib", M[c], w).reshape(-1)

        def scale(x, axes, first):
            """x / (1 - dt (sum of the axes' eigenvalues)), `first` already holding the pencil's part."""
            den = first
            for j in axes:
                lam = eig[j][0][torch.from_numpy(self.c1[:, j]).cuda()]
                den = den - dt * lam.reshape(self.cells, *([1] * j), N1, *([1] * (d - 1 - j)))
            return (x.reshape(self.cells, *([N1] * d)) / den).reshape(-1)

        z = v
        for i, k in enumerate(ops):
            if i:
                z = z - dt * sum(cellwise(z, j, ops[j].diagonal(dim1=0, dim2=1).permute(2, 0, 1)) for j in ops)
            others = [j for j in ops if j != k]
            for j in others:
                z = cellwise(z, j, eig[j][1].transpose(1, 2).contiguous())
            Q, theta = {}, torch.zeros((self.cells, N1), dtype=torch.float64, device="cuda")
            for ids, cells in self.pencils(k):
                m = len(ids)
                t, q = torch.linalg.eigh(ops[k][ids][:, ids].permute(0, 2, 1, 3).reshape(m * N1, m * N1))
                Q[tuple(ids.tolist())] = q
                theta[cells] = t.reshape(1, m, N1)
            z = self.along(z, k, lambda ids: Q[tuple(ids.tolist())].T.contiguous())
            first = 1 - dt * theta.reshape(self.cells, *([1] * k), N1, *([1] * (d - 1 - k)))
            z = scale(z, others, first)
            z = self.along(z, k, lambda ids: Q[tuple(ids.tolist())])
            for j in others:
                z = cellwise(z, j, eig[j][1])
        return z


def exact(case, seed):
    """run's outputs in FP64 by plain torch."""
    call = case["call"]
    if call == "cgs":
        V, w = basis(case, seed)
        h = torch.mv(V, w)
        w = w - torch.mv(V.T, h)
        return {"h": h, "w": w, "norm": float(torch.linalg.vector_norm(w))}
    ref, n = Reference(case), size(case)
    if call == "apply":
        x, y0 = (v.double() for v in uniform(seed, n, torch.float32 if case["vectors"] == "f32"
                                             else torch.float64, 2))
        kx = ref.euler(x) if case["euler"] else ref.apply(x)
        return case["alpha"] * kx + (case["beta"] * y0 if case["beta"] != 0.0 else 0.0)
    if call == "line":
        return ref.line(uniform(seed, n)[0])
    if call == "solve":
        b, = uniform(seed, n)
        return ref.solve(b, torch.zeros_like(b))
    x, f = uniform(seed, n, count=2)
    for _ in range(case["steps"]):
        x = x + ref.dt * f
        x = ref.solve(x, x)
    return x
