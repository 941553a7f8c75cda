"""Plans of different sizes at work in two host threads at once: each plan
sees one call at a time, and neither thread's calls fail or change because of
the other's."""
import threading
import time

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _side_by_side(jobs, seconds=2.0):
    """Runs every job over and over in a thread and on a stream of its own,
    all at the same time; each call's result must be the first one's bits."""
    import torch
    expect = [job().clone() for job in jobs]
    torch.cuda.synchronize()
    start, stop, wrong = threading.Barrier(len(jobs)), time.monotonic() + seconds, []

    def work(i):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                start.wait(10)
                while time.monotonic() < stop and not wrong:
                    if not torch.equal(jobs[i](), expect[i]):
                        wrong.append((i, "other values"))
        except Exception as e:      # the calls' own errors
            wrong.append((i, repr(e)))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join(60)
    assert not any(t.is_alive() for t in threads)
    assert not wrong, wrong


def _uniform(n, seed=0):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.rand(n, dtype=torch.float64, device="cuda", generator=g) * 2 - 1


@pytest.mark.parametrize("kernel", ["gram-schmidt step", "line factor", "generic operator"])
def test_launches_of_different_sizes(cuda, kernel):
    """One kernel at two dynamic shared-memory sizes: a size that a thread
    asks for must not take the larger one away from the other thread."""
    import asgard_b200 as ab
    import torch

    def solve_job(level, restart):
        mat = ab.SparseGridOperator(2, level, 2, kind="advdiff").kronmult_matrix()
        b = _uniform(mat.output_size())

        def job():
            x = torch.zeros_like(b)
            info = ab.simple_gmres_euler(1e-3, mat, x, b, restart, 400, 1e-10, tol_mode="rel")
            assert info.status == 0
            return x
        return job

    def line_job(level):
        mat = ab.SparseGridOperator(4, level, 4, kind="advdiff").kronmult_matrix(mode="global")
        pc = ab.JacobiPreconditioner(mat, 1e-3, kind="line")
        v = _uniform(mat.output_size())
        return lambda: pc.apply(v, torch.empty_like(v))

    def generic_job(n):
        cells = 20
        data = oracle.make_kronmult_data(2, n, cells, 2, 9)
        mat = ab.kronmult_matrix.from_csr(2, n, cells, cells, 2, data["pntr"], data["indx"], data["iA"],
                                          data["vA"])
        x = _uniform(mat.input_size())

        def job():
            y = torch.empty_like(x)
            mat.apply(1.0, x, 0.0, y)
            return y
        return job

    old = ab.gmres_settings(graphs=False)       # every step launched from the host
    try:
        if kernel == "gram-schmidt step":
            _side_by_side([solve_job(6, 200), solve_job(3, 20)])
        elif kernel == "line factor":
            _side_by_side([line_job(5), line_job(4), line_job(6)])
        else:
            _side_by_side([generic_job(8), generic_job(4)])
    finally:
        ab.gmres_settings(**old)


# (d, level, terms, vectors): pair plans whose kernels held nothing between
# calls, as lists that are applied one by one and as whole grids
SHARED = [(2, 5, 2, "f64"), (2, 7, 4, "f64"), (5, 4, 2, "f64"), (6, 4, 1, "f64"), (3, 6, 3, "f32")]


@pytest.mark.parametrize("d,L,T,vectors", SHARED)
def test_one_plan_on_two_streams(cuda, d, L, T, vectors):
    """Applies and solves of one plan that are enqueued on two streams, with
    nothing between them, give the values of one after the other."""
    import asgard_b200 as ab
    import torch
    mat = ab.SparseGridOperator(d, L, T, kind="random", seed=1).kronmult_matrix()
    dtype = torch.float32 if vectors == "f32" else torch.float64
    xs = [_uniform(mat.output_size(), s).to(dtype) for s in range(2)]
    expect = [torch.empty_like(x) for x in xs]
    for x, y in zip(xs, expect):
        mat.apply(1.0, x, 0.0, y)
    b = _uniform(mat.output_size(), 2)
    dt = 1e-3 / float(expect[0].abs().max())
    u0 = torch.zeros_like(b)
    assert ab.simple_gmres_euler(dt, mat, u0, b, 20, 40, 1e-10, tol_mode="rel").status == 0
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in xs]
    got = [[torch.empty_like(x) for _ in range(20)] for x in xs]
    u = torch.zeros_like(b)
    torch.cuda.synchronize()
    for i in range(20):
        for k in range(2):
            with torch.cuda.stream(streams[k]):
                mat.apply(1.0, xs[k], 0.0, got[k][i])
    with torch.cuda.stream(streams[0]):
        assert ab.simple_gmres_euler(dt, mat, u, b, 20, 40, 1e-10, tol_mode="rel").status == 0
    torch.cuda.synchronize()
    assert all(torch.equal(y, expect[k]) for k in range(2) for y in got[k])
    assert torch.equal(u, u0)
