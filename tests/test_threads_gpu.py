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
