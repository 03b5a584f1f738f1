"""Resident Jacobi-PCG solves of several contexts at once, from several threads
(each a cooperative launch that may fill the GPU), next to loops whose OC update
is one too: every solve gives the bits it gives alone."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GRIDS = [(32, 16, 16), (48, 20, 21), (70, 30, 30), (9, 5, 4)]


def solve(gpu, c, design):
    c.set_design(design)
    u, info = c.solve(gpu.solve_opts(gpu.JACOBI_PCG, rtol=1e-10, maxit=20000))
    return u.copy(), info.iterations, info.status


def loop(gpu, c):
    c.loop_init(0.3, method="oc", filter_radius=1.5, solve=gpu.solve_opts(gpu.JACOBI_PCG))
    info = [c.loop_step() for _ in range(3)]
    return c.loop_get("x"), [i.cg_iterations for i in info], [i.status for i in info]


def test_solves_at_once(gpu):
    ctx = [gpu.Context(*g) for g in GRIDS]
    rho = [np.random.default_rng(q).uniform(0.1, 1.0, c.nelx) for q, c in enumerate(ctx)]
    jobs = [lambda c=c, r=r: solve(gpu, c, r) for c, r in zip(ctx, rho)]
    jobs += [lambda c=gpu.Context(16, 8, 8): loop(gpu, c) for _ in range(2)]
    alone = [j() for j in jobs]
    got = [[] for _ in jobs]
    failed = []

    def work(q):
        try:
            for _ in range(4):
                got[q].append(jobs[q]())
        except Exception as e:  # reported below, in the test's own thread
            failed.append((q, e))

    threads = [threading.Thread(target=work, args=(q,)) for q in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
    for a, runs in zip(alone, got):
        assert len(runs) == 4
        for r in runs:
            assert np.array_equal(r[0], a[0]) and r[1] == a[1] and r[2] == a[2]
