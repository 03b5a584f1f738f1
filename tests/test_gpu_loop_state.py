"""A loop's iterates depend on its own steps alone: not on an earlier loop,
solve or load cases of the same context, with the options that carry state from
one step to the next (warm_start, coarse_lag).  Same kernels on the same inputs
in the same order: compared bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def run(gpu, G, steps, grid_kw):
    opts = gpu.solve_opts(gpu.MG_PCG, rtol=1e-8, mg_levels=3, warm_start=1,
                          coarse_lag=grid_kw.get("lag", 1))
    G.loop_init(0.3, method="mma", filter_radius=grid_kw.get("radius", 1.5),
                use_threshold=grid_kw.get("threshold", False), solve=opts,
                filter=grid_kw.get("filter", "radius"))
    return finish(G, steps)


def finish(G, steps):
    info = [G.loop_step() for _ in range(steps)]
    assert all(i.status == 0 for i in info), [(i.status, i.cg_iterations) for i in info]
    return ([(i.cg_iterations, i.compliance) for i in info], G.loop_get("x"), G.loop_get("dfds"))


def same(a, b):
    assert a[0] == b[0]
    assert np.array_equal(a[1], b[1]) and np.array_equal(a[2], b[2])


# the second: six steps leave voids whose factor is no preconditioner for a
# uniform design
@pytest.mark.parametrize("dims,steps,kw", [
    ((16, 8, 8), 4, {}),
    ((48, 16, 24), 6, dict(radius=1.772, threshold=True)),
    ((16, 8, 8), 3, dict(filter="helmholtz", threshold=True)),
])
def test_second_loop_repeats_the_first(gpu, dims, steps, kw):
    G = gpu.Context(*dims)
    a = run(gpu, G, steps, kw)
    same(run(gpu, G, steps, kw), a)


def test_loop_after_a_solve_is_a_fresh_one(gpu):
    F = gpu.Context(16, 8, 8)
    a = run(gpu, F, 3, {})
    G = gpu.Context(16, 8, 8)
    G.set_design(np.random.default_rng(1).uniform(1e-4, 1.0, G.nelx))
    G.solve(gpu.solve_opts(gpu.MG_PCG, rtol=1e-8, mg_levels=3))
    same(run(gpu, G, 3, {}), a)


def test_load_cases_start_anew(gpu):
    """(coarse_lag 0: with it a later case takes the new factor as soon as the
    other stream has finished it)"""
    G = gpu.Context(16, 8, 8)
    cases = np.random.default_rng(2).standard_normal((2, G.numeq))
    G.set_load_cases(cases)
    kw = dict(lag=0, threshold=True)
    a = run(gpu, G, 3, kw)
    same(run(gpu, G, 3, kw), a)


def test_resume_on_a_used_context(gpu, tmp_path):
    """a snapshot loaded where another loop has run continues as on a new context"""
    path = str(tmp_path / "loop.bin")
    G = gpu.Context(16, 8, 8)
    run(gpu, G, 3, {})
    G.loop_save(path)
    finish(G, 3)
    G.loop_load(path)
    a = finish(G, 3)
    F = gpu.Context(16, 8, 8)
    F.loop_load(path)
    same(a, finish(F, 3))
