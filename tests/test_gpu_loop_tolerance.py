"""MMA loops on small multigrid grids, where a solve to rtol 1e-8 takes 25 and more
iterations from the fifth step on and its iterate depends on the rounding of
every sum before it.  What holds there:

- at rtol 1e-12 the loop is the oracle's (solved to 1e-13) to 1e-10 in
  compliance and design and 1e-9 in dc/drho: solver errors of 1e-12 carried
  through six updates;
- at rtol 1e-8 compliance, design and dc/drho are as near to that as the
  reference's own solver stopped at 1e-8 comes, within a factor of 4 (the bound
  of the headline trajectory's test), and so they are when the loop is started
  again on the same context.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STEPS = 6


def rel(a, b):
    return float(np.linalg.norm(np.asarray(a) - b) / np.linalg.norm(b))


def oracle_rows(oracle, dims, R, tol):
    P = oracle.Problem(*dims)
    L = oracle.Loop(P, oracle.Filter(P, R), method="mma", x0=0.3, move=0.2, cg_tol=tol)
    rows = []
    for _ in range(STEPS):
        L.step()
        rows.append((L.scalars()["compliance"], L.get("x").copy(), L.get("dfds").copy()))
    return rows


def gpu_rows(gpu, G, R, levels, rtol):
    G.loop_init(0.3, method="mma", filter_radius=R, move=0.2,
                solve=gpu.solve_opts(gpu.MG_PCG, rtol=rtol, mg_levels=levels, warm_start=1,
                                     coarse_lag=1))
    rows = []
    for _ in range(STEPS):
        info = G.loop_step()
        assert info.status == gpu.OK and info.cg_rel_residual < rtol
        rows.append((info.compliance, G.loop_get("x"), G.loop_get("dfds")))
    return rows


def worst(rows, exact):
    d = [(abs(a[0] - b[0]) / b[0], rel(a[1], b[1]), rel(a[2], b[2])) for a, b in zip(rows, exact)]
    return np.max(d, axis=0)


@pytest.mark.parametrize("dims,R,levels", [((24, 8, 8), 1.595, 3), ((48, 16, 16), 1.746, 4)])
def test_loop_at_loose_tolerance(gpu, oracle, dims, R, levels):
    exact = oracle_rows(oracle, dims, R, 1e-13)
    G = gpu.Context(*dims)
    tight = worst(gpu_rows(gpu, G, R, levels, 1e-12), exact)
    assert tight[0] <= 1e-10 and tight[1] <= 1e-10 and tight[2] <= 1e-9, tight
    allowed = 4.0 * worst(oracle_rows(oracle, dims, R, 1e-8), exact) + 1e-12
    for _ in range(2):
        got = worst(gpu_rows(gpu, G, R, levels, 1e-8), exact)
        assert np.all(got <= allowed), (got, allowed)
