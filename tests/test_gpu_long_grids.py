"""Multigrid on strips with more node planes, or rows, than a launch grid's
second and third axes can number (65,535), clamped along both sides so that the
coarsest level keeps no unknown: the displacement holds K u = f, and the
loaded part agrees with a shorter strip's (the load decays within a few
cells).  Tolerances: 1e-10 is the solver's; K^-1 of a strip two cells wide
amplifies it by less than 100."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def strip(gpu, dims):
    nx, ny, nz = dims
    sides = [((1, 1, 1), (0.0, 0.0, 0.0), ((x, x), (0, ny), (0, nz))) for x in (0, nx)]
    return gpu.Context(*dims, dirichlet=sides, loads=[((0.3, 1.0, -0.5), ((1, 1), (1, 1), (1, 1)))])


@pytest.mark.parametrize("method", ["mg", "mixed"])
@pytest.mark.parametrize("dims,short", [((2, 2, 65536), (2, 2, 64)), ((2, 262144, 2), (2, 64, 2))])
def test_more_planes_than_a_grid_axis(gpu, dims, short, method):
    o = gpu.solve_opts(gpu.MG_PCG if method == "mg" else gpu.MIXED_IR, rtol=1e-10, mg_levels=2)
    sol = []  # the strip, and one of 64 planes
    for d in (dims, short):
        G = strip(gpu, d)
        G.set_design(np.full(G.nelx, 0.5))
        u, info = G.solve(o)
        assert info.status == 0
        f = G.fext()
        assert np.linalg.norm(G.apply_K(u) - f) <= 2e-10 * np.linalg.norm(f)
        sol.append(G.node_values().reshape(d[2] + 1, d[1] + 1, d[0] + 1, 3))
    cut = tuple(min(a, 16) for a in sol[1].shape[:2])
    a, b = (s[:cut[0], :cut[1]] for s in sol)
    assert np.abs(a - b).max() <= 1e-8 * np.abs(b).max()
