"""Order of the coarsest level's direct solver: K_c x = b through W^T W for
trees of 0 to 5 levels of separators, one to many 64-column steps, and planes of
unequal size (point supports).  ||b - K_c x|| is bounded by about eps times the
condition number, at most some 1e8 for the longest beam here, times ||b||:
1e-7; an entry in the wrong place gives O(1)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("galerkin", [0, 1])
@pytest.mark.parametrize("grid", [
    (2, 2, 2),      # one coarse element: one leaf
    (4, 2, 2),      # two planes: still one leaf
    (6, 4, 4),      # three planes: two leaves and a separator
    (8, 18, 8),     # y longest, leaves of one and two planes
    (14, 8, 30),    # z longest, planes of 120: two steps each
    (60, 6, 2),     # planes of 24
    (80, 2, 2),     # planes of 12, several per leaf
    (130, 2, 4),
])
def test_tree_of_planes(gpu, grid, galerkin):
    G = gpu.Context(*grid)
    G.set_design(np.random.default_rng(sum(grid)).uniform(0.3, 1.0, G.nelx))
    if galerkin:  # one product on the coarsest level builds that hierarchy
        o = gpu.solve_opts(gpu.MG_PCG, mg_levels=2, coarse_op=gpu.COARSE_GALERKIN)
        G.mg_level_apply(1, np.zeros(3 * int(np.prod([q // 2 + 1 for q in grid]))), o)
    rel, n = G.coarse_check(2)
    assert n > 0 and rel <= 1e-7, (rel, n)


def test_planes_of_unequal_size(gpu):
    # single supports in the middle of the body: no plane is constrained whole
    nx, ny, nz = 24, 8, 8
    at = [(0, 0, 0), (12, 8, 8), (24, 0, 8), (12, 0, 0)]
    d = [((1, 1, 1), (0.0, 0.0, 0.0), tuple((p, p) for p in q)) for q in at]
    lo = [((0.0, 0.0, -1.0), ((nx / 2, nx / 2), (ny / 2, ny / 2), (nz, nz)))]
    G = gpu.Context(nx, ny, nz, dirichlet=d, loads=lo)
    G.set_design(np.random.default_rng(3).uniform(0.3, 1.0, G.nelx))
    rel, n = G.coarse_check(2)
    assert n == 3 * (13 * 5 * 5 - 4) and rel <= 1e-7
