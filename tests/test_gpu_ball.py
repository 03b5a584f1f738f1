"""The radius filter and the OC bisection on compiled balls (radii up to 3
voxels) against the oracle, which sums the reference's neighbour list.

Radii: one of every ball (squared radius in voxels 1, 2, 3, 4, 5, 6, 8, 9) and
one beyond them; grids: one tile of 32 x 8 x 4 elements and its edges, thin in
each axis, ragged, and enough elements that the ball is taken (1e5 taps).
Filters: bit-exact, as the reference sums them.  OC: the same bisection steps
(the volume sum differs by rounding) and densities to 1e-12.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RADII = [1.0, 1.5, 1.8, 2.0, 2.3, 2.5, 2.9, 3.0, 3.2]
GRIDS = [(32, 8, 64), (33, 9, 61), (129, 41, 3), (3, 70, 80), (95, 2, 90), (64, 33, 9)]


@pytest.mark.parametrize("grid", GRIDS)
@pytest.mark.parametrize("R", RADII)
def test_filters_bit_exact(gpu, oracle, grid, R):
    P = oracle.Problem(*grid)
    F = oracle.Filter(P, R)
    G = gpu.Context(*grid)
    G.filter_setup(R)
    rng = np.random.default_rng(int(10 * R) + grid[0])
    x = rng.uniform(0.0, 1.0, P.nelx)
    g = rng.standard_normal(P.nelx) * 10.0 ** rng.uniform(-6.0, 6.0, P.nelx)
    assert np.array_equal(G.density_filter(x), F.density_filter(x))
    assert np.array_equal(G.density_filter(g, True), F.density_filter(g, True))


@pytest.mark.parametrize("R", [1.5, 2.5, 3.0])
def test_selection_bit_exact(gpu, oracle, R):
    """removed elements of an L-bracket are nobody's neighbour"""
    from oracle import submesh as S
    N, T, NZ = 36, 12, 10
    boxes = [((0, N), (0, T), (0, NZ)), ((0, T), (0, N), (0, NZ))]
    d = [((1, 1, 1), (0.0, 0.0, 0.0), ((0, T), (N, N), (0, NZ)))]
    loads = [((0.0, -1.0, 0.0), ((N, N), (T / 2, T / 2), (NZ / 2, NZ / 2)))]
    Q = S.SelProblem(N, N, NZ, boxes, d, loads)
    G = gpu.Context(N, N, NZ, dirichlet=d, loads=loads, selection=boxes)
    F = oracle.Filter(centroids=Q.centroids, radius=R)
    G.filter_setup(R)
    x = np.random.default_rng(4).uniform(0.0, 1.0, Q.nelx)
    assert np.array_equal(G.density_filter(x), F.density_filter(x))
    assert np.array_equal(G.density_filter(x, True), F.density_filter(x, True))


@pytest.mark.parametrize("grid", [(33, 9, 13), (5, 3, 2), (70, 20, 21)])
@pytest.mark.parametrize("R", [1.0, 2.5, 3.0, 3.2])
def test_oc_matches_oracle(gpu, oracle, grid, R):
    P = oracle.Problem(*grid)
    F = oracle.Filter(P, R)
    G = gpu.Context(*grid)
    G.filter_setup(R)
    rng = np.random.default_rng(grid[0])
    x = rng.uniform(0.2, 0.6, P.nelx)
    df, dg = -rng.uniform(0.1, 3.0, P.nelx), np.ones(P.nelx)
    lo, hi = np.full(P.nelx, 1e-4), np.ones(P.nelx)
    a, sa = oracle.oc_update(x, df, 0.4 * P.nelx, dg, lo, hi,
                             lambda xk: F.density_filter(xk).sum())
    b, sb = G.oc_update(x, df, 0.4 * P.nelx, dg, lo, hi)
    assert sa == sb
    assert np.abs(b - a).max() <= 1e-12 * np.abs(a).max()
