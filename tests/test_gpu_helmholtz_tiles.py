"""Helmholtz filter at the edges of its tiles, 32 nodes along x by 8 (grids of up
to 8 nodes along y) or 16 (wider ones), against the oracle: tolerances as in
test_gpu_helmholtz.py."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GRIDS = [(31, 1, 9), (32, 6, 5), (40, 7, 33), (33, 8, 6), (30, 15, 4), (64, 16, 3), (3, 1, 150)]


@pytest.mark.parametrize("grid", GRIDS)
@pytest.mark.parametrize("is_sens", [False, True])
def test_tile_edges(oracle, gpu, grid, is_sens):
    G = gpu.Context(*grid, dirichlet=[], loads=[])
    G.helmholtz_setup(2.2)
    x = np.random.default_rng(sum(grid)).uniform(1e-3, 1.0, G.nelx)
    a, info = G.helmholtz_filter(x, is_sens, rtol=1e-12)
    b, its = oracle.helmholtz_filter(*grid, 2.2, x, is_sens=is_sens, tol=1e-12)
    assert info.status == 0 and info.rel_residual < 1e-12
    assert np.abs(a - b).max() <= 1e-9 * np.abs(b).max()
    assert abs(info.iterations - its) <= 2
