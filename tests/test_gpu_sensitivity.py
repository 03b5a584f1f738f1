"""Compliance sensitivity from the parity blocks of Ke0, against the CPU
restatement's dense element products: whole and fractional penalties (products
and pow), box elements of unequal edges, prescribed displacements, ragged element
counts.  Both sides round a form whose terms cancel by (displacement / element
strain)^2, some 1e3 here: 2.2e-16 sqrt(576) 1e3 = 5e-12, bound 1e-11."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("penalty", [1.0, 2.0, 2.5, 3.0])
@pytest.mark.parametrize("grid,size", [((1, 1, 1), (1.0, 1.0, 1.0)),
                                       ((7, 3, 5), (7.0, 3.0, 5.0)),
                                       ((9, 5, 4), (4.5, 5.0, 8.0))])
def test_sensitivity_matches_dense_products(oracle, gpu, grid, size, penalty):
    lx, ly, lz = size
    d = [((1, 1, 1), (0.0, 0.0, 0.0), ((0.0, 0.0), (0.0, ly), (0.0, lz))),
         ((0, 1, 0), (0.0, 0.02, 0.0), ((lx, lx), (0.0, ly), (0.0, lz)))]
    kw = dict(lx=lx, ly=ly, lz=lz, dirichlet=d, loads=[])
    P = oracle.Problem(*grid, penal=penalty, **kw)
    G = gpu.Context(*grid, penalty=penalty, **kw)
    rho = np.random.default_rng(len(grid) + grid[0]).uniform(0.05, 1.0, P.nelx)
    G.set_design(rho)
    G.solve(gpu.solve_opts(rtol=1e-12))
    dfds, dgds = G.sensitivity(0.5)
    rdf, rdg = P.sensitivity(rho, G.node_values(), 0.5)
    assert np.linalg.norm(dfds - rdf) <= 1e-11 * np.linalg.norm(rdf)
    assert np.array_equal(dgds, rdg)
