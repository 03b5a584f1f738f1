"""Jacobi-PCG resident on the SMs (grids of up to about 1000 nodes per SM).

Grids: one element, thin ones whose blocks own a single layer or row, ragged
splits, one near the capacity and one beyond it (which keeps the launches per
iteration).  Against the oracle's Jacobi-PCG to the same tolerance: the same
equations, so at rtol 1e-12 solutions agree to 1e-8 of the largest
displacement (the tolerance of the other solver tests).  A solve cut into
launches of 7 iterations resumes exactly: bit-identical solution and count.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid", [(1, 1, 1), (2, 1, 40), (40, 1, 1), (3, 50, 2), (17, 16, 15),
                                  (32, 16, 16), (61, 11, 7), (29, 30, 31)])
def test_matches_oracle_and_resumes(gpu, oracle, grid):
    P = oracle.Problem(*grid)
    rho = np.random.default_rng(sum(grid)).uniform(0.1, 1.0, P.nelx)
    ref, _, _ = P.solve(rho, tol=1e-12)
    G = gpu.Context(*grid)
    G.set_design(rho)
    val, info = G.solve(gpu.solve_opts(gpu.JACOBI_PCG, rtol=1e-12, maxit=20000))
    assert info.status == gpu.OK
    assert np.abs(val - ref).max() <= 1e-8 * np.abs(ref).max()
    cut, info7 = G.solve(gpu.solve_opts(gpu.JACOBI_PCG, rtol=1e-12, maxit=20000, chunk=7))
    assert info7.iterations == info.iterations
    assert np.array_equal(cut, val)


def test_cap_and_zero_load(gpu):
    G = gpu.Context(12, 6, 6)
    G.set_design(np.full(G.nelx, 0.5))
    _, info = G.solve(gpu.solve_opts(gpu.JACOBI_PCG, rtol=1e-14, maxit=3))
    assert info.status == gpu.WARN_MAXITER and info.iterations == 4
    u, info = G.solve_rhs(np.zeros(G.numeq), gpu.solve_opts(gpu.JACOBI_PCG))
    assert info.iterations == 0 and not u.any()


@pytest.mark.parametrize("grid", [(80, 40, 40), (100, 40, 33)])
def test_near_and_beyond_capacity(gpu, grid):
    """131 k nodes (886 per SM) and 141 k: the residual of the returned
    solution, by the FP64 operator, is the one the solve stopped on."""
    G = gpu.Context(*grid)
    G.set_design(np.random.default_rng(1).uniform(0.1, 0.5, G.nelx))
    val, info = G.solve(gpu.solve_opts(gpu.JACOBI_PCG, rtol=1e-9))
    f = G.fext()
    assert info.status == gpu.OK
    assert np.linalg.norm(f - G.apply_K(val)) <= 1.1e-9 * np.linalg.norm(f)
