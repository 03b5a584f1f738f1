"""Marches with more work items than blocks: the kernels that sum partial values
launch at most 2048 blocks, each of which then takes several tiles one after
another.  A tile has at most 192 (FP64) or 256 (FP32) node columns, so a plate
of 1025 x 513 columns has more than 2048 of either.  Both plate faces are
clamped (the free middle plane makes a well-conditioned system).

The product in place takes the capped launch and must repeat the uncapped one's
bits; the solvers' solutions must have the residual they stopped on, by the
uncapped product (2 rtol: the recurrence residual the stop test reads drifts by
rounding, far below rtol = 1e-9)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NX, NY, NZ = 1024, 512, 2


@pytest.fixture(scope="module")
def plate(gpu):
    assert (NX + 1) * (NY + 1) > 2048 * 256
    faces = [((1, 1, 1), (0.0,) * 3, ((0, NX), (0, NY), (z, z))) for z in (0, NZ)]
    G = gpu.Context(NX, NY, NZ, dirichlet=faces,
                    loads=[((0.3, -1.0, 0.5), ((0, NX), (0, NY), (1, 1)))])
    G.set_design(np.random.default_rng(3).uniform(0.3, 1.0, G.nelx))
    return G


def test_product_in_place(plate):
    import torch
    u = torch.tensor(np.random.default_rng(4).standard_normal(plate.numeq), device="cuda")
    y = torch.full_like(u, float("nan"))
    torch.cuda.synchronize()
    plate.apply_K_dev(u.data_ptr(), y.data_ptr())
    plate.apply_K_dev(u.data_ptr(), u.data_ptr())
    plate.synchronize()
    assert np.array_equal(u.cpu().numpy(), y.cpu().numpy())


@pytest.mark.parametrize("method", ["JACOBI_PCG", "MG_PCG", "MIXED_IR"])
@pytest.mark.parametrize("warm", [0, 1])
def test_solvers(gpu, plate, method, warm):
    f = plate.fext()
    o = gpu.solve_opts(getattr(gpu, method), rtol=1e-9, mg_levels=2, warm_start=warm)
    rng = np.random.default_rng(5 + warm)
    if warm:  # the next design from this one's solution
        plate.set_design(rng.uniform(0.3, 1.0, plate.nelx))
        plate.solve(o)
    plate.set_design(rng.uniform(0.3, 1.0, plate.nelx))
    u, info = plate.solve(o)
    assert info.status == gpu.OK and info.iterations > 1
    assert np.linalg.norm(f - plate.apply_K(u)) <= 2e-9 * np.linalg.norm(f)
    g = rng.standard_normal(plate.numeq)
    if not warm:
        u, info = plate.solve_rhs(g, o)
        assert info.status == gpu.OK
        assert np.linalg.norm(g - plate.apply_K(u)) <= 2e-9 * np.linalg.norm(g)
