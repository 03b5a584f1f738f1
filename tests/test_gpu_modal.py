"""The parity-block stiffness march at the edges of its tiles.

A block takes W x H <= 192 (FP64) or 256 (FP32) element columns with sides of
at most 32, and a z chunk of one or more layers: grids of one element, of one
tile less, exactly and more, thin in each axis, and one with more tiles than
reduction blocks (the blocks then loop).  Reference: the oracle's assembled
K u; for the largest grid (whose FP64 launch is capped at the reduction
blocks) the FP32 product, whose launch is not, to its rounding.
Tolerances (max |y - y_ref| / max |y_ref|): FP64 sums of 24 products per row
and 8 elements in another order, 1e-14; FP32 rounding of Ke0, E, u and the
sums, 1e-6.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GRIDS = [(1, 1, 1), (1, 40, 2), (2, 2, 70), (15, 12, 1), (16, 11, 5), (17, 3, 33), (31, 5, 4),
         (32, 6, 7), (33, 31, 2), (64, 12, 13), (70, 33, 3)]


@pytest.mark.parametrize("grid", GRIDS)
@pytest.mark.parametrize("lengths", [(1.0, 1.0, 1.0), (1.5, 0.7, 2.0)])
def test_product_matches_oracle(gpu, oracle, grid, lengths):
    nx, ny, nz = grid
    box = dict(lx=nx * lengths[0], ly=ny * lengths[1], lz=nz * lengths[2])
    bc = gpu.cantilever_bc(nx, ny, nz, **box)
    P = oracle.Problem(nx, ny, nz, dirichlet=bc[0], loads=bc[1], **box)
    G = gpu.Context(nx, ny, nz, dirichlet=bc[0], loads=bc[1], **box)
    rng = np.random.default_rng(nx + 100 * ny + 10000 * nz)
    rho = rng.uniform(0.05, 1.0, P.nelx)
    u = rng.standard_normal(P.numeq)
    P.assemble(rho)
    G.set_design(rho)
    ref = P.apply_K(u)
    top = np.abs(ref).max()
    assert np.abs(G.apply_K(u) - ref).max() <= 1e-14 * top
    assert np.abs(G.apply_K_op(u, gpu.OP_FP32) - ref).max() <= 1e-6 * top


def test_more_tiles_than_blocks(gpu):
    G = gpu.Context(1100, 420, 1)
    rng = np.random.default_rng(7)
    G.set_design(rng.uniform(0.05, 1.0, G.nelx))
    u = rng.standard_normal(G.numeq)
    ref = G.apply_K_op(u, gpu.OP_FP32)
    assert np.abs(G.apply_K(u) - ref).max() <= 1e-6 * np.abs(ref).max()


def test_equation_vectors_partly_fixed_nodes(gpu, oracle):
    """nodes with one, two or all components fixed on four faces, device
    pointers, and the product in place (which keeps the scattered form)"""
    import torch
    nx, ny, nz = 21, 13, 17
    faces = [((1, 1, 1), (0.0,) * 3, ((0.0, 0.0), (0.0, ny), (0.0, nz))),
             ((0, 1, 0), (0.0,) * 3, ((0.0, nx), (0.0, 0.0), (0.0, nz))),
             ((1, 0, 1), (0.0,) * 3, ((0.0, nx), (ny, ny), (0.0, nz))),
             ((0, 0, 1), (0.0,) * 3, ((nx, nx), (0.0, ny), (0.0, 0.0)))]
    loads = [((0.0, 0.0, -1.0), ((nx, nx), (6.0, 6.0), (9.0, 9.0)))]
    P = oracle.Problem(nx, ny, nz, dirichlet=faces, loads=loads)
    G = gpu.Context(nx, ny, nz, dirichlet=faces, loads=loads)
    rng = np.random.default_rng(2)
    rho, u = rng.uniform(0.05, 1.0, P.nelx), rng.standard_normal(P.numeq)
    P.assemble(rho)
    G.set_design(rho)
    ref = P.apply_K(u)
    d_u = torch.tensor(u, device="cuda")
    d_y = torch.full_like(d_u, float("nan"))
    torch.cuda.synchronize()
    G.apply_K_dev(d_u.data_ptr(), d_y.data_ptr())
    G.synchronize()
    top = np.abs(ref).max()
    assert np.abs(d_y.cpu().numpy() - ref).max() <= 1e-14 * top
    assert np.abs(G.apply_K(u) - ref).max() <= 1e-14 * top
    G.apply_K_dev(d_u.data_ptr(), d_u.data_ptr())
    G.synchronize()
    assert np.array_equal(d_u.cpu().numpy(), d_y.cpu().numpy())
