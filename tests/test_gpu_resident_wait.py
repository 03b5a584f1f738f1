"""A bounded wait of the resident Jacobi-PCG that runs out is reported as an
error, whichever block it happens in: the kernel is launched on a grid with one
block too few, so the neighbour of the missing tile waits for values that
nothing sends.  The sums do not need them, so block 0 finishes its one iteration
without a fault.  The wait ends by its own limit (seconds), and a launch with
all blocks on the same buffers succeeds afterwards."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SYMBOL = ("_ZN11icarat_b20011resident_cgEP11CUstream_stRKNS_12ResidentPlanERKNS_7GridDevERKNS_"
          "7KhParamIdEEPKdSD_PdSE_SE_SE_SE_SE_PNS_9CgScalarsEi")


class Plan(C.Structure):
    _fields_ = [(n, C.c_int) for n in ("BX", "BY", "S", "kc", "nbx", "nby", "nbz", "blocks")] + \
               [("smem", C.c_size_t)]


class Grid(C.Structure):
    _fields_ = [(n, C.c_int) for n in ("nx", "ny", "nz", "NX", "NY", "NZ", "numnp", "nelx")]


SCALARS = np.dtype([(n, "f8") for n in ("alpha", "beta", "zr", "zr_new", "pAp", "rr", "rnorm",
                                        "bnorm", "tol")] +
                   [(n, "i4") for n in ("iter", "maxit", "done", "status", "counter", "pad")])


def test_lost_wait_is_an_error(gpu):
    import torch
    launch = getattr(gpu.load_library(), SYMBOL)
    launch.restype = None
    grid = Grid(63, 3, 3, 64, 4, 4, 64 * 16, 63 * 9)  # eight tiles of 8 x 4 x 4 nodes along x
    cells, nodes = 10 * 6 * 6, 8 * 4 * 4
    smem = 8 * (6 * cells + 12 * nodes + 18 * 384) + 4 * (cells + 2 * nodes)
    kh = np.zeros(33)  # 1 on the diagonals of the parity blocks
    kh[[0, 3, 5, 6, 9, 11, 30, 31, 32]] = 1.0
    kh[12:30:3] = kh[14:30:3] = 1.0
    n = 3 * grid.numnp
    rng = np.random.default_rng(0)
    r0 = rng.standard_normal(n)

    def run(blocks):
        d = lambda a: torch.tensor(a, device="cuda")  # noqa: E731
        E, invd, x, r, p = d(np.ones(grid.nelx)), d(np.ones(n)), d(np.zeros(n)), d(r0), d(r0)
        z, Ap, work = d(np.zeros(n)), d(np.zeros(n)), d(np.zeros(1024))
        s = np.zeros(1, SCALARS)
        s["zr"], s["bnorm"], s["tol"], s["maxit"] = r0 @ r0, 1.0, 1e-30, 1000
        ds = torch.tensor(np.frombuffer(s.tobytes(), np.uint8).copy(), device="cuda")
        torch.cuda.synchronize()
        plan = Plan(8, 4, 4, 1, 8, 1, 1, blocks, smem)
        ptr = [C.c_void_p(t.data_ptr()) for t in (E, invd, x, r, z, Ap, p, work, ds)]
        launch(C.c_void_p(0), C.byref(plan), C.byref(grid), kh.ctypes.data_as(C.c_void_p), *ptr,
               C.c_int(1))
        torch.cuda.synchronize()
        return np.frombuffer(ds.cpu().numpy().tobytes(), SCALARS)[0], x.cpu().numpy()

    s, _ = run(7)
    assert s["status"] == gpu.ERR_CUDA and s["done"] == 1
    s, x = run(8)
    assert s["status"] == gpu.OK and s["done"] == 0 and s["iter"] == 1
    assert np.array_equal(x, s["alpha"] * r0)
