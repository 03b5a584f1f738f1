"""The work this framework is used for, case by case, through its public entry points.

Every case is a voxel cantilever (x = 0 face clamped, point load on the right face)
as the tests, the bench and the reference's samples use it: the stiffness product, the
density filters, one linear analysis with its sensitivities in FP64 and in mixed
precision, whole runs of the optimisation loops, a batch of designs and one training
step of the preconditioner network.

listed() names the cases, draw() gives others of the same ranges, prepare() makes what a
program holds before the call, run() is one pass, work() the bytes and operations a pass
cannot do without, exact() the same outputs from plain torch in 64 bits.
"""
import math

import numpy as np
import torch

import icarat2_b200 as G

DEV = "cuda"
YOUNG, POISSON, PENALTY = (1e-9, 1.0), 0.3, 3.0


def _case(name, kind, nx, ny, nz, **kw):
    return dict(name=name, kind=kind, nx=nx, ny=ny, nz=nz, **kw)


def listed():
    return [
        # one K u on the reference's small OC sample: three launches, latency only
        _case("ku_32x16x16", "ku", 32, 16, 16),
        # one K u on the grid of the reference's largest sample: ragged in every axis
        _case("ku_250x50x50", "ku", 250, 50, 50),
        # density filter of the design and transposed filter of its sensitivities
        _case("filter_128x64x64", "filter", 128, 64, 64, radius=2.5),
        # the same pair by the Helmholtz equation, the bench's grid
        _case("helm_256x128x128", "helm", 256, 128, 128, radius=2.0),
        # the OC sample from its start: Jacobi-PCG to 1e-10, bisection over the filter
        _case("oc_32x16x16", "loop", 32, 16, 16, method="oc", filter="radius", radius=1.5,
              threshold=False, solver="jacobi", levels=0, rtol=1e-10, galerkin=False, loads=1,
              steps=10),
        # the MMA loop the bench's headline times, from its start
        _case("mma_128x64x64", "loop", 128, 64, 64, method="mma", filter="radius", radius=2.5,
              threshold=False, solver="mg", levels=4, rtol=1e-8, galerkin=False, loads=1,
              steps=6),
        # several load cases, Helmholtz filter, threshold, Galerkin coarse operators
        _case("loads3_128x64x64", "loop", 128, 64, 64, method="mma", filter="helmholtz",
              radius=2.0, threshold=True, solver="mg", levels=4, rtol=1e-8, galerkin=True,
              loads=3, steps=4),
        # a linear analysis and its sensitivities on a new design, host arrays in and out:
        # Jacobi-PCG where the divisions do not halve (a third of the largest sample),
        # multigrid and mixed precision on the bench's largest grid
        _case("jacobi_125x25x25", "analysis", 125, 25, 25, solver="jacobi", levels=0, rtol=1e-8),
        _case("mg_256x128x128", "analysis", 256, 128, 128, solver="mg", levels=6, rtol=1e-8),
        _case("mixed_256x128x128", "analysis", 256, 128, 128, solver="mixed", levels=6,
              rtol=1e-10),
        # designs of even and uneven sizes solved together
        _case("batch_64x32x32", "batch", 64, 32, 32, designs=10, method="mixed", levels=4,
              rtol=1e-10),
        # one optimiser step of the network on one sample (a warm-up learning rate)
        _case("train_96x48x48", "train", 96, 48, 48, lr=1e-6),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _any_grid(rng, most):
    """Divisions of any size, odd ones among them, elongated along x."""
    n = int(_log(rng, 8, most))
    return max(4, int(n * rng.uniform(0.8, 1.0))), max(3, int(n * rng.uniform(0.2, 0.55))), \
        max(3, int(n * rng.uniform(0.2, 0.55)))


def _mg_grid(rng, levels, most):
    """Divisions a multigrid of that many levels can halve."""
    s = 2 ** (levels - 1)
    a = max(4, int(_log(rng, 4 * s, most)) // s)
    b = max(2, int(a * rng.uniform(0.3, 0.55)))
    c = max(2, int(a * rng.uniform(0.3, 0.55)))
    return a * s, b * s, c * s


def draw(rng):
    kind = rng.choice(["ku", "ku", "filter", "filter", "helm", "oc", "mma", "loads", "jacobi", "mg",
                       "mixed", "batch", "train"])
    if kind == "ku":
        nx, ny, nz = _any_grid(rng, 256)
        return dict(kind="ku", nx=nx, ny=ny, nz=nz)
    if kind == "filter":
        nx, ny, nz = _any_grid(rng, 200)
        return dict(kind="filter", nx=nx, ny=ny, nz=nz, radius=round(rng.uniform(1.5, 3.0), 3))
    if kind == "helm":
        nx, ny, nz = _any_grid(rng, 256)
        return dict(kind="helm", nx=nx, ny=ny, nz=nz, radius=round(rng.uniform(1.0, 3.0), 3))
    if kind == "oc":
        nx, ny, nz = _any_grid(rng, 40)
        return dict(kind="loop", nx=nx, ny=ny, nz=nz, method="oc", filter="radius",
                    radius=round(rng.uniform(1.5, 3.0), 3), threshold=rng.random() < 0.5,
                    solver="jacobi", levels=0, rtol=1e-10, galerkin=False, loads=1,
                    steps=rng.choice([4, 6, 10]))
    if kind == "mma":
        levels = rng.choice([3, 4])
        nx, ny, nz = _mg_grid(rng, levels, 8 * 2 ** levels)
        return dict(kind="loop", nx=nx, ny=ny, nz=nz, method="mma", filter="radius",
                    radius=round(rng.uniform(1.5, 3.0), 3), threshold=rng.random() < 0.5,
                    solver="mg", levels=levels, rtol=1e-8, galerkin=False, loads=1,
                    steps=rng.choice([3, 4, 6]))
    if kind == "loads":
        levels = rng.choice([3, 4])
        nx, ny, nz = _mg_grid(rng, levels, 6 * 2 ** levels)
        return dict(kind="loop", nx=nx, ny=ny, nz=nz, method="mma", filter="helmholtz",
                    radius=round(rng.uniform(1.0, 2.5), 3), threshold=True, solver="mg",
                    levels=levels, rtol=1e-8, galerkin=rng.random() < 0.5,
                    loads=rng.choice([2, 3]), steps=rng.choice([2, 4]))
    if kind == "jacobi":
        nx, ny, nz = _any_grid(rng, 100)
        return dict(kind="analysis", nx=nx, ny=ny, nz=nz, solver="jacobi", levels=0, rtol=1e-8)
    if kind in ("mg", "mixed"):
        levels = rng.choice([3, 4, 5])
        nx, ny, nz = _mg_grid(rng, levels, min(192, 9 * 2 ** levels))
        return dict(kind="analysis", nx=nx, ny=ny, nz=nz, solver=kind, levels=levels,
                    rtol=1e-8 if kind == "mg" else 1e-10)
    if kind == "batch":
        levels = rng.choice([3, 4])
        nx, ny, nz = _mg_grid(rng, levels, 64)
        return dict(kind="batch", nx=nx, ny=ny, nz=nz, designs=rng.randint(3, 10),
                    method=rng.choice(["mixed", "mg"]), levels=levels, rtol=1e-10)
    nx = int(_log(rng, 24, 97))
    ny, nz = (int(nx * rng.uniform(0.3, 0.5)) for _ in range(2))
    return dict(kind="train", nx=nx, ny=ny, nz=nz, lr=1e-6)


# ------------------------------------------------------------------ inputs
def _dims(case):
    return case["nx"], case["ny"], case["nz"]


def _load_nodes(case, rng, count):
    """Nodes of the right face the loads act on."""
    nx, ny, nz = _dims(case)
    return [(nx, int(rng.integers(0, ny + 1)), int(rng.integers(0, nz + 1))) for _ in range(count)]


def _bc(dims, node):
    return G.cantilever_bc(*dims, load_node=node)


def _context(case, node):
    dirichlet, loads = _bc(_dims(case), node)
    return G.Context(*_dims(case), young=YOUNG, poisson=POISSON, penalty=PENALTY,
                     dirichlet=dirichlet, loads=loads)


def _pinned(n):
    return torch.empty(max(n, 1), dtype=torch.float64, pin_memory=True).numpy()


def _opts(case, **kw):
    method = {"jacobi": G.JACOBI_PCG, "mg": G.MG_PCG, "mixed": G.MIXED_IR}[case["solver"]]
    return G.solve_opts(method, rtol=case["rtol"], mg_levels=case["levels"] or 4, **kw)


def _batch_problems(case, rng):
    """The listed grid for two designs of three, half of it (as far as its levels allow)
    for the others, loads uniform over the right face, densities U[0.1, 0.5]."""
    problems, s = [], 2 ** (case["levels"] - 1)
    for q in range(case["designs"]):
        dims = _dims(case)
        if q % 3 == 2:
            dims = tuple(max(s, v // (2 * s) * s) for v in dims)
        node = _load_nodes(dict(nx=dims[0], ny=dims[1], nz=dims[2]), rng, 1)[0]
        nelx = dims[0] * dims[1] * dims[2]
        problems.append((dims, node, rng.uniform(0.1, 0.5, nelx)))
    return problems


def _inputs(case, seed):
    """What both prepare() and exact() start from, from the seed alone (host arrays)."""
    rng = np.random.default_rng(seed)
    nx, ny, nz = _dims(case)
    nelx, numnp, numeq = nx * ny * nz, (nx + 1) * (ny + 1) * (nz + 1), 3 * nx * (ny + 1) * (nz + 1)
    kind = case["kind"]
    d = {"node": (nx, ny // 2, 0)}
    if kind == "ku":
        d["rho"], d["u"] = rng.uniform(0.1, 0.5, nelx), rng.standard_normal(numeq)
    elif kind in ("filter", "helm"):
        d["x"], d["df"] = rng.uniform(1e-4, 1.0, nelx), -rng.exponential(1.0, nelx)
    elif kind == "loop":
        d["nodes"] = _load_nodes(case, rng, case["loads"])
        d["node"] = d["nodes"][0]
        d["x0"] = np.full(nelx, 0.3)
    elif kind == "analysis":
        d["node"] = _load_nodes(case, rng, 1)[0]
        d["rho"] = rng.uniform(0.1, 0.5, nelx)
    elif kind == "batch":
        d["problems"] = _batch_problems(case, rng)
    elif kind == "train":
        d["rho"], d["u"] = rng.uniform(0.1, 0.5, nelx), rng.standard_normal(numeq)
        d["node"] = _load_nodes(case, rng, 1)[0]
        d["net_seed"] = int(seed) % 100000
    d.update(nelx=nelx, numnp=numnp, numeq=numeq)
    return d


def prepare(case, seed):
    d = _inputs(case, seed)
    kind = case["kind"]
    s = {"case": case}
    if kind == "batch":
        B = G.Batch([dims + _bc(dims, node) for dims, node, _ in d["problems"]], young=YOUNG,
                    poisson=POISSON, penalty=PENALTY)
        s["batch"], s["rho"] = B, [rho for _, _, rho in d["problems"]]
        s["opts"] = B.opts(rtol=case["rtol"], mg_levels=case["levels"],
                           method=G.MIXED_IR if case["method"] == "mixed" else G.MG_PCG)
        return s
    c = s["ctx"] = _context(case, d["node"])
    if kind == "ku":
        c.set_design(d["rho"])
        s["u"] = torch.tensor(d["u"], device=DEV)
        s["y"] = torch.empty_like(s["u"])
    elif kind in ("filter", "helm"):
        (c.filter_setup if kind == "filter" else c.helmholtz_setup)(case["radius"])
        s["x"], s["df"] = torch.tensor(d["x"], device=DEV), torch.tensor(d["df"], device=DEV)
        s["xf"], s["dff"] = torch.empty_like(s["x"]), torch.empty_like(s["x"])
    elif kind == "loop":
        s["x0"] = d["x0"]
        if case["loads"] > 1:
            cases = []
            for node in d["nodes"]:  # one unit load each, in the equation numbering
                f = np.zeros(c.numeq)
                f[_equation(case, node, 2)] = -1.0
                cases.append(f)
            c.set_load_cases(np.array(cases))
        mg = case["solver"] == "mg"
        s["opts"] = _opts(case, warm_start=int(mg), coarse_lag=int(mg),
                          coarse_op=G.COARSE_GALERKIN if case["galerkin"]
                          else G.COARSE_REDISCRETISED)
    elif kind == "analysis":
        s["rho"] = _pinned(c.nelx)
        s["rho"][:] = d["rho"]
        s["val"], s["sens"] = _pinned(c.numeq), (_pinned(c.nelx), _pinned(c.nelx))
        s["opts"] = _opts(case)
    else:  # train
        s["net"] = G.Net(seed=d["net_seed"])
        s["rho"], s["f"], s["u"] = d["rho"], c.fext(), d["u"]
    torch.cuda.synchronize()
    return s


def _equation(case, node, comp):
    """Equation number of a free component (x = 0 nodes carry none)."""
    nx, ny, _ = _dims(case)
    return 3 * ((node[0] - 1) + nx * (node[1] + (ny + 1) * node[2])) + comp


# ------------------------------------------------------------------ one pass
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "batch":
        B = s["batch"]
        for q, rho in enumerate(s["rho"]):
            B[q].set_design(rho)
        B.solve(s["opts"])
        return [B.solution(q) for q in range(len(B))]
    c = s["ctx"]
    if kind == "ku":
        c.apply_K_dev(s["u"].data_ptr(), s["y"].data_ptr())
        return s["y"]
    if kind == "filter":
        _filter_dev(c, s["x"], s["xf"], 0)
        _filter_dev(c, s["df"], s["dff"], 1)
        return s["xf"], s["dff"]
    if kind == "helm":
        c.helmholtz_filter_dev(s["x"].data_ptr(), s["xf"].data_ptr())
        c.helmholtz_filter_dev(s["df"].data_ptr(), s["dff"].data_ptr(), is_sens=True)
        return s["xf"], s["dff"]
    if kind == "loop":
        c.loop_init(s["x0"], method=case["method"], filter_radius=case["radius"],
                    use_threshold=case["threshold"], solve=s["opts"], filter=case["filter"])
        steps = [c.loop_step() for _ in range(case["steps"])]
        return {"x": c.loop_get("x"), "dfds": c.loop_get("dfds"),
                "compliance": [i.compliance for i in steps]}
    if kind == "analysis":
        c.set_design(s["rho"])
        val, _ = c.solve(s["opts"], out=s["val"])
        dfds, dgds = c.sensitivity(out=s["sens"])
        return {"val": val, "dfds": dfds, "dgds": dgds, "compliance": c.compliance()}
    loss = s["net"].train_step(c, s["rho"], s["f"], s["u"], case["lr"])
    return {"loss": loss, "grads": s["net"].grads(), "params": s["net"].params()}


def _filter_dev(c, x, out, is_sens):
    """icarat_density_filter_dev on device tensors."""
    st = c.lib.icarat_density_filter_dev(c.h, x.data_ptr(), out.data_ptr(), is_sens)
    if st < 0:
        raise G.IcaratError(st, "density_filter_dev")


# ------------------------------------------------------------------ least work
_NET = ((4, 16), (16, 16), (16, 32), (32, 32), (32, 64), (64, 64), (64, 128), (128, 128),
        (192, 64), (64, 64), (96, 32), (32, 32), (48, 16), (16, 16))
_NET_LEVEL = (0, 0, 1, 1, 2, 2, 3, 3, 2, 2, 1, 1, 0, 0)


def work(case):
    """Inputs read once and outputs written once; the element products of one K u
    (1152 per element); for the network the three passes of its convolutions.  A
    solve's iterations are the solver's business and are not counted."""
    nx, ny, nz = _dims(case)
    nelx, ndof = nx * ny * nz, 3 * (nx + 1) * (ny + 1) * (nz + 1)
    kind = case["kind"]
    if kind == "ku":
        return {"bytes": 16.0 * ndof + 8.0 * nelx, "flops": 1152.0 * nelx}
    if kind == "filter":
        reach = (4.0 / 3.0) * math.pi * case["radius"] ** 3
        return {"bytes": 32.0 * nelx, "flops": 4.0 * reach * nelx}
    if kind == "helm":
        return {"bytes": 32.0 * nelx, "flops": 2 * 54.0 * nelx}
    if kind == "loop":
        n = case["steps"] * case["loads"]
        return {"bytes": n * (24.0 * ndof + 40.0 * nelx), "flops": n * 3 * 1152.0 * nelx}
    if kind == "analysis":
        return {"bytes": 16.0 * ndof + 24.0 * nelx, "flops": 2 * 1152.0 * nelx}
    if kind == "batch":
        return {"bytes": case["designs"] * (16.0 * ndof + 8.0 * nelx),
                "flops": case["designs"] * 1152.0 * nelx}
    pad = [-(-(v + 1) // 8) * 8 for v in (nx, ny, nz)]
    flops = sum(3 * 2 * 27.0 * ci * co * pad[0] * pad[1] * pad[2] / 8 ** lv
                for (ci, co), lv in zip(_NET, _NET_LEVEL))
    return {"bytes": 16.0 * ndof + 8.0 * nelx + 20.0 * sum(27 * a * b for a, b in _NET),
            "flops": flops}


# ------------------------------------------------------------------ 64-bit answers
def _corner(a):
    return a & 1, (a >> 1) & 1, (a >> 2) & 1


def _unit_stiffness():
    """24 x 24 stiffness of the unit cube at E = 1 (2 x 2 x 2 Gauss points), corners in
    bit order x + 2 y + 4 z."""
    lam = POISSON / ((1 + POISSON) * (1 - 2 * POISSON))
    mu = 0.5 / (1 + POISSON)
    D = np.zeros((6, 6))
    D[:3, :3] = lam
    D[range(3), range(3)] += 2 * mu
    D[range(3, 6), range(3, 6)] = mu
    K = np.zeros((24, 24))
    g = 0.5 / math.sqrt(3.0)
    for ip in range(8):
        p = [0.5 + (g if b else -g) for b in _corner(ip)]
        B = np.zeros((6, 24))
        for a in range(8):
            s = _corner(a)
            f = [p[d] if s[d] else 1 - p[d] for d in range(3)]
            df = [1.0 if s[d] else -1.0 for d in range(3)]
            gx, gy, gz = df[0] * f[1] * f[2], f[0] * df[1] * f[2], f[0] * f[1] * df[2]
            B[:, 3 * a:3 * a + 3] = [[gx, 0, 0], [0, gy, 0], [0, 0, gz], [gy, gx, 0],
                                     [0, gz, gy], [gz, 0, gx]]
        K += B.T @ D @ B / 8
    return K


def _device():
    return DEV if torch.cuda.is_available() else "cpu"


def _views(t, dims):
    """The 8 corner slices of a node field [..., z, y, x]."""
    nx, ny, nz = dims
    for a in range(8):
        ax, ay, az = _corner(a)
        yield t[..., az:az + nz, ay:ay + ny, ax:ax + nx]


class _Elastic:
    """K, solves and sensitivities of one design, fields [3, z, y, x]."""

    def __init__(self, dims, rho):
        self.dims = nx, ny, nz = dims
        self.K0 = torch.tensor(_unit_stiffness(), device=_device())
        self.rho = torch.as_tensor(rho, dtype=torch.float64, device=_device()).reshape(nz, ny, nx)
        rp = self.rho ** PENALTY
        self.E = (1 - rp) * YOUNG[0] + rp * YOUNG[1]
        self.shape = (3, nz + 1, ny + 1, nx + 1)

    def gather(self, u):
        return torch.cat(list(_views(u, self.dims))).reshape(24, -1)

    def scatter(self, f):
        out = torch.zeros(self.shape, dtype=torch.float64, device=f.device)
        for a, v in enumerate(_views(out, self.dims)):
            v += f[3 * a:3 * a + 3].reshape((3,) + tuple(self.E.shape))
        return out

    def apply(self, u):
        y = self.scatter((self.K0 @ self.gather(u)) * self.E.reshape(1, -1))
        y[..., 0] = 0
        return y

    def solve(self, f):
        d = self.scatter(torch.diagonal(self.K0)[:, None] * self.E.reshape(1, -1))
        m = 1 / d
        m[..., 0] = 0
        x, r = torch.zeros_like(f), f.clone()
        z = m * r
        p, zr, stop = z.clone(), (z * r).sum(), 1e-13 * f.norm()
        for it in range(20000):
            q = self.apply(p)
            al = zr / (p * q).sum()
            x += al * p
            r -= al * q
            if it % 20 == 0 and r.norm() < stop:
                break
            z = m * r
            new = (z * r).sum()
            p = z + (new / zr) * p
            zr = new
        return x

    def energy(self, u):
        U = self.gather(u)
        return (U * (self.K0 @ U)).sum(0).reshape(self.E.shape)

    def dfds(self, u):
        return -PENALTY * self.rho ** (PENALTY - 1) * (YOUNG[1] - YOUNG[0]) * self.energy(u)

    def load(self, node):
        f = torch.zeros(self.shape, dtype=torch.float64, device=_device())
        f[2, node[2], node[1], node[0]] = -1.0
        return f

    def field(self, numeq):
        nx, ny, nz = self.dims
        u = torch.zeros(self.shape, dtype=torch.float64, device=_device())
        t = torch.as_tensor(numeq, device=_device()).reshape(nz + 1, ny + 1, nx, 3)
        u[..., 1:] = t.permute(3, 0, 1, 2)
        return u

    @staticmethod
    def numeq(u):
        return u[..., 1:].permute(1, 2, 3, 0).reshape(-1)


class _Radius:
    """The radius filter and its transpose on [z, y, x] fields."""

    def __init__(self, dims, R):
        r = math.ceil(R)
        self.taps = [(dz, dy, dx, R - math.sqrt(dx * dx + dy * dy + dz * dz))
                     for dz in range(-r, r + 1) for dy in range(-r, r + 1)
                     for dx in range(-r, r + 1) if math.sqrt(dx * dx + dy * dy + dz * dz) <= R]
        self.r = r
        self.sum = self.conv(torch.ones(dims[::-1], dtype=torch.float64, device=_device()))

    def conv(self, x):
        r, (nz, ny, nx) = self.r, x.shape
        p = torch.nn.functional.pad(x, (r,) * 6)
        return sum(w * p[r + dz:r + dz + nz, r + dy:r + dy + ny, r + dx:r + dx + nx]
                   for dz, dy, dx, w in self.taps)

    def forward(self, x):
        return self.conv(x) / self.sum

    def back(self, x):
        return self.conv(x / self.sum)


def _helmholtz(dims, R, s, sens):
    """The nodal Helmholtz solve by Jacobi-PCG to the last bits."""
    nx, ny, nz = dims
    m1, s1 = np.array([[2.0, 1.0], [1.0, 2.0]]) / 6, np.array([[1.0, -1.0], [-1.0, 1.0]])
    c = (R / (2 * math.sqrt(3.0))) ** 2

    def kron(a, b, d):  # corner bit order: z slowest
        return np.kron(d, np.kron(b, a))

    Ke = kron(m1, m1, m1) + c * (kron(s1, m1, m1) + kron(m1, s1, m1) + kron(m1, m1, s1))
    Ke = torch.tensor(Ke, device=_device())
    shape = (nz + 1, ny + 1, nx + 1)

    def scatter(f):
        out = torch.zeros(shape, dtype=torch.float64, device=_device())
        for a, v in enumerate(_views(out, dims)):
            v += f[a].reshape(nz, ny, nx)
        return out

    def apply(p):
        return scatter(Ke @ torch.stack(list(_views(p, dims))).reshape(8, -1))

    # integrals of the shape functions: 1/8 of the element each, their Gauss sums 1
    b = scatter(s.reshape(1, -1).expand(8, -1) / 8) / (8 if sens else 1)
    d = scatter(torch.diagonal(Ke)[:, None].expand(8, s.numel()))
    x, r = torch.zeros_like(b), b.clone()
    z = r / d
    p, zr = z.clone(), (z * r).sum()
    for _ in range(500):
        q = apply(p)
        al = zr / (p * q).sum()
        x += al * p
        r -= al * q
        if r.norm() < 1e-15 * b.norm():
            break
        z = r / d
        new = (z * r).sum()
        p = z + (new / zr) * p
        zr = new
    return sum(_views(x, dims)) / (1 if sens else 8)


def _exact_oc(case, d):
    """The OC loop without a threshold or with it, radius filter, one load."""
    dims = _dims(case)
    F = _Radius(dims, case["radius"])
    x = torch.full(dims[::-1], 0.3, dtype=torch.float64, device=_device())
    beta, T, move = 1.0, 0.5, 0.15

    def project(t):
        if not case["threshold"]:
            return t
        return 0.5 * (math.tanh(T * beta) + torch.tanh(beta * (t - T))) / math.tanh(T * beta)

    V0, comp, df = None, [], None
    for _ in range(case["steps"]):
        xf = F.forward(x)
        E = _Elastic(dims, project(xf))
        f = E.load(d["node"])
        u = E.solve(f)
        comp.append(float((u * f).sum()))
        V0 = float(E.rho.sum()) if V0 is None else V0
        thr = 0.5 * beta * (1 - torch.tanh(beta * (xf - T)) ** 2) / math.tanh(T * beta) \
            if case["threshold"] else torch.ones_like(xf)
        df, dg = F.back(E.dfds(u) * thr), F.back(thr)
        lo = torch.maximum(torch.full_like(x, 1e-4), (1 - move) * x)
        hi = torch.minimum(torch.ones_like(x), (1 + move) * x)
        l0, l1, new, it = 0.0, 1e4, torch.zeros_like(x), 0
        while (l1 - l0) / (l1 + l0) > 1e-5 and it < 100:
            lam = 0.5 * (l0 + l1)
            new = torch.sqrt(torch.clamp(-df / (dg * lam), min=0)) * x
            new = torch.minimum(torch.maximum(new, lo), hi)
            if float(project(F.forward(new)).sum()) - V0 > 0:
                l0 = lam
            else:
                l1 = lam
            it += 1
        x = new
    return {"x": x.reshape(-1), "dfds": df.reshape(-1), "compliance": comp}


def _exact_train(case, d):
    """Loss and gradients of the network with its BF16 storage (weights and activations
    rounded to nearest) and every sum in 64 bits; the first update's weights are not given
    (a step of Adam divides by the gradient's own size)."""
    dims = _dims(case)
    nx, ny, nz = dims
    dev = _device()
    net = G.Net(seed=d["net_seed"])
    flat = torch.tensor(net.params(), device=dev)
    net.close()

    class Round(torch.autograd.Function):  # storage rounding, gradient passed through
        @staticmethod
        def forward(ctx, t):
            return t.to(torch.bfloat16).to(torch.float64)

        @staticmethod
        def backward(ctx, g):
            return g

    sizes = [(co, ci, 3) for ci, co in _NET] + [(3, 16, 1)]
    W, o = [], 0
    for co, ci, k in sizes:
        n = co * ci * k ** 3
        w = flat[o:o + n].reshape(co, ci, k, k, k).to(torch.bfloat16).double().requires_grad_()
        b = flat[o + n:o + n + co].double().requires_grad_()
        W.append((w, b))
        o += n + co
    pad = [-(-(v + 1) // 8) * 8 - (v + 1) for v in (nx, ny, nz)]
    pads = (0, pad[0], 0, pad[1], 0, pad[2])
    f = np.zeros(d["numeq"])
    f[_equation(case, d["node"], 2)] = -1.0
    E = _Elastic(dims, d["rho"])
    ones = torch.ones((nz, ny, nx), dtype=torch.float64, device=dev)

    def nodal(t):
        out = torch.zeros(E.shape[1:], dtype=torch.float64, device=dev)
        for v in _views(out, dims):
            v += t
        return out

    node_rho = (nodal(E.rho) / nodal(ones)).float().double()
    x = torch.cat([E.field(f), node_rho[None]])[None]
    x = torch.nn.functional.pad(Round.apply(x), pads)

    def conv(i, t):
        w, b = W[i]
        out = 0  # tap by tap: a double convolution as 27 matrix products
        p = torch.nn.functional.pad(t, (1,) * 6)
        Z, Y, X = t.shape[2:]
        for tap in range(27):
            dz, dy, dx = tap // 9, tap // 3 % 3, tap % 3
            out = out + torch.einsum("oc,czyx->ozyx", w[:, :, dz, dy, dx],
                                     p[0, :, dz:dz + Z, dy:dy + Y, dx:dx + X])
        return Round.apply(torch.relu(out + b[:, None, None, None]))[None]

    def pool(t):
        return Round.apply(torch.nn.functional.avg_pool3d(t, 2))

    def up(t):
        return t.repeat_interleave(2, 2).repeat_interleave(2, 3).repeat_interleave(2, 4)

    s0 = conv(1, conv(0, x))
    s1 = conv(3, conv(2, pool(s0)))
    s2 = conv(5, conv(4, pool(s1)))
    b3 = conv(7, conv(6, pool(s2)))
    d2 = conv(9, conv(8, torch.cat([up(b3), s2], 1)))
    d1 = conv(11, conv(10, torch.cat([up(d2), s1], 1)))
    d0 = conv(13, conv(12, torch.cat([up(d1), s0], 1)))
    w, b = W[14]
    y = torch.einsum("oc,czyx->ozyx", w[:, :, 0, 0, 0], d0[0]) + b[:, None, None, None]
    y = y[:, :nz + 1, :ny + 1, 1:nx + 1]
    t = E.field(d["u"])[..., 1:]
    yt, yy, tt = (y * t).sum(), (y * y).sum(), (t * t).sum()
    loss = 1 - yt * yt / (yy * tt) + 1e-2 * (yy - 1) ** 2
    loss.backward()
    grads = torch.cat([torch.cat([w.grad.reshape(-1), b.grad.reshape(-1)]) for w, b in W])
    return {"loss": float(loss), "grads": grads, "params": None}


def exact(case, seed):
    d = _inputs(case, seed)
    kind, dims = case["kind"], _dims(case)
    dev = _device()
    if kind == "ku":
        E = _Elastic(dims, d["rho"])
        return E.numeq(E.apply(E.field(d["u"])))
    if kind in ("filter", "helm"):
        x, df = (torch.tensor(d[k], device=dev).reshape(dims[::-1]) for k in ("x", "df"))
        if kind == "filter":
            F = _Radius(dims, case["radius"])
            return F.forward(x).reshape(-1), F.back(df).reshape(-1)
        return tuple(_helmholtz(dims, case["radius"], t, sens).reshape(-1)
                     for t, sens in ((x, False), (df, True)))
    if kind == "analysis":
        E = _Elastic(dims, d["rho"])
        f = E.load(d["node"])
        u = E.solve(f)
        return {"val": E.numeq(u), "dfds": E.dfds(u).reshape(-1),
                "dgds": torch.ones(d["nelx"], dtype=torch.float64), "compliance":
                float((u * f).sum())}
    if kind == "batch":
        out = []
        for bdims, node, rho in d["problems"]:
            E = _Elastic(bdims, rho)
            out.append(E.numeq(E.solve(E.load(node))))
        return out
    if kind == "train":
        return _exact_train(case, d)
    if case["method"] == "oc":
        return _exact_oc(case, d)
    return None  # the MMA loops: a dual interior-point solve per step
