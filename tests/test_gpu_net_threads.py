"""Two nets trained from two threads at once, the first use of their kernels
included, give the losses and gradients they give alone (every sum has a fixed
order: bit for bit)."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def train(gpu, seed, grid, out):
    G = gpu.Context(*grid)
    rng = np.random.default_rng(seed)
    rho, f, u = rng.uniform(0.1, 1.0, G.nelx), G.fext(), rng.standard_normal(G.numeq)
    net = gpu.Net(seed=seed)
    for _ in range(3):
        out.append((net.train_step(G, rho, f, u, 1e-4), net.grads().copy()))


def test_two_nets_at_once(gpu):
    jobs = [(1, (24, 9, 13)), (2, (15, 15, 7))]
    at_once = [[], []]
    threads = [threading.Thread(target=train, args=(gpu, s, g, o))
               for (s, g), o in zip(jobs, at_once)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for (s, g), got in zip(jobs, at_once):
        alone = []
        train(gpu, s, g, alone)
        assert len(got) == 3
        for a, b in zip(got, alone):
            assert a[0] == b[0] and np.array_equal(a[1], b[1])
