"""Gradients of the network on grids whose levels cut the backward kernels'
16 x 4 x 4 voxel tiles everywhere: extents that are not multiples of the tile,
levels of one or a few voxels, one tile and many.

The weights are sparse powers of two and the inputs few-bit values, so every
forward sum is exact in FP32 and the GPU's BF16 activations are the numpy
oracle's bit for bit (with dense random weights a sum next to a rounding
boundary rounds either way and moves whole layers' gradients by per cent).
What remains is the FP32 rounding of the backward sums, up to 1e4 terms a sum
(about 1e-6) through 14 layers: 1e-4 per layer, L2 relative.
"""
import numpy as np
import pytest
from test_gpu_net import NO, layer_slices, oracle_sample

pytestmark = pytest.mark.gpu


def exact_weights(rng):
    """three power-of-two weights per output channel, mostly positive"""
    parts = []
    for ci, co, k in NO.LAYERS:
        w = np.zeros((co, ci * k ** 3), dtype=np.float32)
        for o in range(co):
            at = rng.choice(ci * k ** 3, size=3, replace=False)
            w[o, at] = rng.choice([1.0, 0.5, 0.5, -0.5], size=3)
        parts += [w.ravel(), np.zeros(co, dtype=np.float32)]
    return np.concatenate(parts)


@pytest.mark.parametrize("grid", [(15, 7, 7), (23, 9, 17), (40, 5, 20), (33, 16, 8)])
def test_gradients_match_oracle(gpu, grid):
    G = gpu.Context(*grid)
    rng = np.random.default_rng(sum(grid))
    rho = rng.choice([0.25, 0.5, 0.75, 1.0], size=G.nelx)
    f = np.zeros(G.numeq)
    f[rng.choice(G.numeq, size=256, replace=False)] = rng.choice([-1.0, 1.0], size=256)
    u = rng.standard_normal(G.numeq)
    net = gpu.Net(seed=5)
    w = exact_weights(rng)
    net.set_params(w)
    loss = net.train_step(G, rho, f, u, 0.0)
    g = net.grads()
    xin, t, m = oracle_sample(G, rho, f, u)
    loss_ref, g_ref, _ = NO.loss_and_grads(w, xin, t, m, bf=True)
    assert abs(loss - loss_ref) <= 1e-5 * loss_ref
    for i, sl in enumerate(layer_slices()):
        a, b = g[sl].astype(np.float64), g_ref[sl].astype(np.float64)
        assert np.linalg.norm(b) > 0.0
        assert np.linalg.norm(a - b) <= 1e-4 * np.linalg.norm(b), i
    # repeated: bit-identical (every sum has a fixed order)
    net.train_step(G, rho, f, u, 0.0)
    assert np.array_equal(net.grads(), g)
