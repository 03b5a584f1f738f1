"""K u on equation vectors where nodes keep some of their components: every
combination of free components in one grid, on the whole box and on a
selection with removed nodes, against the scattered form (the product in place
takes it).  The same sums in both: bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 9


def clamped_lines():
    """node lines along z, the eight combinations in turn over (x, y)"""
    lines = []
    for x in range(N + 1):
        for y in range(N + 1):
            q = (x + 3 * y) % 8
            flag = tuple((q >> k) & 1 for k in range(3))
            if any(flag):
                lines.append((flag, (0.0,) * 3, ((x, x), (y, y), (0, N))))
    return lines


@pytest.mark.parametrize("selection", [None, [((0, N), (0, 4), (0, N)), ((0, 4), (0, N), (0, N))]])
def test_equation_form_is_the_scattered_form(gpu, selection):
    import torch
    kw = dict(selection=selection) if selection else {}
    loads = [((0.0, 0.0, -1.0), ((1, 1), (1, 1), (3, 3)))]
    G = gpu.Context(N, N, N, dirichlet=clamped_lines(), loads=loads, **kw)
    rng = np.random.default_rng(5)
    G.set_design(rng.uniform(0.05, 1.0, G.nelx))
    u = torch.tensor(rng.standard_normal(G.numeq), device="cuda")
    y = torch.full_like(u, float("nan"))
    torch.cuda.synchronize()
    G.apply_K_dev(u.data_ptr(), y.data_ptr())
    G.apply_K_dev(u.data_ptr(), u.data_ptr())
    G.synchronize()
    assert np.array_equal(u.cpu().numpy(), y.cpu().numpy())
