"""A loop started again on the same context keeps its buffers (filter set-up,
MMA work vectors): it must run as the first one did, also after a loop with
another radius, filter or method in between."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def run(G, gpu, **kw):
    G.loop_init(0.4, solve=gpu.solve_opts(gpu.MG_PCG, rtol=1e-10, mg_levels=3), **kw)
    steps = [G.loop_step() for _ in range(4)]
    return [s.compliance for s in steps], G.loop_get("x"), G.loop_get("dfds")


@pytest.mark.parametrize("between", [None, dict(method="oc", filter_radius=2.5),
                                     dict(method="mma", filter_radius=1.5, filter="helmholtz")])
@pytest.mark.parametrize("kw", [dict(method="mma", filter_radius=1.5),
                                dict(method="mma", filter_radius=2.0, filter="helmholtz"),
                                dict(method="oc", filter_radius=1.5)])
def test_second_run_repeats_the_first(gpu, kw, between):
    G = gpu.Context(16, 8, 8)
    a = run(G, gpu, **kw)
    if between:
        run(G, gpu, **between)
    b = run(G, gpu, **kw)
    assert a[0] == b[0]
    assert np.array_equal(a[1], b[1]) and np.array_equal(a[2], b[2])


def test_setup_again_needs_a_forward_call(gpu):
    G = gpu.Context(6, 4, 4)
    G.filter_setup(1.5)
    x = np.full(G.nelx, 0.3)
    G.density_filter(x)
    G.filter_setup(1.5)
    with pytest.raises(gpu.IcaratError) as e:
        G.density_filter(x, True)
    assert e.value.status == gpu.ERR_STATE
