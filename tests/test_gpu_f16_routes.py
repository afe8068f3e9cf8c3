"""FP16 batches on each of their routes: fused steps, and past 2^23 cells steps whose warps claim their rows or
walk fixed ones (rows of two 64-cell blocks; few rows a warp), replayed as graphs and as direct launches.
The bits of the single calls, or of one another."""
import numpy as np
import pytest

import nlos_lbm
from nlos_lbm import abi
from test_gpu_step_shapes import case

pytestmark = pytest.mark.gpu

ROUTES = {"fused": (97, 41, 30), "claimed": (257, 200, 230), "fixed_two_blocks": (128, 300, 250),
          "fixed_few_rows": (900, 200, 50)}


def solver(size, graphs):
    cfg, srcs, probes, tris = case(size, abi.LBM_STORE_F16, ground=True)
    cfg.use_graphs = graphs
    return nlos_lbm.Solver(cfg, srcs, probes, triangles=tris)


@pytest.mark.parametrize("route", list(ROUTES))
def test_graphs_equal_direct_launches(route, gpu):
    a, b = solver(ROUTES[route], 1), solver(ROUTES[route], 0)
    for n in (1, 6, 2, 9):
        a.step(n)
        b.step(n)
    assert np.array_equal(a.get_probes(), b.get_probes())
    assert np.array_equal(a.get_probe_energy(), b.get_probe_energy())
    assert np.array_equal(a.get_rho(), b.get_rho())
    assert np.max(np.abs(a.get_rho())) > 0
    a.close()
    b.close()


@pytest.mark.parametrize("route", ["fixed_two_blocks", "fixed_few_rows"])
def test_fixed_rows_equal_single_calls(route, gpu):
    a, b = solver(ROUTES[route], 1), solver(ROUTES[route], 1)
    for s in range(15):
        a.apply_source(s * a.dt)
        a.exchange_halos()
        a.step_collision_bgk()
        a.record_probes()
    for n in (1, 4, 7, 3):
        b.step(n)
    assert np.array_equal(a.get_probes(), b.get_probes())
    assert np.array_equal(a.get_probe_energy(), b.get_probe_energy())
    assert np.array_equal(a.get_rho(), b.get_rho())
    assert np.max(np.abs(a.get_rho())) > 0
    a.close()
    b.close()
