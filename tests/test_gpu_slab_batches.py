"""lbm_step on a z-slab handle is batched as on a whole grid: at most three launches a step (source, ghost fill,
step with its probes), the bits of the single calls, on a slab that is the whole grid and on one with cuts."""
import numpy as np
import pytest

from nlos_lbm import Solver, abi
from test_gpu_step_shapes import case

pytestmark = pytest.mark.gpu


def handles(size, storage, slab):
    cfg, srcs, probes, tris = case(size, storage, ground=True)
    cfg.slab_k0, cfg.slab_nz = slab
    return [Solver(cfg, srcs, probes, triangles=tris) for _ in range(2)]


@pytest.mark.parametrize("size,slab", [((33, 10, 8), (0, 8)), ((65, 13, 16), (0, 9)), ((97, 9, 20), (7, 6)),
                                       ((130, 6, 18), (10, 8))], ids=str)
@pytest.mark.parametrize("storage", [abi.LBM_STORE_F32, abi.LBM_STORE_F16], ids=["f32", "f16"])
def test_slab_batches_equal_single_calls(size, slab, storage, gpu):
    a, b = handles(size, storage, slab)
    for s in range(23):
        a.apply_source(s * a.dt)
        a.exchange_halos()
        a.step_collision_bgk()
        a.record_probes()
    for n in (1, 5, 2, 15):
        before = b.launch_count
        b.step(n)
        assert b.launch_count - before <= 3 * n
    assert np.array_equal(a.get_probes(), b.get_probes(), equal_nan=True)
    assert np.array_equal(a.get_probe_energy(), b.get_probe_energy(), equal_nan=True)
    assert np.array_equal(a.get_f(), b.get_f())
    assert np.array_equal(a.get_rho(), b.get_rho())
    assert np.max(np.abs(a.get_rho())) > 0
    a.close()
    b.close()


@pytest.mark.parametrize("storage", [abi.LBM_STORE_F32, abi.LBM_STORE_F16], ids=["f32", "f16"])
def test_slab_of_the_whole_grid_equals_the_grid(storage, gpu):
    size = (65, 13, 16)
    a = handles(size, storage, (0, 0))[0]
    b = handles(size, storage, (0, 16))[0]
    a.step(30)
    b.step(30)
    assert np.array_equal(a.get_probes(), b.get_probes())
    assert np.array_equal(a.get_f(), b.get_f())
    a.close()
    b.close()
