"""Grids so long in y that the blocks beside a step (probes, halo copies) do not fit the rows of blocks that the
step leaves of gridDim.y (65535): the FP32 step takes a split with fewer rows of blocks, scheme A a launch of
their own.  Tolerance of the scheme-A run: that of tests/test_gpu_family_a.py."""
import numpy as np
import pytest

import nlos_lbm
import oracle
import scenarios
from nlos_lbm import abi
from scenarios import rel_l2
from test_gpu_family_a_shapes import TOL, case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(193, 65535, 1), (40, 65533, 1)], ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("storage", [abi.LBM_STORE_F32, abi.LBM_STORE_F16], ids=["f32", "f16"])
def test_longest_rows_step_in_batches(size, storage, gpu):
    nx, ny, nz = size
    cfg = scenarios.lattice_config(nx, ny, nz, 0.52, face_bc=(abi.LBM_BC_NSCBC,) * 6, use_geometry=0, storage=storage,
                                   f16_scale=1e5)
    src = abi.reference_source(sx=20.3, sy=ny - 6.4, sz=0.5, ex=20.3, ey=ny - 6.4, ez=0.5, amp=1e-3, freq=1 / 20.0,
                               waveform=abi.LBM_WAVE_SINE)
    probes = np.array([[21.5, ny - 0.5, 0.5], [23.5, ny - 5.5, 0.5], [3.5, 0.5, 0.5]])
    a = nlos_lbm.Solver(cfg, [src], probes)
    b = nlos_lbm.Solver(cfg, [src], probes)
    for s in range(7):
        a.apply_source(s * a.dt)
        a.exchange_halos()
        a.step_collision_bgk()
        a.record_probes()
    for n in (1, 4, 2):
        b.step(n)
    assert np.max(np.abs(a.get_probes())) > 0
    assert np.array_equal(a.get_probes(), b.get_probes())
    assert np.array_equal(a.get_rho(), b.get_rho())
    a.close()
    b.close()


@pytest.mark.parametrize("size", [(64, 40000, 1), (130, 40000, 2)], ids=lambda s: "x".join(map(str, s)))
def test_scheme_a_with_more_halo_copies_than_rows_left(size, gpu):
    cfg, src, probes, mask, _ = case("copy_flow", size)
    g = nlos_lbm.Solver(cfg, [src], probes, mask=mask)
    o = oracle.OracleSolver(cfg, [src], probes, mask=mask)
    steps = 5
    g.step(steps)
    o.step(steps)
    assert np.max(np.abs(o.get_probes())) > 0
    assert rel_l2(g.get_probes(), o.get_probes()) <= TOL
    h = nlos_lbm.Solver(cfg, [src], probes, mask=mask)
    for s in range(steps):
        h.apply_source(s * h.dt)
        h.exchange_halos()
        h.step_collision_bgk()
        h.record_probes()
    assert np.array_equal(h.get_probes(), g.get_probes())
    assert np.array_equal(h.get_rho(), g.get_rho())
    g.close()
    h.close()
