"""A gradient whose reverse pass recomputes every segment against one that stores every step: bit for bit, since
both run the same operations on the same data.  The sources lie in the first layer of an open face, so the last
launch of a recompute is the ghost fill, which writes the face moments that the first reverse launch reads, and
the receivers off it, each in a cell of its own."""
import numpy as np
import pytest

import scenarios
from nlos_lbm import Solver, abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(48, 40, 30), (130, 33, 21), (200, 90, 60)], ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("outer,inner", [(6, 2), (8, 8), (5, 1)])
def test_recomputed_segments_give_the_stored_gradient(size, outer, inner, gpu):
    nx, ny, nz = size
    cfg = scenarios.lattice_config(nx, ny, nz, 0.53, face_bc=(abi.LBM_BC_NSCBC,) * 6)
    src = abi.reference_source(sx=1.3, sy=ny / 2, sz=nz - 1.4, ex=1.3, ey=ny / 2, ez=nz - 1.4, amp=1e-3, freq=1 / 12.0,
                               t0=10.0, waveform=abi.LBM_WAVE_RICKER, injection=abi.LBM_INJECT_TRILINEAR)
    probes = np.array([[6.5, ny / 2 + 0.5, nz - 4.5], [4.5, ny / 2 - 3.5, nz - 5.5], [9.5, ny / 2 + 4.5, nz - 7.5]])
    steps = 60
    observed = 2e-5 * np.random.default_rng(5).standard_normal((steps, len(probes)))
    g = Solver(cfg, [src], probes)
    L, gp, gs, pred = g.adjoint_grad(observed)
    assert np.max(np.abs(gp)) > 0
    for _ in range(3):
        L2, gp2, gs2, pred2 = g.adjoint_grad(observed, ckpt_outer=outer, ckpt_inner=inner)
        assert L2 == L and np.array_equal(pred2, pred)
        assert np.array_equal(gp2, gp) and np.array_equal(gs2, gs)
    g.close()
