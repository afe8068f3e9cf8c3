"""lbm_adjoint_grad where its launches split differently: rows of two to five
warps, sources and receivers in the first layer of an open face (which the ghost
fill and its adjoint touch) and away from it, several receivers in one cell, grids
without an open face, and the one-launch forward pass against a checkpointed one.

Tolerance: the 1e-4 gradient bar and the 1e-5 probe bar of tests/test_gpu_adjoint.py.
"""
import numpy as np
import pytest

import scenarios
from nlos_lbm import Solver, abi
from oracle import OracleSolver
from scenarios import rel_l2

pytestmark = pytest.mark.gpu

GRAD_TOL = 1e-4
PROBE_TOL = 1e-5


def case(size, where, faces):
    nx, ny, nz = size
    bc = {"open": (abi.LBM_BC_NSCBC,) * 4 + (abi.LBM_BC_WALL, abi.LBM_BC_NSCBC), "rest": (abi.LBM_BC_REST,) * 6}[faces]
    cfg = scenarios.lattice_config(nx, ny, nz, 0.53, face_bc=bc, sponge_faces=(1 << 6) - 1, sponge_width=3.0)
    tris = scenarios.boxes_to_triangles([(nx // 2, 4, 0, nx // 2 + 5, 9, 5)])
    c = np.array([4.3, 5.6, 5.2]) if where == "inside" else np.array([1.2, 5.6, nz - 1.4])
    src = abi.reference_source(sx=c[0], sy=c[1], sz=c[2], ex=c[0] + 2, ey=c[1] + 1, ez=c[2], speed=0.05, amp=1e-3,
                               freq=1 / 12.0, t0=10.0, waveform=abi.LBM_WAVE_RICKER,
                               injection=abi.LBM_INJECT_TRILINEAR)
    probes = c + np.array([[5.1, 1.2, -0.3], [3.3, 3.1, -2.0], [5.4, 1.4, -0.1], [2.2, 4.4, -1.0]])
    if where == "face":
        probes = np.vstack([probes, [[0.5, 8.5, nz - 3.5], [4.5, 8.5, nz - 0.5], [nx - 0.5, 6.5, 6.5], [-3.0, 5.0, 5.0]]])
    return cfg, src, probes, tris


@pytest.mark.parametrize("size", [(40, 24, 20), (150, 14, 13), (200, 13, 12), (301, 13, 11)],
                         ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("where,faces", [("inside", "open"), ("face", "open"), ("inside", "rest")])
def test_gradient_matches_fp64_adjoint(size, where, faces, gpu):
    cfg, src, probes, tris = case(size, where, faces)
    steps = 36
    rng = np.random.default_rng(3)
    observed = 2e-5 * rng.standard_normal((steps, len(probes)))
    o = OracleSolver(cfg, [src], probes, triangles=tris)
    L0, gp0, gs0, pred0 = o.adjoint_grad(observed, K=8)
    g = Solver(cfg, [src], probes, triangles=tris)
    L, gp, gs, pred = g.adjoint_grad(observed)
    owned = ~np.isnan(pred0[0])
    assert np.max(np.abs(pred0[:, owned])) > 0
    assert rel_l2(pred[:, owned], pred0[:, owned]) <= PROBE_TOL
    assert L == pytest.approx(L0, rel=GRAD_TOL)
    assert np.max(np.abs(gp - gp0)) <= GRAD_TOL * np.max(np.abs(gp0))
    assert rel_l2(gs, gs0) <= GRAD_TOL
    # a checkpointed schedule runs the forward pass in separate launches
    L2, gp2, gs2, pred2 = g.adjoint_grad(observed, ckpt_outer=9, ckpt_inner=4)
    assert L2 == L and np.array_equal(pred2[:, owned], pred[:, owned])
    g.step(steps)
    assert np.array_equal(g.get_probes()[:, owned], pred[:, owned])
    # receivers that share a cell add their residuals in any order
    assert np.max(np.abs(gp2 - gp)) <= 1e-6 * np.max(np.abs(gp))
    assert rel_l2(gs2, gs) <= 1e-6
    g.close()
