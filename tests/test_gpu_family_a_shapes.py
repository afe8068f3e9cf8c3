"""Scheme-A steps against the FP64 oracle at the sizes where the blocks beside a
step (halo copies, probe record) do not fill a row of blocks or a layer, with
zero-gradient halos on every face, with periodic z and with per-column fields
(whose instance leaves those blocks to a launch of their own).

Tolerance: that of tests/test_gpu_family_a.py.
"""
import numpy as np
import pytest

import nlos_lbm
import oracle
import scenarios
from nlos_lbm import abi
from scenarios import rel_l2

pytestmark = pytest.mark.gpu

TOL = 1e-5

SIZES = [(16, 9, 6), (33, 7, 12), (64, 21, 5), (129, 6, 8), (257, 5, 6)]
# more warps than a wave holds: blocks of two, three, four and five warps along a row
WIDE = [(66, 80, 40), (139, 50, 31), (208, 40, 30), (310, 33, 31)]


def case(kind, size):
    nx, ny, nz = size
    dx, cs = 0.25, abi.CS
    kw, solid, cols = {}, None, None
    src = dict(amp=0.01, freq=1.0 / (20.0 * cs * dx), waveform=abi.LBM_WAVE_SINE, injection=abi.LBM_INJECT_FIELD,
               sigma_cells=1.5, field_mode=abi.LBM_FIELD_FORCE)
    if kind.startswith("copy"):
        # (no reference program has both SOLID cells and a flow)
        kw = dict(face_bc=(abi.LBM_BC_COPY,) * 6, sponge_faces=(1 << 6) - 1, sponge_width=2.0, tau_sponge_max=0.9,
                  flow=(0.05, 0.0, 0.1) if kind == "copy_flow" else (0.0, 0.0, 0.0))
        solid = np.zeros((nz + 2, ny + 2, nx + 2), np.uint8)
        solid[2:4, 3:5, 4:7] = kind != "copy_flow"
    else:
        kw = dict(face_bc=(abi.LBM_BC_REST,) * 4 + (abi.LBM_BC_PERIODIC,) * 2, sponge_faces=15, sponge_width=2.0,
                  sponge_strength=0.5, sponge_blend=1)
        solid = np.zeros((nz + 2, ny + 2, nx + 2), np.uint8)
        solid[:, 2:4, 5:8] = 1
        src["field_mode"] = abi.LBM_FIELD_DST
    if kind.endswith("columns"):
        y, x = np.mgrid[0:ny, 0:nx]
        cols = np.exp(-0.2 * ((x - nx / 2) ** 2 + (y - ny / 2) ** 2))
    cfg = scenarios.lattice_config(nx, ny, nz, 0.53, x_max=nx * dx, y_max=ny * dx, z_max=nz * dx, dx=dx, c_phys=1.0,
                                   use_geometry=0, scheme=abi.LBM_SCHEME_A, dt=cs * dx, **kw)
    ctr = np.array([nx / 2, ny / 2, nz / 2]) * dx
    s = abi.reference_source(sx=ctr[0], sy=ctr[1], sz=ctr[2], ex=ctr[0], ey=ctr[1], ez=ctr[2], **src)
    probes = np.array([[0.1, 0.1, 0.1], [nx * dx - 0.1, ny * dx - 0.1, nz * dx - 0.1], ctr + 0.01,
                       [nx * dx - 0.1, 0.1, ctr[2]], [ctr[0], ny * dx - 0.1, 0.1]])
    return cfg, s, probes, solid.ravel(), cols


@pytest.mark.parametrize("size", SIZES + WIDE, ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("kind", ["copy", "copy_flow", "copy_columns", "periodic", "periodic_columns"])
def test_scheme_a_matches_oracle(kind, size, gpu):
    cfg, src, probes, mask, cols = case(kind, size)
    g = nlos_lbm.Solver(cfg, [src], probes, mask=mask, field_xy=cols)
    o = oracle.OracleSolver(cfg, [src], probes, mask=mask, field_xy=cols)
    steps = 21
    g.step(steps)
    o.step(steps)
    assert np.max(np.abs(o.get_probes())) > 0
    assert rel_l2(g.get_probes(), o.get_probes()) <= TOL
    nx, ny, nz = g.dims
    rho = o.get_rho().reshape(nz + 2, ny + 2, nx + 2)[1:-1, 1:-1, 1:-1] - 1.0
    rho = np.where(mask.reshape(nz + 2, ny + 2, nx + 2)[1:-1, 1:-1, 1:-1] != 0, 0.0, rho)
    assert np.max(np.abs(g.get_rho() - rho)) <= TOL * np.max(np.abs(rho))
    # single calls take the same route for the copies and their own for the probes
    h = nlos_lbm.Solver(cfg, [src], probes, mask=mask, field_xy=cols)
    for s in range(steps):
        h.apply_source(s * h.dt)
        h.exchange_halos()
        h.step_collision_bgk()
        h.record_probes()
    assert np.array_equal(h.get_probes(), g.get_probes())
    assert np.array_equal(h.get_rho(), g.get_rho())
    g.close()
    h.close()
