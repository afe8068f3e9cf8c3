"""The fused step's launch shapes against the FP64 oracle at the sizes where a
row's columns or a plane's rows do not fill a block: one warp and less per row,
two, three, four and five 64-column segments, odd widths, and row counts that
leave rows of a block without cells.

Tolerances: those of tests/test_gpu_parity.py for FP32 and FP16 storage.
"""
import numpy as np
import pytest

import nlos_lbm
import oracle
import scenarios
from nlos_lbm import abi
from scenarios import rel_l2

pytestmark = pytest.mark.gpu

FP32_PROBE_TOL = 1e-5
FP32_STATE_TOL = 1e-4
FP16_PROBE_TOL = 1e-3

SIZES = [(17, 9, 7), (33, 10, 8), (63, 11, 9), (64, 8, 12), (65, 13, 6), (97, 9, 10), (128, 10, 9), (129, 6, 11),
         (191, 7, 8), (257, 5, 7), (320, 6, 6)]


def case(size, storage, ground):
    """A box crossing a segment edge, a source against the low x face, open faces (and a ground plane)."""
    nx, ny, nz = size
    faces = [abi.LBM_BC_NSCBC] * 6
    if ground:
        faces[abi.FACE_ZLO] = abi.LBM_BC_WALL
    cfg = scenarios.lattice_config(nx, ny, nz, 0.52, face_bc=tuple(faces), sponge_faces=(1 << 6) - 1,
                                   sponge_width=2.0, storage=storage, f16_scale=1e5)
    x0 = min(60, nx // 2)
    tris = scenarios.boxes_to_triangles([(x0, ny // 2, 0, min(x0 + 6, nx - 1), ny - 1, nz // 2)])
    src = abi.reference_source(sx=2.3, sy=2.1, sz=nz / 2 + 0.2, ex=2.3, ey=2.1, ez=nz / 2 + 0.2, amp=1e-3,
                               freq=1 / 20.0, waveform=abi.LBM_WAVE_SINE)
    far = abi.reference_source(sx=nx - 1.6, sy=ny / 2, sz=nz - 2.2, ex=nx / 2, ey=1.4, ez=nz - 1.2, speed=0.3, amp=1e-3,
                               freq=1 / 16.0, waveform=abi.LBM_WAVE_SINE, injection=abi.LBM_INJECT_TRILINEAR)
    probes = np.array([[0.5, 2.5, nz / 2], [3.5, 3.5, nz / 2], [nx - 0.5, ny / 2, nz - 1.5],
                       [nx - 2.5, 1.5, nz - 0.5], [1.5, 0.5, nz - 0.5]])
    return cfg, [src, far], probes, tris


@pytest.mark.parametrize("size", SIZES, ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("storage", [abi.LBM_STORE_F32, abi.LBM_STORE_F16], ids=["f32", "f16"])
def test_step_matches_oracle(size, storage, gpu):
    steps = 24
    cfg, srcs, probes, tris = case(size, storage, ground=size[2] % 2 == 0)
    g = nlos_lbm.Solver(cfg, srcs, probes, triangles=tris)
    o = oracle.OracleSolver(cfg, srcs, probes, triangles=tris)
    assert np.array_equal(g.get_mask(), o.get_mask())
    g.step(steps)
    o.step(steps)
    assert rel_l2(g.get_probes(), o.get_probes()) <= (FP32_PROBE_TOL if storage == abi.LBM_STORE_F32 else FP16_PROBE_TOL)
    if storage == abi.LBM_STORE_F32:
        w = np.array(abi.W)
        nx, ny, nz = g.dims_halo
        dg, do = (s.get_f().reshape(nz, ny, nx, 19)[1:-1, 1:-1, 1:-1] - w for s in (g, o))
        assert np.max(np.abs(dg - do)) <= FP32_STATE_TOL * np.max(np.abs(do))
    g.close()


@pytest.mark.parametrize("size", [(33, 10, 8), (65, 13, 6), (128, 10, 9), (191, 7, 8)], ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("storage", [abi.LBM_STORE_F32, abi.LBM_STORE_F16], ids=["f32", "f16"])
@pytest.mark.parametrize("split", [(13,), (1, 1, 1, 2, 1, 7), (2, 11), (5, 8)], ids=str)
def test_batches_equal_single_calls(size, storage, split, gpu):
    """However a run is split into batches, every batched step (which applies the next step's sources and
    ghosts to its own results) gives the bits of the single calls, sources against the open faces included."""
    cfg, srcs, probes, tris = case(size, storage, ground=True)
    a = nlos_lbm.Solver(cfg, srcs, probes, triangles=tris)
    b = nlos_lbm.Solver(cfg, srcs, probes, triangles=tris)
    for s in range(sum(split)):
        a.apply_source(s * a.dt)
        a.exchange_halos()
        a.step_collision_bgk()
        a.record_probes()
    for n in split:
        b.step(n)
    assert np.array_equal(a.get_probes(), b.get_probes())
    assert np.array_equal(a.get_probe_energy(), b.get_probe_energy())
    assert np.array_equal(a.get_f(), b.get_f())
    assert np.array_equal(a.get_rho(), b.get_rho())
    # single calls after a batch, and a batch after single calls
    for s in range(sum(split), sum(split) + 2):
        b.apply_source(s * b.dt)
        b.exchange_halos()
        b.step_collision_bgk()
        b.record_probes()
    a.step(2)
    assert np.array_equal(a.get_f(), b.get_f())
    assert np.array_equal(a.get_probes(), b.get_probes())
    a.close()
    b.close()


@pytest.mark.parametrize("size", [(129, 204, 320), (192, 200, 222), (257, 181, 190), (299, 174, 173)],
                         ids=lambda s: "x".join(map(str, s)))
def test_claimed_rows_equal_single_calls(size, gpu):
    """Large FP16 grids with many rows a warp, three blocks a row and more: batched steps, whose warps claim
    their rows, give the bits of the single calls, whose warps walk fixed rows."""
    cfg, srcs, probes, tris = case(size, abi.LBM_STORE_F16, ground=True)
    a = nlos_lbm.Solver(cfg, srcs, probes, triangles=tris)
    b = nlos_lbm.Solver(cfg, srcs, probes, triangles=tris)

    def single(g, n):
        for _ in range(n):
            g.apply_source(g.step_count * g.dt)
            g.exchange_halos()
            g.step_collision_bgk()
            g.record_probes()

    single(a, 14)
    for n in (1, 4, 9):
        b.step(n)
    single(a, 1)
    single(b, 1)   # the field is read from the state before the last step
    assert np.array_equal(a.get_rho(), b.get_rho())
    assert np.array_equal(a.get_probes(), b.get_probes())
    assert np.max(np.abs(a.get_rho())) > 0
    a.close()
    b.close()


def test_large_f32_batches_equal_single_calls(gpu):
    """FP32 past the fused step's size: source, ghost fill and step as chained launches."""
    cfg, srcs, probes, tris = case((199, 151, 145), abi.LBM_STORE_F32, ground=True)
    a = nlos_lbm.Solver(cfg, srcs, probes, triangles=tris)
    b = nlos_lbm.Solver(cfg, srcs, probes, triangles=tris)
    for s in range(12):
        a.apply_source(s * a.dt)
        a.exchange_halos()
        a.step_collision_bgk()
        a.record_probes()
    for n in (1, 4, 7):
        b.step(n)
    assert np.array_equal(a.get_probes(), b.get_probes())
    assert np.array_equal(a.get_probe_energy(), b.get_probe_energy())
    assert np.array_equal(a.get_rho(), b.get_rho())
    a.step(3)
    b.step(3)
    assert np.array_equal(a.get_rho(), b.get_rho())
    assert np.max(np.abs(a.get_rho())) > 0
    a.close()
    b.close()
