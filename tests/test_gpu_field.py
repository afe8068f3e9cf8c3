"""lbm_get_rho's staged download at the sizes where its parts, threads and pages
can go wrong: less than one part, one part and a row more, several parts with a
short last one, rows of odd length, and a caller's array that starts off a page
boundary.  lbm_get_rho_noalloc, which fills one device array in one launch,
gives the same values.
"""
import ctypes

import numpy as np
import pytest

import nlos_lbm
import scenarios
from nlos_lbm import abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(5, 4, 3), (97, 83, 20), (163, 101, 10), (163, 101, 11), (333, 70, 61), (700, 90, 33)],
                         ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("scheme", [abi.LBM_SCHEME_B, abi.LBM_SCHEME_A], ids=["b", "a"])
def test_field_parts(size, scheme, gpu):
    nx, ny, nz = size
    kw = dict(face_bc=(abi.LBM_BC_REST,) * 6, scheme=scheme) if scheme == abi.LBM_SCHEME_A else {}
    cfg = scenarios.lattice_config(nx, ny, nz, 0.55, sponge_width=0.0, **kw)
    src = abi.reference_source(sx=nx / 2, sy=ny / 2, sz=nz / 2, ex=nx / 2, ey=ny / 2, ez=nz / 2, amp=1e-3, freq=0.1,
                               waveform=abi.LBM_WAVE_SINE,
                               **(dict(injection=abi.LBM_INJECT_FIELD, sigma_cells=40.0, field_mode=abi.LBM_FIELD_DST)
                                  if scheme == abi.LBM_SCHEME_A else dict(radius=1)))
    g = nlos_lbm.Solver(cfg, [src], None)
    g.step(7)
    n = nx * ny * nz
    whole = np.full(n, np.nan, np.float32)
    p = ctypes.POINTER(ctypes.c_float)
    assert g.lib.lbm_get_rho_noalloc(g.h, whole.ctypes.data_as(p), n) == 0
    assert np.max(np.abs(whole)) > 0
    buf = np.full(n + 64, 7.0, np.float32)
    part = buf[13:13 + n]
    assert g.lib.lbm_get_rho(g.h, part.ctypes.data_as(p), n) == 0
    assert np.array_equal(part, whole)
    assert np.all(buf[:13] == 7.0) and np.all(buf[13 + n:] == 7.0)
    assert np.array_equal(g.get_rho().ravel(), whole)
    g.close()
