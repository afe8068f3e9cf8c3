"""The characteristic open boundary's ghost values (exchange_halos 06:684-835), bit for bit: one ghost fill
of a random state against the same FP32 operations in numpy, with IEEE divisions and the multiply-adds that
round once.  No tolerance: series in FP16 storage repeat only if these values do.
"""
import numpy as np
import pytest

import nlos_lbm
import scenarios
from nlos_lbm import abi

pytestmark = pytest.mark.gpu

E = np.array([[0, 1, -1, 0, 0, 0, 0, 1, 1, -1, -1, 1, 1, -1, -1, 0, 0, 0, 0],
              [0, 0, 0, 1, -1, 0, 0, 1, -1, 1, -1, 0, 0, 0, 0, 1, 1, -1, -1],
              [0, 0, 0, 0, 0, 1, -1, 0, 0, 0, 0, 1, -1, 1, -1, 1, -1, 1, -1]])
W = np.array(abi.W)
F = np.float32


def fma(x, y, z):
    """x y + z with one rounding: the product is exact in the 64-bit significand."""
    return (np.longdouble(x) * np.longdouble(y) + np.longdouble(z)).astype(F)


def ghosts(G, axis, side, inv_scale):
    """Ghost values of the directions into the grid from interior values G [cells][19]; {q: values}."""
    m = [np.zeros(len(G), F) for _ in range(4)]
    for q in range(19):
        m[0] = m[0] + G[:, q]
        for a in range(3):
            if E[a, q]:
                m[a + 1] = m[a + 1] + G[:, q] if E[a, q] > 0 else m[a + 1] - G[:, q]
    rho, inv_scale, cs, cs2 = m[0], F(inv_scale), F(abi.CS), F(1.0 / 3.0)
    r = fma(rho, inv_scale, F(1))
    assert np.all(r > 0)
    u = [j / r for j in m[1:]]
    p = (cs2 * rho) / cs
    w = u[axis] + p if side else u[axis] - p
    rho_b = (F(0.5 if side else -0.5) * cs * w) / cs2
    r_b = fma(rho_b, inv_scale, F(1))
    b = list(u)
    b[axis] = F(0.5) * w
    square = lambda v: fma(v[2], v[2], fma(v[0], v[0], v[1] * v[1]))   # noqa: E731
    k45 = F(4.5) * inv_scale
    d = fma(F(-1.5) * inv_scale, fma(r_b, square(b), -(r * square(u))), rho_b - rho)
    qv, pv = [r_b * v for v in b], [r * v for v in u]
    out = {}
    for q in range(19):
        if E[axis, q] != (-1 if side else 1):
            continue
        e, c = d, E[:, q]
        for a in range(3):
            if c[a]:
                e = fma(k45, fma(qv[a], b[a], -(pv[a] * u[a])), e)
        for a, a2 in ((0, 1), (0, 2), (1, 2)):
            if c[a] * c[a2]:
                e = fma(F(2 * c[a] * c[a2]) * k45, fma(qv[a], b[a2], -(pv[a] * u[a2])), e)
        for a in range(3):
            if c[a]:
                e = fma(F(3 * c[a]), qv[a] - pv[a], e)
        out[q] = fma(F(W[q]), e, G[:, q])
    return out


@pytest.mark.parametrize("size", [(33, 10, 8), (64, 21, 12), (130, 7, 9)], ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("storage", [abi.LBM_STORE_F32, abi.LBM_STORE_F16], ids=["f32", "f16"])
def test_ghost_fill_to_the_bit(size, storage, gpu):
    nx, ny, nz = size
    half = storage == abi.LBM_STORE_F16
    scale = 2.0 ** 14 if half else 1.0
    cfg = scenarios.lattice_config(nx, ny, nz, 0.52, face_bc=(abi.LBM_BC_NSCBC,) * 6, storage=storage, f16_scale=scale)
    src = abi.reference_source(sx=nx / 2, sy=ny / 2, sz=nz / 2, ex=nx / 2, ey=ny / 2, ez=nz / 2, amp=1e-3, freq=0.05,
                               waveform=abi.LBM_WAVE_SINE)
    s = nlos_lbm.Solver(cfg, [src], np.array([[nx / 2, ny / 2, nz / 2]]))
    rng = np.random.default_rng(list(size))
    # a wave of up to 5 % of the density and of Mach 0.1, with some non-equilibrium
    shape = (nz + 2, ny + 2, nx + 2)
    mom = 0.05 * rng.uniform(-1, 1, (4, *shape))
    G = W * (mom[0][..., None] + 3 * np.einsum("a...,aq->...q", mom[1:], E.astype(float)) +
             0.01 * rng.uniform(-1, 1, (*shape, 19)))
    G = (G * scale).astype(np.float16 if half else F).astype(F)   # as stored
    s.set_f((W + G.astype(np.float64) / scale).ravel())
    s.exchange_halos()
    got = ((s.get_f().reshape(*shape, 19) - W) * scale).astype(F)
    inner = G[1:-1, 1:-1, 1:-1]
    assert np.array_equal(got[1:-1, 1:-1, 1:-1], inner)
    for axis in range(3):
        for side in (0, 1):
            cells = np.take(inner, -side, axis=2 - axis)
            halo = np.take(got, -side, axis=2 - axis)[1:-1, 1:-1]
            for q, v in ghosts(cells.reshape(-1, 19), axis, side, 1.0 / scale).items():
                if half and axis > 0:   # x ghosts are kept in FP32
                    v = v.astype(np.float16).astype(F)
                assert np.array_equal(halo[..., q].ravel(), v), (axis, side, q)
    s.close()
