// Device parts shared by the fused scheme-B steps (FP32 and FP16) and by the
// kernels that do the same work on their own for single calls: the source
// stencil (apply_source, 06:576-667), the characteristic ghost values
// (exchange_halos, 06:684-835) and the probe record (06:1085-1092).
//
// A batched step applies the next step's source and ghost fill to its own
// results while they are in registers.  What surrounded a step before were
// four launches (source, ghosts, step, probes) whose small kernels are chains
// of dependent loads: on grids of up to a few million cells they and the
// gaps between them took as long as the step.  Every value is formed by the
// same operations in the same order as by the separate kernels, with explicit
// FMAs, so both routes give the same bits.
#pragma once

#include <cuda_fp16.h>

#include <cstdint>

#include "check.cuh"
#include "device.hpp"
#include "lattice.cuh"

namespace lbm {
namespace {

// e_q components as 2-bit fields of one immediate, for per-lane q
__host__ __device__ constexpr unsigned long long pack_e(int axis)
{
    unsigned long long v = 0;
    for (int q = 0; q < Q; ++q)
        v |= (unsigned long long)((axis == 0 ? ex(q) : axis == 1 ? ey(q) : ez(q)) + 1) << (2 * q);
    return v;
}
template <int AXIS>
__device__ __forceinline__ int e_of(int q)
{
    constexpr unsigned long long t = pack_e(AXIS);
    return (int)((t >> (2 * q)) & 3ull) - 1;
}
__host__ __device__ constexpr unsigned long long pack_inv(int part)   // 5-bit fields, 12 per word
{
    unsigned long long v = 0;
    for (int q = 12 * part; q < Q && q < 12 * part + 12; ++q) v |= (unsigned long long)inv(q) << (5 * (q - 12 * part));
    return v;
}
__device__ __forceinline__ int inv_of(int q)
{
    constexpr unsigned long long lo = pack_inv(0), hi = pack_inv(1);
    return (int)((q < 12 ? lo >> (5 * q) : hi >> (5 * (q - 12))) & 31ull);
}

// ---------------------------------------------------------------- source
// Stencil of one source at one step, by a whole block of a multiple of 32
// threads: weights of the (2R+1)^3 Gaussian stencil (or the 8 trilinear
// weights) normalised over the FLUID cells of the grid, A = mass / sum_w; each
// FLUID cell gains w_q * A * w_cell in direction q.  put(cell, amounts) gets
// every cell of the box, i fastest, amounts = what directions 0, 1-6 and 7-18
// gain, w = 1 for a FLUID cell of the grid.  False when nothing is injected.
// The sum is taken per 32 cells by a shuffle tree and then over the groups in
// order, whatever the block size.
template <typename Put>
__device__ __forceinline__ bool source_stencil(const SourceEntry& e, const SourceStatic& st, const SourceArgs& a,
                                               const Layout& L, const uint32_t* __restrict__ links, double* red,
                                               SourceBox& box, Put&& put)
{
    constexpr int kRounds = (kStencilCells + 127) / 128;   // blocks have at least 128 threads
    box = SourceBox{0, 0, 0, 0};
    if (e.mass == 0.0) return false;
    int n, i0, j0, k0;
    double tx = 0.0, ty = 0.0, tz = 0.0;
    if (st.injection == 1)
    {
        const double fx = (e.cx - a.x_min) / a.dx - 0.5;
        const double fy = (e.cy - a.y_min) / a.dx - 0.5;
        const double fz = (e.cz - a.z_min) / a.dx - 0.5;
        i0 = (int)floor(fx), j0 = (int)floor(fy), k0 = (int)floor(fz);
        tx = fx - i0, ty = fy - j0, tz = fz - k0;
        n = 2;
    }
    else
    {
        const int R = st.radius;
        const int ic = (int)floor((e.cx - a.x_min) / a.dx);
        const int jc = (int)floor((e.cy - a.y_min) / a.dx);
        const int kc = (int)floor((e.cz - a.z_min) / a.dx);
        if (ic < -R || ic >= L.nx + R || jc < -R || jc >= L.ny + R || kc - a.k_off < -R || kc - a.k_off >= L.nz + R)
            return false;
        i0 = ic - R, j0 = jc - R, k0 = kc - R;
        n = 2 * R + 1;
    }
    const int ncell = n * n * n;
    double ww[kRounds];
    bool fluid[kRounds];
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int r = 0; r < kRounds; ++r)
    {
        const int c = (int)threadIdx.x + r * (int)blockDim.x;
        ww[r] = 0.0;
        fluid[r] = false;
        if (r * (int)blockDim.x >= ncell) continue;
        if (c < ncell)
        {
            const int di = c % n, dj = (c / n) % n, dk = c / (n * n);
            const int gi = i0 + di, gj = j0 + dj, gk = k0 + dk;
            if (st.injection == 1)
            {
                ww[r] = (di ? tx : 1.0 - tx) * (dj ? ty : 1.0 - ty) * (dk ? tz : 1.0 - tz);
            }
            else
            {
                const double x = a.x_min + (gi + 0.5) * a.dx;
                const double y = a.y_min + (gj + 0.5) * a.dx;
                const double z = a.z_min + (gk + 0.5) * a.dx;
                const double ddx = x - e.cx, ddy = y - e.cy, ddz = z - e.cz;
                const double r2 = ddx * ddx + ddy * ddy + ddz * ddz;
                ww[r] = exp(-0.5 * r2 / st.sigma2);
            }
            // weights in the coordinates of the whole grid; a z-slab holds layers k_off..
            const int lk = gk - a.k_off;
            if (gi >= 0 && gi < L.nx && gj >= 0 && gj < L.ny && lk >= 0 && lk < L.nz)
                fluid[r] = (links[L.cell(gi + 1, gj + 1, lk + 1)] & kSolidSelfBit) == 0u;
        }
        double v = fluid[r] ? ww[r] : 0.0;
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0 && c < ncell) red[c >> 5] = v;
    }
    __syncthreads();
    double bsum = 0.0;
    for (int g = 0; g < (ncell + 31) / 32; ++g) bsum += red[g];
    __syncthreads();   // before the next source's sums
    const double sum = e.wsum > 0.0 ? e.wsum : bsum;   // a stencil across a z-slab cut
    if (sum < 1e-30) return false;
    box = SourceBox{i0 + 1, j0 + 1, k0 - a.k_off + 1, n};
    const double A = e.mass / sum;
#pragma unroll
    for (int r = 0; r < kRounds; ++r)
    {
        const int c = (int)threadIdx.x + r * (int)blockDim.x;
        if (c >= ncell) continue;
        const double add = A * ww[r] * (double)a.scale;
        put(c, make_float4((float)(wd(0) * add), (float)(wd(1) * add), (float)(wd(7) * add), fluid[r] ? 1.0f : 0.0f));
    }
    return true;
}
__device__ __forceinline__ float source_gain(const float4& v, int q) { return q == 0 ? v.x : (q < 7 ? v.y : v.z); }

// Sources of step t into *out, by one block: what the step before applies to its results.
__device__ __forceinline__ void prepare_sources(SourceNext* out, const SourceArgs& a, long long t, bool fill,
                                                const Layout& L, const uint32_t* links, double* red)
{
    if (threadIdx.x == 0) out->fill = fill ? 1 : 0;
    if (!fill) return;
    for (int s = 0; s < a.nsrc; ++s)
    {
        const SourceEntry e = a.ctl ? a.table[(t - a.ctl->table_base) * a.nsrc + s] : a.direct[s];
        SourceBox box{};
        source_stencil(e, a.st[s], a, L, links, red, box, [&](int c, const float4& v) { out->add[s][c] = v; });
        if (threadIdx.x == 0) out->box[s] = box;
    }
}

// Bits of the sources whose box holds cells of row (j, k) (whole warp).
__device__ __forceinline__ unsigned sources_of_row(const SourceNext* __restrict__ nx, int nsrc, int lane, int j, int k)
{
    bool hit = false;
    if (lane < nsrc)
    {
        const SourceBox b = nx->box[lane];
        hit = j >= b.j0 && j < b.j0 + b.n && k >= b.k0 && k < b.k0 + b.n;
    }
    return __ballot_sync(0xffffffffu, hit);
}

// ---------------------------------------------------------------- ghosts
// Characteristic open boundary (exchange_halos 06:684-835, MPI size 1): the
// ghost cell next to interior cell I gets
//   f_B = feq(rho_B, u_B) + (f_I - feq(rho_I, u_I)),
// where u_B keeps the tangential velocity of I, and the normal velocity and
// pressure carry only the outgoing invariant (incoming invariant zero).  In
// stored deviation units (Gs = scale * g):
//   geq(rho', r, u) = w (rho' + r (3 c.u + (4.5 (c.u)^2 - 1.5 u^2) / scale)).
//
// Only the 5 directions that point from the ghost into the interior (e_axis =
// +1 on the low side, -1 on the high side) are ever pulled from a ghost cell
// (by the step, the probes, the field output, the slab messages and the
// adjoint); the fill computes and stores those and leaves the other 14 of the
// ghost cell as they are.
template <int AXIS, int SIDE>
__host__ __device__ constexpr bool inward(int q)
{
    return (AXIS == 0 ? ex(q) : AXIS == 1 ? ey(q) : ez(q)) == (SIDE ? -1 : 1);
}

// (rho', J) of one cell, get(q) its stored populations
template <typename Get>
__device__ __forceinline__ float4 cell_moments(Get&& get)
{
    float4 m = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int q = 0; q < Q; ++q)
    {
        const float g = get(q);
        m.x += g;
        if (ex(q) > 0) m.y += g;
        if (ex(q) < 0) m.y -= g;
        if (ey(q) > 0) m.z += g;
        if (ey(q) < 0) m.z -= g;
        if (ez(q) > 0) m.w += g;
        if (ez(q) < 0) m.w -= g;
    }
    return m;
}

// Quotients as IEEE division rounds them, by Markstein's correction of an approximate one (Computation of
// elementary functions on the IBM RISC System/6000 processor, 1990): q + y (x - q b), exact where q is within a
// unit of its last place and the remainder does not underflow.  Division itself branches on zeros and tiny
// numerators, as quiet cells have: with it the scatter box 128^3 took 55.9 us a step in FP16 against 50.2,
// 256x128x128 FP32 127 against 117.  Compared with division bit for bit: `quotient` over 2^33 pairs of |x| in
// 2^-97 .. 2^90 and every x at b = 1 (smaller moments come with a density of 1), `over` for every |x| to 2^98.
//
// x / b, y = 1 / b rounded: two steps, the product alone may be two units off.
__device__ __forceinline__ float quotient(float x, float b, float y)
{
    float q = __fmul_rn(x, y);
    q = __fmaf_rn(__fmaf_rn(-q, b, x), y, q);
    return __fmaf_rn(__fmaf_rn(-q, b, x), y, q);
}
// x / c for c = cs or cs^2, z = 1 / c rounded: one step, the remainder scaled up so that it is exact for any x and
// a quotient below the normal range is rounded once.
__device__ __forceinline__ float over(float x, float c, float z)
{
    const float q = __fmul_rn(x, z);
    const float r = __fmaf_rn(-__fmul_rn(q, 0x1p28f), c, __fmul_rn(x, 0x1p28f));
    return __fmaf_rn(r, z * 0x1p-28f, q);
}

// What the ghosts of cell I take from its moments m, whichever face they lie on: rho', density and velocity, and
// p / cs with p = cs^2 rho'.  (A product with a rounded reciprocal has a rounding of its own, and an FP16 ghost on
// the other side of a rounding step is stored one unit away.)
struct GhostState
{
    float rho, r, ux, uy, uz, pc;
};
__device__ __forceinline__ GhostState ghost_state(const float4& m, float inv_scale)
{
    constexpr float cs = (float)kCs, cs2 = (float)kCs2;
    GhostState g{m.x, __fmaf_rn(m.x, inv_scale, 1.0f), 0.0f, 0.0f, 0.0f, 0.0f};
    const bool fluid = g.r > 1e-30f;
    if (!fluid)
    {
        g.r = 1.0f;
        g.rho = 0.0f;
    }
    // (taken for every cell: as a branch they cost the FP32 step 16 bytes of spills, 256x128x128 127 us against 117)
    const float iv = __frcp_rn(g.r);
    g.ux = quotient(m.y, g.r, iv);
    g.uy = quotient(m.z, g.r, iv);
    g.uz = quotient(m.w, g.r, iv);
    g.pc = over(__fmul_rn(cs2, g.rho), cs, 1.0f / cs);
    if (!fluid) g.ux = g.uy = g.uz = 0.0f;
    return g;
}

// Ghost values of the inward directions of face (AXIS, SIDE) from cell I, through put(q, value).
template <int AXIS, int SIDE, typename Get, typename Put>
__device__ __forceinline__ void nscbc(const GhostState& g, float inv_scale, Get&& get, Put&& put)
{
    const auto mul = [](float x, float y) { return __fmul_rn(x, y); };
    const auto add = [](float x, float y) { return __fadd_rn(x, y); };
    const auto sub = [](float x, float y) { return __fsub_rn(x, y); };
    const auto fma = [](float x, float y, float z) { return __fmaf_rn(x, y, z); };
    const float rho = g.rho, rI = g.r, ux = g.ux, uy = g.uy, uz = g.uz;
    // the outgoing invariant w = u_n -+ p / cs (06:694-698 low side, 06:721-725 high side),
    // u_B = w / 2, p_B = -+ cs w / 2 and rho_B' = p_B / cs^2
    constexpr float cs = (float)kCs, cs2 = (float)kCs2;
    const float un = AXIS == 0 ? ux : (AXIS == 1 ? uy : uz);
    const float w = SIDE == 0 ? sub(un, g.pc) : add(un, g.pc);
    const float unB = mul(0.5f, w);
    const float rhoB = over(mul(SIDE == 0 ? -0.5f * cs : 0.5f * cs, w), cs2, 1.0f / cs2);
    const float rB = fma(rhoB, inv_scale, 1.0f);
    const float bx = AXIS == 0 ? unB : ux, by = AXIS == 1 ? unB : uy, bz = AXIS == 2 ? unB : uz;
    // geq(B) - geq(I) = w_q (d0 + c.v + c^T M c), a quadratic form in
    // c_q whose ten coefficients are taken once per cell
    const float k45 = mul(4.5f, inv_scale), k90 = mul(9.0f, inv_scale);
    const float b2 = fma(bz, bz, fma(bx, bx, mul(by, by))), u2 = fma(uz, uz, fma(ux, ux, mul(uy, uy)));
    const float d0 = fma(mul(-1.5f, inv_scale), fma(rB, b2, -mul(rI, u2)), sub(rhoB, rho));
    const float qx = mul(rB, bx), qy = mul(rB, by), qz = mul(rB, bz);
    const float px = mul(rI, ux), py = mul(rI, uy), pz = mul(rI, uz);
    const float vx = sub(qx, px), vy = sub(qy, py), vz = sub(qz, pz);
    const float mxx = fma(qx, bx, -mul(px, ux)), myy = fma(qy, by, -mul(py, uy)), mzz = fma(qz, bz, -mul(pz, uz));
    const float mxy = fma(qx, by, -mul(px, uy)), mxz = fma(qx, bz, -mul(px, uz)), myz = fma(qy, bz, -mul(py, uz));
#pragma unroll
    for (int q = 0; q < Q; ++q)
    {
        if (!inward<AXIS, SIDE>(q)) continue;
        float e = d0;
        if (ex(q)) e = fma(k45, mxx, e);
        if (ey(q)) e = fma(k45, myy, e);
        if (ez(q)) e = fma(k45, mzz, e);
        if (ex(q) * ey(q)) e = fma(ex(q) * ey(q) > 0 ? k90 : -k90, mxy, e);
        if (ex(q) * ez(q)) e = fma(ex(q) * ez(q) > 0 ? k90 : -k90, mxz, e);
        if (ey(q) * ez(q)) e = fma(ey(q) * ez(q) > 0 ? k90 : -k90, myz, e);
        if (ex(q)) e = fma(ex(q) > 0 ? 3.0f : -3.0f, vx, e);
        if (ey(q)) e = fma(ey(q) > 0 ? 3.0f : -3.0f, vy, e);
        if (ez(q)) e = fma(ez(q) > 0 ? 3.0f : -3.0f, vz, e);
        put(q, fma(wf(q), e, get(q)));
    }
}

// ---------------------------------------------------------------- probes
// rho - 1 at probe p for the step whose pre-step buffer is `f` (the value
// LBMSolver::run records, 06:1085-1092; SOLID cells read 0).  One warp per
// probe, lane q pulls direction q (halfway bounce-back included, x-halo
// sources from the x-face ghosts), so a probe is three dependent loads; the
// sum is taken in direction order.  (One thread per probe pulled its 19
// values one after another: 6-17 us a launch beside or after each step.)
template <typename S>
__device__ __forceinline__ float probe_value(const S* p);
template <>
__device__ __forceinline__ float probe_value<float>(const float* p) { return __ldg(p); }
template <>
__device__ __forceinline__ float probe_value<__half>(const __half* p) { return __half2float(__ldg(p)); }

__device__ __forceinline__ float sum_directions(float g)
{
    float rho = 0.f;
#pragma unroll
    for (int q = 0; q < Q; ++q) rho += __shfl_sync(0xffffffffu, g, q);
    return rho;
}
__device__ __forceinline__ void record_probe(const ProbeArgs& a, long long row, int p, bool owned, double val)
{
    if (owned)
    {
        a.energy[p] += val * val;
        if (!isfinite(val)) *a.nonfinite = 1;
    }
    a.out[row * a.n + p] = val;
}

template <typename S>
__device__ __forceinline__ void probe_warp(const S* __restrict__ f, const Layout& L, const uint32_t* __restrict__ links,
                                           const float* __restrict__ xgh, const ProbeArgs& a, long long row, int p,
                                           int lane)
{
    const int i = a.ijk[3 * p], j = a.ijk[3 * p + 1], k = a.ijk[3 * p + 2];
    if (i < 0)
    {
        if (lane == 0) record_probe(a, row, p, false, __longlong_as_double(0x7ff8000000000000LL));
        return;
    }
    const uint32_t lk = links[L.cell(i, j, k)];
    float g = 0.f;
    if (lane < Q)
    {
        const int q = lane, si = i - e_of<0>(q), sj = j - e_of<1>(q), sk = k - e_of<2>(q);
        const bool back = (lk >> q) & 1u;
        if (!back && (si == 0 || si == L.nx + 1))
        {
            g = xgh[XFace{nullptr, nullptr}.gh_index(si == 0 ? 0 : 1, q, sj, sk, L.ny, L.nz)];
        }
        else
        {
            const long long e = back ? L.elem(inv_of(q), i, j, k) : L.elem(q, si, sj, sk);
            if (LBM_IN(kChkProbe, e, L.total)) g = probe_value<S>(f + e);
        }
    }
    const float rho = sum_directions(g);
    if (lane == 0)
    {
        const float rp = rho * (1.0f / a.scale);
        double val;
        if ((lk & kSolidSelfBit) != 0u) val = 0.0;
        else if (1.0f + rp <= 0.f) val = 1e-12 - 1.0;
        else val = (double)rp;
        record_probe(a, row, p, true, val);
    }
}

}  // namespace
}  // namespace lbm
