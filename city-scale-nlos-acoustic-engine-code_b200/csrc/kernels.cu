// sm_100a kernels of the D3Q19 acoustic step (family-B semantics of
// 06_transient_localization_dx1.cpp).  Storage is FP32 or FP16 deviations from
// rest equilibrium in the block-interleaved layout of device.hpp; arithmetic
// is FP32 (packed FP32x2 where two cells go together), with FP64 for the
// source-weight reduction and the probe accumulators.
#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <mutex>
#include <type_traits>

#include "check.cuh"
#include "device.hpp"
#include "epilogue.cuh"
#include "lattice.cuh"

namespace lbm {
namespace {

constexpr unsigned kFull = 0xffffffffu;

#ifdef LBM_CHECK
// Extents of the side arrays (elements), for the bounds-checked build.
__device__ __forceinline__ long long links_extent(const Layout& L) { return L.plane * (L.nz + 2); }
__device__ __forceinline__ long long near_extent(const Layout& L)
{
    return (long long)L.words_per_row * (L.ny + 2) * (L.nz + 2);
}
__device__ __forceinline__ long long xgh_extent(const Layout& L) { return 2LL * 19 * (L.nz + 2) * (L.ny + 2); }
__device__ __forceinline__ long long xexp_extent(const Layout& L) { return 2LL * 19 * L.nz * L.ny; }
#endif

// Scalar access.  ld: read-only path (arrays the kernel does not write);
// ldw: coherent load for arrays the same kernel also writes.
template <typename S>
struct Io;

template <>
struct Io<float>
{
    static __device__ __forceinline__ float ld(const float* p) { return __ldg(p); }
    static __device__ __forceinline__ float ldw(const float* p) { return *p; }
    static __device__ __forceinline__ void st(float* p, float v) { *p = v; }
};

template <>
struct Io<__half>
{
    static __device__ __forceinline__ float ld(const __half* p) { return __half2float(__ldg(p)); }
    static __device__ __forceinline__ float ldw(const __half* p) { return __half2float(*p); }
    static __device__ __forceinline__ void st(__half* p, float v) { *p = __float2half_rn(v); }
};

// Two x-adjacent FP32 cells as one aligned vector.
struct PairIo
{
    using V = float2;
    static __device__ __forceinline__ V ld(const float* p) { return __ldg(reinterpret_cast<const float2*>(p)); }
    static __device__ __forceinline__ void st(float* p, float2 v) { *reinterpret_cast<float2*>(p) = v; }
    // cells (c-1, c) from the previous pair's high element and cur = (c, c+1)
    static __device__ __forceinline__ float2 left(float prev_hi, V cur) { return make_float2(prev_hi, cur.x); }
    // cells (c+1, c+2) from cur = (c, c+1) and the next pair's low element
    static __device__ __forceinline__ float2 right(V cur, float next_lo) { return make_float2(cur.y, next_lo); }
};

__device__ __forceinline__ uint32_t near_bits(const StepArgs& a, const Layout& L, int col, int j, int k)
{
    return a.near[((long long)k * (L.ny + 2) + j) * L.words_per_row + (col >> 5)] >> (col & 31);
}

// Pulled populations of one cell (halo-inclusive coordinates i, j, k),
// halfway bounce-back included (06:918-931); x-halo sources read the x-face
// ghosts.  Used by the probe and field kernels.
template <typename S>
__device__ __forceinline__ void pull_cell(const S* __restrict__ f, const Layout& L, const StepArgs& sa, int i, int j,
                                          int k, float (&G)[Q], bool& solid)
{
    const uint32_t lk = sa.links[L.cell(i, j, k)];
    solid = (lk & kSolidSelfBit) != 0u;
#pragma unroll
    for (int q = 0; q < Q; ++q)
    {
        const int si = i - ex(q);
        long long e = -1;
        G[q] = 0.f;
        if ((lk >> q) & 1u) e = L.elem(inv(q), i, j, k);
        else if (si == 0) G[q] = sa.xf.xgh[sa.xf.gh_index(0, q, j - ey(q), k - ez(q), L.ny, L.nz)];
        else if (si == L.nx + 1) G[q] = sa.xf.xgh[sa.xf.gh_index(1, q, j - ey(q), k - ez(q), L.ny, L.nz)];
        else e = L.elem(q, si, j - ey(q), k - ez(q));
        if (e >= 0 && LBM_IN(kChkProbe, e, L.total)) G[q] = Io<S>::ld(f + e);
    }
}

// y and z components of the velocities, for per-lane index arithmetic
__constant__ signed char c_ey[19] = {0, 0, 0, 1, -1, 0, 0, 1, -1, 1, -1, 0, 0, 0, 0, 1, 1, -1, -1};
__constant__ signed char c_ez[19] = {0, 0, 0, 0, 0, 1, -1, 0, 0, 0, 0, 1, -1, 1, -1, 1, -1, 1, -1};

// ---------------------------------------------------------------- step
// Packed FP32x2 arithmetic (sm_100): both cells of a thread's pair in one
// instruction.
__device__ __forceinline__ float2 f2(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, f2(-1.0f), a); }

// BGK + sponge of two cells in lockstep, in place, deviation form (06:940-967).
// With stored G = scale * (f - w):
//   rho' = sum G, J = sum c G, r = 1 + rho'/scale (guard r <= 0 -> 1e-12, 06:948)
//   Geq_q = w_q (rho' + 3 c.J + (4.5 (c.J)^2 - 1.5 J^2) / (scale r))
//   G'    = (1 - sigma) (G - omega (G - Geq))      [sponge blend toward w_q, 06:955-965]
// A SOLID cell gets cA = 1, cB = 0, so its pulled values pass through
// unchanged (06:933-938).  on_moments(rho', jx, jy, jz) receives the moments
// of the pulled populations as soon as they are summed (the adjoint's forward
// data), so nothing beyond the collision's own values stays live for them.
template <typename OnMoments>
__device__ __forceinline__ void collide2(float2 (&G)[Q], float inv_scale, float omega, float2 sigma, bool solid0,
                                         bool solid1, OnMoments&& on_moments)
{
    // rho' and J in the family-B order (06:21-23)
    const float2 rho = add2(add2(add2(add2(G[0], G[1]), add2(G[2], G[3])), add2(add2(G[4], G[5]), add2(G[6], G[7]))),
                            add2(add2(add2(G[8], G[9]), add2(G[10], G[11])),
                                 add2(add2(add2(G[12], G[13]), add2(G[14], G[15])), add2(add2(G[16], G[17]), G[18]))));
    const float2 jx = sub2(add2(add2(add2(G[1], G[7]), add2(G[8], G[11])), G[12]),
                           add2(add2(add2(G[2], G[9]), add2(G[10], G[13])), G[14]));
    const float2 jy = sub2(add2(add2(add2(G[3], G[7]), add2(G[9], G[15])), G[16]),
                           add2(add2(add2(G[4], G[8]), add2(G[10], G[17])), G[18]));
    const float2 jz = sub2(add2(add2(add2(G[5], G[11]), add2(G[13], G[15])), G[17]),
                           add2(add2(add2(G[6], G[12]), add2(G[14], G[16])), G[18]));
    on_moments(rho, jx, jy, jz);
    float2 r = fma2(rho, f2(inv_scale), f2(1.0f));
    if (r.x <= 0.f) r.x = 1e-12f;   // 06:948
    if (r.y <= 0.f) r.y = 1e-12f;
    const float2 irs = make_float2(__fdividef(inv_scale, r.x), __fdividef(inv_scale, r.y));
    const float2 j2 = fma2(jz, jz, fma2(jy, jy, mul2(jx, jx)));
    const float2 base = fma2(mul2(irs, j2), f2(-1.5f), rho);
    const float2 k45 = mul2(irs, f2(4.5f));
    const float2 keep = sub2(f2(1.0f), sigma);
    float2 cA = mul2(keep, f2(1.0f - omega));
    float2 cB = mul2(keep, f2(omega));
    if (solid0) cA.x = 1.0f, cB.x = 0.0f;
    if (solid1) cA.y = 1.0f, cB.y = 0.0f;
    const float2 cBw1 = mul2(cB, f2(wf(1))), cBw2 = mul2(cB, f2(wf(7)));
    const float2 cBt1 = mul2(cB, f2(3.0f * wf(1))), cBt2 = mul2(cB, f2(3.0f * wf(7)));
    G[0] = fma2(cA, G[0], mul2(mul2(cB, f2(wf(0))), base));
#pragma unroll
    for (int p = 0; p < 9; ++p)
    {
        const int q = pair_head(p);
        const int qb = inv(q);
        float2 cj;
        if (p == 0) cj = jx;                  // q = 1  ( 1, 0, 0)
        else if (p == 1) cj = jy;             // q = 3  ( 0, 1, 0)
        else if (p == 2) cj = jz;             // q = 5  ( 0, 0, 1)
        else if (p == 3) cj = add2(jx, jy);   // q = 7  ( 1, 1, 0)
        else if (p == 4) cj = sub2(jx, jy);   // q = 8  ( 1,-1, 0)
        else if (p == 5) cj = add2(jx, jz);   // q = 11 ( 1, 0, 1)
        else if (p == 6) cj = sub2(jx, jz);   // q = 12 ( 1, 0,-1)
        else if (p == 7) cj = add2(jy, jz);   // q = 15 ( 0, 1, 1)
        else cj = sub2(jy, jz);               // q = 16 ( 0, 1,-1)
        const float2 cBw = q < 7 ? cBw1 : cBw2;
        const float2 cBt = q < 7 ? cBt1 : cBt2;
        const float2 e = mul2(cBw, fma2(k45, mul2(cj, cj), base));
        const float2 o = mul2(cBt, cj);
        G[q] = fma2(cA, G[q], add2(e, o));
        G[qb] = fma2(cA, G[qb], sub2(e, o));
    }
}

// What a step launch does beyond the update: nothing (single calls); the
// blocks beside it (probe record, step counter); those and the next step's
// sources and ghosts.
enum StepMode { kPlain = 0, kSide = 1, kFused = 2 };

// Blocks beside a batched step's own: block 0 prepares the sources of the step
// after the next (fused) and advances the step counter, the others record this
// step's probes, a warp each.  They read what the step only reads.
__host__ __device__ constexpr int side_blocks(int nprobe, int warps) { return 1 + (nprobe + warps - 1) / warps; }

template <typename S, int MODE>
__device__ __forceinline__ void side_block(const S* __restrict__ fin, const Layout& L, const StepArgs& a,
                                           const FusedArgs& fa, int block, double* red)
{
    const long long s = fa.ctl ? fa.ctl->step[fa.parity] : fa.direct_step;
    if (block == 0)
    {
        if (MODE == kFused) prepare_sources(fa.prep, fa.src, s + 2, s + 1 < fa.ctl->last, L, a.links, red);
        if (fa.ctl && threadIdx.x == 0)
        {
            fa.ctl->step[fa.parity ^ 1] = s + 1;
            fa.ctl->rows[fa.parity ^ 1] = 0;
        }
        return;
    }
    const int p = (block - 1) * (int)(blockDim.x >> 5) + (int)(threadIdx.x >> 5);
    if (p < fa.probe.n)
        probe_warp<S>(fin, L, a.links, a.xf.xgh, fa.probe, fa.ctl ? s - fa.ctl->probe_base : fa.probe.direct_row, p,
                      threadIdx.x & 31);
}

// The next step's sources on a pair's results (kernel of FP32 storage).
__device__ __forceinline__ void add_sources(float2 (&G)[Q], const SourceNext* __restrict__ nx, unsigned sources, int c0,
                                            int j, int k, const Layout& L)
{
    while (sources)
    {
        const int s = __ffs(sources) - 1;
        sources &= sources - 1;
        const SourceBox b = nx->box[s];
        const int row = ((k - b.k0) * b.n + (j - b.j0)) * b.n, d = c0 + 1 - b.i0;
        const bool in0 = d >= 0 && d < b.n, in1 = d + 1 >= 0 && d + 1 < b.n && c0 + 1 < L.nx;
        float4 a0 = make_float4(0.f, 0.f, 0.f, 0.f), a1 = a0;
        if (in0 && LBM_IN(kChkSource, row + d, kStencilCells)) a0 = nx->add[s][row + d];
        if (in1 && LBM_IN(kChkSource, row + d + 1, kStencilCells)) a1 = nx->add[s][row + d + 1];
        if (a0.w != 0.f)
        {
#pragma unroll
            for (int q = 0; q < Q; ++q) G[q].x += source_gain(a0, q);
        }
        if (a1.w != 0.f)
        {
#pragma unroll
            for (int q = 0; q < Q; ++q) G[q].y += source_gain(a1, q);
        }
    }
}

// The next step's ghosts of an open y or z face from a pair's results; `ghost`
// is the pair's place in the halo row of buffer `f`.
template <int AXIS, int SIDE>
__device__ __forceinline__ void ghost_pair(const float2 (&G)[Q], const GhostState& s0, const GhostState& s1, float* ghost,
                                           [[maybe_unused]] const float* f, [[maybe_unused]] long long total)
{
    constexpr int BC = block_cells(sizeof(float));
    float2 o[Q];
    nscbc<AXIS, SIDE>(s0, 1.0f, [&](int q) { return G[q].x; }, [&](int q, float v) { o[q].x = v; });
    nscbc<AXIS, SIDE>(s1, 1.0f, [&](int q) { return G[q].y; }, [&](int q, float v) { o[q].y = v; });
#pragma unroll
    for (int q = 0; q < Q; ++q)
        if (inward<AXIS, SIDE>(q) && LBM_IN(kChkGhost, ghost - f + q * BC, total - 1))
            *reinterpret_cast<float2*>(ghost + q * BC) = o[q];
}
// ... and of an open x face, from the cell at the row's end.
template <int SIDE, typename Get>
__device__ __forceinline__ void ghost_end(const GhostState& s, float inv_scale, const FusedArgs& fa, const XFace& xf,
                                          const Layout& L, int j, int k, Get&& get)
{
    nscbc<0, SIDE>(s, inv_scale, get, [&](int q, float v) {
        const long long e = xf.gh_index(SIDE, q, j, k, L.ny, L.nz);
        if (LBM_IN(kChkGhost, e, xgh_extent(L))) fa.xgh_out[e] = v;
    });
}

// Moments of the ghosts' interior cells, for the adjoint: the pair (c0, c0 + 1)
// of row (j, k), `row` its open y and z faces, `ends` the x faces that its first
// (bits 0-1) and second cell (bits 2-3) border.
__device__ __forceinline__ void keep_face_moments(const FusedArgs& fa, const Layout& L, unsigned row, unsigned ends, int c0,
                                                  int j, int k, const float4& m0, const float4& m1)
{
    const long long xc = (long long)(k - 1) * L.ny + (j - 1), yc = (long long)(k - 1) * L.nx + c0,
                    zc = (long long)(j - 1) * L.nx + c0;
    const auto put = [&](long long t, const float4& m) {
        if (LBM_IN(kChkGhost, t, fa.face_total)) fa.face_mom[t] = m;
    };
#pragma unroll
    for (int f = 2; f < 6; ++f)
    {
        if (!((row >> f) & 1u)) continue;
        put(fa.face_first[f] + (f < 4 ? yc : zc), m0);
        if (c0 + 1 < L.nx) put(fa.face_first[f] + (f < 4 ? yc : zc) + 1, m1);
    }
    if (ends & 1u) put(fa.face_first[0] + xc, m0);
    if (ends & 2u) put(fa.face_first[1] + xc, m0);
    if (ends & 8u) put(fa.face_first[1] + xc, m1);
}

// Open y and z faces that row (j, k) borders.
__device__ __forceinline__ unsigned row_faces(unsigned open, int j, int k, const Layout& L)
{
    return open & ((j == 1 ? 4u : 0u) | (j == L.ny ? 8u : 0u) | (k == 1 ? 16u : 0u) | (k == L.nz ? 32u : 0u));
}

// Fused pull-stream + halfway bounce-back + BGK + sponge (06:906-972), two
// x-adjacent cells per thread.  Direction q of the pair comes from the row
// (j - ey, k - ez) of the block-interleaved layout as one aligned vector at
// a compile-time offset from that row's base; the +-1 x shift of directions
// with ex != 0 takes the missing neighbour element from the adjacent lane
// (warp shuffle) and, at the warp edge, from one extra aligned load.  Cells
// next to the x faces take their x-halo sources from the x-face ghosts and
// export their results for the next ghost fill.
// MOM: also write the moments (rho', J) of every cell's pulled populations to
// `mom` (PairMoments: 12-bit floats, one record per x pair), the forward data
// the adjoint's BGK Jacobian needs.
// FP16 bits of x rounded to nearest-even at their 4 lowest mantissa bits:
// sign at bit 11, exponent at bits 6-10, 6 mantissa bits (finite values only).
__device__ __forceinline__ unsigned to_f12(float x)
{
    const unsigned h = (unsigned)__half_as_ushort(__float2half_rn(x));
    const unsigned mag = h & 0x7fffu;
    const unsigned r = min((mag + 7u + ((mag >> 4) & 1u)) >> 4, 0x7bfu);
    return ((h >> 15) << 11) | r;
}
__device__ __forceinline__ PairMoments pack_moments(float4 m0, float4 m1)
{
    const unsigned v0 = to_f12(m0.x), v1 = to_f12(m0.y), v2 = to_f12(m0.z), v3 = to_f12(m0.w);
    const unsigned v4 = to_f12(m1.x), v5 = to_f12(m1.y), v6 = to_f12(m1.z), v7 = to_f12(m1.w);
    return PairMoments{{v0 | (v1 << 12) | (v2 << 24), (v2 >> 8) | (v3 << 4) | (v4 << 16) | (v5 << 28),
                        (v5 >> 4) | (v6 << 8) | (v7 << 20)}};
}

// MODE: the last side_rows rows of blocks of every layer are the blocks beside
// the step (a block's own row and plane stay plain block indices); a fused
// step writes the x-face exports only where its results stay as they are.
// 80 registers (24 warps per SM) for the fused step: at the plain step's 72 it
// spills 40 bytes, 256x256x128 233 us a step against 218; at 96 250 us.
template <int BX, bool MOM, int MODE>
__global__ void __launch_bounds__(kPairBlock, MODE == kFused ? 6 : 0) k_step(const float* __restrict__ fin, float* __restrict__ fout, Layout L,
                                                      StepArgs a, PairMoments* __restrict__ mom,
                                                      const __grid_constant__ FusedArgs fa, int side_rows)
{
    using S = float;
    using P = PairIo;
    constexpr bool FUSED = MODE == kFused;
    if constexpr (MODE != kPlain) fin = chain_wait(fin);
    if constexpr (MODE != kPlain)
    {
        const int row0 = (int)gridDim.y - side_rows;
        if ((int)blockIdx.y >= row0)
        {
            __shared__ double red[16];
            const int block =
                ((int)blockIdx.z * side_rows + (int)blockIdx.y - row0) * (int)gridDim.x + (int)blockIdx.x;
            if (block < side_blocks(fa.probe.n, kPairBlock / 32)) side_block<S, MODE>(fin, L, a, fa, block, red);
            return;
        }
    }
    constexpr int BC = block_cells(sizeof(S));   // cells per interleaved block
    constexpr int BE = 19 * BC;                   // elements per block
    const int lane = threadIdx.x & 31;
    const int c0r = pair_column<BX>();                        // first column (0-based) of the pair
    const bool active = c0r < L.nx;
    const int c0 = active ? c0r : ((L.nx - 1) & ~1);         // inactive lanes shadow a valid pair
    const int j = pair_row<BX>();
    const int k = blockIdx.z + 1;
    if (BX < 4 && j > L.ny) return;   // whole warps
    const long long e0 = L.elem(0, c0 + 1, j, k);
    const S* own = fin + e0;
    const long long rs = L.row_stride, ps = L.plane_stride;

    // pair load (the bounds-checked build tests the index first)
    const auto ldp = [&](const S* p) -> typename P::V {
        if (LBM_IN(kChkStepLoad, p - fin, L.total - 1)) return P::ld(p);
        return typename P::V{};
    };

    uint32_t lk0 = 0, lk1 = 0;
    if (active)
    {
        const uint32_t b = near_bits(a, L, c0, j, k) & 3u;
        const long long cl = L.cell(c0 + 1, j, k);
        if (b & 1u) lk0 = a.links[cl];
        if (b & 2u) lk1 = a.links[cl + 1];
    }
    const bool any_link = __any_sync(kFull, (lk0 | lk1) != 0u);
    float2 G[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q)
    {
        const S* row = own - (ey(q) * rs + ez(q) * ps);
        const typename P::V cur = ldp(row + q * BC);
        if (ex(q) == 0)
        {
            G[q] = cur;
        }
        else if (ex(q) > 0)
        {
            // lane 0 sits at the start of a block: its left neighbour pair is
            // the last pair of the previous block
            auto prev = __shfl_up_sync(kFull, cur.y, 1);
            if (lane == 0) prev = ldp(row + q * BC - BE + (BC - 2)).y;
            G[q] = P::left(prev, cur);
        }
        else
        {
            // lane 31 sits at the last pair of a block: its right neighbour
            // pair is the first pair of the next block
            auto next = __shfl_down_sync(kFull, cur.x, 1);
            if (lane == 31) next = ldp(row + q * BC + BE - (BC - 2)).x;
            G[q] = P::right(cur, next);
        }
    }
    if (any_link)
    {
#pragma unroll
        for (int q = 0; q < Q; ++q)
        {
            if (((lk0 | lk1) >> q) & 1u)
            {
                const float2 o = ldp(own + inv(q) * BC);
                if ((lk0 >> q) & 1u) G[q].x = o.x;
                if ((lk1 >> q) & 1u) G[q].y = o.y;
            }
        }
    }
    // FUSED: bits 0-7 the sources whose cells the row holds, bit 8 that results take sources and ghosts at all
    unsigned todo = 0u;
    if constexpr (FUSED)
    {
        if (fa.next->fill != 0)
        {
            todo = 256u;
            if (fa.src.nsrc > 0) todo |= sources_of_row(fa.next, fa.src.nsrc, lane, j, k);
        }
    }

    // x faces: sources in the x halo come from the x-face ghosts.
    const bool xlo = active && c0 == 0;
    const bool xhi0 = active && c0 == L.nx - 1;       // nx odd: first cell of the pair is the last
    const bool xhi1 = active && c0 + 1 == L.nx - 1;   // nx even: second cell is the last
    if (xlo | xhi0 | xhi1)
    {
#pragma unroll
        for (int q = 0; q < Q; ++q)
        {
            if (ex(q) == 0) continue;
            const float g = a.xf.xgh[a.xf.gh_index(ex(q) > 0 ? 0 : 1, q, j - ey(q), k - ez(q), L.ny, L.nz)];
            if (ex(q) > 0 && xlo && !((lk0 >> q) & 1u)) G[q].x = g;
            if (ex(q) < 0 && xhi0 && !((lk0 >> q) & 1u)) G[q].x = g;
            if (ex(q) < 0 && xhi1 && !((lk1 >> q) & 1u)) G[q].y = g;
        }
    }
    if (!active) return;

    const float syz = fmaxf(a.sig_y[j - 1], a.sig_z[k - 1]);
    const float2 sg = make_float2(fmaxf(a.sig_x[c0], syz), fmaxf(c0 + 1 < L.nx ? a.sig_x[c0 + 1] : 0.f, syz));
    collide2(G, 1.0f, a.omega, sg, (lk0 & kSolidSelfBit) != 0u, (lk1 & kSolidSelfBit) != 0u,
             [&](float2 rho, float2 jx, float2 jy, float2 jz) {
                 if constexpr (MOM)
                 {
                     const long long pi = ((long long)(k - 1) * L.ny + (j - 1)) * ((L.nx + 1) >> 1) + (c0 >> 1);
                     mom[pi] = pack_moments(make_float4(rho.x, jx.x, jy.x, jz.x),
                                            c0 + 1 < L.nx ? make_float4(rho.y, jx.y, jy.y, jz.y)
                                                          : make_float4(0.f, 0.f, 0.f, 0.f));
                 }
             });

    S* out = fout + e0;
    if (FUSED && (todo & 255u)) add_sources(G, fa.next, todo & 255u, c0, j, k, L);
#pragma unroll
    for (int q = 0; q < Q; ++q)
        if (LBM_IN(kChkStepStore, e0 + q * BC, L.total - 1)) P::st(out + q * BC, G[q]);

    if constexpr (FUSED)
    {
        if (todo & 256u)
        {
            const unsigned row = row_faces(fa.open, j, k, L);
            const unsigned ends = (xlo ? fa.open & 1u : 0u) | (xhi0 ? fa.open & 2u : 0u) | (xhi1 ? (fa.open & 2u) << 2 : 0u);
            if (!(row | ends)) return;
            // a row's end takes the moments of its own cell only, unless the whole row is a face
            float4 m0 = make_float4(0.f, 0.f, 0.f, 0.f), m1 = m0;
            if (row | (ends & 3u)) m0 = cell_moments([&](int q) { return G[q].x; });
            if (row | (ends & 8u)) m1 = cell_moments([&](int q) { return G[q].y; });
            const GhostState s0 = ghost_state(m0, 1.0f), s1 = ghost_state(m1, 1.0f);
            // halo rows of the pair; within the buffer, as every pulled row is
            if (row & 4u) ghost_pair<1, 0>(G, s0, s1, out - rs, fout, L.total);
            if (row & 8u) ghost_pair<1, 1>(G, s0, s1, out + rs, fout, L.total);
            if (row & 16u) ghost_pair<2, 0>(G, s0, s1, out - ps, fout, L.total);
            if (row & 32u) ghost_pair<2, 1>(G, s0, s1, out + ps, fout, L.total);
            if (ends & 1u) ghost_end<0>(s0, 1.0f, fa, a.xf, L, j, k, [&](int q) { return G[q].x; });
            if (ends & 10u)
                ghost_end<1>(xhi0 ? s0 : s1, 1.0f, fa, a.xf, L, j, k, [&](int q) { return xhi0 ? G[q].x : G[q].y; });
            if (fa.face_mom) keep_face_moments(fa, L, row, ends, c0, j, k, m0, m1);
            return;
        }
    }

    if (xlo | xhi0 | xhi1)
    {
#pragma unroll
        for (int q = 0; q < Q; ++q)
        {
            if (xlo) a.xf.xexp[a.xf.exp_index(0, q, j, k, L.ny, L.nz)] = G[q].x;
            if (xhi0) a.xf.xexp[a.xf.exp_index(1, q, j, k, L.ny, L.nz)] = G[q].x;
            if (xhi1) a.xf.xexp[a.xf.exp_index(1, q, j, k, L.ny, L.nz)] = G[q].y;
        }
    }
}

// ---------------------------------------------------------------- FP16 step
// FP16 storage keeps the 19 directions of a cell pair packed as half2 words
// through the whole update: the moment pass and the update pass each convert
// a word to float2 right before use, so no 19 x float2 array is ever live and
// the kernel needs far fewer registers (more warps, more loads in flight).
__device__ __forceinline__ float2 h2f(unsigned u)
{
    __half2 h;
    *reinterpret_cast<unsigned*>(&h) = u;
    return __half22float2(h);
}
__device__ __forceinline__ unsigned f2h(float2 v)
{
    const __half2 h = __float22half2_rn(v);
    return *reinterpret_cast<const unsigned*>(&h);
}
__device__ __forceinline__ unsigned set_lo(unsigned w, float v)
{
    return (w & 0xffff0000u) | (unsigned)__half_as_ushort(__float2half_rn(v));
}
__device__ __forceinline__ unsigned set_hi(unsigned w, float v)
{
    return (w & 0x0000ffffu) | ((unsigned)__half_as_ushort(__float2half_rn(v)) << 16);
}

// collide2() on packed FP16 words: each word is converted to FP32 once; the moments share partial sums
// (rho = g0 + rest + S(x+) + S(x-), jx = S(x+) - S(x-)); each direction of a
// pair (q, inv q) is two FMAs from the pair's equilibrium term
//   e = (cB w k45) (c.J)^2 + cB w base,   G'_q = cA G_q + e +- 3 cB w (c.J).
// Same formulas as collide2(); the rounding order differs.
__device__ __forceinline__ void collide2_grouped(unsigned (&w)[Q], float inv_scale, float omega, float2 sigma,
                                                 bool solid0, bool solid1)
{
    float2 g[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) g[q] = h2f(w[q]);
    const float2 sxp = add2(add2(add2(g[1], g[7]), add2(g[8], g[11])), g[12]);
    const float2 sxn = add2(add2(add2(g[2], g[9]), add2(g[10], g[13])), g[14]);
    const float2 rest = add2(add2(add2(g[3], g[4]), add2(g[5], g[6])), add2(add2(g[15], g[16]), add2(g[17], g[18])));
    const float2 rho = add2(add2(g[0], rest), add2(sxp, sxn));
    const float2 jx = sub2(sxp, sxn);
    const float2 jy = sub2(add2(add2(add2(g[3], g[7]), add2(g[9], g[15])), g[16]),
                           add2(add2(add2(g[4], g[8]), add2(g[10], g[17])), g[18]));
    const float2 jz = sub2(add2(add2(add2(g[5], g[11]), add2(g[13], g[15])), g[17]),
                           add2(add2(add2(g[6], g[12]), add2(g[14], g[16])), g[18]));
    float2 r = fma2(rho, f2(inv_scale), f2(1.0f));
    if (r.x <= 0.f) r.x = 1e-12f;   // 06:948
    if (r.y <= 0.f) r.y = 1e-12f;
    const float2 irs = make_float2(__fdividef(inv_scale, r.x), __fdividef(inv_scale, r.y));
    const float2 j2 = fma2(jz, jz, fma2(jy, jy, mul2(jx, jx)));
    const float2 base = fma2(mul2(irs, j2), f2(-1.5f), rho);
    const float2 k45 = mul2(irs, f2(4.5f));
    const float2 keep = sub2(f2(1.0f), sigma);
    float2 cA = mul2(keep, f2(1.0f - omega));
    float2 cB = mul2(keep, f2(omega));
    if (solid0) cA.x = 1.0f, cB.x = 0.0f;
    if (solid1) cA.y = 1.0f, cB.y = 0.0f;
    const float2 cBw1 = mul2(cB, f2(wf(1))), cBw2 = mul2(cB, f2(wf(7)));
    const float2 K1 = mul2(cBw1, k45), K2 = mul2(cBw2, k45);
    const float2 B1 = mul2(cBw1, base), B2 = mul2(cBw2, base);
    const float2 T1 = mul2(cB, f2(3.0f * wf(1))), T2 = mul2(cB, f2(3.0f * wf(7)));
    const float2 N1 = mul2(cB, f2(-3.0f * wf(1))), N2 = mul2(cB, f2(-3.0f * wf(7)));
    w[0] = f2h(fma2(cA, g[0], mul2(mul2(cB, f2(wf(0))), base)));
#pragma unroll
    for (int p = 0; p < 9; ++p)
    {
        const int q = pair_head(p);
        const int qb = inv(q);
        float2 cj;
        if (p == 0) cj = jx;
        else if (p == 1) cj = jy;
        else if (p == 2) cj = jz;
        else if (p == 3) cj = add2(jx, jy);
        else if (p == 4) cj = sub2(jx, jy);
        else if (p == 5) cj = add2(jx, jz);
        else if (p == 6) cj = sub2(jx, jz);
        else if (p == 7) cj = add2(jy, jz);
        else cj = sub2(jy, jz);
        const float2 e = fma2(q < 7 ? K1 : K2, mul2(cj, cj), q < 7 ? B1 : B2);
        w[q] = f2h(fma2(q < 7 ? T1 : T2, cj, fma2(cA, g[q], e)));
        w[qb] = f2h(fma2(q < 7 ? N1 : N2, cj, fma2(cA, g[qb], e)));
    }
}

// ---------------------------------------------------------------- FP16 step, warp pipelines
// Each warp walks whole rows one interleaved block (64 cells, two per lane)
// at a time and keeps the source lines of its next P blocks in flight as
// cp.async copies into its own ring of shared-memory slots: the bytes in
// flight no longer depend on registers or on resident warps, and no barrier
// couples the warps of a CTA.  A block's 19 source lines (direction q from
// row (j - ey, k - ez)) are 152 16-byte pieces, five copy instructions per
// lane.  The x neighbour of the block's first / last cell is the last /
// first element of the previous / next block of the same row, which the ring
// still / already holds (at the row ends the x-face ghosts replace it).  The
// near-solid words of a block are loaded one block ahead of its copies and
// its links words travel with the copies when any bit is set.
namespace wp {
constexpr int kPopBytes = 19 * 128;           // one block's 19 source lines
constexpr int kLinkOff = kPopBytes;           // 64 links words
constexpr int kNearOff = kPopBytes + 256;     // the block's 2 near-solid words
constexpr int kGhostOff = kNearOff + 16;      // x-face ghosts of a row-end block: 5 per side
constexpr int kSlotBytes = kGhostOff + 48;
// A warp's ring has P + 1 slots; of the block before the one being updated it keeps the last words (the
// directions with ex > 0), in the place of the low x face's ghosts, which only a row's first block has.  With a
// slot for that block (11.0 instead of 8.3 KB a warp) the L1 cache had 28 KB left, and the bounce-back words of
// near-solid blocks, up to 18 lines at a time, waited for room in it: a 1024x1024x256 city step 3898 us against
// 3836 (both with fixed rows).
// Directions with ex > 0 (ghosts of the low x face) and ex < 0 (high face).
__device__ __forceinline__ int ghost_dir(int i) { return i < 5 ? (i < 1 ? 1 : i < 3 ? i + 6 : i + 8) : (i < 6 ? 2 : i < 8 ? i + 3 : i + 5); }
}  // namespace wp

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async8(uint32_t dst, const void* src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async4(uint32_t dst, const void* src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait()
{
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// Position of direction q (ex != 0) in a slot's x-face ghosts (inverse of wp::ghost_dir).
__host__ __device__ constexpr int ghost_slot(int q)
{
    constexpr int t[Q] = {-1, 0, 5, -1, -1, -1, -1, 1, 2, 6, 7, 3, 4, 8, 9, -1, -1, -1, -1};
    return t[q];
}

// The next step's sources on a word of results: as stored, one source after another.
__device__ __forceinline__ void add_sources(unsigned (&w)[Q], const SourceNext* __restrict__ nx, unsigned sources,
                                            int c0, int j, int k, const Layout& L)
{
    while (sources)
    {
        const int s = __ffs(sources) - 1;
        sources &= sources - 1;
        const SourceBox b = nx->box[s];
        const int row = ((k - b.k0) * b.n + (j - b.j0)) * b.n, d = c0 + 1 - b.i0;
        const bool in0 = d >= 0 && d < b.n, in1 = d + 1 >= 0 && d + 1 < b.n && c0 + 1 < L.nx;
        float4 a0 = make_float4(0.f, 0.f, 0.f, 0.f), a1 = a0;
        if (in0 && LBM_IN(kChkSource, row + d, kStencilCells)) a0 = nx->add[s][row + d];
        if (in1 && LBM_IN(kChkSource, row + d + 1, kStencilCells)) a1 = nx->add[s][row + d + 1];
        if (a0.w != 0.f)
        {
#pragma unroll
            for (int q = 0; q < Q; ++q) w[q] = set_lo(w[q], h2f(w[q]).x + source_gain(a0, q));
        }
        if (a1.w != 0.f)
        {
#pragma unroll
            for (int q = 0; q < Q; ++q) w[q] = set_hi(w[q], h2f(w[q]).y + source_gain(a1, q));
        }
    }
}

template <int AXIS, int SIDE>
__device__ __forceinline__ void ghost_pair(const unsigned (&w)[Q], const float4& m0, const float4& m1, float inv_scale,
                                           unsigned* ghost, [[maybe_unused]] const __half* f,
                                           [[maybe_unused]] long long total)
{
    float lo[Q];
    nscbc<AXIS, SIDE>(ghost_state(m0, inv_scale), inv_scale, [&](int q) { return h2f(w[q]).x; }, [&](int q, float v) { lo[q] = v; });
    nscbc<AXIS, SIDE>(ghost_state(m1, inv_scale), inv_scale, [&](int q) { return h2f(w[q]).y; },
                              [&](int q, float v) {
                                  if (LBM_IN(kChkGhost, 2 * (ghost - reinterpret_cast<const unsigned*>(f)) + 64 * q, total - 1))
                                      ghost[32 * q] = f2h(make_float2(lo[q], v));
                              });
}

// MODE: as k_step, the first `side` blocks beside the pipelines.
// CLAIM: a warp's first row is given, every further one is claimed from a
// counter when the copy cursor reaches the last block of the row before it.
// The SMs do not run at one speed (near-solid rows, distance to memory, the
// blocks beside the step), and with fixed rows the step waited for the slowest
// warps: 1024x1024x256 city 3833 -> 3645 us a step (82 -> 86 % of the measured
// copy bandwidth), 512x512x128 536 -> 522, 256x256x256 310 -> 302.  Which warp
// updates a row does not change its bits.  With more than P blocks in a row
// the update cursor is at most one row behind the copy cursor, so one word
// carries the next row over.
template <int P, int WARPS, int MINB, int MODE, bool CLAIM>
__global__ void __launch_bounds__(32 * WARPS, MINB) k_step_hw(const __half* __restrict__ fin,
                                                               __half* __restrict__ fout, Layout L, StepArgs a,
                                                               float inv_scale, const __grid_constant__ FusedArgs fa,
                                                               int side)
{
    constexpr int S = P + 1;   // ring slots: blocks t .. t + P
    constexpr uint32_t kDirBits = (1u << Q) - 2u;   // (a SOLID cell's direction 0 pulls its own value anyway)
    extern __shared__ __align__(128) unsigned char wp_smem[];
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    unsigned char* ring = wp_smem + warp * (S * wp::kSlotBytes);
    const uint32_t ring_s = (uint32_t)__cvta_generic_to_shared(ring);
    constexpr bool FUSED = MODE == kFused;
    if constexpr (MODE != kPlain)
    {
        if ((int)blockIdx.x < side)
        {
            side_block<__half, MODE>(fin, L, a, fa, blockIdx.x, reinterpret_cast<double*>(wp_smem));
            return;
        }
    }
    const int nrows = L.ny * L.nz;
    const int all_warps = ((int)gridDim.x - (MODE != kPlain ? side : 0)) * WARPS;
    const int r0 = ((int)blockIdx.x - (MODE != kPlain ? side : 0)) * WARPS + warp;   // rows r0, r0 + all_warps, ...; r = (k-1) ny + (j-1)
    if (r0 >= nrows) return;
    [[maybe_unused]] int claimed = 0;   // lane 0: the claimed row, less all_warps
    [[maybe_unused]] volatile int* next_row = reinterpret_cast<int*>(ring + wp::kNearOff + 8);   // of the update cursor
    const auto claim = [&]() {
        if (lane == 0) claimed = atomicAdd(&fa.ctl->rows[fa.parity], 1);
    };

    // element offsets of this lane's five 16-byte pieces from the destination block
    int poff[5];
#pragma unroll
    for (int i = 0; i < 5; ++i)
    {
        const int p = i * 32 + lane;
        const int q = min(p >> 3, 18);
        poff[i] = -(c_ey[q] * (int)L.row_stride + c_ez[q] * (int)L.plane_stride) + q * 64 + (p & 7) * 8;
    }

    // lanes 0-4 copy the low-face ghosts of a row-start block, lanes 5-9 the
    // high-face ghosts of a row-end block: ghost of direction q for row
    // (j, k) is xgh[gh_index(side, q, j - ey, k - ez)] = row (k (ny+2) + j) + goff
    const int gq = wp::ghost_dir(lane < 10 ? lane : 0);
    const int goff = (lane < 5 ? 0 : 19) * (L.nz + 2) * (L.ny + 2) + gq * (L.nz + 2) * (L.ny + 2) -
                     c_ez[gq] * (L.ny + 2) - c_ey[gq];

    // ---- copy cursor: the next block whose lines are copied
    [[maybe_unused]] int ci_r = r0;
    int ci_b = 0;
    const __half* ci_src = nullptr;     // the block's own position (lines are offset by poff)
    const uint32_t* ci_near = nullptr;  // the block's two near-solid words
    const uint32_t* ci_link = nullptr;  // links words of this lane's two cells
    const float* ci_gh = nullptr;       // this lane's x-face ghost of the row
    const auto ci_row = [&](int r) {
        const int k = 1 + r / L.ny, j = 1 + r - (k - 1) * L.ny;
        ci_src = fin + L.elem(0, 1, j, k);
        ci_near = a.near + ((long long)k * (L.ny + 2) + j) * L.words_per_row;
        ci_link = a.links + L.cell(1, j, k) + 2 * lane;
        ci_gh = a.xf.xgh + ((long long)k * (L.ny + 2) + j) + goff;
    };
    const auto ci_next = [&]() {
        ci_src += 19 * 64;
        ci_near += 2;
        ci_link += 64;
        if (++ci_b == L.nb)
        {
            ci_b = 0;
            if constexpr (CLAIM)
            {
                const int r = all_warps + __shfl_sync(kFull, claimed, 0);
                __syncwarp();   // every lane has read the row before
                if (lane == 0) *next_row = r;
                if (r < nrows) ci_row(r);
                else ci_b = -1;
            }
            else
            {
                ci_r += all_warps;
                if (ci_r < nrows) ci_row(ci_r);
            }
        }
        if (CLAIM && ci_b == L.nb - 1) claim();
    };
    const auto ci_more = [&]() { return CLAIM ? ci_b >= 0 : ci_r < nrows; };
    uint32_t n0 = 0u, n1 = 0u;   // near words of the copy cursor's block, loaded one block ahead
    const auto load_near = [&]() {
        n0 = LBM_IN(kChkHwNear, ci_near - a.near, near_extent(L)) ? __ldg(ci_near) : 0u;
        n1 = ci_b * 64 + 32 < L.nx && LBM_IN(kChkHwNear, ci_near + 1 - a.near, near_extent(L)) ? __ldg(ci_near + 1)
                                                                                                   : 0u;
    };
    const auto issue = [&](int slot) {
        const uint32_t dst = ring_s + slot * wp::kSlotBytes;
#pragma unroll
        for (int i = 0; i < 5; ++i)
            if ((i < 4 || lane < 24) && LBM_IN(kChkHwLine, (ci_src - fin) + poff[i], L.total - 7))
                cp_async16(dst + (i * 32 + lane) * 16, ci_src + poff[i]);
        if (lane < 2) reinterpret_cast<uint32_t*>(ring + slot * wp::kSlotBytes + wp::kNearOff)[lane] = lane ? n1 : n0;
        if ((n0 | n1) != 0u && ci_b * 64 + 2 * lane < L.nx &&
            LBM_IN(kChkHwLinks, ci_link - a.links, links_extent(L) - 1))
            cp_async8(dst + wp::kLinkOff + lane * 8, ci_link);
        if (((ci_b == 0 && lane < 5) || (ci_b == L.nb - 1 && lane >= 5 && lane < 10)) &&
            LBM_IN(kChkHwGhost, ci_gh - a.xf.xgh, xgh_extent(L)))
            cp_async4(dst + wp::kGhostOff + lane * 4, ci_gh);
    };

    // ---- update cursor: the block being updated
    [[maybe_unused]] int cc_r = r0;
    int cc_b = 0, cc_j = 0, cc_k = 0, c0 = 0;
    const unsigned* own = nullptr;   // this lane's word of line 0 of the block (line q: own[32 q])
    unsigned* outp = nullptr;
    float syz = 0.f;
    // FUSED: what the row's results still take: bits 0-7 sources, bits 8-13 the open faces that the row or
    // one of its ends borders, bit 14 the x-face exports of a step that leaves its results as they are
    unsigned todo = 1u << 14;
    const auto cc_row = [&](int r) {
        cc_k = 1 + r / L.ny;
        cc_j = 1 + r - (cc_k - 1) * L.ny;
        const long long e = L.elem(0, 1, cc_j, cc_k);
        own = reinterpret_cast<const unsigned*>(fin + e) + lane;
        outp = reinterpret_cast<unsigned*>(fout + e) + lane;
        c0 = 2 * lane;
        syz = fmaxf(__ldg(a.sig_y + cc_j - 1), __ldg(a.sig_z + cc_k - 1));
        if constexpr (FUSED)
        {
            if (fa.next->fill != 0)
            {
                todo = (row_faces(fa.open, cc_j, cc_k, L) | (fa.open & 3u)) << 8;
                if (fa.src.nsrc > 0) todo |= sources_of_row(fa.next, fa.src.nsrc, lane, cc_j, cc_k);
            }
        }
    };
    const auto cc_more = [&]() { return CLAIM ? cc_k > 0 : cc_r < nrows; };
    const auto cc_next = [&]() {
        own += 19 * 32;
        outp += 19 * 32;
        c0 += 64;
        if (++cc_b == L.nb)
        {
            cc_b = 0;
            if constexpr (CLAIM)
            {
                const int r = *next_row;
                if (r < nrows) cc_row(r);
                else cc_k = 0;
            }
            else
            {
                cc_r += all_warps;
                if (cc_r < nrows) cc_row(cc_r);
            }
        }
    };

    ci_row(r0);
    cc_row(r0);
#pragma unroll 1
    for (int p = 0; p < P; ++p)
    {
        if (ci_more())
        {
            load_near();
            issue(p);
            ci_next();
        }
        cp_async_commit();
    }
    if (ci_more()) load_near();

    int st = 0;   // slot of block t
#pragma unroll 1
    while (cc_more())
    {
        const int sn = st == S - 1 ? 0 : st + 1;
        int si = st + P;
        if (si >= S) si -= S;
        if (ci_more())
        {
            issue(si);
            ci_next();
            if (ci_more()) load_near();
        }
        cp_async_commit();
        cp_async_wait<P - 1>();   // blocks up to t + 1 have landed
        __syncwarp();

        const int j = cc_j, k = cc_k;
        const bool active = c0 < L.nx;
        const int last = L.nx - 1 - c0;
        const bool xlo = c0 == 0;
        const bool xhi = last >= 0 && last < 2;
        const bool edge = cc_b == 0 || cc_b == L.nb - 1;
        const unsigned char* slot = ring + st * wp::kSlotBytes;

        // links words of block t (they came with its lines, when a near-solid bit is set)
        // sponge strengths of the two cells, first so that the loads are in flight early
        const float sx0 = active ? __ldg(a.sig_x + c0) : 0.f;
        const float sx1 = c0 + 1 < L.nx ? __ldg(a.sig_x + c0 + 1) : 0.f;
        const uint2 nw = *reinterpret_cast<const uint2*>(slot + wp::kNearOff);
        uint32_t lk0 = 0u, lk1 = 0u;
        bool any_link = false;
        if ((nw.x | nw.y) != 0u)
        {
            const uint32_t bits = active ? ((lane < 16 ? nw.x : nw.y) >> ((2 * lane) & 31)) & 3u : 0u;
            const uint32_t* lw = reinterpret_cast<const uint32_t*>(slot + wp::kLinkOff) + 2 * lane;
            lk0 = (bits & 1u) ? lw[0] : 0u;
            lk1 = (bits & 2u) ? lw[1] : 0u;
            any_link = __any_sync(kFull, ((lk0 | lk1) & kDirBits) != 0u);
        }
        const uint32_t lka = (lk0 | lk1) & kDirBits;

        // pulled words: line q of the slot, shifted by ex(q) across lanes / blocks
        const unsigned* cur = reinterpret_cast<const unsigned*>(slot) + lane;   // line q: cur[32 q]
        const unsigned* end = reinterpret_cast<const unsigned*>(slot + wp::kGhostOff);   // last words of block t - 1
        const unsigned* nxt =
            lane < 31 ? cur + 1
                      : (cc_b + 1 < L.nb ? reinterpret_cast<const unsigned*>(ring + sn * wp::kSlotBytes) : cur);
        unsigned w[Q];
#pragma unroll
        for (int q = 0; q < Q; ++q)
        {
            const unsigned v = cur[32 * q];
            if (ex(q) == 0) w[q] = v;
            else if (ex(q) > 0) w[q] = __byte_perm(lane > 0 ? cur[32 * q - 1] : end[ghost_slot(q)], v, 0x5432);
            else w[q] = __byte_perm(v, nxt[32 * q], 0x5432);
        }
        if (any_link)
        {
            // halfway bounce-back: the own cell's word of the opposite direction
#pragma unroll
            for (int q = 1; q < Q; ++q)
            {
                const unsigned o =
                    ((lka >> q) & 1u) &&
                            LBM_IN(kChkHwBounce, 2 * (own - reinterpret_cast<const unsigned*>(fin)) + inv(q) * 64,
                                   L.total - 1)
                        ? __ldg(own + inv(q) * 32)
                        : 0u;
                const unsigned m = ((0u - ((lk0 >> q) & 1u)) & 0x0000ffffu) | ((0u - ((lk1 >> q) & 1u)) & 0xffff0000u);
                w[q] = (w[q] & ~m) | (o & m);
            }
        }
        if (edge)
        {
            // x-face ghosts of the row ends (they came with the block's lines)
            const float* gs = reinterpret_cast<const float*>(slot + wp::kGhostOff);
#pragma unroll
            for (int q = 0; q < Q; ++q)
            {
                if (ex(q) == 0) continue;
                const float g = gs[ghost_slot(q)];
                if (ex(q) > 0 && xlo && !((lk0 >> q) & 1u)) w[q] = set_lo(w[q], g);
                if (ex(q) < 0 && xhi && last == 0 && !((lk0 >> q) & 1u)) w[q] = set_lo(w[q], g);
                if (ex(q) < 0 && xhi && last == 1 && !((lk1 >> q) & 1u)) w[q] = set_hi(w[q], g);
            }
        }
        if (active)
        {
            const float2 sg = make_float2(fmaxf(sx0, syz), fmaxf(sx1, syz));
            collide2_grouped(w, inv_scale, a.omega, sg, (lk0 & kSolidSelfBit) != 0u, (lk1 & kSolidSelfBit) != 0u);
            if (FUSED && (todo & 0xffu)) add_sources(w, fa.next, todo & 0xffu, c0, j, k, L);
#pragma unroll
            for (int q = 0; q < Q; ++q)
                if (LBM_IN(kChkHwStore, 2 * (outp - reinterpret_cast<unsigned*>(fout)) + 64 * q, L.total - 1))
                    outp[32 * q] = w[q];
            if ((todo & (1u << 14)) && edge && (xlo | xhi))
            {
#pragma unroll
                for (int q = 0; q < Q; ++q)
                {
                    if (!LBM_IN(kChkHwExport, a.xf.exp_index(xlo ? 0 : 1, q, j, k, L.ny, L.nz), xexp_extent(L)))
                        continue;
                    if (xlo) a.xf.xexp[a.xf.exp_index(0, q, j, k, L.ny, L.nz)] = h2f(w[q]).x;
                    if (xhi && last == 0) a.xf.xexp[a.xf.exp_index(1, q, j, k, L.ny, L.nz)] = h2f(w[q]).x;
                    if (xhi && last == 1) a.xf.xexp[a.xf.exp_index(1, q, j, k, L.ny, L.nz)] = h2f(w[q]).y;
                }
            }
            if (FUSED && ((todo & (60u << 8)) || edge))
            {
                // from the values as stored; a row's end takes the moments of its own cell only, unless the
                // whole row is a face
                const unsigned row = (todo >> 8) & 60u, open = (todo >> 8) & 3u;
                const unsigned ends = (xlo ? open & 1u : 0u) | (last == 0 ? open & 2u : 0u) |
                                      (last == 1 ? (open & 2u) << 2 : 0u);
                float4 m0 = make_float4(0.f, 0.f, 0.f, 0.f), m1 = m0;
                if (row | (ends & 3u)) m0 = cell_moments([&](int q) { return h2f(w[q]).x; });
                if (row | (ends & 8u)) m1 = cell_moments([&](int q) { return h2f(w[q]).y; });
                // (with 32-bit offsets nvcc 12.9 stored the low faces' rows one row inside the grid in a variant of
                // this code that kept both cells' GhostState for all faces)
                const long long rsw = L.row_stride >> 1, psw = L.plane_stride >> 1;
                if (row & 4u) ghost_pair<1, 0>(w, m0, m1, inv_scale, outp - rsw, fout, L.total);
                if (row & 8u) ghost_pair<1, 1>(w, m0, m1, inv_scale, outp + rsw, fout, L.total);
                if (row & 16u) ghost_pair<2, 0>(w, m0, m1, inv_scale, outp - psw, fout, L.total);
                if (row & 32u) ghost_pair<2, 1>(w, m0, m1, inv_scale, outp + psw, fout, L.total);
                if (ends & 1u)
                    ghost_end<0>(ghost_state(m0, inv_scale), inv_scale, fa, a.xf, L, j, k, [&](int q) { return h2f(w[q]).x; });
                if (ends & 10u)
                    ghost_end<1>(ghost_state(last == 0 ? m0 : m1, inv_scale), inv_scale, fa, a.xf, L, j, k,
                                 [&](int q) { return last == 0 ? h2f(w[q]).x : h2f(w[q]).y; });
            }
        }
        if (cc_b + 1 < L.nb && lane < 5)   // the row goes on: its next block's first cells pull this one's last words
            reinterpret_cast<unsigned*>(ring + sn * wp::kSlotBytes + wp::kGhostOff)[lane] =
                reinterpret_cast<const unsigned*>(slot)[32 * wp::ghost_dir(lane) + 31];
        __syncwarp();   // every lane is done with slot t before the next copy lands there
        cc_next();
        st = sn;
    }
    cp_async_wait<0>();
}

// ---------------------------------------------------------------- z-slab messages
// The populations that cross a z cut: the 5 directions with ez = +1 leave a
// slab's top plane for the upper neighbour's halo plane 0, the 5 with ez = -1
// its bottom plane for the lower neighbour's halo plane nz + 1.  A message holds
// those directions of every row of the plane (y-halo rows included) as whole
// 128-byte lines, [5][ny + 2][nb], then the two x-face ghost rows of the plane
// that the receiving plane's row-end cells pull (the two of the five with
// ex != 0), [2][ny + 2] floats.  The same kernel packs (plane -> message) and
// unpacks (message -> plane); it moves bytes, whatever the storage type.
__host__ __device__ constexpr int cross_dir(int up, int d)
{
    constexpr int u[5] = {5, 11, 13, 15, 17};   // ez = +1
    constexpr int w[5] = {6, 12, 14, 16, 18};   // ez = -1
    return up ? u[d] : w[d];
}
// the x-face ghost directions among them: side 0 (low face, ex > 0), side 1 (high face, ex < 0)
__host__ __device__ constexpr int cross_ghost_dir(int up, int side) { return up ? (side ? 13 : 11) : (side ? 14 : 12); }

template <bool PACK>
__global__ void __launch_bounds__(256) k_slab_msg(unsigned char* __restrict__ f, float* __restrict__ xgh,
                                                  unsigned char* __restrict__ msg, Layout L, int k, int up, int esz)
{
    const long long nl = 5LL * (L.ny + 2) * L.nb * 8;   // 16-byte pieces of the lines
    const long long ng = 2LL * (L.ny + 2);
    for (long long u = blockIdx.x * (long long)blockDim.x + threadIdx.x; u < nl + ng;
         u += (long long)gridDim.x * blockDim.x)
    {
        if (u < nl)
        {
            const int piece = (int)(u & 7);
            long long line = u >> 3;
            const int b = (int)(line % L.nb);
            line /= L.nb;
            const int j = (int)(line % (L.ny + 2));
            const int d = (int)(line / (L.ny + 2));
            const long long e = kFrontElems + ((long long)k * (L.ny + 2) + j) * L.row_stride + (long long)b * 19 * L.bc +
                                (long long)cross_dir(up, d) * L.bc;
            uint4* fp = reinterpret_cast<uint4*>(f + e * esz) + piece;
            uint4* mp = reinterpret_cast<uint4*>(msg) + u;
            if (PACK) *mp = *fp;
            else *fp = *mp;
        }
        else
        {
            const long long g = u - nl;
            const int side = (int)(g / (L.ny + 2)), j = (int)(g % (L.ny + 2));
            const long long gi = ((long long)(side * 19 + cross_ghost_dir(up, side)) * (L.nz + 2) + k) * (L.ny + 2) + j;
            float* mp = reinterpret_cast<float*>(msg + nl * 16) + g;
            if (PACK) *mp = xgh[gi];
            else xgh[gi] = *mp;
        }
    }
}

// ---------------------------------------------------------------- links
// Per interior cell: bit q set when the pull source cell - e_q is SOLID,
// bit 19 when the cell itself is SOLID (mask semantics 06:923, 06:933).
// The near-solid bitmap gets one bit per cell (a warp ballot), so the step
// kernel reads the links word only in warps that touch a solid.
__global__ void __launch_bounds__(128) k_build_links(const uint8_t* __restrict__ m, uint32_t* __restrict__ links,
                                                     uint32_t* __restrict__ near, Layout L)
{
    const int i0 = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y + 1;
    const int k = blockIdx.z + 1;
    const bool active = i0 < L.nx;
    const long long nxt = L.nx + 2, nyt = L.ny + 2;
    uint32_t lk = 0;
    if (active)
    {
        const int i = i0 + 1;
#pragma unroll
        for (int q = 0; q < Q; ++q)
        {
            const long long src = (long long)(i - ex(q)) + (long long)(j - ey(q)) * nxt + (long long)(k - ez(q)) * nxt * nyt;
            if (m[src]) lk |= 1u << q;
        }
        if (m[(long long)i + (long long)j * nxt + (long long)k * nxt * nyt]) lk |= kSolidSelfBit;
        links[L.cell(i, j, k)] = lk;
    }
    const uint32_t ball = __ballot_sync(kFull, active && lk != 0u);
    if ((threadIdx.x & 31) == 0 && i0 < L.pitch)
        near[((long long)k * (L.ny + 2) + j) * L.words_per_row + (i0 >> 5)] = ball;
}

// ---------------------------------------------------------------- source
// Source injection (LBMSolver::apply_source 06:576-667), block 0: every FLUID
// cell of a source's stencil gains its amounts.  One block; sources run in order.
// Cells next to the x faces also update their x-face export.  Block 1, at the
// start of a batch of fused steps: the sources of the next step.
template <typename S>
__global__ void __launch_bounds__(512) k_source(S* __restrict__ f, Layout L, StepArgs sa, SourceArgs a, int parity,
                                                SourceNext* __restrict__ next)
{
    __shared__ double red[32];
    f = chain_wait(f);
    if (blockIdx.x == 1)
    {
        const long long s = a.ctl->step[parity];
        prepare_sources(next, a, s + 1, s < a.ctl->last, L, sa.links, red);
        return;
    }
    for (int s = 0; s < a.nsrc; ++s)
    {
        SourceEntry e;
        if (a.ctl)
        {
            const long long row = a.ctl->step[parity] - a.ctl->table_base;
            e = a.table[row * a.nsrc + s];
        }
        else
        {
            e = a.direct[s];
        }
        SourceBox b{};
        source_stencil(e, a.st[s], a, L, sa.links, red, b, [&](int c, const float4& add) {
            const int i = b.i0 + c % b.n, j = b.j0 + (c / b.n) % b.n, k = b.k0 + c / (b.n * b.n);
            // (the bounds-checked build skips a cell whose 19 directions leave the buffer)
            if (add.w == 0.f || !LBM_IN(kChkSource, L.elem(18, i, j, k), L.total)) return;
            // the 19 directions of one cell are 19 distinct elements: every load
            // first (one round trip), then the stores
            S* p = f + L.elem(0, i, j, k);   // direction q at p + q * bc
            float v[Q];
#pragma unroll
            for (int q = 0; q < Q; ++q) v[q] = Io<S>::ldw(p + q * L.bc);
#pragma unroll
            for (int q = 0; q < Q; ++q)
            {
                Io<S>::st(p + q * L.bc, v[q] + source_gain(add, q));
                if (i == 1 || i == L.nx)
                {
                    const float gs = Io<S>::ldw(p + q * L.bc);   // the stored value, as the step would export it
                    if (i == 1) sa.xf.xexp[sa.xf.exp_index(0, q, j, k, L.ny, L.nz)] = gs;
                    if (i == L.nx) sa.xf.xexp[sa.xf.exp_index(1, q, j, k, L.ny, L.nz)] = gs;
                }
            }
        });
        __syncthreads();
    }
}

// ---------------------------------------------------------------- ghosts
// G: the populations of cell I in, its ghost's inward directions out
template <int AXIS, int SIDE>
__device__ __forceinline__ void ghost_values(float (&G)[Q], float inv_scale, float4* face_mom, long long t)
{
    const float4 m = cell_moments([&](int q) { return G[q]; });
    if (face_mom) face_mom[t] = m;
    nscbc<AXIS, SIDE>(ghost_state(m, inv_scale), inv_scale, [&](int q) { return G[q]; },
                         [&](int q, float v) { G[q] = v; });
}

// One face cell (two x-adjacent ones in FP16 y and z faces) of face (AXIS, SIDE).
template <typename S, int AXIS, int SIDE>
__device__ __forceinline__ void ghost_cell(S* __restrict__ f, const Layout& L, const GhostArgs& a, const GhostFace& F,
                                           long long t, int lt)
{
    const int v = lt / F.nu, u = lt - v * F.nu;
    const float inv_scale = 1.0f / a.scale;
    float G[Q];
    if constexpr (AXIS == 0)
    {
        // x faces: compact export -> compact ghost, both coalesced along j
        const int j = 1 + u, k = 1 + v;
        if (!LBM_IN(kChkGhost, a.xf.exp_index(SIDE, 18, j, k, L.ny, L.nz), xexp_extent(L)) ||
            !LBM_IN(kChkGhost, a.xf.gh_index(SIDE, 18, j, k, L.ny, L.nz), xgh_extent(L)))
            return;
#pragma unroll
        for (int q = 0; q < Q; ++q) G[q] = a.xf.xexp[a.xf.exp_index(SIDE, q, j, k, L.ny, L.nz)];
        ghost_values<AXIS, SIDE>(G, inv_scale, a.face_mom, t);
#pragma unroll
        for (int q = 0; q < Q; ++q)
            if (inward<AXIS, SIDE>(q)) a.xf.xgh[a.xf.gh_index(SIDE, q, j, k, L.ny, L.nz)] = G[q];
        return;
    }
    else if constexpr (std::is_same<S, __half>::value)
    {
        // y and z faces in FP16: the first half of the face's threads take two
        // x-adjacent cells each, one half2 per direction (a 64-cell block
        // holds both cells of an even-aligned pair); same values as one cell
        // per thread, half as many 2-byte accesses
        const int npair = (F.nu + 1) >> 1;
        if (lt >= npair * F.nv) return;
        const int vp = lt / npair, up = 2 * (lt - vp * npair);
        const bool two = up + 1 < F.nu;
        const int pi = 1 + up;
        const int pj = AXIS == 1 ? (SIDE ? L.ny : 1) : 1 + vp, pk = AXIS == 1 ? 1 + vp : (SIDE ? L.nz : 1);
        const int qj = AXIS == 1 ? (SIDE ? L.ny + 1 : 0) : pj, qk = AXIS == 1 ? pk : (SIDE ? L.nz + 1 : 0);
        constexpr int BCH = block_cells(sizeof(S));
        if (!LBM_IN(kChkGhost, L.elem(18, pi + (two ? 1 : 0), pj, pk), L.total) ||
            !LBM_IN(kChkGhost, L.elem(18, pi + (two ? 1 : 0), qj, qk), L.total))
            return;
        const __half* I = f + L.elem(0, pi, pj, pk);
        __half* B = f + L.elem(0, pi, qj, qk);
        float G1[Q];
#pragma unroll
        for (int q = 0; q < Q; ++q)
        {
            if (two)
            {
                const float2 v2 = __half22float2(__ldg(reinterpret_cast<const __half2*>(I + q * BCH)));
                G[q] = v2.x;
                G1[q] = v2.y;
            }
            else
            {
                G[q] = Io<S>::ld(I + q * BCH);
                G1[q] = 0.f;
            }
        }
        const long long cell = F.first + (long long)vp * F.nu + up;   // the face enumeration of one cell a thread
        ghost_values<AXIS, SIDE>(G, inv_scale, a.face_mom, cell);
        if (two)
        {
            ghost_values<AXIS, SIDE>(G1, inv_scale, a.face_mom, cell + 1);
#pragma unroll
            for (int q = 0; q < Q; ++q)
                if (inward<AXIS, SIDE>(q)) *reinterpret_cast<__half2*>(B + q * BCH) = __floats2half2_rn(G[q], G1[q]);
        }
        else
        {
#pragma unroll
            for (int q = 0; q < Q; ++q)
                if (inward<AXIS, SIDE>(q)) Io<S>::st(B + q * BCH, G[q]);
        }
    }
    else
    {
        const int ci = 1 + u;
        const int cj = AXIS == 1 ? (SIDE ? L.ny : 1) : 1 + v, gj = AXIS == 1 ? (SIDE ? L.ny + 1 : 0) : cj;
        const int ck = AXIS == 1 ? 1 + v : (SIDE ? L.nz : 1), gk = AXIS == 1 ? ck : (SIDE ? L.nz + 1 : 0);
        constexpr int BC = block_cells(sizeof(S));
        if (!LBM_IN(kChkGhost, L.elem(18, ci, cj, ck), L.total) ||
            !LBM_IN(kChkGhost, L.elem(18, ci, gj, gk), L.total) || !LBM_IN(kChkGhost, L.elem(0, ci, gj, gk), L.total))
            return;
        const S* I = f + L.elem(0, ci, cj, ck);
        S* B = f + L.elem(0, ci, gj, gk);
#pragma unroll
        for (int q = 0; q < Q; ++q) G[q] = Io<S>::ld(I + q * BC);
        ghost_values<AXIS, SIDE>(G, inv_scale, a.face_mom, t);
#pragma unroll
        for (int q = 0; q < Q; ++q)
            if (inward<AXIS, SIDE>(q)) Io<S>::st(B + q * BC, G[q]);
    }
}

template <typename S>
__global__ void __launch_bounds__(128) k_ghost(S* __restrict__ f, Layout L, GhostArgs a)
{
    f = chain_wait(f);
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= a.total) return;
    int fi = 0;
    while (fi + 1 < a.nfaces && t >= a.face[fi + 1].first) ++fi;
    const GhostFace F = a.face[fi];
    const int lt = (int)(t - F.first);   // a face has fewer than 2^31 cells (nu, nv are ints of one grid)
    switch (F.axis * 2 + F.side)
    {
    case 0: ghost_cell<S, 0, 0>(f, L, a, F, t, lt); break;
    case 1: ghost_cell<S, 0, 1>(f, L, a, F, t, lt); break;
    case 2: ghost_cell<S, 1, 0>(f, L, a, F, t, lt); break;
    case 3: ghost_cell<S, 1, 1>(f, L, a, F, t, lt); break;
    case 4: ghost_cell<S, 2, 0>(f, L, a, F, t, lt); break;
    default: ghost_cell<S, 2, 1>(f, L, a, F, t, lt); break;
    }
}

// ---------------------------------------------------------------- probes
// One step's probe record on its own (single calls), one warp per probe.
template <typename S>
__global__ void __launch_bounds__(128) k_probe(const S* __restrict__ f, Layout L, StepArgs sa, ProbeArgs a)
{
    const long long row = a.ctl ? a.ctl->step[a.parity] - a.ctl->probe_base : a.direct_row;
    const int p = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    if (p < a.n) probe_warp<S>(f, L, sa.links, sa.xf.xgh, a, row, p, threadIdx.x & 31);
}

// (float)(rho - 1) of rows [row0, row0 + gridDim.y) of the interior, row r =
// (k - 1) ny + j - 1, dense into `out` (device memory, or pinned host memory).
template <typename S>
__global__ void __launch_bounds__(128) k_field_rho(const S* __restrict__ f, float* __restrict__ out, Layout L,
                                                   StepArgs sa, float inv_scale, int row0)
{
    const int i0 = blockIdx.x * blockDim.x + threadIdx.x;
    if (i0 >= L.nx) return;
    const int row = row0 + (int)blockIdx.y, k = 1 + row / L.ny, j = 1 + row - (k - 1) * L.ny;
    bool solid;
    float G[Q];
    pull_cell<S>(f, L, sa, i0 + 1, j, k, G, solid);
    float rho = 0.f;
#pragma unroll
    for (int q = 0; q < Q; ++q) rho += G[q];
    out[(long long)blockIdx.y * L.nx + i0] = solid ? 0.f : rho * inv_scale;
}

// ---------------------------------------------------------------- import/export
// Conversions between the device state and FP64 f in the reference's AoS
// halo-inclusive layout; the x-halo columns map to the x-face ghosts and the
// cells next to the x faces are mirrored into the x-face exports.
template <typename S>
__global__ void k_export_f(const S* __restrict__ f, double* __restrict__ out, Layout L, XFace xf, float inv_scale)
{
    const long long nxt = L.nx + 2, nyt = L.ny + 2, n = nxt * nyt * (L.nz + 2);
    for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < n;
         idx += (long long)gridDim.x * blockDim.x)
    {
        const int i = (int)(idx % nxt);
        const int j = (int)((idx / nxt) % nyt);
        const int k = (int)(idx / (nxt * nyt));
#pragma unroll
        for (int q = 0; q < Q; ++q)
        {
            float g;
            if (i == 0) g = xf.xgh[xf.gh_index(0, q, j, k, L.ny, L.nz)];
            else if (i == L.nx + 1) g = xf.xgh[xf.gh_index(1, q, j, k, L.ny, L.nz)];
            else g = Io<S>::ld(f + L.elem(q, i, j, k));
            out[idx * Q + q] = wd(q) + (double)g * (double)inv_scale;
        }
    }
}

template <typename S>
__global__ void k_import_f(S* __restrict__ f, const double* __restrict__ in, Layout L, XFace xf, float scale)
{
    const long long nxt = L.nx + 2, nyt = L.ny + 2, n = nxt * nyt * (L.nz + 2);
    for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < n;
         idx += (long long)gridDim.x * blockDim.x)
    {
        const int i = (int)(idx % nxt);
        const int j = (int)((idx / nxt) % nyt);
        const int k = (int)(idx / (nxt * nyt));
        const bool inner = j >= 1 && j <= L.ny && k >= 1 && k <= L.nz;
#pragma unroll
        for (int q = 0; q < Q; ++q)
        {
            const float g = (float)((in[idx * Q + q] - wd(q)) * (double)scale);
            if (i == 0)
            {
                xf.xgh[xf.gh_index(0, q, j, k, L.ny, L.nz)] = g;
                continue;
            }
            if (i == L.nx + 1)
            {
                xf.xgh[xf.gh_index(1, q, j, k, L.ny, L.nz)] = g;
                continue;
            }
            S* p = f + L.elem(q, i, j, k);
            Io<S>::st(p, g);
            const float gs = Io<S>::ldw(p);   // the stored (rounded) value
            if (inner && i == 1) xf.xexp[xf.exp_index(0, q, j, k, L.ny, L.nz)] = gs;
            if (inner && i == L.nx) xf.xexp[xf.exp_index(1, q, j, k, L.ny, L.nz)] = gs;
        }
    }
}

// Self-test of the bounds-checked build: lane 5 tests an index one past its
// extent (nothing is accessed), which must be recorded as site kChkSelfTest.
__global__ void k_check_selftest()
{
    const int lane = threadIdx.x & 31;
    if (lane == 5 && !LBM_IN(kChkSelfTest, 32 + lane, 37)) return;
}

// Statically reserved device array for lbm_get_rho_noalloc: the field of
// (rho - 1) passes through it instead of a temporary cudaMalloc buffer.  It
// exists on every GPU that loads this library, for the life of the process.
static __device__ __align__(256) float g_field_scratch[kNoAllocFieldCells];
static_assert(sizeof(g_field_scratch) == sizeof(float) * LBM_NOALLOC_MAX_CELLS,
              "the static field array must hold the grid size lbm_get_rho_noalloc accepts");

dim3 row_grid(const Layout& L) { return dim3((unsigned)((L.nx + 127) / 128), (unsigned)L.ny, (unsigned)L.nz); }

// Warp-pipelined FP16 step: dynamic shared memory (one ring per warp) and a
// grid of as many CTAs as the GPU holds at once (every warp then walks rows
// all_warps apart, or claims them).  The attribute and the occupancy are set up once per device.
template <int P, int WARPS, int MINB, int MODE, bool CLAIM>
cudaError_t hw_ctas(int* out)
{
    constexpr int smem = WARPS * (P + 1) * wp::kSlotBytes;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
    static std::mutex mu;
    static int ctas[kMaxDevices] = {};
    std::lock_guard<std::mutex> lock(mu);
    if (!ctas[dev])
    {
        const auto kernel = k_step_hw<P, WARPS, MINB, MODE, CLAIM>;
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        int per_sm = 0, sms = 0;
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, 32 * WARPS, smem);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (e != cudaSuccess) return e;
        if (per_sm < 1) return cudaErrorInvalidConfiguration;
        ctas[dev] = per_sm * sms;
    }
    *out = ctas[dev];
    return cudaSuccess;
}

template <int P, int WARPS, int MINB, int MODE, bool CLAIM>
cudaError_t launch_hw(const __half* fin, __half* fout, const Layout& L, const StepArgs& a, float inv_scale,
                      const FusedArgs& fa, cudaStream_t stream)
{
    // the per-lane source offsets are 32-bit
    if (L.plane_stride + L.row_stride + 19 * 64 > 0x7fffffffLL) return cudaErrorInvalidValue;
    int ctas = 0;
    const cudaError_t e = hw_ctas<P, WARPS, MINB, MODE, CLAIM>(&ctas);
    if (e != cudaSuccess) return e;
    const long long need = ((long long)L.ny * L.nz + WARPS - 1) / WARPS;
    const int side = MODE != kPlain ? side_blocks(fa.probe.n, WARPS) : 0;
    const int grid = (int)(need < ctas ? need : ctas) + side;
    // (not chained: with the next launch's blocks waiting on the SMs a 256x128x128 step took 84.9 us, 80.3 without)
    constexpr size_t smem = WARPS * (P + 1) * wp::kSlotBytes;
    k_step_hw<P, WARPS, MINB, MODE, CLAIM><<<grid, 32 * WARPS, smem, stream>>>(fin, fout, L, a, inv_scale, fa, side);
    return cudaGetLastError();
}

template <bool MOM, int MODE>
cudaError_t launch_pair_step(const float* fin, float* fout, const Layout& L, const StepArgs& a, PairMoments* mom,
                             const FusedArgs& fa, cudaStream_t stream)
{
    const PairLaunch g = pair_launch(L, MODE != kPlain ? side_blocks(fa.probe.n, kPairBlock / 32) : 0);
    if (g.grid.y > (unsigned)kMaxGridY && MODE != kPlain && fa.probe.n > 0)
    {
        // more probes than rows of blocks are left for: they follow the step, whose input it only reads
        FusedArgs rest = fa;
        rest.probe.n = 0;
        const cudaError_t e = launch_pair_step<MOM, MODE>(fin, fout, L, a, mom, rest, stream);
        return e != cudaSuccess ? e : launch_probe(0, fin, L, a, fa.probe, stream);
    }
    const auto kernel = g.bx == 4 ? k_step<4, MOM, MODE> : g.bx == 2 ? k_step<2, MOM, MODE> : k_step<1, MOM, MODE>;
    if (MODE != kPlain)
        return launch_chained(kernel, g.grid, kPairBlock, 0, stream, fin, fout, L, a, mom, fa, g.side_rows);
    kernel<<<g.grid, kPairBlock, 0, stream>>>(fin, fout, L, a, mom, fa, g.side_rows);
    return cudaGetLastError();
}

}  // namespace

cudaError_t field_scratch_address(int device, float** ptr)
{
    // Host code cannot use the array's name as a device address; the address
    // is looked up once per device, with that device current (the caller
    // sets it), and cached.
    static std::mutex mu;
    static float* cached[kMaxDevices] = {};
    if (device < 0 || device >= kMaxDevices) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lock(mu);
    if (!cached[device])
    {
        void* p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, g_field_scratch);
        if (e != cudaSuccess) return e;
        cached[device] = static_cast<float*>(p);
    }
    *ptr = cached[device];
    return cudaSuccess;
}

long long slab_message_bytes(const Layout& L) { return 5LL * (L.ny + 2) * L.nb * 128 + 8LL * (L.ny + 2); }

cudaError_t launch_slab_msg(bool pack, void* f, float* xgh, void* msg, const Layout& L, int k, int up, int esz,
                            cudaStream_t stream)
{
    const long long n = 5LL * (L.ny + 2) * L.nb * 8 + 2LL * (L.ny + 2);
    const unsigned blocks = (unsigned)std::min<long long>((n + 255) / 256, 148LL * 16);
    if (pack)
        k_slab_msg<true><<<blocks, 256, 0, stream>>>((unsigned char*)f, xgh, (unsigned char*)msg, L, k, up, esz);
    else
        k_slab_msg<false><<<blocks, 256, 0, stream>>>((unsigned char*)f, xgh, (unsigned char*)msg, L, k, up, esz);
    return cudaGetLastError();
}

cudaError_t check_read_kernels(check::Status* out) { return check::read_and_clear(out); }

cudaError_t launch_check_selftest(cudaStream_t stream)
{
    k_check_selftest<<<1, 32, 0, stream>>>();
    return cudaGetLastError();
}

cudaError_t launch_build_links(const uint8_t* mask_ref, uint32_t* links, uint32_t* near, const Layout& L,
                               cudaStream_t stream)
{
    k_build_links<<<row_grid(L), 128, 0, stream>>>(mask_ref, links, near, L);
    return cudaGetLastError();
}

cudaError_t prepare_step(int storage)
{
    if (storage == 0) return cudaSuccess;
    int ctas = 0;
    cudaError_t e = hw_ctas<2, 4, 5, kPlain, false>(&ctas);
    if (e == cudaSuccess) e = hw_ctas<2, 4, 5, kSide, false>(&ctas);
    if (e == cudaSuccess) e = hw_ctas<2, 4, 5, kSide, true>(&ctas);
    return e != cudaSuccess ? e : hw_ctas<2, 4, 5, kFused, false>(&ctas);
}

namespace {
template <int MODE>
cudaError_t launch_step_mode(int storage, const void* fin, void* fout, const Layout& L, const StepArgs& a, float scale,
                             const FusedArgs& fa, PairMoments* mom, cudaStream_t stream)
{
    if (storage == 0 && mom) return launch_pair_step<true, MODE>((const float*)fin, (float*)fout, L, a, mom, fa, stream);
    if (storage == 0) return launch_pair_step<false, MODE>((const float*)fin, (float*)fout, L, a, nullptr, fa, stream);
    if (mom) return cudaErrorInvalidValue;
    if constexpr (MODE == kSide)
    {
        // Claimed rows pay from about ten rows a warp on: 400x350x128 (15 rows) 328 -> 323 us, 900x700x60 (14)
        // 610 -> 605, 700x300x90 (9) 306 and 306.5, 900x200x50 (3.4) 164 -> 167, and on the fused step's
        // grids 320x200x100 (7) 113 -> 116, 256x256x128 (11) 148 -> 151: there the order in which the
        // warps start says which SMs get the last rows, and fixed rows spread those evenly.
        int ctas = 0;
        const cudaError_t e = hw_ctas<2, 4, 5, MODE, true>(&ctas);
        if (e != cudaSuccess) return e;
        if (fa.ctl && L.nb > 2 && (long long)L.ny * L.nz >= 10LL * 4 * ctas)
            return launch_hw<2, 4, 5, MODE, true>((const __half*)fin, (__half*)fout, L, a, 1.0f / scale, fa, stream);
    }
    return launch_hw<2, 4, 5, MODE, false>((const __half*)fin, (__half*)fout, L, a, 1.0f / scale, fa, stream);
}
}  // namespace

cudaError_t launch_step(int storage, const void* fin, void* fout, const Layout& L, const StepArgs& a,
                        float scale, PairMoments* mom, cudaStream_t stream)
{
    return launch_step_mode<kPlain>(storage, fin, fout, L, a, scale, FusedArgs{}, mom, stream);
}

cudaError_t launch_batched_step(int storage, const void* fin, void* fout, const Layout& L, const StepArgs& a,
                                float scale, const FusedArgs& fa, bool fused, PairMoments* mom, cudaStream_t stream)
{
    if (fused) return launch_step_mode<kFused>(storage, fin, fout, L, a, scale, fa, mom, stream);
    return launch_step_mode<kSide>(storage, fin, fout, L, a, scale, fa, mom, stream);
}

cudaError_t launch_source(int storage, void* f, const Layout& L, const StepArgs& sa, const SourceArgs& a,
                          int parity, SourceNext* next, cudaStream_t stream, bool chained)
{
    const unsigned blocks = next ? 2 : 1;
    if (storage == 0 && chained)
        return launch_chained(k_source<float>, dim3(blocks), 512, 0, stream, (float*)f, L, sa, a, parity, next);
    if (storage == 0) k_source<float><<<blocks, 512, 0, stream>>>((float*)f, L, sa, a, parity, next);
    else k_source<__half><<<blocks, 512, 0, stream>>>((__half*)f, L, sa, a, parity, next);
    return cudaGetLastError();
}

cudaError_t launch_ghost(int storage, void* f, const Layout& L, const GhostArgs& a, cudaStream_t stream, bool chained)
{
    if (a.total <= 0) return cudaSuccess;
    const unsigned blocks = (unsigned)((a.total + 127) / 128);
    if (storage == 0 && chained)
        return launch_chained(k_ghost<float>, dim3(blocks), 128, 0, stream, (float*)f, L, a);
    if (storage == 0) k_ghost<float><<<blocks, 128, 0, stream>>>((float*)f, L, a);
    else k_ghost<__half><<<blocks, 128, 0, stream>>>((__half*)f, L, a);
    return cudaGetLastError();
}

cudaError_t launch_probe(int storage, const void* f, const Layout& L, const StepArgs& sa, const ProbeArgs& a,
                         cudaStream_t stream)
{
    if (a.n <= 0) return cudaSuccess;
    const unsigned blocks = (unsigned)((a.n + 3) / 4);
    if (storage == 0) k_probe<float><<<blocks, 128, 0, stream>>>((const float*)f, L, sa, a);
    else k_probe<__half><<<blocks, 128, 0, stream>>>((const __half*)f, L, sa, a);
    return cudaGetLastError();
}

cudaError_t launch_field_rho(int storage, const void* f, float* out, const Layout& L, const StepArgs& sa,
                             float scale, int row0, int rows, cudaStream_t stream)
{
    // the rows of a launch are its blocks along y
    for (int r = 0; r < rows; r += kFieldRows)
    {
        const dim3 g((unsigned)((L.nx + 127) / 128), (unsigned)std::min(kFieldRows, rows - r));
        float* o = out + (long long)r * L.nx;
        if (storage == 0) k_field_rho<float><<<g, 128, 0, stream>>>((const float*)f, o, L, sa, 1.0f / scale, row0 + r);
        else k_field_rho<__half><<<g, 128, 0, stream>>>((const __half*)f, o, L, sa, 1.0f / scale, row0 + r);
    }
    return cudaGetLastError();
}

cudaError_t launch_export_f(int storage, const void* f, double* out, const Layout& L, const XFace& xf, float scale,
                            cudaStream_t stream)
{
    if (storage == 0) k_export_f<float><<<1184, 256, 0, stream>>>((const float*)f, out, L, xf, 1.0f / scale);
    else k_export_f<__half><<<1184, 256, 0, stream>>>((const __half*)f, out, L, xf, 1.0f / scale);
    return cudaGetLastError();
}

cudaError_t launch_import_f(int storage, void* f, const double* in, const Layout& L, const XFace& xf, float scale,
                            cudaStream_t stream)
{
    if (storage == 0) k_import_f<float><<<1184, 256, 0, stream>>>((float*)f, in, L, xf, scale);
    else k_import_f<__half><<<1184, 256, 0, stream>>>((__half*)f, in, L, xf, scale);
    return cudaGetLastError();
}

}  // namespace lbm
