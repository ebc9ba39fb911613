// Shared device code for the EDGE sm_100a library: field geometry, the
// quadratic B-spline MAC sampler, the trilinear dye sampler, the three cubic
// Hermite flow-map interpolants and the RK4 point marches.
//
// Layout (identical to the reference's ti.field / to_numpy() order): scalar
// fields are row-major (i, j, k) with k fastest; vec3/vec4 fields store their
// components last (AoS).  Face grids of an (nx, ny, nz) cell grid are u_x
// (nx+1, ny, nz), u_y (nx, ny+1, nz), u_z (nx, ny, nz+1).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "../../include/edge_b200.h"

#define EDGE_HD __host__ __device__ __forceinline__
#define EDGE_D __device__ __forceinline__

namespace edge {

// taichi_utils.py:3 eps = 1e-6.  The reference clamps sample coordinates to
// [1, dim-2-eps] (B-spline, Hermite) or [1, dim-1-eps] (trilinear); Taichi
// folds that Python constant in double and narrows it to float32, so at
// dim >= ~64 the bound is exactly dim-2 (resp. dim-1).  Host code computes the
// bounds the same way and passes them in.
static inline float clamp_bound(int dim, int minus) { return (float)((double)(dim - minus) - 1e-6); }

EDGE_HD int idx3(int i, int j, int k, int n1, int n2) { return (i * n1 + j) * n2 + k; }
// x / dx as the reference writes it; when dx is a power of two (every grid
// spacing 1/res or 256/res of the drivers) the quotient is the exact scaling
// x * (1/dx), so the multiply gives the same float
static inline bool pow2f(float x) {
    int e;
    return x > 0.0f && frexpf(x, &e) == 0.5f;
}
EDGE_D float over_dx(float x, float dx, float inv_dx, bool pow2) { return pow2 ? x * inv_dx : x / dx; }
// A sampler struct with its power-of-two flag fixed at compile time: the hot
// kernels are built for both cases (P2 = pow2f(dx), chosen at launch), so
// over_dx is the exact multiply by 1/dx or the division with no run-time
// select between them (which made every sample evaluate the division too).
template <bool P2, class T>
EDGE_D T with_pow2(T s) {
    s.pow2 = P2 ? 1 : 0;
    return s;
}
// v[a] with constant indices only (a run-time index into a register array
// or a kernel-parameter array puts it in local memory)
EDGE_D float sel3(const float v[3], int a) { return a == 0 ? v[0] : (a == 1 ? v[1] : v[2]); }
EDGE_D int clampi(int v, int lo, int hi) { return v < lo ? lo : (v > hi ? hi : v); }

// ---------------------------------------------------------------------------
// Two floats in one 64-bit register, for the packed FP32 instructions of
// sm_100 (fma.rn.f32x2 and mul.rn.f32x2).  They have the FP32 peak of the
// scalar ones (67 against 65 TFLOP/s, independent chains) but take half the
// issue slots, and an operand that is one float in both halves (`both`) needs
// no instruction of its own.  Each half rounds as the scalar instruction does.
// A multiply-add whose three operands are different registers is bound by the
// register ports: measured 1.84 cycles scalar, 2.71 cycles per pair.
// ---------------------------------------------------------------------------
struct f2 {
    unsigned long long v;
};
EDGE_D f2 pair(float lo, float hi) {
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(lo), "f"(hi));
    return r;
}
EDGE_D f2 both(float a) { return pair(a, a); }
EDGE_D float lo(f2 a) {
    float x;
    asm("mov.b64 {%0, _}, %1;" : "=f"(x) : "l"(a.v));
    return x;
}
EDGE_D float hi(f2 a) {
    float x;
    asm("mov.b64 {_, %0}, %1;" : "=f"(x) : "l"(a.v));
    return x;
}
EDGE_D f2 fma2(f2 a, f2 b, f2 c) {
    f2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return d;
}
EDGE_D f2 mul2(f2 a, f2 b) {
    f2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d.v) : "l"(a.v), "l"(b.v));
    return d;
}
EDGE_D f2 add2(f2 a, f2 b) {
    f2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d.v) : "l"(a.v), "l"(b.v));
    return d;
}
// a0 b0 + a1 b1 + a2 b2 with the roundings of the scalar expression as nvcc
// contracts it (the products of the inner sum: the first is fused)
EDGE_D f2 dot3(f2 a0, f2 b0, f2 a1, f2 b1, f2 a2, f2 b2) { return fma2(a2, b2, fma2(a0, b0, mul2(a1, b1))); }
EDGE_D float dot3(float a0, float b0, float a1, float b1, float a2, float b2) {
    return __fmaf_rn(a2, b2, __fmaf_rn(a0, b0, __fmul_rn(a1, b1)));
}

// ---------------------------------------------------------------------------
// quadratic B-spline (taichi_utils.py:230-251) evaluated separably on the three
// non-zero taps of each axis
// ---------------------------------------------------------------------------
EDGE_D float N2(float x) {
    float a = fabsf(x);
    float r = 0.0f;
    if (a < 0.5f) r = 0.75f - a * a;
    else if (a < 1.5f) { float t = 1.5f - a; r = 0.5f * (t * t); }
    return r;
}

// One axis of interp_2 / interp_grad_2 (taichi_utils.py:254-319): the clamped
// grid coordinate, the first of the three taps that carry weight (the 4th tap
// of the reference's -1..2 loop is always zero) and their weights; with GRAD
// each weight is paired with its derivative, w[t] = (N2, N2').
template <bool GRAD>
struct Axis3;
template <>
struct Axis3<false> {
    int base;
    float w[3];
};
template <>
struct Axis3<true> {
    int base;
    f2 w[3];
};
EDGE_D void set_tap(float& w, float v, float) { w = v; }
EDGE_D void set_tap(f2& w, float v, float d) { w = pair(v, d); }

template <bool GRAD>
EDGE_D Axis3<GRAD> bspline_axis(float u, float hi_) {
    Axis3<GRAD> a;
    const float s = fmaxf(1.0f, fminf(u, hi_));
    // the first tap, an integer held exactly; s >= 1, so s - 0.5 is exact
    const float bf = floorf(s - 0.5f);
    const float x0 = s - bf;
    a.base = (int)bf;
    // x0 lies in [0.5, 1.5) (exactly: s - bf is exact), so the branches of
    // N2 and its derivative at x0, x0 - 1 and x0 - 2 are known: the same values
    // as the general functions', without their compares.  The third tap's zero
    // branch (|x0 - 2| = 1.5, i.e. x0 = 0.5) needs no select either: there
    // t2 = x0 - 0.5 = 0.  Every difference below is exact, so the first and
    // third derivatives (2 |x| - 3) / 2 are x0 - 1.5 and x0 - 0.5.
    const float x1 = x0 - 1.0f, t0 = 1.5f - x0, t2 = x0 - 0.5f;
    set_tap(a.w[0], (0.5f * t0) * t0, x0 - 1.5f);
    set_tap(a.w[1], __fmaf_rn(-x1, x1, 0.75f), -2.0f * x1);
    set_tap(a.w[2], (0.5f * t2) * t2, t2);
    return a;
}

// Tap row (i, j) of a sample, tap k by [k].  In global memory: one 32-bit byte
// offset per sample (grids have less than 2^30 faces per component) added to
// the row's uniform address, so that a row costs one add and its taps are
// immediate offsets.
struct GRow {
    const float* p;
    EDGE_D float operator[](int k) const { return __ldg(p + k); }
};
struct GRows {
    const float* f;
    int e, n1, n2;
    EDGE_D GRow operator()(int i, int j) const {
        return GRow{reinterpret_cast<const float*>(reinterpret_cast<const char*>(f + (i * n1 + j) * n2) +
                                                   4u * (unsigned)e)};
    }
};
EDGE_D GRows grows(const float* f, int x, int y, int z, int n1, int n2) {
    return GRows{f, idx3(x, y, z, n1, n2), n1, n2};
}

// The taps of samples at scattered points, which take 64-bit addresses.  Where
// a warp's points are in no order, its load costs a wavefront for every point
// or two, whatever its width: WIDE takes a row's three taps in the aligned 16
// bytes that hold the first and, where these do not hold the third, the 8 bytes
// after them.
struct VRow {
    float q[3];
    EDGE_D float operator[](int k) const { return q[k]; }
};
template <bool WIDE>
struct VRows {
    const float* f;  // the sample's first tap
    int n1, n2;
    EDGE_D VRow operator()(int i, int j) const {
        const float* p = f + (i * n1 + j) * n2;
        if (!WIDE) return VRow{{__ldg(p), __ldg(p + 1), __ldg(p + 2)}};
        const unsigned o = (unsigned)(reinterpret_cast<size_t>(p) >> 2) & 3;
        const float4 a = __ldg(reinterpret_cast<const float4*>(p - o));
        float2 b = make_float2(0.f, 0.f);
        if (o >= 2) b = __ldg(reinterpret_cast<const float2*>(p - o + 4));
        const float s0 = (o & 1) ? a.y : a.x, s1 = (o & 1) ? a.z : a.y, s2 = (o & 1) ? a.w : a.z, s3 = (o & 1) ? b.x : a.w;
        const float s4 = (o & 1) ? b.y : b.x;
        return (o & 2) ? VRow{{s2, s3, s4}} : VRow{{s0, s1, s2}};
    }
};
template <bool WIDE>
EDGE_D VRows<WIDE> vrows(const float* f, int x, int y, int z, int n1, int n2) {
    return VRows<WIDE>{f + (((long long)x * n1 + y) * n2 + z), n1, n2};
}

// 27-tap separable contraction of one scalar field, z then y then x, value and
// gradient (already multiplied by 1/dx).  (weight, derivative) pairs against
// taps in both halves give each row's value and z derivative in one packed
// multiply-add per tap, and the y and x sums carry the same pair.  The kernels
// this runs in are bound by FP32 register ports and issue slots: 690 thread
// instructions per three-component sample with scalar multiply-adds and 64-bit
// row addresses, 515 in this form (RK4 with Jacobian of 128^3 cells, 12
// samples each: 0.611 -> 0.508 ms, the same bits).
template <class Rows>
EDGE_D float bspline_sum(const Rows& rows, const Axis3<true>& X, const Axis3<true>& Y, const Axis3<true>& Z,
                         float inv_dx, float* g) {
    f2 vz = both(0.0f);  // (value, z derivative)
    float gx = 0.0f, gy = 0.0f;
#pragma unroll
    for (int i = 0; i < 3; i++) {
        f2 c = both(0.0f);
        float cy = 0.0f;
#pragma unroll
        for (int j = 0; j < 3; j++) {
            const auto q = rows(i, j);
            const f2 a = dot3(Z.w[0], both(q[0]), Z.w[1], both(q[1]), Z.w[2], both(q[2]));
            c = fma2(both(lo(Y.w[j])), a, c);
            cy = __fmaf_rn(hi(Y.w[j]), lo(a), cy);
        }
        vz = fma2(both(lo(X.w[i])), c, vz);
        gx = __fmaf_rn(hi(X.w[i]), lo(c), gx);
        gy = __fmaf_rn(lo(X.w[i]), cy, gy);
    }
    g[0] = gx * inv_dx;
    g[1] = gy * inv_dx;
    g[2] = hi(vz) * inv_dx;
    return lo(vz);
}

// The value alone: rows of equal j are paired over i = 0, 1 and the first two
// rows of i = 2 over j, so that the 27 row products take 15 instructions.  All
// 27 taps are loaded before the first is used: the kernels that take one
// sample per thread wait for their gathers (velocity pullback at 256x128x128
// 344 us row by row, 322 us so, 343 us with the scalar sampler).
template <class Rows>
EDGE_D float bspline_sum(const Rows& rows, const Axis3<false>& X, const Axis3<false>& Y, const Axis3<false>& Z, float,
                         float*) {
    float q[3][3][3];
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) {
            const auto row = rows(i, j);
#pragma unroll
            for (int k = 0; k < 3; k++) q[i][j][k] = row[k];
        }
    auto pairs = [&](const float (&a)[3], const float (&b)[3]) {
        return dot3(both(Z.w[0]), pair(a[0], b[0]), both(Z.w[1]), pair(a[1], b[1]), both(Z.w[2]), pair(a[2], b[2]));
    };
    f2 c01 = both(0.0f);
#pragma unroll
    for (int j = 0; j < 3; j++) c01 = fma2(both(Y.w[j]), pairs(q[0][j], q[1][j]), c01);
    const f2 a2 = pairs(q[2][0], q[2][1]);
    float c2 = __fmaf_rn(Y.w[0], lo(a2), 0.0f);
    c2 = __fmaf_rn(Y.w[1], hi(a2), c2);
    c2 = __fmaf_rn(Y.w[2], dot3(Z.w[0], q[2][2][0], Z.w[1], q[2][2][1], Z.w[2], q[2][2][2]), c2);
    float v = __fmaf_rn(X.w[0], lo(c01), 0.0f);
    v = __fmaf_rn(X.w[1], hi(c01), v);
    return __fmaf_rn(X.w[2], c2, v);
}

// The same value row by row: fewer registers, for the samplers at scattered
// points, where more warps in flight are worth more than a warp's loads ahead.
template <class Rows>
EDGE_D float bspline_rows(const Rows& rows, const Axis3<false>& X, const Axis3<false>& Y, const Axis3<false>& Z) {
    float v = 0.0f;
#pragma unroll
    for (int i = 0; i < 3; i++) {
        float c = 0.0f;
#pragma unroll
        for (int j = 0; j < 3; j++) {
            const auto q = rows(i, j);
            c = __fmaf_rn(Y.w[j], dot3(Z.w[0], q[0], Z.w[1], q[1], Z.w[2], q[2]), c);
        }
        v = __fmaf_rn(X.w[i], c, v);
    }
    return v;
}

// MAC velocity field + the clamp bounds of its three staggered components.
struct Mac {
    const float* __restrict__ u[3];
    int nx, ny, nz;
    float dx, inv_dx;
    int pow2;      // dx is a power of two
    float hi0[3];  // axis d, BL = 0   (the face field normal to d): dim = n_d + 1
    float hi5[3];  // axis d, BL = 0.5 (a face field tangential to d): dim = n_d
};

static inline Mac make_mac(const float* ux, const float* uy, const float* uz, int nx, int ny, int nz, float dx) {
    Mac m;
    m.u[0] = ux; m.u[1] = uy; m.u[2] = uz;
    m.nx = nx; m.ny = ny; m.nz = nz;
    m.dx = dx; m.inv_dx = 1.0f / dx; m.pow2 = pow2f(dx);
    int n[3] = {nx, ny, nz};
    for (int d = 0; d < 3; d++) {
        m.hi0[d] = clamp_bound(n[d] + 1, 2);
        m.hi5[d] = clamp_bound(n[d], 2);
    }
    return m;
}

// The six axes of a sample at p: A0 where the component is normal to the axis,
// A5 where it is tangential.
template <bool GRAD>
EDGE_D void mac_axes(const Mac& m, const float p[3], float q[3], Axis3<GRAD> A0[3], Axis3<GRAD> A5[3]) {
#pragma unroll
    for (int d = 0; d < 3; d++) {
        q[d] = over_dx(p[d], m.dx, m.inv_dx, m.pow2);
        A0[d] = bspline_axis<GRAD>(q[d], m.hi0[d]);
        A5[d] = bspline_axis<GRAD>(q[d] - 0.5f, m.hi5[d]);
    }
}
template <bool GRAD>
EDGE_D void mac_sums(const Mac& m, const Axis3<GRAD> A0[3], const Axis3<GRAD> A5[3], float v[3], float G[3][3]) {
    v[0] = bspline_sum(grows(m.u[0], A0[0].base, A5[1].base, A5[2].base, m.ny, m.nz), A0[0], A5[1], A5[2],
                       m.inv_dx, GRAD ? G[0] : nullptr);
    v[1] = bspline_sum(grows(m.u[1], A5[0].base, A0[1].base, A5[2].base, m.ny + 1, m.nz), A5[0], A0[1], A5[2],
                       m.inv_dx, GRAD ? G[1] : nullptr);
    v[2] = bspline_sum(grows(m.u[2], A5[0].base, A5[1].base, A0[2].base, m.ny, m.nz + 1), A5[0], A5[1], A0[2],
                       m.inv_dx, GRAD ? G[2] : nullptr);
}

// interp_u_MAC at a scattered point; mask: the warp's lanes that sample.  A
// warp's points in no order are bound by wavefronts and take wide loads; points
// that follow one another in space (sorted particles, a lattice) share their
// lines, and there a 16-byte load, which goes by quarters of a warp, costs more
// wavefronts than three scalar ones.  So a warp takes wide loads where more than
// kPointGroups of its points lie apart from the one before.  us, always wide,
// always scalar and so: 10^6 points at random in 128x256x128 135, 164, 131; in
// a ball 113, 148, 111; on a lattice 92, 31, 35; sorted by cell 88, 49, 51; in
// runs of two 92, 87, 76, of four 88, 52, 53.
constexpr int kPointGroups = 10;
EDGE_D void mac_sample_points(const Mac& m, const float p[3], unsigned mask, float v[3]) {
    float q[3];
    Axis3<false> A0[3], A5[3];
    mac_axes<false>(m, p, q, A0, A5);
    const int x0 = A0[0].base, y0 = A0[1].base, z0 = A0[2].base, x5 = A5[0].base, y5 = A5[1].base, z5 = A5[2].base;
    // apart: not within a cell or so in x and y of the lane before
    const unsigned xy = ((unsigned)x0 << 16) + (unsigned)y0, step = xy - __shfl_up_sync(mask, xy, 1) + 0x00010001u;
    const bool apart = (step & 0xfffcfffcu) != 0;
    auto sums = [&](auto wide) {
        constexpr bool W = decltype(wide)::value;
        v[0] = bspline_rows(vrows<W>(m.u[0], x0, y5, z5, m.ny, m.nz), A0[0], A5[1], A5[2]);
        v[1] = bspline_rows(vrows<W>(m.u[1], x5, y0, z5, m.ny + 1, m.nz), A5[0], A0[1], A5[2]);
        v[2] = bspline_rows(vrows<W>(m.u[2], x5, y5, z0, m.ny, m.nz + 1), A5[0], A5[1], A0[2]);
    };
    if (__popc(__ballot_sync(mask, apart)) > kPointGroups &&
        __all_sync(mask, (x5 > 0 || y5 > 0) && (x0 + 3 < m.nx || y0 + 3 < m.ny)))
        sums(std::true_type{});
    else
        sums(std::false_type{});
}
// the lanes of a warp (of a one-dimensional block) whose index is below n, for
// a thread e that is one of them
EDGE_D unsigned lanes_below(int e, int n) {
    const int left = n - (e - (int)(threadIdx.x & 31));
    return left >= 32 ? 0xffffffffu : (1u << left) - 1u;
}

// interp_u_MAC / interp_u_MAC_grad (taichi_utils.py:322-341).  G rows are the
// gradients of u_x, u_y, u_z.
template <bool GRAD>
EDGE_D void mac_sample(const Mac& m, const float p[3], float v[3], float G[3][3]) {
    float q[3];
    Axis3<GRAD> A0[3], A5[3];
    mac_axes<GRAD>(m, p, q, A0, A5);
    mac_sums<GRAD>(m, A0, A5, v, G);
}

// Component a of interp_u_MAC alone (mac_sample's arithmetic for that
// component): the semi-Lagrangian advection keeps only the face's own
// component of its last sample.
EDGE_D float mac_sample_comp(const Mac& m, const float p[3], int a) {
    Axis3<false> A[3];
#pragma unroll
    for (int d = 0; d < 3; d++) {
        const float q = over_dx(p[d], m.dx, m.inv_dx, m.pow2);
        A[d] = d == a ? bspline_axis<false>(q, m.hi0[d]) : bspline_axis<false>(q - 0.5f, m.hi5[d]);
    }
    const int n1 = m.ny + (a == 1), n2 = m.nz + (a == 2);
    const float* u = a == 0 ? m.u[0] : (a == 1 ? m.u[1] : m.u[2]);
    return bspline_sum(grows(u, A[0].base, A[1].base, A[2].base, n1, n2), A[0], A[1], A[2], m.inv_dx, nullptr);
}

// ---------------------------------------------------------------------------
// The velocity around a block of TI x TJ x TK cells in shared memory, for the
// marches that take some ten samples within a cell of where they start.  Row
// strides are constants there, so a tap is one instruction, and a warp's 32
// consecutive taps are one wavefront at any alignment (1.43 in global memory).
// Two nodes on each side of the block hold every tap of a sample whose
// coordinate is in (i - 1, i + 1.5) on each axis, i the thread's cell: tap
// nodes floor(q - 0.5) .. + 2 and, staggered, floor(q - 1) .. + 2, and the
// clamped ones near the walls (a cell index is at most n - 1).  A warp with a
// sample outside that takes it from global memory.  A step of up to a cell, as
// the CFL condition gives, stays inside; what larger ones cost stands at the
// rules that choose the tile.
// ---------------------------------------------------------------------------
// Blocks of 4 x 4 x 8 cells: 2 x 2 x 32 stage more nodes per cell, were slower
// and leave more of a ragged grid's threads idle.
template <int TI, int TJ, int TK>
struct Tile {
    static constexpr int I = TI, J = TJ, K = TK, threads = TI * TJ * TK;
    static constexpr int N0 = TI + 4, N1 = TJ + 4, N2 = TK + 4;
    // rows of eight cells: the four rows of a warp start 24 words apart, 0, 24,
    // 16, 8 modulo 32, and a row holds two components' twelve nodes
    static_assert(TK == 8, "two components per row of 24 words");
    static constexpr int S2 = 2 * N2, S1 = N1 * S2;
    static constexpr int at(int a) { return a == 1 ? N2 : (a == 2 ? N0 * S1 : 0); }
    static constexpr int size = 2 * N0 * S1;
};
struct SRow {
    const float* p;
    EDGE_D float operator[](int k) const { return p[k]; }
};
template <class T>
struct SRows {
    const float* p;
    EDGE_D SRow operator()(int i, int j) const { return SRow{p + i * T::S1 + j * T::S2}; }
};
template <class T>
struct MacTile {
    Mac m;
    const float* sm;  // component a at T::at(a)
    int off;          // node (0, 0, 0) is at sm - off
    float c[3];       // the thread's cell + 0.25
    unsigned mask;    // the warp's threads that sample
    EDGE_D SRows<T> rows(int a, int x, int y, int z) const {
        return SRows<T>{sm + T::at(a) + ((x * T::N1 + y) * T::S2 + z - off)};
    }
    EDGE_D bool holds(const float q[3]) const {
        const bool in = fabsf(q[0] - c[0]) < 1.25f && fabsf(q[1] - c[1]) < 1.25f && fabsf(q[2] - c[2]) < 1.25f;
        return __all_sync(mask, in);
    }
};
// thread 16 b + c loads node (a, b, c) of every plane a
template <class T>
EDGE_D void stage_tile(const Mac& m, float* sm, int i0, int j0, int k0) {
    static_assert(T::N1 * 16 == T::threads && T::N2 <= 16, "sixteen threads per row of nodes");
    const int c = threadIdx.x & 15, b = threadIdx.x >> 4;
    if (c >= T::N2) return;
    const int j = max(j0 - 2 + b, 0), k = max(k0 - 2 + c, 0);
    const int jc = min(j, m.ny - 1), kc = min(k, m.nz - 1);
    const float* ux = m.u[0] + jc * m.nz + kc;
    const float* uy = m.u[1] + min(j, m.ny) * m.nz + kc;
    const float* uz = m.u[2] + jc * (m.nz + 1) + min(k, m.nz);
    float* d = sm + b * T::S2 + c;
#pragma unroll
    for (int a = 0; a < T::N0; a++) {
        const int i = max(i0 - 2 + a, 0), ic = min(i, m.nx - 1);
        d[T::at(0) + a * T::S1] = __ldg(ux + min(i, m.nx) * (m.ny * m.nz));
        d[T::at(1) + a * T::S1] = __ldg(uy + ic * ((m.ny + 1) * m.nz));
        d[T::at(2) + a * T::S1] = __ldg(uz + ic * (m.ny * (m.nz + 1)));
    }
}
// Stages cell tile `block` (in k, j, i order over the grid) and finds the
// thread's cell; false for a thread past the grid.  All threads of the block.
template <class T>
EDGE_D bool enter_tile(const Mac& m, float* sm, unsigned block, MacTile<T>& t, int& i, int& j, int& k) {
    const unsigned nk = (unsigned)(m.nz + T::K - 1) / T::K, nj = (unsigned)(m.ny + T::J - 1) / T::J;
    const unsigned bj = block / nk, bi = bj / nj;
    const int k0 = (int)(block - bj * nk) * T::K, j0 = (int)(bj - bi * nj) * T::J, i0 = (int)bi * T::I;
    stage_tile<T>(m, sm, i0, j0, k0);
    __syncthreads();
    k = k0 + (int)threadIdx.x % T::K;
    j = j0 + (int)threadIdx.x / T::K % T::J;
    i = i0 + (int)threadIdx.x / (T::K * T::J);
    const bool in = i < m.nx && j < m.ny && k < m.nz;
    t.m = m;
    t.sm = sm;
    t.off = ((i0 - 2) * T::N1 + (j0 - 2)) * T::S2 + (k0 - 2);
    t.c[0] = (float)i + 0.25f;
    t.c[1] = (float)j + 0.25f;
    t.c[2] = (float)k + 0.25f;
    t.mask = __ballot_sync(0xffffffffu, in);
    return in;
}
template <class T>
static inline int tile_blocks(int nx, int ny, int nz) {
    return (nx + T::I - 1) / T::I * ((ny + T::J - 1) / T::J) * ((nz + T::K - 1) / T::K);
}
template <class T>
EDGE_D float mac_sample_comp(const MacTile<T>& t, const float p[3], int a) {
    float q[3];
    Axis3<false> A[3];
#pragma unroll
    for (int d = 0; d < 3; d++) {
        q[d] = over_dx(p[d], t.m.dx, t.m.inv_dx, t.m.pow2);
        A[d] = d == a ? bspline_axis<false>(q[d], t.m.hi0[d]) : bspline_axis<false>(q[d] - 0.5f, t.m.hi5[d]);
    }
    if (t.holds(q))
        return bspline_sum(t.rows(a, A[0].base, A[1].base, A[2].base), A[0], A[1], A[2], t.m.inv_dx, nullptr);
    return mac_sample_comp(t.m, p, a);
}
template <bool GRAD, class T>
EDGE_D void mac_sample(const MacTile<T>& t, const float p[3], float v[3], float G[3][3]) {
    float q[3];
    Axis3<GRAD> A0[3], A5[3];
    mac_axes<GRAD>(t.m, p, q, A0, A5);
    if (t.holds(q)) {
        v[0] = bspline_sum(t.rows(0, A0[0].base, A5[1].base, A5[2].base), A0[0], A5[1], A5[2], t.m.inv_dx,
                           GRAD ? G[0] : nullptr);
        v[1] = bspline_sum(t.rows(1, A5[0].base, A0[1].base, A5[2].base), A5[0], A0[1], A5[2], t.m.inv_dx,
                           GRAD ? G[1] : nullptr);
        v[2] = bspline_sum(t.rows(2, A5[0].base, A5[1].base, A0[2].base), A5[0], A5[1], A0[2], t.m.inv_dx,
                           GRAD ? G[2] : nullptr);
    } else {
        mac_sums<GRAD>(t.m, A0, A5, v, G);
    }
}

// ---------------------------------------------------------------------------
// trilinear dye sampler on 4-channel cell fields (taichi_utils.py:172-227)
// ---------------------------------------------------------------------------
struct Dye {
    int nx, ny, nz;
    float dx, inv_dx;
    int pow2;
    float hi[3];  // dim-1-eps
};
static inline Dye make_dye(int nx, int ny, int nz, float dx) {
    Dye d;
    d.nx = nx; d.ny = ny; d.nz = nz; d.dx = dx; d.inv_dx = 1.0f / dx; d.pow2 = pow2f(dx);
    d.hi[0] = clamp_bound(nx, 1);
    d.hi[1] = clamp_bound(ny, 1);
    d.hi[2] = clamp_bound(nz, 1);
    return d;
}
struct Lin8 {
    int i0, j0, k0, i1, j1, k1;
    float wx[2], wy[2], wz[2];
};
EDGE_D Lin8 lin_setup(const Dye& d, const float p[3]) {
    Lin8 L;
    float s[3];
    float u[3] = {over_dx(p[0], d.dx, d.inv_dx, d.pow2) - 0.5f, over_dx(p[1], d.dx, d.inv_dx, d.pow2) - 0.5f,
                  over_dx(p[2], d.dx, d.inv_dx, d.pow2) - 0.5f};
#pragma unroll
    for (int a = 0; a < 3; a++) s[a] = fmaxf(1.0f, fminf(u[a], d.hi[a]));
    float iu = floorf(s[0]), iv = floorf(s[1]), iw = floorf(s[2]);
    L.i0 = (int)iu; L.j0 = (int)iv; L.k0 = (int)iw;
    // sample() clamps the +1 corner (it can reach dim when s hits the bound)
    L.i1 = min(L.i0 + 1, d.nx - 1);
    L.j1 = min(L.j0 + 1, d.ny - 1);
    L.k1 = min(L.k0 + 1, d.nz - 1);
    L.wx[0] = 1.0f - fabsf(s[0] - iu); L.wx[1] = 1.0f - fabsf(s[0] - (iu + 1.0f));
    L.wy[0] = 1.0f - fabsf(s[1] - iv); L.wy[1] = 1.0f - fabsf(s[1] - (iv + 1.0f));
    L.wz[0] = 1.0f - fabsf(s[2] - iw); L.wz[1] = 1.0f - fabsf(s[2] - (iw + 1.0f));
    return L;
}
EDGE_D float4 ld4(const float* __restrict__ f, int e) { return __ldg(reinterpret_cast<const float4*>(f) + e); }

EDGE_D float4 dye_interp(const float* __restrict__ f, const Dye& d, const Lin8& L) {
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int c = 0; c < 8; c++) {
        int a = c >> 2, b = (c >> 1) & 1, q = c & 1;
        float4 v = ld4(f, idx3(a ? L.i1 : L.i0, b ? L.j1 : L.j0, q ? L.k1 : L.k0, d.ny, d.nz));
        float w = L.wx[a] * L.wy[b] * L.wz[q];
        acc.x += v.x * w; acc.y += v.y * w; acc.z += v.z * w; acc.w += v.w * w;
    }
    return acc;
}
EDGE_D void dye_minmax(const float* __restrict__ f, const Dye& d, const Lin8& L, float4& mn, float4& mx) {
#pragma unroll
    for (int c = 0; c < 8; c++) {
        int a = c >> 2, b = (c >> 1) & 1, q = c & 1;
        float4 v = ld4(f, idx3(a ? L.i1 : L.i0, b ? L.j1 : L.j0, q ? L.k1 : L.k0, d.ny, d.nz));
        if (c == 0) { mn = v; mx = v; }
        else {
            mn.x = fminf(mn.x, v.x); mn.y = fminf(mn.y, v.y); mn.z = fminf(mn.z, v.z); mn.w = fminf(mn.w, v.w);
            mx.x = fmaxf(mx.x, v.x); mx.y = fmaxf(mx.y, v.y); mx.z = fmaxf(mx.z, v.z); mx.w = fmaxf(mx.w, v.w);
        }
    }
}
EDGE_D float4 clamp4(float4 v, float4 lo, float4 hi) {
    return make_float4(fminf(fmaxf(v.x, lo.x), hi.x), fminf(fmaxf(v.y, lo.y), hi.y), fminf(fmaxf(v.z, lo.z), hi.z),
                       fminf(fmaxf(v.w, lo.w), hi.w));
}

// ---------------------------------------------------------------------------
// cubic Hermite flow-map interpolation (hermite.py:4-607)
// ---------------------------------------------------------------------------
enum Variant { HV_FD = EDGE_HERMITE_FD, HV_GARM = EDGE_HERMITE_GARM, HV_FULL = EDGE_HERMITE_FULL };

// Flow-map fields on the cell grid: psi (vec3), rows T_c = grad psi_c (vec3),
// dT_c = (psi_c,yz, psi_c,xz, psi_c,xy) (vec3) and d2T_c = psi_c,xyz (scalar).
struct MapF {
    const float* __restrict__ psi;
    const float* __restrict__ T[3];
    const float* __restrict__ dT[3];
    const float* __restrict__ d2T[3];
    int nx, ny, nz;
    float dx, inv_dx;
    int pow2;
    float hi[3];  // dim-2-eps
};
static inline MapF make_map(const float* psi, const float* const T[3], const float* const dT[3],
                            const float* const d2T[3], int nx, int ny, int nz, float dx) {
    MapF m;
    m.psi = psi;
    for (int c = 0; c < 3; c++) {
        m.T[c] = T[c];
        m.dT[c] = dT ? dT[c] : nullptr;
        m.d2T[c] = d2T ? d2T[c] : nullptr;
    }
    m.nx = nx; m.ny = ny; m.nz = nz; m.dx = dx; m.inv_dx = 1.0f / dx; m.pow2 = pow2f(dx);
    m.hi[0] = clamp_bound(nx, 2);
    m.hi[1] = clamp_bound(ny, 2);
    m.hi[2] = clamp_bound(nz, 2);
    return m;
}

// Basis of one axis at the two corners (i = 0, 1): hermite_f/g and their
// derivatives at x = s - (iu + i).
struct HAxis {
    int c0, cm, cp, cpp;   // iu, iu-1, iu+1, iu+2 (clamped as sample() does)
    float f[2], g[2], df[2], dg[2];
};
// hermite_f/g and derivatives at x with |x| <= 1 (haxis passes x in [0, 1)
// and [-1, 0)).  The reference's |x| >= 1 branch gives 0; at |x| = 1 every
// polynomial below is exactly 0 as well, so no select is needed.
EDGE_D void hbasis(float x, float& f, float& g, float& df, float& dg) {
    float a = fabsf(x);
    float a2 = a * a, a3 = a2 * a;
    f = 2.0f * a3 - 3.0f * a2 + 1.0f;
    float gg = a3 - 2.0f * a2 + a;
    float dff = 6.0f * a2 - 6.0f * a;
    dg = 3.0f * a2 - 4.0f * a + 1.0f;
    g = x < 0.0f ? -gg : gg;
    df = x < 0.0f ? -dff : dff;
}
EDGE_D HAxis haxis(float u, float hi, int n) {
    HAxis h;
    float s = fmaxf(1.0f, fminf(u, hi));
    float iu = floorf(s);
    int b = (int)iu;
    h.c0 = b;
    h.cm = b - 1;
    h.cp = min(b + 1, n - 1);
    h.cpp = min(b + 2, n - 1);
    hbasis(s - iu, h.f[0], h.g[0], h.df[0], h.dg[0]);
    hbasis(s - (iu + 1.0f), h.f[1], h.g[1], h.df[1], h.dg[1]);
    return h;
}

EDGE_D float ldv(const float* __restrict__ f, int e, int c) { return __ldg(f + 3 * e + c); }

// The 8 Hermite coefficients t[a][b][c] (a, b, c = 0 for f, 1 for g basis on
// x, y, z) of component `comp` at corner (ii, jj, kk); term scaling as in the
// reference (value, grad*dx, mixed*dx^2, triple*dx^3).
template <int VARIANT>
EDGE_D void hcoef(const MapF& m, int comp, int ii, int jj, int kk, int im, int ip, int jm, int jp, int km, int kp,
                  float t[8]) {
    const int n1 = m.ny, n2 = m.nz;
    const float dx = m.dx;
    const float* __restrict__ G = m.T[comp];
    int e = idx3(ii, jj, kk, n1, n2);
    t[0] = ldv(m.psi, e, comp);                  // fff
    t[4] = ldv(G, e, 0) * dx;                    // gff
    t[2] = ldv(G, e, 1) * dx;                    // fgf
    t[1] = ldv(G, e, 2) * dx;                    // ffg
    if (VARIANT == HV_FD) {
        // hermite.py:104-148 (FD of the stored gradient)
        int ekp = idx3(ii, jj, kp, n1, n2), ekm = idx3(ii, jj, km, n1, n2);
        int ejp = idx3(ii, jp, kk, n1, n2), ejm = idx3(ii, jm, kk, n1, n2);
        int eip = idx3(ip, jj, kk, n1, n2), eim = idx3(im, jj, kk, n1, n2);
        t[3] = ((ldv(G, ekp, 1) - ldv(G, ekm, 1)) + (ldv(G, ejp, 2) - ldv(G, ejm, 2))) / 4.0f * dx;   // fgg
        t[5] = ((ldv(G, ekp, 0) - ldv(G, ekm, 0)) + (ldv(G, eip, 2) - ldv(G, eim, 2))) / 4.0f * dx;   // gfg
        t[6] = ((ldv(G, ejp, 0) - ldv(G, ejm, 0)) + (ldv(G, eip, 1) - ldv(G, eim, 1))) / 4.0f * dx;   // ggf
        float v30 = ((ldv(G, idx3(ip, jj, kp, n1, n2), 1) - ldv(G, idx3(ip, jj, km, n1, n2), 1)) +
                     (ldv(G, idx3(ip, jp, kk, n1, n2), 2) - ldv(G, idx3(ip, jm, kk, n1, n2), 2))) / 4.0f;
        float v31 = ((ldv(G, idx3(im, jj, kp, n1, n2), 1) - ldv(G, idx3(im, jj, km, n1, n2), 1)) +
                     (ldv(G, idx3(im, jp, kk, n1, n2), 2) - ldv(G, idx3(im, jm, kk, n1, n2), 2))) / 4.0f;
        float v32 = ((ldv(G, idx3(ii, jp, kp, n1, n2), 0) - ldv(G, idx3(ii, jp, km, n1, n2), 0)) +
                     (ldv(G, idx3(ip, jp, kk, n1, n2), 2) - ldv(G, idx3(im, jp, kk, n1, n2), 2))) / 4.0f;
        float v33 = ((ldv(G, idx3(ii, jm, kp, n1, n2), 0) - ldv(G, idx3(ii, jm, km, n1, n2), 0)) +
                     (ldv(G, idx3(ip, jm, kk, n1, n2), 2) - ldv(G, idx3(im, jm, kk, n1, n2), 2))) / 4.0f;
        float v34 = ((ldv(G, idx3(ii, jp, kp, n1, n2), 0) - ldv(G, idx3(ii, jm, kp, n1, n2), 0)) +
                     (ldv(G, idx3(ip, jj, kp, n1, n2), 1) - ldv(G, idx3(im, jj, kp, n1, n2), 1))) / 4.0f;
        float v35 = ((ldv(G, idx3(ii, jp, km, n1, n2), 0) - ldv(G, idx3(ii, jm, km, n1, n2), 0)) +
                     (ldv(G, idx3(ip, jj, km, n1, n2), 1) - ldv(G, idx3(im, jj, km, n1, n2), 1))) / 4.0f;
        t[7] = (v30 - v31 + v32 - v33 + v34 - v35) / 6.0f * dx;  // ggg
    } else {
        const float* __restrict__ GG = m.dT[comp];
        t[3] = ldv(GG, e, 0) * dx * dx;  // fgg
        t[5] = ldv(GG, e, 1) * dx * dx;  // gfg
        t[6] = ldv(GG, e, 2) * dx * dx;  // ggf
        if (VARIANT == HV_GARM) {
            // hermite.py:346-351 (FD of the stored mixed derivatives)
            t[7] = ((ldv(GG, idx3(ip, jj, kk, n1, n2), 0) - ldv(GG, idx3(im, jj, kk, n1, n2), 0)) +
                    (ldv(GG, idx3(ii, jp, kk, n1, n2), 1) - ldv(GG, idx3(ii, jm, kk, n1, n2), 1)) +
                    (ldv(GG, idx3(ii, jj, kp, n1, n2), 2) - ldv(GG, idx3(ii, jj, km, n1, n2), 2))) / 6.0f * dx * dx;
        } else {
            t[7] = __ldg(m.d2T[comp] + e) * dx * dx * dx;  // hermite.py:508-509
        }
    }
}

// Hermite value (and gradient, already divided by dx, when GRAD) of all three
// components of psi at p.  Tensor-product evaluation: the 64 coefficients of
// the 2x2x2 corner stencil are contracted axis by axis (z, then y, then x).
template <int VARIANT, bool GRAD>
EDGE_D void hermite3(const MapF& m, const float p[3], float val[3], float grad[3][3]) {
    float q[3] = {over_dx(p[0], m.dx, m.inv_dx, m.pow2) - 0.5f, over_dx(p[1], m.dx, m.inv_dx, m.pow2) - 0.5f,
                  over_dx(p[2], m.dx, m.inv_dx, m.pow2) - 0.5f};
    HAxis X = haxis(q[0], m.hi[0], m.nx), Y = haxis(q[1], m.hi[1], m.ny), Z = haxis(q[2], m.hi[2], m.nz);
#pragma unroll
    for (int comp = 0; comp < 3; comp++) {
        float v = 0.0f, gx = 0.0f, gy = 0.0f, gz = 0.0f;
#pragma unroll
        for (int i = 0; i < 2; i++) {
            int ii = i ? X.cp : X.c0, im = i ? X.c0 : X.cm, ip = i ? X.cpp : X.cp;
            // per x-corner partial sums over (j, b) and (k, c)
            float Ax[2] = {0.f, 0.f}, dAx[2] = {0.f, 0.f}, Bx[2] = {0.f, 0.f}, dBx[2] = {0.f, 0.f};
            // Ax[a] = sum_{j,b,k,c} Y Z t[a][b][c]; Bx: with dY; dAx: with dZ
#pragma unroll
            for (int j = 0; j < 2; j++) {
                int jj = j ? Y.cp : Y.c0, jm = j ? Y.c0 : Y.cm, jp = j ? Y.cpp : Y.cp;
#pragma unroll
                for (int k = 0; k < 2; k++) {
                    int kk = k ? Z.cp : Z.c0, km = k ? Z.c0 : Z.cm, kp = k ? Z.cpp : Z.cp;
                    float t[8];
                    hcoef<VARIANT>(m, comp, ii, jj, kk, im, ip, jm, jp, km, kp, t);
                    // contract z (c): P[a][b] = Zf t[a][b][0] + Zg t[a][b][1]
#pragma unroll
                    for (int a = 0; a < 2; a++) {
                        float P0 = Z.f[k] * t[a * 4 + 0] + Z.g[k] * t[a * 4 + 1];
                        float P1 = Z.f[k] * t[a * 4 + 2] + Z.g[k] * t[a * 4 + 3];
                        float Q = Y.f[j] * P0 + Y.g[j] * P1;
                        Ax[a] += Q;
                        if (GRAD) {
                            float dP0 = Z.df[k] * t[a * 4 + 0] + Z.dg[k] * t[a * 4 + 1];
                            float dP1 = Z.df[k] * t[a * 4 + 2] + Z.dg[k] * t[a * 4 + 3];
                            Bx[a] += Y.df[j] * P0 + Y.dg[j] * P1;
                            dAx[a] += Y.f[j] * dP0 + Y.g[j] * dP1;
                        }
                    }
                }
            }
            v += X.f[i] * Ax[0] + X.g[i] * Ax[1];
            if (GRAD) {
                gx += X.df[i] * Ax[0] + X.dg[i] * Ax[1];
                gy += X.f[i] * Bx[0] + X.g[i] * Bx[1];
                gz += X.f[i] * dAx[0] + X.g[i] * dAx[1];
            }
            (void)dBx;
        }
        val[comp] = v;
        if (GRAD) {
            float inv = 1.0f / m.dx;
            grad[comp][0] = gx * inv;
            grad[comp][1] = gy * inv;
            grad[comp][2] = gz * inv;
        }
    }
}

// ---------------------------------------------------------------------------
// packed map layout: float4 planes, one cell per float4, components (x, y, z)
// in .x .y .z:
//   plane 0: psi
//   planes 1..3: d psi / dx, d psi / dy, d psi / dz   (columns of grad psi)
//   planes 4..6: psi_yz, psi_xz, psi_xy               (EDGE dT, ED8 dT)
//   plane 7: psi_xyz                                   (ED8 d2T)
// One 128-bit load then serves all three components of a Hermite stencil
// point.  The ED4 and EDGE maps carry fewer state planes (4 and 7); their
// remaining planes hold the Hermite coefficients the reference derives by
// finite differences at every evaluation (ED4: the fgg, gfg, ggf, ggg terms
// from the gradient, hermite.py:104-148; EDGE: the ggg term from the mixed
// derivatives, hermite.py:346-351), computed once per map by k_coef_p up to
// their final multiplications by dx, which the evaluation applies.  The
// corners a Hermite evaluation visits are cells 1..n-1 of each axis and the
// reference's neighbour indices there are the cell's own +-1 clamped to the
// grid, so a per-cell table with clamped neighbours holds exactly the values
// the reference computes per corner.  Every packed map is 8 planes.
// ---------------------------------------------------------------------------
constexpr int kPlanesED4 = 4, kPlanesEDGE = 7, kPlanesED8 = 8;  // state planes
constexpr int kPlanesStored = 8;
// internal variants: ED4 / EDGE Hermite reading the precomputed planes
constexpr int HV_FD_P = 3, HV_GARM_P = 4;

struct MapP {
    const float4* __restrict__ g;  // planes, plane q at g + q * n
    int n;                          // cells
    int nx, ny, nz;
    float dx, inv_dx;
    int pow2;
    float hi[3];
};
static inline MapP make_mapp(const float* planes, int nx, int ny, int nz, float dx) {
    MapP m;
    m.g = reinterpret_cast<const float4*>(planes);
    m.n = nx * ny * nz;
    m.nx = nx; m.ny = ny; m.nz = nz; m.dx = dx; m.inv_dx = 1.0f / dx; m.pow2 = pow2f(dx);
    m.hi[0] = clamp_bound(nx, 2);
    m.hi[1] = clamp_bound(ny, 2);
    m.hi[2] = clamp_bound(nz, 2);
    return m;
}
EDGE_D float4 ldp(const MapP& m, int q, int e) { return __ldg(m.g + (size_t)q * m.n + e); }
EDGE_D float c4(const float4& v, int c) { return c == 0 ? v.x : (c == 1 ? v.y : v.z); }

// Coefficients t[comp][8] of cell e from the packed planes (same terms and
// scaling as hcoef; the derived planes take their last products by dx here).
template <int VARIANT>
EDGE_D void hcoef_p(const MapP& m, int e, float t[3][8]) {
    const float dx = m.dx;
    float4 P = ldp(m, 0, e), G0 = ldp(m, 1, e), G1 = ldp(m, 2, e), G2 = ldp(m, 3, e);
    float4 A = ldp(m, 4, e), B = ldp(m, 5, e), C = ldp(m, 6, e), D = ldp(m, 7, e);
#pragma unroll
    for (int c = 0; c < 3; c++) {
        t[c][0] = c4(P, c);
        t[c][4] = c4(G0, c) * dx;
        t[c][2] = c4(G1, c) * dx;
        t[c][1] = c4(G2, c) * dx;
        if (VARIANT == HV_FD_P) {
            t[c][3] = c4(A, c) * dx;
            t[c][5] = c4(B, c) * dx;
            t[c][6] = c4(C, c) * dx;
            t[c][7] = c4(D, c) * dx;
        } else {
            t[c][3] = c4(A, c) * dx * dx;
            t[c][5] = c4(B, c) * dx * dx;
            t[c][6] = c4(C, c) * dx * dx;
            t[c][7] = VARIANT == HV_GARM_P ? c4(D, c) * dx * dx : c4(D, c) * dx * dx * dx;
        }
    }
}

// The coefficients of hcoef_p divided by dx^(number of g factors), for a
// power-of-two dx (every such scaling is then exact): the g basis functions
// carry the factor dx instead (hermite3p), which gives every product of the
// contraction the same value with 3 multiplications per corner instead of 33.
template <int VARIANT>
EDGE_D void hcoef_p_unscaled(const MapP& m, int e, float t[3][8]) {
    const float inv = m.inv_dx;
    float4 P = ldp(m, 0, e), G0 = ldp(m, 1, e), G1 = ldp(m, 2, e), G2 = ldp(m, 3, e);
    float4 A = ldp(m, 4, e), B = ldp(m, 5, e), C = ldp(m, 6, e), D = ldp(m, 7, e);
#pragma unroll
    for (int c = 0; c < 3; c++) {
        t[c][0] = c4(P, c);
        t[c][4] = c4(G0, c);
        t[c][2] = c4(G1, c);
        t[c][1] = c4(G2, c);
        if (VARIANT == HV_FD_P) {  // planes 4-7 hold the terms over dx (hcoef_p multiplies by dx once)
            t[c][3] = c4(A, c) * inv;
            t[c][5] = c4(B, c) * inv;
            t[c][6] = c4(C, c) * inv;
            t[c][7] = c4(D, c) * inv * inv;
        } else {
            t[c][3] = c4(A, c);
            t[c][5] = c4(B, c);
            t[c][6] = c4(C, c);
            t[c][7] = VARIANT == HV_GARM_P ? c4(D, c) * inv : c4(D, c);  // GARM_P plane 7 holds psi_xyz over dx
        }
    }
}

// hermite3 on the packed layout: the 8 corners are visited once and feed all
// three components.
template <int VARIANT, bool GRAD>
EDGE_D void hermite3p(const MapP& m, const float p[3], float val[3], float grad[3][3]) {
    float q[3] = {over_dx(p[0], m.dx, m.inv_dx, m.pow2) - 0.5f, over_dx(p[1], m.dx, m.inv_dx, m.pow2) - 0.5f,
                  over_dx(p[2], m.dx, m.inv_dx, m.pow2) - 0.5f};
    HAxis X = haxis(q[0], m.hi[0], m.nx), Y = haxis(q[1], m.hi[1], m.ny), Z = haxis(q[2], m.hi[2], m.nz);
    // power-of-two dx: the g basis functions carry dx and the coefficients
    // come unscaled (hcoef_p_unscaled); the same products, fewer multiplies
    const bool fold = m.pow2;
    if (fold) {
#pragma unroll
        for (int c = 0; c < 2; c++) {
            X.g[c] *= m.dx; X.dg[c] *= m.dx;
            Y.g[c] *= m.dx; Y.dg[c] *= m.dx;
            Z.g[c] *= m.dx; Z.dg[c] *= m.dx;
        }
    }
    float v[3] = {0.f, 0.f, 0.f}, gx[3] = {0.f, 0.f, 0.f}, gy[3] = {0.f, 0.f, 0.f}, gz[3] = {0.f, 0.f, 0.f};
#pragma unroll
    for (int i = 0; i < 2; i++) {
        const int ii = i ? X.cp : X.c0;
        float Ax[3][2] = {{0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}};
        float Bx[3][2] = {{0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}};
        float dAx[3][2] = {{0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}};
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const int jj = j ? Y.cp : Y.c0;
#pragma unroll
            for (int k = 0; k < 2; k++) {
                const int e = idx3(ii, jj, k ? Z.cp : Z.c0, m.ny, m.nz);
                float t[3][8];
                if (fold) hcoef_p_unscaled<VARIANT>(m, e, t);
                else hcoef_p<VARIANT>(m, e, t);
#pragma unroll
                for (int c = 0; c < 3; c++)
#pragma unroll
                    for (int a = 0; a < 2; a++) {
                        float P0 = Z.f[k] * t[c][a * 4 + 0] + Z.g[k] * t[c][a * 4 + 1];
                        float P1 = Z.f[k] * t[c][a * 4 + 2] + Z.g[k] * t[c][a * 4 + 3];
                        Ax[c][a] += Y.f[j] * P0 + Y.g[j] * P1;
                        if (GRAD) Bx[c][a] += Y.df[j] * P0 + Y.dg[j] * P1;
                        if (GRAD) {
                            float dP0 = Z.df[k] * t[c][a * 4 + 0] + Z.dg[k] * t[c][a * 4 + 1];
                            float dP1 = Z.df[k] * t[c][a * 4 + 2] + Z.dg[k] * t[c][a * 4 + 3];
                            dAx[c][a] += Y.f[j] * dP0 + Y.g[j] * dP1;
                        }
                    }
            }
        }
#pragma unroll
        for (int c = 0; c < 3; c++) {
            v[c] += X.f[i] * Ax[c][0] + X.g[i] * Ax[c][1];
            if (GRAD) gx[c] += X.df[i] * Ax[c][0] + X.dg[i] * Ax[c][1];
            if (GRAD) gy[c] += X.f[i] * Bx[c][0] + X.g[i] * Bx[c][1];
            if (GRAD) gz[c] += X.f[i] * dAx[c][0] + X.g[i] * dAx[c][1];
        }
    }
    const float inv = 1.0f / m.dx;
#pragma unroll
    for (int c = 0; c < 3; c++) {
        val[c] = v[c];
        if (GRAD) grad[c][0] = gx[c] * inv;
        if (GRAD) grad[c][1] = gy[c] * inv;
        if (GRAD) grad[c][2] = gz[c] * inv;
    }
}

// The 8 Hermite coefficients of one corner, bit 2 / 1 / 0 of the index = the g
// basis along x / y / z, components x and y as a pair.
struct HCorner {
    f2 xy[8];
    float z[8];
};
EDGE_D void set_coef(HCorner& t, int q, const float4& v) {
    t.xy[q] = pair(v.x, v.y);
    t.z[q] = v.z;
}
EDGE_D void set_coef(HCorner& t, int q, const float4& v, float s) {
    t.xy[q] = mul2(pair(v.x, v.y), both(s));
    t.z[q] = v.z * s;
}
// hcoef_p and hcoef_p_unscaled
template <int VARIANT>
EDGE_D void hcorner(const MapP& m, int e, HCorner& t) {
    const float dx = m.dx;
    set_coef(t, 0, ldp(m, 0, e));
    set_coef(t, 4, ldp(m, 1, e), dx);
    set_coef(t, 2, ldp(m, 2, e), dx);
    set_coef(t, 1, ldp(m, 3, e), dx);
    constexpr int slot[4] = {3, 5, 6, 7};
#pragma unroll
    for (int q = 0; q < 4; q++) {
        set_coef(t, slot[q], ldp(m, 4 + q, e), dx);
        if (VARIANT != HV_FD_P) {
            const int more = q == 3 && VARIANT == HV_FULL ? 2 : 1;
#pragma unroll
            for (int r = 0; r < more; r++) {
                t.xy[slot[q]] = mul2(t.xy[slot[q]], both(dx));
                t.z[slot[q]] = t.z[slot[q]] * dx;
            }
        }
    }
}

template <int VARIANT>
EDGE_D void hcorner_unscaled(const MapP& m, int e, HCorner& t) {
    const float inv = m.inv_dx;
    set_coef(t, 0, ldp(m, 0, e));
    set_coef(t, 4, ldp(m, 1, e));
    set_coef(t, 2, ldp(m, 2, e));
    set_coef(t, 1, ldp(m, 3, e));
    if (VARIANT == HV_FD_P) {  // planes 4-7 hold the terms over dx (hcoef_p multiplies by dx once)
        set_coef(t, 3, ldp(m, 4, e), inv);
        set_coef(t, 5, ldp(m, 5, e), inv);
        set_coef(t, 6, ldp(m, 6, e), inv);
        set_coef(t, 7, ldp(m, 7, e), inv);
        t.xy[7] = mul2(t.xy[7], both(inv));
        t.z[7] = t.z[7] * inv;
    } else {
        set_coef(t, 3, ldp(m, 4, e));
        set_coef(t, 5, ldp(m, 5, e));
        set_coef(t, 6, ldp(m, 6, e));
        if (VARIANT == HV_GARM_P) set_coef(t, 7, ldp(m, 7, e), inv);  // plane 7 holds psi_xyz over dx
        else set_coef(t, 7, ldp(m, 7, e));
    }
}

// f a + g b (+ acc) with the roundings of the scalar expressions as nvcc
// contracts them
EDGE_D float mix(float f, float a, float g, float b) { return __fmaf_rn(f, a, __fmul_rn(g, b)); }
EDGE_D f2 mix(float f, f2 a, float g, f2 b) { return fma2(both(f), a, mul2(both(g), b)); }
EDGE_D float mix(float f, float a, float g, float b, float acc) { return __fadd_rn(acc, mix(f, a, g, b)); }
EDGE_D f2 mix(float f, f2 a, float g, f2 b, f2 acc) { return add2(acc, mix(f, a, g, b)); }

// The contraction of one corner for one component (T = float) or two (f2).
template <class T>
EDGE_D void hcontract(const T t[8], const HAxis& Y, const HAxis& Z, int j, int k, T (&A)[2], T (&B)[2], T (&dA)[2]) {
#pragma unroll
    for (int a = 0; a < 2; a++) {
        const T P0 = mix(Z.f[k], t[a * 4 + 0], Z.g[k], t[a * 4 + 1]);
        const T P1 = mix(Z.f[k], t[a * 4 + 2], Z.g[k], t[a * 4 + 3]);
        A[a] = mix(Y.f[j], P0, Y.g[j], P1, A[a]);
        B[a] = mix(Y.df[j], P0, Y.dg[j], P1, B[a]);
        const T dP0 = mix(Z.df[k], t[a * 4 + 0], Z.dg[k], t[a * 4 + 1]);
        const T dP1 = mix(Z.df[k], t[a * 4 + 2], Z.dg[k], t[a * 4 + 3]);
        dA[a] = mix(Y.f[j], dP0, Y.g[j], dP1, dA[a]);
    }
}

// hermite3p with the gradient, components x and y as pairs: the same values
// with two thirds of the contraction's issue slots, for more registers; what
// it gives depends on the register cap.  EDGE march at 4 blocks of 128 threads
// per SM: 256x128x128 2979 us in the scalar form at its best, 2684 us so; GE
// march at 5 blocks: 96^3 184 -> 166 us.  The value alone is better off in the
// scalar form (ED8 march 2967 against 3169 us).
template <int VARIANT>
EDGE_D void hermite3p_pairs(const MapP& m, const float p[3], float val[3], float grad[3][3]) {
    float q[3] = {over_dx(p[0], m.dx, m.inv_dx, m.pow2) - 0.5f, over_dx(p[1], m.dx, m.inv_dx, m.pow2) - 0.5f,
                  over_dx(p[2], m.dx, m.inv_dx, m.pow2) - 0.5f};
    HAxis X = haxis(q[0], m.hi[0], m.nx), Y = haxis(q[1], m.hi[1], m.ny), Z = haxis(q[2], m.hi[2], m.nz);
    // power-of-two dx: the g basis functions carry dx and the coefficients
    // come unscaled (hcoef_p_unscaled); the same products, fewer multiplies
    const bool fold = m.pow2;
    if (fold) {
#pragma unroll
        for (int c = 0; c < 2; c++) {
            X.g[c] *= m.dx; X.dg[c] *= m.dx;
            Y.g[c] *= m.dx; Y.dg[c] *= m.dx;
            Z.g[c] *= m.dx; Z.dg[c] *= m.dx;
        }
    }
    f2 v2 = both(0.f), gx2 = v2, gy2 = v2, gz2 = v2;       // components x, y
    float v1 = 0.f, gx1 = 0.f, gy1 = 0.f, gz1 = 0.f;       // component z
#pragma unroll
    for (int i = 0; i < 2; i++) {
        const int ii = i ? X.cp : X.c0;
        f2 A2[2] = {both(0.f), both(0.f)}, B2[2] = {both(0.f), both(0.f)}, dA2[2] = {both(0.f), both(0.f)};
        float A1[2] = {0.f, 0.f}, B1[2] = {0.f, 0.f}, dA1[2] = {0.f, 0.f};
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const int jj = j ? Y.cp : Y.c0;
#pragma unroll
            for (int k = 0; k < 2; k++) {
                const int kk = k ? Z.cp : Z.c0;
                HCorner t;
                if (fold) hcorner_unscaled<VARIANT>(m, idx3(ii, jj, kk, m.ny, m.nz), t);
                else hcorner<VARIANT>(m, idx3(ii, jj, kk, m.ny, m.nz), t);
                hcontract(t.xy, Y, Z, j, k, A2, B2, dA2);
                hcontract(t.z, Y, Z, j, k, A1, B1, dA1);
            }
        }
        v2 = mix(X.f[i], A2[0], X.g[i], A2[1], v2);
        v1 = mix(X.f[i], A1[0], X.g[i], A1[1], v1);
        gx2 = mix(X.df[i], A2[0], X.dg[i], A2[1], gx2);
        gx1 = mix(X.df[i], A1[0], X.dg[i], A1[1], gx1);
        gy2 = mix(X.f[i], B2[0], X.g[i], B2[1], gy2);
        gy1 = mix(X.f[i], B1[0], X.g[i], B1[1], gy1);
        gz2 = mix(X.f[i], dA2[0], X.g[i], dA2[1], gz2);
        gz1 = mix(X.f[i], dA1[0], X.g[i], dA1[1], gz1);
    }
    val[0] = lo(v2); val[1] = hi(v2); val[2] = v1;
    const float inv = 1.0f / m.dx;
    grad[0][0] = lo(gx2) * inv; grad[1][0] = hi(gx2) * inv; grad[2][0] = gx1 * inv;
    grad[0][1] = lo(gy2) * inv; grad[1][1] = hi(gy2) * inv; grad[2][1] = gy1 * inv;
    grad[0][2] = lo(gz2) * inv; grad[1][2] = hi(gz2) * inv; grad[2][2] = gz1 * inv;
}

// ---------------------------------------------------------------------------
// RK4 marches (hermite.py:786-860, run_edge.py:337-357)
// ---------------------------------------------------------------------------
// M: Mac or MacTile.  The stages run as a loop: one copy of the sampler keeps
// the kernels inside the instruction cache.
template <class M>
EDGE_D void rk4_pos(const M& mac, float psi[3], float dt) {
    float u[3], q[3], su[3] = {0.0f, 0.0f, 0.0f};
    const float h = 0.5f * dt;
#pragma unroll
    for (int c = 0; c < 3; c++) q[c] = psi[c];
#pragma unroll 1
    for (int stage = 0; stage < 4; stage++) {
        mac_sample<false>(mac, q, u, nullptr);
        const float wt = (stage == 0 || stage == 3) ? 1.0f : 2.0f;
        const float hh = stage < 2 ? h : dt;
#pragma unroll
        for (int c = 0; c < 3; c++) {
            su[c] = __fmaf_rn(wt, u[c], su[c]);
            q[c] = __fmaf_rn(hh, u[c], psi[c]);
        }
    }
    const float w6 = dt * 1.0f / 6.0f;
#pragma unroll
    for (int c = 0; c < 3; c++) psi[c] = __fmaf_rn(w6, su[c], psi[c]);
}

// RK4 of a point with NC Jacobian columns C[a] (dC/dt = grad u . C).  The
// four stages run as a loop (not unrolled): one copy of the 81-tap sampler
// keeps the kernels inside the instruction cache.  Columns 0 and 1 are
// advanced as pairs.
template <int NC, class M>
EDGE_D void rk4_jac(const M& mac, float psi[3], float C[NC][3], float dt) {
    static_assert(NC == 1 || NC == 3, "one column, or all three");
    constexpr int L = NC - 1;  // the column advanced on its own
    float u[3], G[3][3], q[3], su[3], s1[3], S1[3];
    f2 C2[3], s2[3], S2[3];
    const float h = 0.5f * dt;
#pragma unroll
    for (int c = 0; c < 3; c++) {
        q[c] = psi[c];
        su[c] = 0.0f;  // the RK4 sums, started at zero: 0 + 1 * u is u exactly
        s1[c] = C[L][c];
        S1[c] = 0.0f;
        if (NC == 3) {
            C2[c] = s2[c] = pair(C[0][c], C[NC - 2][c]);
            S2[c] = both(0.0f);
        }
    }
#pragma unroll 1
    for (int stage = 0; stage < 4; stage++) {
        mac_sample<true>(mac, q, u, G);
        const float wt = (stage == 0 || stage == 3) ? 1.0f : 2.0f;
        const float hh = stage < 2 ? h : dt;
        // derivative of the columns at this stage, their sums and the next
        // stage's point
        float d1[3];
        f2 d2[3];
#pragma unroll
        for (int r = 0; r < 3; r++) {
            d1[r] = dot3(G[r][0], s1[0], G[r][1], s1[1], G[r][2], s1[2]);
            if (NC == 3) d2[r] = dot3(both(G[r][0]), s2[0], both(G[r][1]), s2[1], both(G[r][2]), s2[2]);
        }
#pragma unroll
        for (int c = 0; c < 3; c++) {
            su[c] = __fmaf_rn(wt, u[c], su[c]);
            q[c] = __fmaf_rn(hh, u[c], psi[c]);
            S1[c] = __fmaf_rn(wt, d1[c], S1[c]);
            s1[c] = __fmaf_rn(hh, d1[c], C[L][c]);
            if (NC == 3) {
                S2[c] = fma2(both(wt), d2[c], S2[c]);
                s2[c] = fma2(both(hh), d2[c], C2[c]);
            }
        }
    }
    const float w6 = dt * 1.0f / 6.0f;
#pragma unroll
    for (int c = 0; c < 3; c++) {
        psi[c] = __fmaf_rn(w6, su[c], psi[c]);
        if (NC == 3) {
            const f2 t = fma2(both(w6), S2[c], C2[c]);
            C[0][c] = lo(t);
            C[NC - 2][c] = hi(t);
        }
        C[L][c] = __fmaf_rn(w6, S1[c], C[L][c]);
    }
}

// products rounded on their own: contracted into a sum that follows (an epsilon
// point), they would round otherwise where dx is no power of two
EDGE_D void cell_pos(int i, int j, int k, float dx, float X[3]) {
    X[0] = __fmul_rn((float)i + 0.5f, dx);
    X[1] = __fmul_rn((float)j + 0.5f, dx);
    X[2] = __fmul_rn((float)k + 0.5f, dx);
}
EDGE_D void face_pos(int axis, int i, int j, int k, float dx, float X[3]) {
    X[0] = __fmul_rn((float)i + (axis == 0 ? 0.0f : 0.5f), dx);
    X[1] = __fmul_rn((float)j + (axis == 1 ? 0.0f : 0.5f), dx);
    X[2] = __fmul_rn((float)k + (axis == 2 ? 0.0f : 0.5f), dx);
}

// Decompose a linear face index over the three face grids (x faces first).
struct FaceIdx {
    int axis, i, j, k, e;
};
EDGE_D FaceIdx face_decompose(long long t, int nx, int ny, int nz) {
    FaceIdx f;
    long long nfx = (long long)(nx + 1) * ny * nz, nfy = (long long)nx * (ny + 1) * nz;
    int n1, n2;
    if (t < nfx) { f.axis = 0; n1 = ny; n2 = nz; }
    else if (t < nfx + nfy) { f.axis = 1; t -= nfx; n1 = ny + 1; n2 = nz; }
    else { f.axis = 2; t -= nfx + nfy; n1 = ny; n2 = nz + 1; }
    // within one face grid the index fits 32 bits (f.e is an int): unsigned
    // 32-bit division instead of the 64-bit one
    const unsigned u = (unsigned)t;
    f.e = (int)u;
    f.k = (int)(u % (unsigned)n2);
    const unsigned r = u / (unsigned)n2;
    f.j = (int)(r % (unsigned)n1);
    f.i = (int)(r / (unsigned)n1);
    return f;
}

EDGE_HD long long n_faces(int nx, int ny, int nz) {
    return (long long)(nx + 1) * ny * nz + (long long)nx * (ny + 1) * nz + (long long)nx * ny * (nz + 1);
}

struct Face3 {
    const float* p[3];
    // select with constant indices only: a run-time index into a kernel
    // parameter array makes the compiler copy the parameter to local memory
    EDGE_D const float* at(int a) const { return a == 0 ? p[0] : (a == 1 ? p[1] : p[2]); }
};
struct Face3W {
    float* p[3];
    EDGE_D float* at(int a) const { return a == 0 ? p[0] : (a == 1 ? p[1] : p[2]); }
};

// ---------------------------------------------------------------------------
// Seven-point stencils over the three face grids (blockIdx.y: the component),
// neighbours clamped to the grid.  A thread takes one (j, k) of `chunk`
// consecutive i's: one division for all of them, and the i neighbours stay in
// registers, five loads a face instead of seven.  Bound by memory.  256x128x128,
// one face per thread and so: clamp 76 -> 43 us, viscous force 83 -> 35 us.
// f(axis, e, centre, low and high neighbour of x, of y, of z).
// ---------------------------------------------------------------------------
struct Star {
    int nx, ny, nz, chunk;
};
template <class F>
EDGE_D void face_star(const Star& g, const Face3& field, F f) {
    const int axis = blockIdx.y;
    const int n0 = g.nx + (axis == 0), n1 = g.ny + (axis == 1), n2 = g.nz + (axis == 2), plane = n1 * n2;
    const float* __restrict__ a = field.at(axis);
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x, c = t / (unsigned)plane;
    const int m = (int)(t - c * (unsigned)plane), i0 = (int)c * g.chunk, i1 = min(i0 + g.chunk, n0);
    if (i0 >= n0) return;
    const unsigned j = (unsigned)m / (unsigned)n2, k = (unsigned)m - j * (unsigned)n2;
    const int jl = j > 0 ? -n2 : 0, jh = (int)j < n1 - 1 ? n2 : 0, kl = k > 0 ? -1 : 0, kh = (int)k < n2 - 1;
    int e = i0 * plane + m;
    float lo = __ldg(a + (i0 > 0 ? e - plane : e)), at = __ldg(a + e);
#pragma unroll 4
    for (int i = i0; i < i1; i++, e += plane) {
        const float hi = i < n0 - 1 ? __ldg(a + e + plane) : at;
        f(axis, e, at, lo, hi, __ldg(a + e + jl), __ldg(a + e + jh), __ldg(a + e + kl), __ldg(a + e + kh));
        lo = at;
        at = hi;
    }
}
// up to eight faces a thread while that leaves a full wave of threads
static inline Star make_star(int nx, int ny, int nz) {
    const long long n = n_faces(nx, ny, nz) / (148LL * 2048);
    return Star{nx, ny, nz, (int)(n < 1 ? 1 : (n > 8 ? 8 : n))};
}
static inline dim3 star_grid(const Star& s, int block) {
    long long most = 0;
    for (int a = 0; a < 3; a++) {
        const long long n0 = s.nx + (a == 0), n1 = s.ny + (a == 1), n2 = s.nz + (a == 2);
        const long long n = (n0 + s.chunk - 1) / s.chunk * n1 * n2;
        if (n > most) most = n;
    }
    return dim3((unsigned)((most + block - 1) / block), 3);
}

}  // namespace edge
