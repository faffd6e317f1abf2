// hex27_tile.cuh — sum-factorised Hex27 stages on tiles of 32 elements.
//
// Mapping: a block of nine warps holds a tile of 32 elements, lane = element, warp = line of
// the 3×3×3 node and quadrature grids. Every 1-D contraction runs along the line a thread
// holds in registers; the lines turn twice between nodes and points through shared memory
// (word [field][line][lane]: conflict-free, no idle lanes). Since a warp's line index is uniform
// and the position along the line is unrolled, every basis coefficient is a compile-time constant
// and the middle point's zeros fold away — the nine-lanes-per-element stages of hex27.cuh
// read them from constant memory, leave five lanes idle and issue a warp instruction for three
// elements where this issues nine for 32.
//
// Roles of warp w, with a = w % 3, b = w / 3:
//   gather, scatter: node line (·, j = a, k = b)        exchanges within the three warps of one b
//   middle         : line (qx = a, ·, k = b)            exchanges within the three warps of one a
//   quadrature     : line (qx = a, qy = b, ·), points q = a + 3b + 9qz
// Each exchange is ordered by a named barrier of the 96 threads it concerns. Between the
// gradient and the transposed contraction of a tile the caller puts a barrier of the whole block
// (both write the buffers that the other reads, in other groups of warps).
#pragma once
#include <type_traits>
#include "common.cuh"

namespace femb {

constexpr int HT_E = 32;                 // elements per tile
constexpr int HT_THREADS = 9 * HT_E;
// words per tile of the two exchange buffers: 18 fields × 9 lines and 27 fields × 9 lines
constexpr int HT_S1 = 18 * 9 * HT_E, HT_S2 = 27 * 9 * HT_E;

// 1-D quadratic Lagrange basis on (−1, 0, 1) at the 3-point Gauss rule ±√(3/5), 0
// (Hex27: src/elements/shape_functions.jl:404-446, Gauss rule integration_points.jl:321).
constexpr double HT_GA = 0.774596669241483377035853079956479922;
FEMB_HD constexpr double ht_x(int q) { return q == 0 ? -HT_GA : (q == 1 ? 0.0 : HT_GA); }
FEMB_HD constexpr double ht_w(int q) { return q == 1 ? 8.0 / 9.0 : 5.0 / 9.0; }
FEMB_HD constexpr double ht_L(int q, int i) {
    return i == 0 ? ht_x(q) * (ht_x(q) - 1.0) * 0.5 : (i == 1 ? 1.0 - ht_x(q) * ht_x(q) : ht_x(q) * (ht_x(q) + 1.0) * 0.5);
}
FEMB_HD constexpr double ht_D(int q, int i) { return i == 0 ? ht_x(q) - 0.5 : (i == 1 ? -2.0 * ht_x(q) : ht_x(q) + 0.5); }
// coordinate and weight at a warp-uniform index
template <class T> FEMB_D T ht_xr(int q) { return q == 0 ? (T)-HT_GA : (q == 1 ? T(0) : (T)HT_GA); }
template <class T> FEMB_D T ht_wr(int q) { return q == 1 ? (T)(8.0 / 9.0) : (T)(5.0 / 9.0); }

// Contractions of one line with compile-time coefficients. Along a line the basis sums to one and
// its derivatives to zero, so values and derivatives at the points are formed from the end
// nodes' differences to the middle one (a constant line has exactly no derivative, and the two
// share the differences), and the derivative's transpose gives the middle node what the ends lack.
template <class T> FEMB_D void ht_val(const T (&x)[3], T (&o)[3]) {   // o[q] = Σ_i L_i(q) x_i
    const T d0 = x[0] - x[1], d2 = x[2] - x[1];
    o[0] = (T)ht_L(0, 0) * d0 + ((T)ht_L(0, 2) * d2 + x[1]);
    o[1] = x[1];
    o[2] = (T)ht_L(2, 2) * d2 + ((T)ht_L(2, 0) * d0 + x[1]);
}
template <class T> FEMB_D void ht_der(const T (&x)[3], T (&o)[3]) {   // o[q] = Σ_i L'_i(q) x_i
    const T d0 = x[0] - x[1], d2 = x[2] - x[1];
    o[0] = (T)ht_D(0, 0) * d0 + (T)ht_D(0, 2) * d2;
    o[1] = T(0.5) * (d2 - d0);
    o[2] = (T)ht_D(2, 0) * d0 + (T)ht_D(2, 2) * d2;
}
template <class T> FEMB_D void ht_val_t(const T (&f)[3], T (&o)[3]) {   // o[i] = Σ_q L_i(q) f_q
    o[0] = (T)ht_L(0, 0) * f[0] + (T)ht_L(2, 0) * f[2];
    o[1] = (T)ht_L(0, 1) * (f[0] + f[2]) + f[1];
    o[2] = (T)ht_L(0, 2) * f[0] + (T)ht_L(2, 2) * f[2];
}
template <class T> FEMB_D void ht_der_t(const T (&f)[3], T (&o)[3]) {   // o[i] = Σ_q L'_i(q) f_q
    o[0] = (T)ht_D(0, 0) * f[0] + ((T)ht_D(2, 0) * f[2] - T(0.5) * f[1]);
    o[2] = (T)ht_D(2, 2) * f[2] + ((T)ht_D(0, 2) * f[0] + T(0.5) * f[1]);
    o[1] = -o[0] - o[2];
}

// The block's warp index in a form the compiler knows to be uniform in the warp: everything
// derived from it (table picks, barrier ids, shared offsets) then stays off the vector pipes.
FEMB_D int ht_warp() { return __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0); }

// Element i of a nodal array by its byte offset: a 32-bit offset from a uniform base costs no
// 64-bit arithmetic per access. Nodal FP32 (FP64) arrays of 2^30 (2^29) nodes do not fit the
// device beside the rest of a state.
template <class T> FEMB_D const T* ht_at(const T* base, uint32_t off) {
    return reinterpret_cast<const T*>(reinterpret_cast<const char*>(base) + off);
}
template <class T> FEMB_D T* ht_at(T* base, uint32_t off) { return reinterpret_cast<T*>(reinterpret_cast<char*>(base) + off); }

// a point's ten entries, two at a time where the array's alignment allows it
template <class T, class TG>
FEMB_D void load10(const TG* p, bool vec, T (&J)[10]) {
    using T2 = std::conditional_t<sizeof(TG) == 8, double2, float2>;
    if (vec) {
#pragma unroll
        for (int r = 0; r < 5; ++r) {
            const T2 x = __ldg(reinterpret_cast<const T2*>(p) + r);
            J[2 * r] = (T)x.x; J[2 * r + 1] = (T)x.y;
        }
    } else {
#pragma unroll
        for (int r = 0; r < 10; ++r) J[r] = (T)ld(p + r);
    }
}

// barrier of the three warps that share b (exchanges along the first direction) or a
FEMB_D void ht_bar_b(int b) { asm volatile("bar.sync %0, 96;" ::"r"(1 + b) : "memory"); }
FEMB_D void ht_bar_a(int a) { asm volatile("bar.sync %0, 96;" ::"r"(4 + a) : "memory"); }

// Reference gradients of NC components at the three points of the owned ζ-line:
// v[c][i] on the owned node line → g[c][d][qz]; d = ξ, η, ζ.
template <class T, int NC>
FEMB_D void ht_gradient(const T (&v)[NC][3], T* S1, T* S2, int a, int b, int lane, T (&g)[NC][3][3]) {
    {
        T* o = S1 + (a + 3 * b) * HT_E + lane;
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            T l[3], d[3];
            ht_val(v[c], l);
            ht_der(v[c], d);
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                o[(q * 2 * NC + 2 * c) * 9 * HT_E] = l[q];
                o[(q * 2 * NC + 2 * c + 1) * 9 * HT_E] = d[q];
            }
        }
    }
    ht_bar_b(b);
    {
        const T* in = S1 + (a * 2 * NC * 9 + 3 * b) * HT_E + lane;
        T* o = S2 + (a + 3 * b) * HT_E + lane;
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            T x0[3], x1[3];
#pragma unroll
            for (int j = 0; j < 3; ++j) { x0[j] = in[(2 * c * 9 + j) * HT_E]; x1[j] = in[((2 * c + 1) * 9 + j) * HT_E]; }
            T y0[3], y1[3], y2[3];
            ht_val(x1, y0);
            ht_der(x0, y1);
            ht_val(x0, y2);
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                o[((q * NC + c) * 3 + 0) * 9 * HT_E] = y0[q];
                o[((q * NC + c) * 3 + 1) * 9 * HT_E] = y1[q];
                o[((q * NC + c) * 3 + 2) * 9 * HT_E] = y2[q];
            }
        }
    }
    ht_bar_a(a);
    {
        const T* in = S2 + (b * 3 * NC * 9 + a) * HT_E + lane;
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            T y[3][3];
#pragma unroll
            for (int f = 0; f < 3; ++f)
#pragma unroll
                for (int k = 0; k < 3; ++k) y[f][k] = in[((c * 3 + f) * 9 + 3 * k) * HT_E];
            ht_val(y[0], g[c][0]);
            ht_val(y[1], g[c][1]);
            ht_der(y[2], g[c][2]);
        }
    }
}

// First half of the transposed contraction: fluxes F[c][d][qz] and value densities
// val(c, qz) (integrated against N, not its gradient) of the owned point line into S2. The
// value shares the ζ flux's ξ and η factors, so it adds no field.
template <class T, int NC, class V>
FEMB_D void ht_scatter_z(const T (&F)[NC][3][3], V val, T* S2, int a, int b, int lane) {
    T* o = S2 + (a + 3 * b) * HT_E + lane;
#pragma unroll
    for (int c = 0; c < NC; ++c) {
        const T w[3] = {val(c, 0), val(c, 1), val(c, 2)};
        T z0[3], z1[3], z2[3], zw[3];
        ht_val_t(F[c][0], z0);
        ht_val_t(F[c][1], z1);
        ht_der_t(F[c][2], z2);
        ht_val_t(w, zw);
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            o[((i * NC + c) * 3 + 0) * 9 * HT_E] = z0[i];
            o[((i * NC + c) * 3 + 1) * 9 * HT_E] = z1[i];
            o[((i * NC + c) * 3 + 2) * 9 * HT_E] = z2[i] + zw[i];
        }
    }
}
// Second half, after a barrier over the warps of one a (ht_bar_a or wider): the nodal
// residual R[c][i] on the owned node line.
template <class T, int NC>
FEMB_D void ht_scatter_yx(T* S1, const T* S2, int a, int b, int lane, T (&R)[NC][3]) {
    {
        const T* in = S2 + (b * 3 * NC * 9 + a) * HT_E + lane;
        T* o = S1 + (a + 3 * b) * HT_E + lane;
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            T z[3][3];
#pragma unroll
            for (int f = 0; f < 3; ++f)
#pragma unroll
                for (int q = 0; q < 3; ++q) z[f][q] = in[((c * 3 + f) * 9 + 3 * q) * HT_E];
            T u0[3], u1[3], u2[3];
            ht_val_t(z[0], u0);
            ht_der_t(z[1], u1);
            ht_val_t(z[2], u2);
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                o[(i * 2 * NC + 2 * c) * 9 * HT_E] = u0[i];
                o[(i * 2 * NC + 2 * c + 1) * 9 * HT_E] = u1[i] + u2[i];
            }
        }
    }
    ht_bar_b(b);
    {
        const T* in = S1 + (a * 2 * NC * 9 + 3 * b) * HT_E + lane;
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            T u0[3], u1[3];
#pragma unroll
            for (int q = 0; q < 3; ++q) { u0[q] = in[(2 * c * 9 + q) * HT_E]; u1[q] = in[((2 * c + 1) * 9 + q) * HT_E]; }
            T r0[3], r1[3];
            ht_der_t(u0, r0);
            ht_val_t(u1, r1);
#pragma unroll
            for (int i = 0; i < 3; ++i) R[c][i] = r0[i] + r1[i];
        }
    }
}

}  // namespace femb
