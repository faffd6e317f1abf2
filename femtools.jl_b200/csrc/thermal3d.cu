// thermal3d.cu — sum-factorised Hex27 heat-diffusion residual and Jacobian diagnostics
// (heat_diffusion/assembly/residual.jl:30-87).
//
// Mapping of hex27.cuh: a warp holds three elements, nine line threads each; the four nodal
// fields (T with its gradient, P, T0 and the source by value) go to the 27 points through
// 1-D contractions, and one transposed contraction carries the rate term and the diffusive
// flux back: the value and the ζ flux share their ξ and η factors, so three blocks cross the
// warp instead of four. The thread-per-element version this replaces evaluated every point as
// 27-node sums with the tables in constant memory and 27-entry local arrays: at 27 × 35 × 22
// cells (FP64, 200 iterations with 5 Jacobian assemblies) the solve went from 81.7 ms to 8.6 ms,
// a coupled solve at 32³ (200 iterations) from 146 ms to 59 ms (5.9 and 30 ms by now, with the residual on
// tiles, fewer launches and dependent ones). What bounds it is the latency
// of the gathers and of the stage exchanges (geometry, 2 160 B a cell, comes from L2). Where no Jacobian
// and no element group is asked for, the residual is thermal3d_tile_kernel's.
//
// The Jacobian diagnostics push the 27 unit vectors through the same transposed contraction:
// column b is the residual's derivative
//   J_ib = Σ_q dΩ [(−1 + δ(s + Φ)) N_b N_i − δ k N_b ∇N_i·∇T − (Δt/ρCp) k ∇N_i·∇N_b],
// δ = (Δt/ρCp)·α ρ0/ρ (the density's temperature dependence), in closed form per point.
#include <algorithm>
#include "hex27.cuh"
#include "hex27_tile.cuh"
#include "kernels.cuh"

namespace femb {
namespace {

constexpr int TH_THREADS = 128;
// five x-stage blocks (T twice, P, T0, source) and six y-stage blocks; the slot stride is
// that of H27Fp64Banked modulo the bank count (539 ≡ 347 ≡ 11 mod 16)
template <class T> struct ThermalStage {
    using LY = H27Layout<T>;
    static constexpr int SLOT = sizeof(T) == 8 ? 347 : 300;
};
static_assert(5 * H27Fp64Banked::K1 + 6 * H27Fp64Banked::K2 <= ThermalStage<double>::SLOT, "thermal stage");
static_assert(5 * H27Compact::K1 + 6 * H27Compact::K2 <= ThermalStage<float>::SLOT, "thermal stage");

template <class T> FEMB_D T sel3(const T (&x)[3], int i) { return i == 0 ? x[0] : (i == 1 ? x[1] : x[2]); }

// Nodal residual on the owned x-line from the value density V and the reference-frame
// fluxes F[d] at the owned z-line: R(a) = Σ_q N_a V + Σ_d ∂_d N_a F_d.
template <class T, class LY>
FEMB_D void scalar_transpose(const Tab1D<T>& t, const T F[3][3], const T V[3], T* E, int m1, int m2, T R[3]) {
#pragma unroll
    for (int iz = 0; iz < 3; ++iz) {
        E[LY::l2(m1, m2, iz)] = t.B[0][iz] * F[0][0] + t.B[1][iz] * F[0][1] + t.B[2][iz] * F[0][2];
        E[LY::K2 + LY::l2(m1, m2, iz)] = t.B[0][iz] * F[1][0] + t.B[1][iz] * F[1][1] + t.B[2][iz] * F[1][2];
        E[2 * LY::K2 + LY::l2(m1, m2, iz)] = (t.Dd[0][iz] * F[2][0] + t.Dd[1][iz] * F[2][1] + t.Dd[2][iz] * F[2][2]) +
                                            (t.B[0][iz] * V[0] + t.B[1][iz] * V[1] + t.B[2][iz] * V[2]);
    }
    __syncwarp();
    T* E1 = E + 3 * LY::K2;
    T A[3], Bv[3], C[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        A[q] = E[LY::l2(m1, q, m2)];
        Bv[q] = E[LY::K2 + LY::l2(m1, q, m2)];
        C[q] = E[2 * LY::K2 + LY::l2(m1, q, m2)];
    }
#pragma unroll
    for (int iy = 0; iy < 3; ++iy) {
        E1[LY::l1(m1, iy, m2)] = t.B[0][iy] * A[0] + t.B[1][iy] * A[1] + t.B[2][iy] * A[2];
        E1[LY::K1 + LY::l1(m1, iy, m2)] = (t.Dd[0][iy] * Bv[0] + t.Dd[1][iy] * Bv[1] + t.Dd[2][iy] * Bv[2]) +
                                         (t.B[0][iy] * C[0] + t.B[1][iy] * C[1] + t.B[2][iy] * C[2]);
    }
    __syncwarp();
    T UA[3], UB[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        UA[q] = E1[LY::l1(q, m1, m2)];
        UB[q] = E1[LY::K1 + LY::l1(q, m1, m2)];
    }
#pragma unroll
    for (int ix = 0; ix < 3; ++ix)
        R[ix] = (t.Dd[0][ix] * UA[0] + t.Dd[1][ix] * UA[1] + t.Dd[2][ix] * UA[2]) +
                (t.B[0][ix] * UB[0] + t.B[1][ix] * UB[1] + t.B[2][ix] * UB[2]);
    __syncwarp();
}

template <class T, class TG, bool JAC>
__global__ void __launch_bounds__(TH_THREADS, JAC ? 3 : 4) thermal3d_kernel(const ThermalArgs<T, TG> a) {
    using LY = typename ThermalStage<T>::LY;
    constexpr int SLOT = ThermalStage<T>::SLOT;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int wpb = TH_THREADS / 32;
    const bool lane_ok = lane < 27;
    // lanes 27..31 carry no element; they work in a private scratch slot (3)
    const int s = lane_ok ? lane / 9 : 3, m = lane_ok ? lane % 9 : LY::IDLE_M, m1 = m % 3, m2 = m / 3;
    T* E = reinterpret_cast<T*>(smem_raw) + ((size_t)warp * 4 + s) * SLOT;
    int* PH = reinterpret_cast<int*>(reinterpret_cast<T*>(smem_raw) + (size_t)wpb * 4 * SLOT) + (warp * 4 + s) * 28;
    Tab1D<T> tb; tb.load();
    // lane-dependent table entries, read once (divergent constant reads serialise)
    int tn_own[3];
    T sumN[3], b1[3], b2[3], d1[3], d2[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        tn_own[i] = c_tab.tn3[tidx(i, m1, m2)];
        sumN[i] = (T)c_tab.sumN3[tidx(m1, m2, i)];
        b1[i] = (T)c_tab.B[m1][i]; b2[i] = (T)c_tab.B[m2][i];
        d1[i] = (T)c_tab.Dd[m1][i]; d2[i] = (T)c_tab.Dd[m2][i];
    }
    const int64_t n = a.group ? a.ngroup : a.nels;
    const int64_t stride = (int64_t)gridDim.x * wpb * 3;
    bool waited = false;
    for (int64_t base = ((int64_t)blockIdx.x * wpb + warp) * 3; base < n; base += stride) {
        const int64_t w = base + (lane_ok ? s : 0);
        const bool act = lane_ok && w < n;
        const int64_t e = !act ? 0 : a.group ? (int64_t)__ldg(a.group + w) - 1 : w;
        int node[3];
        T Tl[3], Pl[3], T0l[3], Sl[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) node[i] = act ? __ldg(a.el2n + 27 * e + tn_own[i]) - 1 : 0;
        if (!waited) { pdl_enter(); waited = true; }
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            Tl[i] = act ? ld_coherent(a.Tn + node[i]) : T(0);
            T0l[i] = act ? ld(a.T0 + node[i]) : T(0);
            Pl[i] = act && a.P ? ld(a.P + node[i]) : T(0);
            Sl[i] = act && a.src ? ld(a.src + node[i]) : T(0);
        }
        // ---- phases: one for the element (the usual case) or one per node ----
        int p0 = 0;
        bool uniform = true;
        if (a.ph && a.ph_layout == FEMB200_PHASE_CELL) {
            p0 = act ? __ldg(a.ph + e) - 1 : 0;
        } else if (a.ph) {
#pragma unroll
            for (int i = 0; i < 3; ++i)
                PH[tidx(i, m1, m2)] = act ? phase_of(a.ph, a.ph_layout, (int64_t)node[i] + 1, tn_own[i], e, 27) : 0;
            __syncwarp();
            p0 = PH[0];
            const bool same = PH[tidx(0, m1, m2)] == p0 && PH[tidx(1, m1, m2)] == p0 && PH[tidx(2, m1, m2)] == p0;
            const unsigned bal = __ballot_sync(0xffffffffu, same || !lane_ok);
            uniform = !lane_ok || ((bal >> (s * 9)) & 0x1ffu) == 0x1ffu;
        }

        // ---- fields at the owned points ----
        T Tq[3], gr[3][3], Pq[3], T0q[3], Sq[3];   // gr[d][qz]
        {
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                const int o = LY::l1(q, m1, m2);
                E[o] = tb.B[q][0] * Tl[0] + tb.B[q][1] * Tl[1] + tb.B[q][2] * Tl[2];
                E[LY::K1 + o] = tb.Dd[q][0] * Tl[0] + tb.Dd[q][1] * Tl[1] + tb.Dd[q][2] * Tl[2];
                E[2 * LY::K1 + o] = tb.B[q][0] * T0l[0] + tb.B[q][1] * T0l[1] + tb.B[q][2] * T0l[2];
                E[3 * LY::K1 + o] = tb.B[q][0] * Pl[0] + tb.B[q][1] * Pl[1] + tb.B[q][2] * Pl[2];
                E[4 * LY::K1 + o] = tb.B[q][0] * Sl[0] + tb.B[q][1] * Sl[1] + tb.B[q][2] * Sl[2];
            }
            __syncwarp();
            T* E1 = E + 5 * LY::K1;
            T X[5][3];
#pragma unroll
            for (int f = 0; f < 5; ++f)
#pragma unroll
                for (int j = 0; j < 3; ++j) X[f][j] = E[f * LY::K1 + LY::l1(m1, j, m2)];
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                const int o = LY::l2(m1, q, m2);
                E1[o] = tb.B[q][0] * X[1][0] + tb.B[q][1] * X[1][1] + tb.B[q][2] * X[1][2];
                E1[LY::K2 + o] = tb.Dd[q][0] * X[0][0] + tb.Dd[q][1] * X[0][1] + tb.Dd[q][2] * X[0][2];
#pragma unroll
                for (int f = 0; f < 4; ++f) {
                    const T* Xf = X[f == 0 ? 0 : f + 1];
                    E1[(2 + f) * LY::K2 + o] = tb.B[q][0] * Xf[0] + tb.B[q][1] * Xf[1] + tb.B[q][2] * Xf[2];
                }
            }
            __syncwarp();
            T Y[6][3];
#pragma unroll
            for (int f = 0; f < 6; ++f)
#pragma unroll
                for (int k = 0; k < 3; ++k) Y[f][k] = E1[f * LY::K2 + LY::l2(m1, m2, k)];
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                gr[0][q] = tb.B[q][0] * Y[0][0] + tb.B[q][1] * Y[0][1] + tb.B[q][2] * Y[0][2];
                gr[1][q] = tb.B[q][0] * Y[1][0] + tb.B[q][1] * Y[1][1] + tb.B[q][2] * Y[1][2];
                gr[2][q] = tb.Dd[q][0] * Y[2][0] + tb.Dd[q][1] * Y[2][1] + tb.Dd[q][2] * Y[2][2];
                Tq[q] = tb.B[q][0] * Y[2][0] + tb.B[q][1] * Y[2][1] + tb.B[q][2] * Y[2][2];
                T0q[q] = tb.B[q][0] * Y[3][0] + tb.B[q][1] * Y[3][1] + tb.B[q][2] * Y[3][2];
                Pq[q] = tb.B[q][0] * Y[4][0] + tb.B[q][1] * Y[4][1] + tb.B[q][2] * Y[4][2];
                Sq[q] = tb.B[q][0] * Y[5][0] + tb.B[q][1] * Y[5][1] + tb.B[q][2] * Y[5][2];
            }
            __syncwarp();
        }

        // ---- rate and diffusive flux at the points ----
        T V[3], F[3][3];                     // F[d][qz]
        T c1[3], h2[3][3], M[3][6];          // JAC: value, N_b·flux and gradient coefficients
#pragma unroll
        for (int qz = 0; qz < 3; ++qz) {
            const int q = tidx(m1, m2, qz);
            T kq, aq, bq, rq, cq;
            if (uniform) {
                kq = (T)c_tmat.k[p0] * sumN[qz]; aq = (T)c_tmat.alpha[p0] * sumN[qz]; bq = (T)c_tmat.beta[p0] * sumN[qz];
                rq = (T)c_tmat.rho0[p0] * sumN[qz]; cq = (T)c_tmat.Cp[p0] * sumN[qz];
            } else {
                kq = aq = bq = rq = cq = T(0);
                for (int k = 0; k < 3; ++k)
                    for (int j = 0; j < 3; ++j)
                        for (int i = 0; i < 3; ++i) {
                            const T N = sel3(b1, i) * sel3(b2, j) * tb.B[qz][k];
                            const int p = PH[tidx(i, j, k)];
                            kq += N * (T)c_tmat.k[p]; aq += N * (T)c_tmat.alpha[p]; bq += N * (T)c_tmat.beta[p];
                            rq += N * (T)c_tmat.rho0[p]; cq += N * (T)c_tmat.Cp[p];
                        }
            }
            const TG* G = a.geo + (e * 27 + q) * 10;
            T Ji[9];
#pragma unroll
            for (int r = 0; r < 9; ++r) Ji[r] = act ? (T)ld(G + r) : T(0);
            const T dO = act ? (T)ld(G + 9) : T(0);
            const T Phi = act && a.src_ip ? ld_coherent(a.src_ip + e * 27 + q) : T(0);
            const T rho = rq * (T(1) - aq * (Tq[qz] - a.Tref) + bq * Pq[qz]);
            const T dtrc = a.dt / (rho * cq);
            T gT[3];
#pragma unroll
            for (int k = 0; k < 3; ++k) gT[k] = gr[0][qz] * Ji[3 * k] + gr[1][qz] * Ji[1 + 3 * k] + gr[2][qz] * Ji[2 + 3 * k];
            V[qz] = (T0q[qz] - Tq[qz] + dtrc * Sq[qz] + dtrc * Phi) * dO;
            const T w3 = dtrc * kq * dO;
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const T hd = Ji[d] * gT[0] + Ji[d + 3] * gT[1] + Ji[d + 6] * gT[2];
                F[d][qz] = -w3 * hd;
                if (JAC) h2[qz][d] = hd;
            }
            if (JAC) {
                const T cfac = dtrc * aq * rq / rho;
                c1[qz] = (cfac * (Sq[qz] + Phi) - T(1)) * dO;
#pragma unroll
                for (int d = 0; d < 3; ++d) h2[qz][d] *= -cfac * kq * dO;
                int r = 0;
#pragma unroll
                for (int d = 0; d < 3; ++d)
#pragma unroll
                    for (int f = d; f < 3; ++f) M[qz][r++] = -w3 * (Ji[d] * Ji[f] + Ji[d + 3] * Ji[f + 3] + Ji[d + 6] * Ji[f + 6]);
            }
        }
        T R[3];
        scalar_transpose<T, LY>(tb, F, V, E, m1, m2, R);
        if (act) {
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                if (a.group) a.R[node[i]] += R[i];
                else atomic_add(a.R + node[i], R[i]);
            }
        }
        if constexpr (JAC) {
            T rows[3] = {T(0), T(0), T(0)}, diag[3] = {T(0), T(0), T(0)};
#pragma unroll 1
            for (int bk = 0; bk < 3; ++bk)
#pragma unroll 1
                for (int bj = 0; bj < 3; ++bj)
#pragma unroll 1
                    for (int bi = 0; bi < 3; ++bi) {
                        const T u1 = sel3(b1, bi), v1 = sel3(d1, bi), u2 = sel3(b2, bj), v2 = sel3(d2, bj);
#pragma unroll
                        for (int qz = 0; qz < 3; ++qz) {
                            const T u3 = tb.B[qz][bk], v3 = tb.Dd[qz][bk];
                            const T N = u1 * u2 * u3;
                            const T g0 = v1 * u2 * u3, g1 = u1 * v2 * u3, g2 = u1 * u2 * v3;
                            V[qz] = c1[qz] * N;
                            F[0][qz] = h2[qz][0] * N + M[qz][0] * g0 + M[qz][1] * g1 + M[qz][2] * g2;
                            F[1][qz] = h2[qz][1] * N + M[qz][1] * g0 + M[qz][3] * g1 + M[qz][4] * g2;
                            F[2][qz] = h2[qz][2] * N + M[qz][2] * g0 + M[qz][4] * g1 + M[qz][5] * g2;
                        }
                        T J[3];
                        scalar_transpose<T, LY>(tb, F, V, E, m1, m2, J);
                        const bool own = bj == m1 && bk == m2;
#pragma unroll
                        for (int i = 0; i < 3; ++i) {
                            rows[i] += fabs(J[i]);
                            if (own && i == bi) diag[i] = fabs(J[i]);
                        }
                    }
            if (act) {
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    if (a.group) {
                        a.dRdT[node[i]] += rows[i];
                        a.PC[node[i]] += diag[i];
                    } else {
                        atomic_add(a.dRdT + node[i], rows[i]);
                        atomic_add(a.PC + node[i], diag[i]);
                    }
                }
            }
        }
    }
    if (!waited) pdl_enter();
}

template <class T, class TG, bool JAC>
cudaError_t launch_t3(const ThermalArgs<T, TG>& a, int64_t n, int num_sms, cudaStream_t st, bool pdl) {
    constexpr int wpb = TH_THREADS / 32;
    const size_t smem = (size_t)wpb * 4 * ThermalStage<T>::SLOT * sizeof(T) + (size_t)wpb * 4 * 28 * sizeof(int);
    static_assert((size_t)wpb * 4 * ThermalStage<T>::SLOT * sizeof(T) + (size_t)wpb * 4 * 28 * sizeof(int) <= 48 * 1024,
                  "within the default shared-memory limit");
    const int64_t groups = (n + 2) / 3;
    const int64_t blocks = std::max<int64_t>(1, std::min<int64_t>((groups + wpb - 1) / wpb, (int64_t)num_sms * 16));
    return launch_pdl(pdl, thermal3d_kernel<T, TG, JAC>, dim3((unsigned)blocks), dim3(TH_THREADS), smem, st, a);
}

// The residual alone: tiles of 32 elements, lane = element, warp = line (hex27_tile.cuh). Bound by the
// latency of the gathers and the atomics and by the geometry, 2 160 B a cell in as many lines as lanes
// (34 us at 27×35×22 from a cold cache, 55 MB from DRAM; 50 us a sweep in a coupled solve at 32³).
// The geometry is read per point also where cells are affine: one J⁻¹ per cell is a quarter faster
// (4.6 against 5.9 ms for 200 iterations at 27×35×22; 6.5 with three elements to a warp), but the
// 27 points agree only to the rounding of the sums that formed them, and the solution at 32³ is then
// seven times further from the 64-bit one (4.5e-14 of T against 6e-15).
template <class T>
struct ThSmem {
    T S1[5 * 3 * 9 * HT_E], S2[6 * 3 * 9 * HT_E];
    T PT[5][MAXPH];   // k, α, β, ρ0, Cp
};
struct ThPhases {   // in the first exchange buffer once its fields are read
    int mask[9][HT_E];
    uint8_t ph[27][HT_E];
};
static_assert(sizeof(ThPhases) <= sizeof(ThSmem<float>::S1), "phases of a tile");

// VEC: the geometry is 16-byte aligned.
template <class T, class TG, bool VEC>
__global__ void __launch_bounds__(HT_THREADS, 2) thermal3d_tile_kernel(const ThermalArgs<T, TG> a) {
    extern __shared__ __align__(16) unsigned char th_smem[];
    ThSmem<T>& S = *reinterpret_cast<ThSmem<T>*>(th_smem);
    const int lane = threadIdx.x & 31, w = ht_warp(), la = w % 3, lb = w / 3;
    const int64_t e0 = (int64_t)blockIdx.x * HT_E;
    const int ne = (int)(a.nels - e0 < HT_E ? a.nels - e0 : HT_E);
    const bool act = lane < ne;
    const int64_t e = e0 + (act ? lane : ne - 1);   // lanes past the end repeat the last element
    int node[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) node[i] = __ldg(a.el2n + 27 * e + c_tab.tn3[i + 3 * w]) - 1;
    if (threadIdx.x < 5 * MAXPH) {
        const int f = threadIdx.x / MAXPH, p = threadIdx.x % MAXPH;
        S.PT[f][p] = (T)(f == 0 ? c_tmat.k[p] : f == 1 ? c_tmat.alpha[p] : f == 2 ? c_tmat.beta[p] : f == 3 ? c_tmat.rho0[p] : c_tmat.Cp[p]);
    }
    const bool nodal = a.ph && a.ph_layout != FEMB200_PHASE_CELL;
    int p0 = a.ph && !nodal ? __ldg(a.ph + e) - 1 : 0, phn[3] = {0, 0, 0};
    if (nodal) {
#pragma unroll
        for (int i = 0; i < 3; ++i) phn[i] = phase_of(a.ph, a.ph_layout, (int64_t)node[i] + 1, c_tab.tn3[i + 3 * w], e, 27);
    }
    pdl_enter();   // everything so far is constant over the iterations

    // ---- T with its gradient, T0, P and the source at the points ----
    T Tq[3], gr[3][3], T0q[3], Pq[3], Sq[3];   // gr[d][qz]
    {
        T* o = S.S1 + w * HT_E + lane;   // field f, point column q at [(5q + f)·9]
        auto values = [&](const T* x, int f) {
            const T v[3] = {ld_coherent(x + node[0]), ld_coherent(x + node[1]), ld_coherent(x + node[2])};
            T l[3];
            ht_val(v, l);
#pragma unroll
            for (int q = 0; q < 3; ++q) o[(5 * q + f) * 9 * HT_E] = l[q];
            if (f == 0) {
                ht_der(v, l);
#pragma unroll
                for (int q = 0; q < 3; ++q) o[(5 * q + 1) * 9 * HT_E] = l[q];
            }
        };
        values(a.Tn, 0);
        values(a.T0, 2);
        if (a.P) values(a.P, 3);
        if (a.src) values(a.src, 4);
    }
    ht_bar_b(lb);
    {
        const T* in = S.S1 + (la * 5 * 9 + 3 * lb) * HT_E + lane;
        T* o = S.S2 + w * HT_E + lane;   // fields L(T_x'), D(T), L(T), L(T0), L(P), L(S) of point row q at [(6q + f)·9]
        auto stage = [&](int f, int fo, bool der) {
            const T x[3] = {in[f * 9 * HT_E], in[(f * 9 + 1) * HT_E], in[(f * 9 + 2) * HT_E]};
            T l[3];
            ht_val(x, l);
#pragma unroll
            for (int q = 0; q < 3; ++q) o[(6 * q + fo) * 9 * HT_E] = l[q];
            if (der) {
                ht_der(x, l);
#pragma unroll
                for (int q = 0; q < 3; ++q) o[(6 * q + 1) * 9 * HT_E] = l[q];
            }
        };
        stage(1, 0, false);
        stage(0, 2, true);
        stage(2, 3, false);
        if (a.P) stage(3, 4, false);
        if (a.src) stage(4, 5, false);
    }
    ht_bar_a(la);
    {
        const T* in = S.S2 + (lb * 6 * 9 + la) * HT_E + lane;
        auto line = [&](int f, T (&x)[3]) {
#pragma unroll
            for (int k = 0; k < 3; ++k) x[k] = in[(f * 9 + 3 * k) * HT_E];
        };
        T x[3];
        line(0, x); ht_val(x, gr[0]);
        line(1, x); ht_val(x, gr[1]);
        line(2, x); ht_val(x, Tq); ht_der(x, gr[2]);
        line(3, x); ht_val(x, T0q);
#pragma unroll
        for (int q = 0; q < 3; ++q) Pq[q] = Sq[q] = T(0);
        if (a.P) { line(4, x); ht_val(x, Pq); }
        if (a.src) { line(5, x); ht_val(x, Sq); }
    }
    __syncthreads();   // the buffers and PT
    bool uniform = true;
    const ThPhases& PH = *reinterpret_cast<const ThPhases*>(S.S1);
    if (nodal) {
        ThPhases& Pw = *reinterpret_cast<ThPhases*>(S.S1);
        int mask = 0;
#pragma unroll
        for (int i = 0; i < 3; ++i) { Pw.ph[i + 3 * w][lane] = (uint8_t)phn[i]; mask |= 1 << phn[i]; }
        Pw.mask[w][lane] = mask;
        __syncthreads();
#pragma unroll
        for (int l = 0; l < 9; ++l) mask |= PH.mask[l][lane];
        uniform = (mask & (mask - 1)) == 0;
        p0 = __ffs(mask) - 1;
    }

    // ---- rate and diffusive flux at the points ----
    T V[3], F[3][3];   // F[d][qz]
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        T kq, aq, bq, rq, cq;
        if (uniform) {
            kq = S.PT[0][p0]; aq = S.PT[1][p0]; bq = S.PT[2][p0]; rq = S.PT[3][p0]; cq = S.PT[4][p0];
        } else {
            kq = aq = bq = rq = cq = T(0);
#pragma unroll 1
            for (int t = 0; t < 27; ++t) {
                const T N = (T)c_tab.N3[w + 9 * q][c_tab.tn3[t]];
                const int p = PH.ph[t][lane];
                kq += N * S.PT[0][p]; aq += N * S.PT[1][p]; bq += N * S.PT[2][p]; rq += N * S.PT[3][p]; cq += N * S.PT[4][p];
            }
        }
        T J[10];
        load10(a.geo + (e * 27 + w + 9 * q) * 10, VEC, J);
        const T dO = J[9];
        const T Phi = a.src_ip ? ld_coherent(a.src_ip + e * 27 + w + 9 * q) : T(0);
        const T rho = rq * (T(1) - aq * (Tq[q] - a.Tref) + bq * Pq[q]);
        const T dtrc = a.dt / (rho * cq);
        T gT[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) gT[k] = gr[0][q] * J[3 * k] + gr[1][q] * J[1 + 3 * k] + gr[2][q] * J[2 + 3 * k];
        V[q] = (T0q[q] - Tq[q] + dtrc * (Sq[q] + Phi)) * dO;
        const T w3 = dtrc * kq * dO;
#pragma unroll
        for (int d = 0; d < 3; ++d) F[d][q] = -w3 * (J[d] * gT[0] + J[d + 3] * gT[1] + J[d + 6] * gT[2]);
    }
    if (nodal) __syncthreads();   // the phases are read: the contraction takes their place
    {
        T Fz[1][3][3];
#pragma unroll
        for (int d = 0; d < 3; ++d)
#pragma unroll
            for (int q = 0; q < 3; ++q) Fz[0][d][q] = F[d][q];
        ht_scatter_z<T, 1>(Fz, [&](int, int q) { return V[q]; }, S.S2, la, lb, lane);
    }
    ht_bar_a(la);
    T R[1][3];
    ht_scatter_yx<T, 1>(S.S1, S.S2, la, lb, lane, R);
    // the next lane's ξ = −1 node, when it is this lane's ξ = +1 node, is added here (stokes3d.cu)
    const int n0n = __shfl_down_sync(0xffffffffu, node[0], 1);
    const bool fold = lane + 1 < ne && n0n == node[2];
    const bool folded = __shfl_up_sync(0xffffffffu, (int)fold, 1) && lane > 0;
    const T r0n = __shfl_down_sync(0xffffffffu, R[0][0], 1);
    if (fold) R[0][2] += r0n;
    if (act) {
        if (!folded) atomic_add(a.R + node[0], R[0][0]);
        atomic_add(a.R + node[1], R[0][1]);
        atomic_add(a.R + node[2], R[0][2]);
    }
}

template <class T, class TG>
cudaError_t launch_t3_tiles(const ThermalArgs<T, TG>& a, cudaStream_t st, bool pdl) {
    const bool vec = (reinterpret_cast<uintptr_t>(a.geo) & 15u) == 0;
    const auto fn = vec ? thermal3d_tile_kernel<T, TG, true> : thermal3d_tile_kernel<T, TG, false>;
    const cudaError_t err = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(ThSmem<T>));
    if (err != cudaSuccess) return err;
    return launch_pdl(pdl, fn, dim3((unsigned)((a.nels + HT_E - 1) / HT_E)), dim3(HT_THREADS), sizeof(ThSmem<T>), st, a);
}

}  // namespace

template <class T, class TG>
cudaError_t launch_thermal3d(const ThermalArgs<T, TG>& a, int num_sms, cudaStream_t st, bool pdl) {
    if (!a.jac && !a.group) return launch_t3_tiles<T, TG>(a, st, pdl);
    const int64_t n = a.group ? a.ngroup : a.nels;
    return a.jac ? launch_t3<T, TG, true>(a, n, num_sms, st, pdl) : launch_t3<T, TG, false>(a, n, num_sms, st, pdl);
}

template cudaError_t launch_thermal3d<double, double>(const ThermalArgs<double, double>&, int, cudaStream_t, bool);
template cudaError_t launch_thermal3d<float, float>(const ThermalArgs<float, float>&, int, cudaStream_t, bool);
template cudaError_t launch_thermal3d<double, float>(const ThermalArgs<double, float>&, int, cudaStream_t, bool);
template cudaError_t launch_thermal3d<float, double>(const ThermalArgs<float, double>&, int, cudaStream_t, bool);

}  // namespace femb
