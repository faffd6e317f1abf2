// q9.cu — Q9/P1-disc plane-strain Stokes sweep and augmented Jacobian diagnostics
// (momentum_residuals.jl:497-528, :929-1117, pressure_residual.jl:132-158, rheology.jl:226-334).
//
// The residual sweep maps 32 elements to a block with one warp per point row; the Jacobian
// diagnostics three elements to a warp, nine lanes each. Both replace one thread per element
// (64² cells were 32 blocks of one long serial thread each); figures beside the kernels.
#include <algorithm>
#include "kernels.cuh"

namespace femb {
namespace {

// ---- nine lanes per element (Jacobian diagnostics) ----------------------------------------
//
// Lane m of an element is its node m (tensor order) in the gather and the scatter and its
// quadrature point m in between. Values cross between nodes and points through a shared slot
// per element (stride ≡ 11 modulo the 16 eight-byte banks: the three slots' broadcasts fall in
// distinct banks), ordered by __syncwarp.
constexpr int Q9_THREADS = 128, Q9_WPB = Q9_THREADS / 32;

// Lane tables of one lane: 1-D basis values and derivatives as a point (row of the lane's
// point over the nodes) and as a node (column of the lane's node over the points).
template <class T>
struct Q9Lane {
    int lane, s, m, m1, m2;
    bool ok;
    T b1[3], d1[3], b2[3], d2[3];     // point: B[m1][i], D[m1][i], B[m2][j], D[m2][j]
    T tb1[3], td1[3], tb2[3], td2[3]; // node:  B[q][m1], …
    T x, y, sumN;
    FEMB_D void load() {
        lane = threadIdx.x & 31;
        ok = lane < 27;
        s = ok ? lane / 9 : 3;
        m = ok ? lane % 9 : 0;
        m1 = m % 3; m2 = m / 3;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            b1[i] = (T)c_tab.B[m1][i]; d1[i] = (T)c_tab.Dd[m1][i];
            b2[i] = (T)c_tab.B[m2][i]; d2[i] = (T)c_tab.Dd[m2][i];
            tb1[i] = (T)c_tab.B[i][m1]; td1[i] = (T)c_tab.Dd[i][m1];
            tb2[i] = (T)c_tab.B[i][m2]; td2[i] = (T)c_tab.Dd[i][m2];
        }
        x = (T)c_tab.qx[m1]; y = (T)c_tab.qx[m2];
        sumN = (T)c_tab.sumN2[m];
    }
};

// Reference gradient at the lane's point of the nodal values u[i + 3j] in shared memory.
template <class T>
FEMB_D void q9_ref_gradient(const Q9Lane<T>& L, const T* u, T& gx, T& gy) {
    gx = gy = T(0);
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        const T u0 = u[3 * j], u1 = u[3 * j + 1], u2 = u[3 * j + 2];
        gx += L.b2[j] * (L.d1[0] * u0 + L.d1[1] * u1 + L.d1[2] * u2);
        gy += L.d2[j] * (L.b1[0] * u0 + L.b1[1] * u1 + L.b1[2] * u2);
    }
}

// Σ_q ∂_ξ N_a Fx + ∂_η N_a Fy at the lane's node, from fluxes at the points.
template <class T>
FEMB_D T q9_transpose(const Q9Lane<T>& L, const T* Fx, const T* Fy) {
    T r = T(0);
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        r += L.tb2[q] * (L.td1[0] * Fx[3 * q] + L.td1[1] * Fx[3 * q + 1] + L.td1[2] * Fx[3 * q + 2]);
        r += L.td2[q] * (L.tb1[0] * Fy[3 * q] + L.tb1[1] * Fy[3 * q + 1] + L.tb1[2] * Fy[3 * q + 2]);
    }
    return r;
}
// Phase of the element when all nine lanes carry one (`uniform`), per-lane phase otherwise;
// every lane of the warp calls it.
FEMB_D bool q9_uniform(int ph, int s, bool ok, int& p0) {
    p0 = __shfl_sync(0xffffffffu, ph, ok ? s * 9 : 27);
    const unsigned bal = __ballot_sync(0xffffffffu, ph == p0 || !ok);
    return !ok || ((bal >> (s * 9)) & 0x1ffu) == 0x1ffu;
}

// Material at the lane's point (interp2ip_phase, utils.jl:37-44): the element's one phase, or
// the nodes' phases weighted by N.
template <class T>
struct Q9Mat {
    T eta, invG, rho0, alpha, beta, cphi, sphi, spsi, C, ereg, Kb;
};
template <class T>
FEMB_D void q9_material(const Q9Lane<T>& L, bool uniform, int p0, int ph, bool plastic, Q9Mat<T>& m) {
    if (__all_sync(0xffffffffu, uniform)) {
        m.eta = (T)c_mat.eta[p0] * L.sumN; m.invG = (T)c_mat.invG[p0] * L.sumN;
        m.rho0 = (T)c_mat.rho0[p0] * L.sumN; m.alpha = (T)c_mat.alpha[p0] * L.sumN; m.beta = (T)c_mat.beta[p0] * L.sumN;
        if (plastic) {
            m.cphi = (T)c_mat.cos_phi[p0] * L.sumN; m.sphi = (T)c_mat.sin_phi[p0] * L.sumN;
            m.spsi = (T)c_mat.sin_psi[p0] * L.sumN; m.C = (T)c_mat.C[p0] * L.sumN;
            m.ereg = (T)c_mat.eta_reg[p0] * L.sumN; m.Kb = (T)c_mat.Kb[p0] * L.sumN;
        }
        return;
    }
    m.eta = m.invG = m.rho0 = m.alpha = m.beta = m.cphi = m.sphi = m.spsi = m.C = m.ereg = m.Kb = T(0);
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const T N = L.b1[i] * L.b2[j];
            const int p = __shfl_sync(0xffffffffu, ph, L.ok ? L.s * 9 + i + 3 * j : 27);
            m.eta += N * (T)c_mat.eta[p]; m.invG += N * (T)c_mat.invG[p];
            m.rho0 += N * (T)c_mat.rho0[p]; m.alpha += N * (T)c_mat.alpha[p]; m.beta += N * (T)c_mat.beta[p];
            if (plastic) {
                m.cphi += N * (T)c_mat.cos_phi[p]; m.sphi += N * (T)c_mat.sin_phi[p]; m.spsi += N * (T)c_mat.sin_psi[p];
                m.C += N * (T)c_mat.C[p]; m.ereg += N * (T)c_mat.eta_reg[p]; m.Kb += N * (T)c_mat.Kb[p];
            }
        }
}

// Plane-strain trial stress and Drucker–Prager return (rheology.jl:226-334); keeps the trial
// state that the linearisation needs.
template <class T>
struct PsState {
    T tt[3], tau[3], twoe, lam, itII, itIIs, iden;
};
template <class T>
FEMB_D void ps_return(PsState<T>& s, bool plastic, T cC, T sphi, T iden, T Peq) {
    s.lam = T(0); s.itII = T(1); s.itIIs = T(1); s.iden = iden;
#pragma unroll
    for (int c = 0; c < 3; ++c) s.tau[c] = s.tt[c];
    if (!plastic) return;
    const T tzz = -s.tt[0] - s.tt[1];
    const T tII = sqrt(T(0.5) * (s.tt[0] * s.tt[0] + s.tt[1] * s.tt[1] + tzz * tzz) + s.tt[2] * s.tt[2] + eps2<T>());
    const T F = tII - cC - sphi * Peq;
    if (!(F > T(0))) return;
    const T lam = F * iden;
    s.lam = lam;
    if (!(lam > T(0))) return;
    s.itII = T(1) / tII;
    s.itIIs = T(1) / (tII + eps2<T>());
    const T f = s.twoe * lam * s.itIIs;
    s.tau[0] = s.tt[0] - f * (s.tt[0] + T(0.5) * s.tt[1]);
    s.tau[1] = s.tt[1] - f * (T(0.5) * s.tt[0] + s.tt[1]);
    s.tau[2] = s.tt[2] - f * s.tt[2];
}
// dτ along the strain-rate increment (dexx, deyy, dexy)
template <class T>
FEMB_D void ps_tangent(const PsState<T>& s, T dexx, T deyy, T dexy, T dtau[3]) {
    const T tr = (dexx + deyy) / T(3);
    const T d[3] = {s.twoe * (dexx - tr), s.twoe * (deyy - tr), s.twoe * dexy};
    if (!(s.lam > T(0))) {
#pragma unroll
        for (int c = 0; c < 3; ++c) dtau[c] = d[c];
        return;
    }
    const T* t = s.tt;
    const T dtII = (T(0.5) * ((T(2) * t[0] + t[1]) * d[0] + (t[0] + T(2) * t[1]) * d[1]) + t[2] * d[2]) * s.itII;
    const T dlam = dtII * s.iden;
    // flow direction and its derivative, in units of 1/τII
    const T q[3] = {t[0] + T(0.5) * t[1], T(0.5) * t[0] + t[1], t[2]};
    const T p[3] = {d[0] + T(0.5) * d[1], T(0.5) * d[0] + d[1], d[2]};
    const T w = dtII * s.itIIs;
#pragma unroll
    for (int c = 0; c < 3; ++c) dtau[c] = d[c] - s.twoe * s.itIIs * (dlam * q[c] + s.lam * (p[c] - q[c] * w));
}

// ---- residual sweep: 32 elements per block, one warp per point row ----------------------
//
// Thread (lane, w) owns the points (·, η_w) of element 32·block + lane on the way in and the
// nodes (·, j = w) on the way out: the 1-D coefficients along ξ are compile-time constants,
// those along η uniform in the warp, and 66 instructions an element replace the 342 of the
// nine-lane mapping, whose lane tables and guards outweighed its arithmetic. The per-point arrays
// (32 elements' geometry, stress history, …, contiguous in memory) come by coalesced cp.async
// into shared memory, where the strides of 45 and 9 words (odd) read conflict-free.
// Measured (FP64): 64² viscous inclusion, 1000 iterations 31.6 -> 12.9 ms (8.1 with dependent launches); 256²
// shear band, 600 iterations with seven assemblies of the diagnostics 54.0 -> 23.2 ms (18.7; 43.3 ms with
// nine lanes per element, 77 us a sweep: 1027 instructions per three elements, 27 % issue). Bound by the
// dependent gathers and the block's three barriers: a sweep of 256² takes 32 us from a cold cache with 14
// warps per SM, 34 % issue and 62 MB from DRAM.
constexpr int QT = 32, QR_THREADS = 3 * QT;
constexpr double QGA = 0.774596669241483377035853079956479922;
FEMB_HD constexpr double q_x(int q) { return q == 0 ? -QGA : (q == 1 ? 0.0 : QGA); }
FEMB_HD constexpr double q_L(int q, int i) {
    return i == 0 ? q_x(q) * (q_x(q) - 1.0) * 0.5 : (i == 1 ? 1.0 - q_x(q) * q_x(q) : q_x(q) * (q_x(q) + 1.0) * 0.5);
}
FEMB_HD constexpr double q_D(int q, int i) { return i == 0 ? q_x(q) - 0.5 : (i == 1 ? -2.0 * q_x(q) : q_x(q) + 0.5); }
// fma with a compile-time coefficient; the middle point's zeros fold away
template <class T> FEMB_D T q_fma(double c, T x, T acc) { return c != 0.0 ? (T)c * x + acc : acc; }

template <class T> FEMB_D void q_cp_async(T* dst, const T* src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    if constexpr (sizeof(T) == 8) asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d), "l"(src) : "memory");
}
template <class T> FEMB_D void q_stage(T* dst, const T* src, int n) {
    for (int i = threadIdx.x; i < n; i += QR_THREADS) q_cp_async(dst + i, src + i);
}

// Shared memory of one block (36.5 KB in FP64, 38.8 KB with a per-point field: five blocks per
// SM): the staged point arrays and per-lane columns. The row fluxes X take the place of what the
// pressure pass has consumed.
template <class T, class TG>
struct Q9Smem {
    TG geo[QT * 45];
    T told[3][QT * 9];
    T P[18][QT], pn[3][QT];   // pressure fields (P, P − P0, T, T − T0, Q, Pf), Pnum
    union {
        struct {
            T V[18][QT], rp[9][QT];   // velocities, row sums of the pressure residual
            TG geoP[QT * 9];          // |det J|·ω of the pressure residual
        };
        T X[45][QT];
    };
    int ph[9][QT];
    T ip[QT * 9];   // viscosity or P_old per point; not allocated when neither is given
};

template <class T, class TG>
__global__ void __launch_bounds__(QR_THREADS, 5) q9_residual_kernel(const H27Args<T, TG> a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Q9Smem<T, TG>& S = *reinterpret_cast<Q9Smem<T, TG>*>(smem_raw);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t e0 = (int64_t)blockIdx.x * QT;
    const int ne = (int)(a.nels - e0 < QT ? a.nels - e0 : QT);   // elements of this tile
    const bool act = lane < ne;
    // lanes past the mesh's end repeat its last element and store nothing
    const int64_t e = e0 + (act ? lane : ne - 1);
    const int el = act ? lane : ne - 1;

    q_stage(S.geo, a.geo_v + e0 * 45, ne * 45);
    q_stage(S.geoP, a.geo_P + e0 * 9, ne * 9);
#pragma unroll
    for (int c = 0; c < 3; ++c)
        if (a.told[c]) q_stage(S.told[c], a.told[c] + e0 * 9, ne * 9);
    const T* ip = a.eta_ip ? a.eta_ip : a.P_old_ip;   // both given: P_old is read from memory
    if (ip) q_stage(S.ip, ip + e0 * 9, ne * 9);
    asm volatile("cp.async.commit_group;\n" ::: "memory");

    int node[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) node[i] = __ldg(a.el2n + 9 * e + c_tab.tn2[i + 3 * w]) - 1;
    const int dof = __ldg(a.dofsP + 3 * e + w) - 1;
    const bool cell = !a.phv || a.phv_layout == FEMB200_PHASE_CELL;
    int p0 = 0;
    if (cell) {
        if (a.phv) p0 = __ldg(a.phv + e) - 1;
    } else {
#pragma unroll
        for (int i = 0; i < 3; ++i)
            S.ph[i + 3 * w][lane] = phase_of(a.phv, a.phv_layout, (int64_t)node[i] + 1, c_tab.tn2[i + 3 * w], e, 9);
    }
    pdl_enter();   // everything so far is constant over the iterations
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        S.V[i + 3 * w][lane] = ld_coherent(a.v[0] + node[i]);
        S.V[9 + i + 3 * w][lane] = ld_coherent(a.v[1] + node[i]);
    }
    // warp w brings pressure DoF w of every element
    const T Pw = ld_coherent(a.P + dof);
    S.P[w][lane] = Pw;
    S.P[3 + w][lane] = a.P_old_ip || !a.P0 ? Pw : Pw - ld(a.P0 + dof);
    if (a.temp || a.temp0) {   // an absent temperature is zero
        const T t = a.temp ? ld_coherent(a.temp + dof) : T(0);
        S.P[6 + w][lane] = t;
        S.P[9 + w][lane] = a.temp0 ? t - ld(a.temp0 + dof) : t;
    }
    if (a.Q) S.P[12 + w][lane] = ld(a.Q + dof);
    if (a.Pf) S.P[15 + w][lane] = ld(a.Pf + dof);
    const T gam = a.gammaP ? ld(a.gammaP + dof) : T(0), mp = a.MP ? ld(a.MP + dof) : T(1);
    const T pin = a.with_pnum && a.Pnum_in ? ld(a.Pnum_in + dof) : T(0);
    int php[3] = {0, 0, 0};
    if (a.php) {
#pragma unroll
        for (int p = 0; p < 3; ++p)
            php[p] = a.php_layout == FEMB200_PHASE_CELL ? __ldg(a.php + e) - 1
                     : a.php_layout == FEMB200_PHASE_ELEMENT_NODE ? __ldg(a.php + 3 * e + p) - 1
                                                                  : __ldg(a.php + __ldg(a.dofsP + 3 * e + p) - 1) - 1;
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();

    bool uniform = true;
    if (!cell) {
        p0 = S.ph[0][lane];
#pragma unroll
        for (int k = 1; k < 9; ++k) uniform = uniform && S.ph[k][lane] == p0;
    }
    const bool plastic = c_mat.plastic != 0, bulk_inf = c_mat.all_bulk_inf != 0;
    const bool consts_ok = c_mat.dt_consts == (double)a.dt || (T)c_mat.dt_consts == a.dt;
    T by[3], dy[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) { by[j] = (T)c_tab.B[w][j]; dy[j] = (T)c_tab.Dd[w][j]; }
    const T et = (T)c_tab.qx[w];
    const TG* geo = S.geo + el * 45 + w * 15;
    const int q0 = el * 9 + 3 * w;                        // the row's first point

    // ---- gradients along the row and the pressure residual ----
    T g[3][2][2];
    {
        T X[2][3], Y[2][3];
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                const T u0 = S.V[9 * c + i][lane], u1 = S.V[9 * c + i + 3][lane], u2 = S.V[9 * c + i + 6][lane];
                X[c][i] = by[0] * u0 + by[1] * u1 + by[2] * u2;
                Y[c][i] = dy[0] * u0 + dy[1] * u1 + dy[2] * u2;
            }
#pragma unroll
        for (int q = 0; q < 3; ++q)
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                T r0 = T(0), r1 = T(0);
#pragma unroll
                for (int i = 0; i < 3; ++i) { r0 = q_fma<T>(q_D(q, i), X[c][i], r0); r1 = q_fma<T>(q_L(q, i), Y[c][i], r1); }
                g[q][c][0] = r0 * (T)geo[5 * q] + r1 * (T)geo[5 * q + 1];
                g[q][c][1] = r0 * (T)geo[5 * q + 2] + r1 * (T)geo[5 * q + 3];
            }
    }
    // a pressure field at the row's point q: linear in ξ
    auto at = [&](int f, int q) {
        const T c0 = S.P[3 * f][lane];
        return (T(1) - (T)q_x(q) - et) * c0 + (T)q_x(q) * S.P[3 * f + 1][lane] + et * S.P[3 * f + 2][lane];
    };
    {
        const bool one_php = php[0] == p0 && php[1] == p0 && php[2] == p0;
        T rp[3] = {T(0), T(0), T(0)};
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const T NP0 = T(1) - (T)q_x(q) - et;
            T f = -(g[q][0][0] + g[q][1][1]);
            if (!bulk_inf) {
                T dPinc = at(1, q);
                if (a.P_old_ip) dPinc -= a.eta_ip ? ld(a.P_old_ip + e * 9 + 3 * w + q) : S.ip[q0 + q];
                if (one_php && consts_ok) f -= dPinc * (T)c_mat.u_inv_bulkdt[p0];
                else f -= dPinc / ((NP0 * (T)c_mat.bulk[php[0]] + (T)q_x(q) * (T)c_mat.bulk[php[1]] + et * (T)c_mat.bulk[php[2]]) * a.dt);
            }
            if (a.temp || a.temp0)
                f += (NP0 * (T)c_mat.alpha[php[0]] + (T)q_x(q) * (T)c_mat.alpha[php[1]] + et * (T)c_mat.alpha[php[2]]) * at(3, q) / a.dt;
            if (a.Q) f += at(4, q);
            f *= (T)S.geoP[q0 + q];
            rp[0] += NP0 * f;
            rp[1] = q_fma<T>(q_x(q), f, rp[1]);
            rp[2] += et * f;
        }
#pragma unroll
        for (int p = 0; p < 3; ++p) S.rp[3 * w + p][lane] = rp[p];
    }
    __syncthreads();
    {
        const T rp = S.rp[w][lane] + S.rp[3 + w][lane] + S.rp[6 + w][lane];
        if (act && a.write_RP) a.RP[dof] = rp;
        T pn = T(0);
        if (a.with_pnum) {
            pn = a.Pnum_in ? pin : gam * rp / mp;
            if (act && a.Pnum_out) a.Pnum_out[dof] = pn;
        }
        S.pn[w][lane] = pn;
    }
    if (!a.do_momentum && !a.phi) return;
    __syncthreads();

    // ---- stress and fluxes, contracted along the row ----
    T A[2][3], Bf[2][3], Ab[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) { A[0][i] = A[1][i] = Bf[0][i] = Bf[1][i] = Ab[i] = T(0); }
    const bool fast = uniform && consts_ok && !a.eta_ip;
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        const T NP0 = T(1) - (T)q_x(q) - et;
        T told[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) told[c] = a.told[c] ? S.told[c][q0 + q] : T(0);
        T twoe, twoe_el, rho0, alpha, beta, cC = T(0), sphi = T(0), iden = T(1);
        T invG = T(0);
        if (fast) {
            twoe = (T)c_mat.u_twoe[p0]; twoe_el = (T)c_mat.u_twoe_el[p0];
            rho0 = (T)c_mat.rho0[p0]; alpha = (T)c_mat.alpha[p0]; beta = (T)c_mat.beta[p0];
            if (plastic) { cC = (T)c_mat.u_cC[p0]; sphi = (T)c_mat.sin_phi[p0]; iden = (T)c_mat.u_inv_den[p0]; }
        } else {
            Q9Mat<T> m;
            if (uniform) {
                const T sN = (T)c_tab.sumN2[q + 3 * w];
                m.eta = (T)c_mat.eta[p0] * sN; m.invG = (T)c_mat.invG[p0] * sN;
                m.rho0 = (T)c_mat.rho0[p0] * sN; m.alpha = (T)c_mat.alpha[p0] * sN; m.beta = (T)c_mat.beta[p0] * sN;
                if (plastic) {
                    m.cphi = (T)c_mat.cos_phi[p0] * sN; m.sphi = (T)c_mat.sin_phi[p0] * sN; m.spsi = (T)c_mat.sin_psi[p0] * sN;
                    m.C = (T)c_mat.C[p0] * sN; m.ereg = (T)c_mat.eta_reg[p0] * sN; m.Kb = (T)c_mat.Kb[p0] * sN;
                }
            } else {
                m.eta = m.invG = m.rho0 = m.alpha = m.beta = m.cphi = m.sphi = m.spsi = m.C = m.ereg = m.Kb = T(0);
#pragma unroll 1
                for (int k = 0; k < 9; ++k) {
                    const T N = (T)c_tab.N2[q + 3 * w][c_tab.tn2[k]];
                    const int p = S.ph[k][lane];
                    m.eta += N * (T)c_mat.eta[p]; m.invG += N * (T)c_mat.invG[p];
                    m.rho0 += N * (T)c_mat.rho0[p]; m.alpha += N * (T)c_mat.alpha[p]; m.beta += N * (T)c_mat.beta[p];
                    if (plastic) {
                        m.cphi += N * (T)c_mat.cos_phi[p]; m.sphi += N * (T)c_mat.sin_phi[p]; m.spsi += N * (T)c_mat.sin_psi[p];
                        m.C += N * (T)c_mat.C[p]; m.ereg += N * (T)c_mat.eta_reg[p]; m.Kb += N * (T)c_mat.Kb[p];
                    }
                }
            }
            if (a.eta_ip) m.eta = S.ip[q0 + q];
            const T etave = T(1) / (T(1) / m.eta + m.invG / a.dt);
            twoe = T(2) * etave;
            invG = m.invG;
            twoe_el = twoe * (invG / (T(2) * a.dt));
            rho0 = m.rho0; alpha = m.alpha; beta = m.beta;
            if (plastic) {
                cC = m.cphi * m.C; sphi = m.sphi;
                iden = T(1) / (etave + m.ereg + m.Kb * a.dt * (-m.spsi) * (-m.sphi));
            }
        }
        const T Pq = at(0, q), Pfq = a.Pf ? at(5, q) : T(0);
        const T Pnq = NP0 * S.pn[0][lane] + (T)q_x(q) * S.pn[1][lane] + et * S.pn[2][lane];
        const T Peq = a.Pf ? Pq - Pfq : Pq;
        const T tr = (g[q][0][0] + g[q][1][1]) * T(1.0 / 3.0);
        PsState<T> st;
        st.twoe = twoe;
        st.tt[0] = twoe * (g[q][0][0] - tr) + twoe_el * told[0];
        st.tt[1] = twoe * (g[q][1][1] - tr) + twoe_el * told[1];
        st.tt[2] = twoe * (T(0.5) * (g[q][0][1] + g[q][1][0])) + twoe_el * told[2];
        ps_return(st, plastic, cC, sphi, iden, Peq);
        const int64_t gp = e * 9 + 3 * w + q;
        if (act && a.tau_store[0]) {
#pragma unroll
            for (int c = 0; c < 3; ++c) a.tau_store[c][gp] = st.tau[c];
        }
        if (act && a.phi) {
            // shear_dissipation, plane strain (shear_heating.jl:79-88)
            const T* t = st.tau;
            const T tzz = -(t[0] + t[1]), tzzo = -(told[0] + told[1]);
            // (1/(2GΔt) from G: 2ηve may be zero)
            const T inv2Gdt = (fast ? (T)c_mat.invG[p0] : invG) / (T(2) * a.dt);
            const T power = t[0] * g[q][0][0] + t[1] * g[q][1][1] + t[2] * (g[q][0][1] + g[q][1][0]);
            const T el_ = (t[0] * (t[0] - told[0]) + t[1] * (t[1] - told[1]) + tzz * (tzz - tzzo) +
                           T(2) * t[2] * (t[2] - told[2])) * inv2Gdt;
            a.phi[gp] = power - el_;
        }
        const T Ptot = (a.Pf ? Peq + Pfq : Pq) + Pnq;
        const T Tq = a.temp ? at(2, q) : T(0);
        const T dO = (T)geo[5 * q + 4];
        const T bq = rho0 * (T(1) - alpha * (Tq - (T)c_mat.Tref) + beta * Pq) * dO;
        const T s00 = (st.tau[0] - Ptot) * dO, s11 = (st.tau[1] - Ptot) * dO, s01 = st.tau[2] * dO;
        const T J00 = (T)geo[5 * q], J10 = (T)geo[5 * q + 1], J01 = (T)geo[5 * q + 2], J11 = (T)geo[5 * q + 3];
        const T F00 = J00 * s00 + J01 * s01, F01 = J10 * s00 + J11 * s01;   // ∂ξ_d/∂x_k σ_kc, c = x
        const T F10 = J00 * s01 + J01 * s11, F11 = J10 * s01 + J11 * s11;   // c = y
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            A[0][i] = q_fma<T>(q_D(q, i), F00, A[0][i]);
            A[1][i] = q_fma<T>(q_D(q, i), F10, A[1][i]);
            Bf[0][i] = q_fma<T>(q_L(q, i), F01, Bf[0][i]);
            Bf[1][i] = q_fma<T>(q_L(q, i), F11, Bf[1][i]);
            Ab[i] = q_fma<T>(q_L(q, i), bq, Ab[i]);
        }
    }
    if (!a.do_momentum) return;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            S.X[15 * w + 3 * c + i][lane] = A[c][i] - (T)c_mat.g[c] * Ab[i];
            S.X[15 * w + 6 + 3 * c + i][lane] = Bf[c][i];
        }
    __syncthreads();
    // ---- nodes (·, j = w): Σ over the point rows, then the scatter ----
    T R[2][3];
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int i = 0; i < 3; ++i) R[c][i] = T(0);
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        const T bl = (T)c_tab.B[r][w], dl = (T)c_tab.Dd[r][w];
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int i = 0; i < 3; ++i)
                R[c][i] += bl * S.X[15 * r + 3 * c + i][lane] + dl * S.X[15 * r + 6 + 3 * c + i][lane];
    }
    // the next lane's ξ = −1 node, when it is this lane's ξ = +1 node, is added here
    const int n0n = __shfl_down_sync(0xffffffffu, node[0], 1);
    const bool fold = lane + 1 < ne && lane < 31 && n0n == node[2];
    const bool folded = __shfl_up_sync(0xffffffffu, (int)fold, 1) && lane > 0;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        const T r0n = __shfl_down_sync(0xffffffffu, R[c][0], 1);
        if (fold) R[c][2] += r0n;
        if (act) {
            if (!folded) atomic_add(a.Rv[c] + node[0], R[c][0]);
            atomic_add(a.Rv[c] + node[1], R[c][1]);
            atomic_add(a.Rv[c] + node[2], R[c][2]);
        }
    }
}

// Augmented Jacobian diagnostics (momentum_residuals.jl:929-1117): |row sums| and |diagonal|
// of the element Jacobian at η_pc. The point's 3 × 3 tangent is formed once; column (b, j) is
// the transposed contraction of its flux along the unit velocity j of node b, two columns per
// exchange.
template <class T, class TG>
__global__ void __launch_bounds__(Q9_THREADS, 3) q9_jacobian_kernel(const H27JacArgs<T, TG> a) {
    // slot: the two columns' fluxes (72), the pressure rows ∂RP/∂v·γ/M (54), velocities (18)
    constexpr int JF = 0, JB = 72, JV = 126, JP = 144, SLOT = 155;   // 155 ≡ 11 mod 16
    __shared__ T smem[Q9_WPB * 4 * SLOT];
    Q9Lane<T> L;
    L.load();
    T* E = smem + ((threadIdx.x >> 5) * 4 + L.s) * SLOT;
    const int tn = c_tab.tn2[L.m];
    const bool plastic = c_mat.plastic != 0;
    const T NP[3] = {T(1) - L.x - L.y, L.x, L.y};
    const int64_t stride = (int64_t)gridDim.x * Q9_WPB * 3;
    for (int64_t base = ((int64_t)blockIdx.x * Q9_WPB + (threadIdx.x >> 5)) * 3; base < a.nels; base += stride) {
        const int64_t e = base + (L.ok ? L.s : 0);
        const bool act = L.ok && e < a.nels;
        const int64_t ec = act ? e : 0;
        const int64_t ip = ec * 9 + L.m;
        const int node = act ? __ldg(a.el2n + 9 * ec + tn) - 1 : 0;
        const TG* G = a.geo_v + ip * 5;
        const T J00 = act ? (T)ld(G) : T(0), J10 = act ? (T)ld(G + 1) : T(0), J01 = act ? (T)ld(G + 2) : T(0),
                J11 = act ? (T)ld(G + 3) : T(0), dO = act ? (T)ld(G + 4) : T(0), dOP = act ? (T)ld(a.geo_P + ip) : T(0);
        E[JV + L.m] = act ? ld(a.v[0] + node) : T(0);
        E[JV + 9 + L.m] = act ? ld(a.v[1] + node) : T(0);
        const int ph = act ? phase_of(a.phv, a.phv_layout, (int64_t)node + 1, tn, ec, 9) : 0;
        T r_own = T(0);   // γ/M of pressure DoF m (lanes m < 3)
        if (act && L.m < 3) {
            const int dof = __ldg(a.dofsP + 3 * ec + L.m) - 1;
            E[JP + L.m] = ld(a.P + dof);
            E[JP + 3 + L.m] = a.Pf ? ld(a.Pf + dof) : T(0);
            r_own = (a.gammaP ? ld(a.gammaP + dof) : T(0)) / (a.MP ? ld(a.MP + dof) : T(1));
        }
        int p0;
        const bool uniform = q9_uniform(ph, L.s, L.ok, p0);
        // η_pc: the largest viscosity of the points (given per point) or of the nodes' phases
        T eta_pc = a.eta_ip ? (act ? ld(a.eta_ip + ip) : T(1)) : (T)c_mat.eta[ph];
        {
            T mx = eta_pc;
#pragma unroll
            for (int k = 0; k < 9; ++k) mx = fmax(mx, __shfl_sync(0xffffffffu, eta_pc, L.ok ? L.s * 9 + k : 27));
            eta_pc = mx;
        }
        T rat[3];
#pragma unroll
        for (int p = 0; p < 3; ++p) rat[p] = __shfl_sync(0xffffffffu, r_own, L.ok ? L.s * 9 + p : 27);
        Q9Mat<T> mt;
        q9_material(L, uniform, p0, ph, plastic, mt);
        __syncwarp();

        // ---- the point's tangent C[·][k]: ∂τ along exx, eyy, exy ----
        T C[3][3];
        {
            T g[2][2];
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                T r0, r1;
                q9_ref_gradient(L, E + JV + 9 * c, r0, r1);
                g[c][0] = r0 * J00 + r1 * J10;
                g[c][1] = r0 * J01 + r1 * J11;
            }
            const T etaq = a.eta_ip ? eta_pc : eta_pc * L.sumN;
            const T etave = T(1) / (T(1) / etaq + mt.invG / a.dt);
            PsState<T> st;
            st.twoe = T(2) * etave;
            const T twoe_el = st.twoe * (mt.invG / (T(2) * a.dt));
            const T tr = (g[0][0] + g[1][1]) / T(3);
            T told[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) told[c] = act && a.told[c] ? ld(a.told[c] + ip) : T(0);
            st.tt[0] = st.twoe * (g[0][0] - tr) + twoe_el * told[0];
            st.tt[1] = st.twoe * (g[1][1] - tr) + twoe_el * told[1];
            st.tt[2] = st.twoe * (T(0.5) * (g[0][1] + g[1][0])) + twoe_el * told[2];
            const T* Pd = E + JP;
            const T Pq = NP[0] * Pd[0] + NP[1] * Pd[1] + NP[2] * Pd[2];
            const T Pfq = NP[0] * Pd[3] + NP[1] * Pd[4] + NP[2] * Pd[5];
            T cC = T(0), sphi = T(0), iden = T(1);
            if (plastic) {
                cC = mt.cphi * mt.C; sphi = mt.sphi;
                iden = T(1) / (etave + mt.ereg + mt.Kb * a.dt * (-mt.spsi) * (-mt.sphi));
            }
            ps_return(st, plastic, cC, sphi, iden, a.Pf ? Pq - Pfq : Pq);
            ps_tangent(st, T(1), T(0), T(0), C[0]);
            ps_tangent(st, T(0), T(1), T(0), C[1]);
            ps_tangent(st, T(0), T(0), T(1), C[2]);
        }
        // ---- pressure rows: B[p][j] at the lane's node = −(γ/M)_p Σ_q N^P_p dΩ_P ∂N/∂x_j ----
#pragma unroll
        for (int p = 0; p < 3; ++p) {
            const T w = NP[p] * dOP;
            T* Fp = E + JF + L.m;
            Fp[0] = w * J00; Fp[9] = w * J10; Fp[18] = w * J01; Fp[27] = w * J11;
            __syncwarp();
            const T r0 = -q9_transpose(L, E + JF, E + JF + 9) * rat[p];
            const T r1 = -q9_transpose(L, E + JF + 18, E + JF + 27) * rat[p];
            E[JB + (p * 2 + 0) * 9 + L.m] = r0;
            E[JB + (p * 2 + 1) * 9 + L.m] = r1;
            __syncwarp();
        }
        // ---- columns ----
        T rows[2] = {T(0), T(0)}, diag[2] = {T(0), T(0)};
#pragma unroll 1
        for (int b = 0; b < 9; ++b) {
            const int bi = b % 3, bj = b / 3;
            const T u1 = bi == 0 ? L.b1[0] : (bi == 1 ? L.b1[1] : L.b1[2]), v1 = bi == 0 ? L.d1[0] : (bi == 1 ? L.d1[1] : L.d1[2]);
            const T u2 = bj == 0 ? L.b2[0] : (bj == 1 ? L.b2[1] : L.b2[2]), v2 = bj == 0 ? L.d2[0] : (bj == 1 ? L.d2[1] : L.d2[2]);
            const T r0 = v1 * u2, r1 = u1 * v2;
            const T n0 = r0 * J00 + r1 * J10, n1 = r0 * J01 + r1 * J11;   // ∂N_b/∂x, ∂N_b/∂y
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const T dexx = j == 0 ? n0 : T(0), deyy = j == 1 ? n1 : T(0), dexy = T(0.5) * (j == 0 ? n1 : n0);
                const T* Bj = E + JB + j * 9 + b;
                const T dPn = NP[0] * Bj[0] + NP[1] * Bj[18] + NP[2] * Bj[36];
                T t[3];
#pragma unroll
                for (int c = 0; c < 3; ++c) t[c] = C[0][c] * dexx + C[1][c] * deyy + C[2][c] * dexy;
                const T s00 = (t[0] - dPn) * dO, s11 = (t[1] - dPn) * dO, s01 = t[2] * dO;
                T* Fp = E + JF + 36 * j + L.m;
                Fp[0] = J00 * s00 + J01 * s01;
                Fp[9] = J10 * s00 + J11 * s01;
                Fp[18] = J00 * s01 + J01 * s11;
                Fp[27] = J10 * s01 + J11 * s11;
            }
            __syncwarp();
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const T* Fj = E + JF + 36 * j;
                const T R0 = fabs(q9_transpose(L, Fj, Fj + 9)), R1 = fabs(q9_transpose(L, Fj + 18, Fj + 27));
                rows[0] += R0;
                rows[1] += R1;
                if (L.m == b) diag[j] = j == 0 ? R0 : R1;
            }
            __syncwarp();
        }
        if (act) {
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                atomic_add(a.dRdv[c] + node, rows[c]);
                atomic_add(a.PC[c] + node, diag[c]);
            }
        }
    }
}

inline unsigned q9_blocks(int64_t nels) {
    // 148 SMs × 16 blocks bounds the grid; larger meshes stride over it
    const int64_t groups = (nels + 2) / 3;
    return (unsigned)std::max<int64_t>(1, std::min<int64_t>((groups + Q9_WPB - 1) / Q9_WPB, 148 * 16));
}

}  // namespace

template <class T, class TG>
cudaError_t launch_q9_residual(const H27Args<T, TG>& args, cudaStream_t st, bool pdl) {
    static_assert(sizeof(Q9Smem<T, TG>) <= 48 * 1024, "within the default shared-memory limit");
    const size_t smem = sizeof(Q9Smem<T, TG>) - (args.eta_ip || args.P_old_ip ? 0 : QT * 9 * sizeof(T));
    count_launch();
    return launch_pdl(pdl, q9_residual_kernel<T, TG>, dim3((unsigned)((args.nels + QT - 1) / QT)), dim3(QR_THREADS), smem, st, args);
}

template <class T, class TG>
cudaError_t launch_q9_jacobian(const H27JacArgs<T, TG>& args, cudaStream_t st) {
    count_launch();
    q9_jacobian_kernel<T, TG><<<q9_blocks(args.nels), Q9_THREADS, 0, st>>>(args);
    return cudaGetLastError();
}

#define FEMB_INSTQ(T, TG)                                                                \
    template cudaError_t launch_q9_residual<T, TG>(const H27Args<T, TG>&, cudaStream_t, bool); \
    template cudaError_t launch_q9_jacobian<T, TG>(const H27JacArgs<T, TG>&, cudaStream_t);
FEMB_INSTQ(double, double)
FEMB_INSTQ(float, float)
FEMB_INSTQ(double, float)
FEMB_INSTQ(float, double)
#undef FEMB_INSTQ

}  // namespace femb
