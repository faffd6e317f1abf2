// stokes3d.cu — Hex27/P1-disc Stokes element sweep for sm_100a.
//
// One kernel evaluates, per element and in one pass over the element's data:
//   the pressure residual  RP  (integrate_PH_pressure_residual,
//                               src/stokes/assemblers/pressure_residual.jl:132-158),
//   Pnum = γP·RP/M_P       (element-local, src/stokes/solvers/DR.jl:674),
//   the momentum residual  Rv  with the visco-elasto-plastic stress
//                               (momentum_residuals.jl:209-258, rheology.jl:413-472),
// optionally storing the integration-point stress (update_stokes_current_stress!,
// DR.jl:820), the shear dissipation (shear_heating.jl:47-103) or the base data of the
// mixed-precision sweep. The nodal residual is scattered with FP64/FP32 atomics into a
// zeroed Rv.
//
// Mapping (hex27_tile.cuh): a block of nine warps owns a tile of 32 elements, lane = element,
// warp = line of the grids. Geometry is per point in the reference layout or, on meshes whose
// cells are affine (the structured boxes and any parallelepipeds), one J⁻¹ and |det J| per
// element, built once per solve by compress_geometry (80 B instead of 2 376 B); the stress history
// (32 elements' values are contiguous) comes by coalesced cp.async into the first exchange buffer
// while the pressure residual is formed. The exchange strides replace the banked node buffers of
// H27Layout<T>. 110 KB of shared memory in FP64: two blocks per SM.
//
// Bound by instruction issue and the latency between its barriers. One solver iteration (sweep, node
// update) at 6×5×7 in three layers 16 us, where three elements to a warp with the next group's loads in
// flight took 23 (both before dependent launches: 20 and 23); 457 us a sweep at 64³ (643); 76 us at 32³ with
// a viscosity per point. One assembly on 40×33×29 distorted cells with a phase per node: 210 us against 432,
// the kernel 155 of it (with the tile's geometry staged in shared memory, which leaves room for one
// block per SM, 5 % more).
#include <type_traits>
#include "hex27_tile.cuh"
#include "kernels.cuh"
#include "rheology.cuh"

namespace femb {
namespace {

enum { PF_P, PF_DP, PF_T, PF_DT, PF_Q, PF_PF, PF_FIELDS };
enum { GEO_POINT, GEO_AFFINE, GEO_DIAG };

template <class T>
struct ResSmem {
    T S1[HT_S1], S2[HT_S2];
    T PF[PF_FIELDS][4][HT_E];    // pressure-DoF fields: P, P − P_old, T, T − T0, Q, Pf
    T pn[4][HT_E];
    T PT[PT_FIELDS][MAXPH];      // per-phase constants of the call's Δt
    int phm[9][HT_E];            // phases of a line's nodes, as a bit mask
    uint8_t PH[27][HT_E], php[4][HT_E];
};
static_assert(2 * (sizeof(ResSmem<double>) + 1024) <= 228 * 1024, "two blocks per SM");
static_assert(sizeof(ResSmem<double>) % 16 == 0 && sizeof(ResSmem<float>) % 16 == 0, "the staged geometry is aligned");
static_assert(HT_S1 == 6 * 27 * HT_E, "the first exchange buffer holds a tile's stress history");

template <class T> FEMB_D void cp_async_el(T* dst, const T* src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    if constexpr (sizeof(T) == 8) asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d), "l"(src) : "memory");
}

// n contiguous entries into shared memory by the whole block; vec: both sides 16-byte aligned
template <class T>
FEMB_D void stage(T* dst, const T* src, int n, bool vec) {
    if (vec) {
        constexpr int K = 16 / sizeof(T);
#pragma unroll 2
        for (int i = threadIdx.x; i < n / K; i += HT_THREADS) {
            const unsigned d = (unsigned)__cvta_generic_to_shared(dst + i * K);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src + i * K) : "memory");
        }
        for (int i = n / K * K + threadIdx.x; i < n; i += HT_THREADS) cp_async_el(dst + i, src + i);
    } else {
        for (int i = threadIdx.x; i < n; i += HT_THREADS) cp_async_el(dst + i, src + i);
    }
}

}  // namespace

// MINB: blocks per SM the registers are cut for. Two in FP64 means 96 registers and spills, which
// pays only where an SM has tiles enough for both.
// MIX: the phases are given per node, so elements may mix them; their properties are interpolated
// through the weights W_p(q) = Σ_{nodes a of phase p} N_a(q), formed by the same line
// contractions from the phases' indicators.
template <class T, class TG, int GEO, int MINB, bool MIX>
__global__ void __launch_bounds__(HT_THREADS, MINB) hex27_residual_kernel(const H27Args<T, TG> a) {
    extern __shared__ __align__(16) unsigned char res_smem[];
    ResSmem<T>& S = *reinterpret_cast<ResSmem<T>*>(res_smem);
    const int lane = threadIdx.x & 31, w = ht_warp(), la = w % 3, lb = w / 3;
    const int64_t tile = a.tile_list ? (int64_t)__ldg(a.tile_list + blockIdx.x) : (int64_t)blockIdx.x;
    const int64_t e0 = tile * HT_E;
    const int ne = (int)(a.nels - e0 < HT_E ? a.nels - e0 : HT_E);
    const bool act = lane < ne;
    // lanes past the mesh's end repeat its last element and store nothing
    const int el = act ? lane : ne - 1;
    const int64_t e = e0 + el;
    const T dt = a.dt;
    const bool plastic = c_mat.plastic != 0, bulk_inf = c_mat.all_bulk_inf != 0;
    const bool consts_ok = c_mat.dt_consts == (double)a.dt || (T)c_mat.dt_consts == a.dt;

    // ---- loads: first what no kernel of the iteration writes ----
    int node[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) node[i] = __ldg(a.el2n + 27 * e + c_tab.tn3[i + 3 * w]) - 1;
    T Ja[10];   // affine cells: the element's J⁻¹ and |det J|
    if constexpr (GEO != GEO_POINT) {
#pragma unroll
        for (int r = 0; r < 10; ++r) Ja[r] = (GEO == GEO_AFFINE || r % 4 == 0 || r == 9) ? ld(a.geo_c + e * 10 + r) : T(0);
    }
    int dof = 0;
    T gam = T(0), mp = T(1), pin = T(0);
    if (w < 4) {   // warp w brings pressure DoF w of every element
        dof = __ldg(a.dofsP + 4 * e + w) - 1;
        if (a.gammaP) gam = ld(a.gammaP + dof);
        if (a.MP) mp = ld(a.MP + dof);
    }
    int p0 = a.phv && !MIX ? __ldg(a.phv + e) - 1 : 0;
    int phn[3];
    if constexpr (MIX) {
        int mask = 0;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            phn[i] = phase_of(a.phv, a.phv_layout, (int64_t)node[i] + 1, c_tab.tn3[i + 3 * w], e, 27);
            S.PH[i + 3 * w][lane] = (uint8_t)phn[i];
            mask |= 1 << phn[i];
        }
        S.phm[w][lane] = mask;
    }
    static_assert(PT_FIELDS * MAXPH <= HT_THREADS, "one entry per thread");
    if (threadIdx.x < PT_FIELDS * MAXPH) (&S.PT[0][0])[threadIdx.x] = (T)(&c_mat.rho0[0])[threadIdx.x];

    // ---- the predecessor's outputs from here on ----
    pdl_enter();
    if (w < 4) {
        const T P = ld_coherent(a.P + dof);
        S.PF[PF_P][w][lane] = P;
        S.PF[PF_DP][w][lane] = a.P_old_ip || !a.P0 ? P : P - ld(a.P0 + dof);
        if (a.temp || a.temp0) {   // an absent temperature is zero
            const T t = a.temp ? ld_coherent(a.temp + dof) : T(0);
            S.PF[PF_T][w][lane] = t;
            S.PF[PF_DT][w][lane] = a.temp0 ? t - ld(a.temp0 + dof) : t;
        }
        if (a.Q) S.PF[PF_Q][w][lane] = ld(a.Q + dof);
        if (a.Pf) S.PF[PF_PF][w][lane] = ld(a.Pf + dof);
        if (a.with_pnum && a.Pnum_in) pin = ld(a.Pnum_in + dof);
        S.php[w][lane] = (uint8_t)phase_of(a.php, a.php_layout, (int64_t)dof + 1, w, e, 4);
    }

    // ---- gradients at the points q = la + 3lb + 9qz ----
    T g[3][3][3];
    {
        T v[3][3];
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int c = 0; c < 3; ++c) v[c][i] = ld_coherent(a.v[c] + node[i]);
        ht_gradient<T, 3>(v, S.S1, S.S2, la, lb, lane, g);
    }
    const TG* Gp = a.geo_v + (e * 27 + w) * 10;   // point qz at Gp + 90·qz
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        T J[10];
#pragma unroll
        for (int r = 0; r < 10; ++r) J[r] = GEO == GEO_POINT ? T(0) : Ja[r];
        if constexpr (GEO == GEO_POINT) load10(Gp + 90 * q, a.geo_vec, J);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const T r0 = g[c][0][q], r1 = g[c][1][q], r2 = g[c][2][q];
#pragma unroll
            for (int k = 0; k < 3; ++k)
                g[c][k][q] = GEO == GEO_DIAG ? (k == 0 ? r0 : k == 1 ? r1 : r2) * J[4 * k]
                                             : r0 * J[3 * k] + r1 * J[1 + 3 * k] + r2 * J[2 + 3 * k];
        }
    }
    __syncthreads();   // PF, PT, the phases; S1 and S2 are free
    // the stress history into S1 ([component][element][point]: odd stride, conflict-free reads)
#pragma unroll
    for (int c = 0; c < 6; ++c)
        if (a.told[c]) stage<T>(S.S1 + c * 27 * HT_E, a.told[c] + e0 * 27, ne * 27, (a.told_vec >> c) & 1);
    asm volatile("cp.async.commit_group;\n" ::: "memory");

    const T xi = ht_xr<T>(la), et = ht_xr<T>(lb);
    const T wxy = ht_wr<T>(la) * ht_wr<T>(lb);
    // a pressure field on the line: F0 + F1·ζ
    auto line = [&](int f, T& c0, T& c1) {
        const T x0 = S.PF[f][0][lane];
        c0 = x0 + xi * (S.PF[f][1][lane] - x0) + et * (S.PF[f][2][lane] - x0);
        c1 = S.PF[f][3][lane] - x0;
    };
    bool uniform = true;
    // phase weights of the thread's points, at WT[(p·3 + qz)·9·32] (the thread's own line of S2,
    // above the pressure parts) for materials of up to WPH phases
    constexpr int WPH = 4;
    T* WT = S.S2 + (12 * 9 + w) * HT_E + lane;
    if constexpr (MIX) {
        int mask = 0;
#pragma unroll
        for (int l = 0; l < 9; ++l) mask |= S.phm[l][lane];
        uniform = (mask & (mask - 1)) == 0;
        p0 = __ffs(mask) - 1;
        if (__syncthreads_or(!uniform) && c_mat.nphases <= WPH) {
            // indicator of phase p through the three stages: x stage at fields 12 + 3p + qx, y stage
            // at fields 3p + qy
            const int np = c_mat.nphases;
            for (int p = 0; p < np; ++p) {
                const T f[3] = {phn[0] == p ? T(1) : T(0), phn[1] == p ? T(1) : T(0), phn[2] == p ? T(1) : T(0)};
                T o[3];
                ht_val(f, o);
#pragma unroll
                for (int q = 0; q < 3; ++q) S.S2[((12 + 3 * p + q) * 9 + w) * HT_E + lane] = o[q];
            }
            ht_bar_b(lb);
            for (int p = 0; p < np; ++p) {
                const T* in = S.S2 + ((12 + 3 * p + la) * 9 + 3 * lb) * HT_E + lane;
                const T f[3] = {in[0], in[HT_E], in[2 * HT_E]};
                T o[3];
                ht_val(f, o);
#pragma unroll
                for (int q = 0; q < 3; ++q) S.S2[((3 * p + q) * 9 + w) * HT_E + lane] = o[q];
            }
            __syncthreads();   // the x-stage fields are free: the weights go there
            for (int p = 0; p < np; ++p) {
                const T* in = S.S2 + ((3 * p + lb) * 9 + la) * HT_E + lane;
                const T f[3] = {in[0], in[3 * HT_E], in[6 * HT_E]};
                T o[3];
                ht_val(f, o);
#pragma unroll
                for (int q = 0; q < 3; ++q) WT[(3 * p + q) * 9 * HT_E] = o[q];
            }
            ht_bar_a(la);   // before the pressure parts overwrite the y stage
        }
    }
    {
        // ---- pressure residual, this line's part ----
        int php[4];
#pragma unroll
        for (int p = 0; p < 4; ++p) php[p] = S.php[p][lane];
        const bool one = php[0] == p0 && php[1] == p0 && php[2] == p0 && php[3] == p0;
        T f[3];
#pragma unroll
        for (int q = 0; q < 3; ++q) f[q] = -(g[0][0][q] + g[1][1][q] + g[2][2][q]);
        if (!bulk_inf) {
            T c0, c1;
            line(PF_DP, c0, c1);
            const T ib = S.PT[PT_INVBULKDT][p0];
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                const T ze = (T)ht_x(q);
                T d = c0 + c1 * ze;
                if (a.P_old_ip) d -= ld(a.P_old_ip + e * 27 + w + 9 * q);
                if (one && consts_ok) f[q] -= d * ib;
                else f[q] -= d / (((T(1) - xi - et - ze) * (T)c_mat.bulk[php[0]] + xi * (T)c_mat.bulk[php[1]] +
                                   et * (T)c_mat.bulk[php[2]] + ze * (T)c_mat.bulk[php[3]]) * dt);
            }
        }
        if (a.temp || a.temp0) {
            T c0, c1;
            line(PF_DT, c0, c1);
            const T a0 = (T)c_mat.alpha[php[0]];
            const T ac = a0 + xi * ((T)c_mat.alpha[php[1]] - a0) + et * ((T)c_mat.alpha[php[2]] - a0), az = (T)c_mat.alpha[php[3]] - a0;
            const T idt = T(1) / dt;
#pragma unroll
            for (int q = 0; q < 3; ++q) f[q] += (ac + az * (T)ht_x(q)) * (c0 + c1 * (T)ht_x(q)) * idt;
        }
        if (a.Q) {
            T c0, c1;
            line(PF_Q, c0, c1);
#pragma unroll
            for (int q = 0; q < 3; ++q) f[q] += c0 + c1 * (T)ht_x(q);
        }
#pragma unroll
        for (int q = 0; q < 3; ++q)
            f[q] *= GEO == GEO_POINT ? (T)ld(a.geo_P + e * 27 + w + 9 * q) : Ja[9] * (wxy * (T)ht_w(q));
        const T s = f[0] + f[1] + f[2], sz = (T)HT_GA * (f[2] - f[0]);
        T* rp = S.S2 + w * HT_E + lane;   // [mode][line][lane]
        rp[0] = (T(1) - xi - et) * s - sz;
        rp[9 * HT_E] = xi * s;
        rp[18 * HT_E] = et * s;
        rp[27 * HT_E] = sz;
    }
    __syncthreads();
    if (w < 4) {
        const T* in = S.S2 + w * 9 * HT_E + lane;
        T rp = in[0];
#pragma unroll
        for (int l = 1; l < 9; ++l) rp += in[l * HT_E];
        if (act && a.write_RP) a.RP[dof] = rp;
        T pn = T(0);
        if (a.with_pnum) {
            pn = a.Pnum_in ? pin : gam * rp / mp;
            if (act && a.Pnum_out) a.Pnum_out[dof] = pn;
        }
        S.pn[w][lane] = pn;
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    if (!a.do_momentum && !a.phi) return;
    __syncthreads();   // Pnum and the stress history

    // ---- stress and reference-frame fluxes; the fluxes take the gradients' place ----
    T bq[3];
    T Pc, Pz, Nc, Nz, fc = T(0), fz = T(0), Tc = T(0), Tz = T(0);
    line(PF_P, Pc, Pz);
    if (a.Pf) line(PF_PF, fc, fz);
    if (a.temp) line(PF_T, Tc, Tz);
    {
        const T x0 = S.pn[0][lane];
        Nc = x0 + xi * (S.pn[1][lane] - x0) + et * (S.pn[2][lane] - x0);
        Nz = S.pn[3][lane] - x0;
    }
    const T EPS2 = eps2<T>();
    const bool fast = uniform && consts_ok && !a.eta_ip;
    T* own = S.S1 + el * 27 + w;   // the line's history: component c, point qz at own[c·27·32 + 9qz]
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        const T ze = (T)ht_x(q);
        const T Pq = Pc + Pz * ze;
        const T Peq = a.Pf ? Pq - (fc + fz * ze) : Pq;
        T twoe, twoe_el, rho0, alpha, beta, cC = T(0), sphi = T(0), inv_den = T(0);
        T invG = T(0);
        if (fast) {
            twoe = S.PT[PT_TWOE][p0]; twoe_el = S.PT[PT_TWOE_EL][p0];
            rho0 = S.PT[PT_RHO0][p0]; alpha = S.PT[PT_ALPHA][p0]; beta = S.PT[PT_BETA][p0];
            if (plastic) { cC = S.PT[PT_CC][p0]; sphi = S.PT[PT_SPHI][p0]; inv_den = S.PT[PT_INVDEN][p0]; }
        } else {
            T eta, rest = T(0);
            if (uniform) {
                const T sN = (T)c_tab.sumN3[w + 9 * q];
                eta = (T)c_mat.eta[p0] * sN; invG = (T)c_mat.invG[p0] * sN;
                rho0 = (T)c_mat.rho0[p0] * sN; alpha = (T)c_mat.alpha[p0] * sN; beta = (T)c_mat.beta[p0] * sN;
                if (plastic) {
                    cC = (T)c_mat.cos_phi[p0] * sN * ((T)c_mat.C[p0] * sN);
                    sphi = (T)c_mat.sin_phi[p0] * sN;
                    rest = (T)c_mat.eta_reg[p0] * sN + (T)c_mat.Kb[p0] * sN * dt * (-(T)c_mat.sin_psi[p0] * sN) * (-sphi);
                }
            } else {
                T cphi = T(0), C = T(0), spsi = T(0), ereg = T(0), Kb = T(0);
                eta = invG = rho0 = alpha = beta = T(0);
                auto add = [&](T N, int p) {
                    eta += N * (T)c_mat.eta[p]; invG += N * (T)c_mat.invG[p];
                    rho0 += N * (T)c_mat.rho0[p]; alpha += N * (T)c_mat.alpha[p]; beta += N * (T)c_mat.beta[p];
                    if (plastic) {
                        cphi += N * (T)c_mat.cos_phi[p]; sphi += N * (T)c_mat.sin_phi[p]; spsi += N * (T)c_mat.sin_psi[p];
                        C += N * (T)c_mat.C[p]; ereg += N * (T)c_mat.eta_reg[p]; Kb += N * (T)c_mat.Kb[p];
                    }
                };
                if (c_mat.nphases <= WPH) {
                    for (int p = 0; p < c_mat.nphases; ++p) add(WT[(3 * p + q) * 9 * HT_E], p);
                } else {
#pragma unroll 1
                    for (int t = 0; t < 27; ++t) add((T)c_tab.N3[w + 9 * q][c_tab.tn3[t]], S.PH[t][lane]);
                }
                cC = cphi * C;
                rest = ereg + Kb * dt * (-spsi) * (-sphi);
            }
            if (a.eta_ip) eta = ld(a.eta_ip + e * 27 + w + 9 * q);
            const T etave = invG == T(0) ? eta : T(1) / (T(1) / eta + invG / dt);
            twoe = T(2) * etave;
            twoe_el = twoe * (invG / (T(2) * dt));
            if (plastic) inv_den = T(1) / (etave + rest);
        }
        const T tr = (g[0][0][q] + g[1][1][q] + g[2][2][q]) * T(1.0 / 3.0);
        T tau[6] = {twoe * (g[0][0][q] - tr), twoe * (g[1][1][q] - tr), twoe * (g[2][2][q] - tr),
                    twoe * (T(0.5) * (g[0][1][q] + g[1][0][q])), twoe * (T(0.5) * (g[0][2][q] + g[2][0][q])),
                    twoe * (T(0.5) * (g[1][2][q] + g[2][1][q]))};
#pragma unroll
        for (int c = 0; c < 6; ++c)
            if (a.told[c]) tau[c] += twoe_el * own[c * 27 * HT_E + 9 * q];
        if (act && a.base_out) {
#pragma unroll
            for (int c = 0; c < 6; ++c) a.base_out[base_index(e, w + 9 * q, c)] = (float)tau[c];
        }
        if (plastic) {
            const T J2 = T(0.5) * (tau[0] * tau[0] + tau[1] * tau[1] + tau[2] * tau[2]) + tau[3] * tau[3] +
                         tau[4] * tau[4] + tau[5] * tau[5];
            const T tII = sqrt(J2 + EPS2);
            const T Fy = tII - cC - sphi * Peq;
            if (act && a.base_out) {
                a.base_out[base_index(e, w + 9 * q, 6)] = (float)Fy;
                // the incremental sweep's apex test (J2 < 1e-6 (C cosϕ)² in FP32) with a margin
                if (!(J2 > T(1.01e-6) * cC * cC)) { a.apex_out[tile] = 1; *a.apex_any = 1; }
            }
            const T lam = Fy * inv_den;
            if (Fy > T(0) && lam > T(0)) {
                const T f = twoe * lam / (tII + EPS2);
                tau[0] -= T(0.5) * f * tau[0]; tau[1] -= T(0.5) * f * tau[1]; tau[2] -= T(0.5) * f * tau[2];
                tau[3] -= f * tau[3]; tau[4] -= f * tau[4]; tau[5] -= f * tau[5];
            }
        }
        if (act && a.phi) {
            // shear_dissipation 3-D (shear_heating.jl:91-103)
            T told[6];
#pragma unroll
            for (int c = 0; c < 6; ++c) told[c] = a.told[c] ? own[c * 27 * HT_E + 9 * q] : T(0);
            // (1/(2GΔt) from G: 2ηve may be zero)
            const T inv2Gdt = (fast ? (T)c_mat.invG[p0] : invG) / (T(2) * dt);
            const T power = tau[0] * g[0][0][q] + tau[1] * g[1][1][q] + tau[2] * g[2][2][q] +
                            tau[3] * (g[0][1][q] + g[1][0][q]) + tau[4] * (g[0][2][q] + g[2][0][q]) +
                            tau[5] * (g[1][2][q] + g[2][1][q]);
            const T el_ = (tau[0] * (tau[0] - told[0]) + tau[1] * (tau[1] - told[1]) + tau[2] * (tau[2] - told[2]) +
                           T(2) * (tau[3] * (tau[3] - told[3]) + tau[4] * (tau[4] - told[4]) + tau[5] * (tau[5] - told[5]))) *
                          inv2Gdt;
            a.phi[e * 27 + w + 9 * q] = power - el_;
        }
        if (act && a.tau_store[0]) {   // in the history's place, copied out coalesced below
#pragma unroll
            for (int c = 0; c < 6; ++c) own[c * 27 * HT_E + 9 * q] = tau[c];
        }
        if (!a.do_momentum) continue;
        const T Ptot = (a.Pf ? Peq + (fc + fz * ze) : Pq) + (Nc + Nz * ze);
        // EOS density (momentum_residuals.jl:11-16)
        const T rhoq = rho0 * (T(1) - alpha * ((Tc + Tz * ze) - (T)c_mat.Tref) + beta * Pq);
        T J[10];
#pragma unroll
        for (int r = 0; r < 10; ++r) J[r] = GEO == GEO_POINT ? T(0) : Ja[r];
        if constexpr (GEO == GEO_POINT) load10(Gp + 90 * q, a.geo_vec, J);
        if constexpr (GEO != GEO_POINT) J[9] = Ja[9] * (wxy * (T)ht_w(q));
        bq[q] = rhoq * J[9];
        // dΩ Σ_k ∂ξ_d/∂x_k σ_kc, σ = τ − Ptot·I
        const T sg[3][3] = {{tau[0] - Ptot, tau[3], tau[4]}, {tau[3], tau[1] - Ptot, tau[5]}, {tau[4], tau[5], tau[2] - Ptot}};
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const T k0 = J[9] * J[GEO == GEO_DIAG ? 4 * d : d];
            const T k1 = J[9] * J[d + 3], k2 = J[9] * J[d + 6];
#pragma unroll
            for (int c = 0; c < 3; ++c)
                g[c][d][q] = GEO == GEO_DIAG ? k0 * sg[d][c] : k0 * sg[0][c] + k1 * sg[1][c] + k2 * sg[2][c];
        }
    }
    if (a.do_momentum)
        ht_scatter_z<T, 3>(g, [&](int c, int q) { return -(T)c_mat.g[c] * bq[q]; }, S.S2, la, lb, lane);
    __syncthreads();
    if (a.tau_store[0]) {
#pragma unroll
        for (int c = 0; c < 6; ++c)
            for (int i = threadIdx.x; i < ne * 27; i += HT_THREADS) a.tau_store[c][e0 * 27 + i] = S.S1[c * 27 * HT_E + i];
        __syncthreads();
    }
    if (!a.do_momentum) return;
    T R[3][3];
    ht_scatter_yx<T, 3>(S.S1, S.S2, la, lb, lane, R);
    // the next lane's ξ = −1 node, when it is this lane's ξ = +1 node (tiles that run along ξ), is
    // added here and one atomic per component saved; any shared node folds correctly
    const int n0n = __shfl_down_sync(0xffffffffu, node[0], 1);
    const bool fold = lane + 1 < ne && n0n == node[2];
    const bool folded = __shfl_up_sync(0xffffffffu, (int)fold, 1) && lane > 0;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const T r0n = __shfl_down_sync(0xffffffffu, R[c][0], 1);
        if (fold) R[c][2] += r0n;
        if (act) {
            if (!folded) atomic_add(a.Rv[c] + node[0], R[c][0]);
            atomic_add(a.Rv[c] + node[1], R[c][1]);
            atomic_add(a.Rv[c] + node[2], R[c][2]);
        }
    }
}

template <class T, class TG>
cudaError_t launch_hex27_residual(const H27Args<T, TG>& args, int num_sms, cudaStream_t st, bool pdl) {
    const int64_t tiles = args.tile_list ? args.tile_count : (args.nels + HT_E - 1) / HT_E;
    if (tiles < 1) return cudaSuccess;
    H27Args<T, TG> a = args;
    auto aligned = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
    a.geo_vec = aligned(a.geo_v);
    a.told_vec = 0;
    for (int c = 0; c < 6; ++c) a.told_vec |= aligned(a.told[c]) ? 1 << c : 0;
    constexpr int TWO = 2;   // blocks per SM where the mesh has tiles for them
    const bool one = sizeof(T) == 8 && tiles <= num_sms;
    const bool mix = a.phv && a.phv_layout != FEMB200_PHASE_CELL;
    constexpr int ONE = sizeof(T) == 8 ? 1 : TWO;
    auto fn = hex27_residual_kernel<T, TG, GEO_POINT, TWO, false>;
    if (!a.geo_c) {
        fn = one ? (mix ? hex27_residual_kernel<T, TG, GEO_POINT, ONE, true> : hex27_residual_kernel<T, TG, GEO_POINT, ONE, false>)
             : mix ? hex27_residual_kernel<T, TG, GEO_POINT, TWO, true> : fn;
    } else if (a.geo_diag) {
        fn = mix ? hex27_residual_kernel<T, TG, GEO_DIAG, ONE, true>
             : one ? hex27_residual_kernel<T, TG, GEO_DIAG, ONE, false> : hex27_residual_kernel<T, TG, GEO_DIAG, TWO, false>;
    } else {
        fn = mix ? hex27_residual_kernel<T, TG, GEO_AFFINE, ONE, true>
             : one ? hex27_residual_kernel<T, TG, GEO_AFFINE, ONE, false> : hex27_residual_kernel<T, TG, GEO_AFFINE, TWO, false>;
    }
    const size_t smem = sizeof(ResSmem<T>);
    const cudaError_t err = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (err != cudaSuccess) return err;
    count_launch();
    return launch_pdl(pdl, fn, dim3((unsigned)tiles), dim3(HT_THREADS), smem, st, a);
}

template cudaError_t launch_hex27_residual<double, double>(const H27Args<double, double>&, int, cudaStream_t, bool);
template cudaError_t launch_hex27_residual<float, float>(const H27Args<float, float>&, int, cudaStream_t, bool);
template cudaError_t launch_hex27_residual<double, float>(const H27Args<double, float>&, int, cudaStream_t, bool);
template cudaError_t launch_hex27_residual<float, double>(const H27Args<float, double>&, int, cudaStream_t, bool);

}  // namespace femb
