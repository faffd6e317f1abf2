// simple.cu — thread-per-element kernels: pressure scaling (setup, once per solve), the
// 2-D thermal-diffusion residual/Jacobian (3-D: thermal3d.cu) and the lithostatic pressure.
#include "kernels.cuh"

namespace femb {

__constant__ DevThermalMaterial c_tmat;

namespace {

template <int DIM> struct Tabs;
template <> struct Tabs<3> {
    static constexpr int NV = 27, NQ = 27, NP = 4;
    FEMB_D static double N(int q, int a) { return c_tab.N3[q][a]; }
    FEMB_D static double dN(int q, int a, int j) { return c_tab.dN3[q][a][j]; }
    FEMB_D static double NPq(int q, int p) { return c_tab.NP3[q][p]; }
    FEMB_D static double sumN(int q) { return c_tab.sumN3[q]; }
};
template <> struct Tabs<2> {
    static constexpr int NV = 9, NQ = 9, NP = 3;
    FEMB_D static double N(int q, int a) { return c_tab.N2[q][a]; }
    FEMB_D static double dN(int q, int a, int j) { return c_tab.dN2[q][a][j]; }
    FEMB_D static double NPq(int q, int p) { return c_tab.NP2[q][p]; }
    FEMB_D static double sumN(int q) { return c_tab.sumN2[q]; }
};

// interp2ip_phase over the element's velocity-node phases (utils.jl:37-44).
template <int DIM, class T>
FEMB_D T interp(int q, const double* var, const int* ph) {
    T out = T(0);
#pragma unroll
    for (int a = 0; a < Tabs<DIM>::NV; ++a) out += (T)Tabs<DIM>::N(q, a) * (T)var[ph[a]];
    return out;
}

// viscosity_weighted_pressure_scaling_kernel! (pressure_scaling.jl:166-211);
// Q9 and Hex27 use the positive Jacobi weight N² (:201-203).
template <int DIM, class T, class TG>
__global__ void pressure_scaling_kernel(const int32_t* el2n, const int32_t* dofsP, const TG* geo_P, const int32_t* phv,
                                        int phv_layout, const T* eta_ip, int use_eta_ip, T* MP, T* gP, int64_t nels,
                                        T gfact, T dt) {
    using TB = Tabs<DIM>;
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= nels) return;
    int ph[TB::NV];
    for (int a = 0; a < TB::NV; ++a)
        ph[a] = phase_of(phv, phv_layout, (int64_t)__ldg(el2n + TB::NV * e + a), a, e, TB::NV);
    int dof[TB::NP];
    for (int p = 0; p < TB::NP; ++p) dof[p] = __ldg(dofsP + TB::NP * e + p) - 1;
    for (int q = 0; q < TB::NQ; ++q) {
        const T dO = (T)ld(geo_P + e * TB::NQ + q);
        const T etaq = use_eta_ip ? ld(eta_ip + e * TB::NQ + q) : interp<DIM, T>(q, c_mat.eta_scaling, ph);
        const T gnum = gfact * etaq;
        const T bq = interp<DIM, T>(q, c_mat.inv_Kscale, ph);
        const T gphy = bq == T(0) ? gnum : dt / bq;
        const T gq = gphy * gnum / (gphy + gnum);
        for (int p = 0; p < TB::NP; ++p) {
            const T NPv = (T)TB::NPq(q, p);
            const T w = NPv * NPv * dO;
            atomic_add(MP + dof[p], w);
            atomic_add(gP + dof[p], w * gq);
        }
    }
}

template <class T>
__global__ void scaling_finalize_kernel(T* gP, const T* MP, int64_t n) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) gP[i] = MP[i] == T(0) ? T(0) : gP[i] / MP[i];
}

// Thermal element residual (heat_diffusion/assembly/residual.jl:58-87; DIM = 2) and the
// exact Jacobian row sums / diagonal of its ForwardDiff diagnostics (:30-48).
template <int DIM, class T, class TG>
__global__ void thermal_kernel(ThermalArgs<T, TG> a) {
    using TB = Tabs<DIM>;
    constexpr int NV = TB::NV, NQ = TB::NQ, S = DIM * DIM + 1;
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (a.group ? a.ngroup : a.nels)) return;
    const int64_t e = a.group ? (int64_t)__ldg(a.group + t) - 1 : t;
    int node[NV], ph[NV];
    T Tl[NV];
    for (int i = 0; i < NV; ++i) {
        node[i] = __ldg(a.el2n + NV * e + i) - 1;
        Tl[i] = ld(a.Tn + node[i]);
        ph[i] = phase_of(a.ph, a.ph_layout, (int64_t)node[i] + 1, i, e, NV);
    }
    const TG* G = a.geo + e * NQ * S;
    T R[NV];
    for (int i = 0; i < NV; ++i) R[i] = T(0);
    for (int q = 0; q < NQ; ++q) {
        const TG* g = G + q * S;
        const T dO = (T)g[DIM * DIM];
        T Tq = T(0), Pq = T(0), T0q = T(0), sq = T(0), kq = T(0), aq = T(0), bq = T(0), rq = T(0), cq = T(0);
        for (int i = 0; i < NV; ++i) {
            const T N = (T)TB::N(q, i);
            const int n = node[i];
            Tq += N * Tl[i];
            Pq += N * (a.P ? ld(a.P + n) : T(0));
            T0q += N * ld(a.T0 + n);
            sq += N * (a.src ? ld(a.src + n) : T(0));
            kq += N * (T)c_tmat.k[ph[i]];
            aq += N * (T)c_tmat.alpha[ph[i]];
            bq += N * (T)c_tmat.beta[ph[i]];
            rq += N * (T)c_tmat.rho0[ph[i]];
            cq += N * (T)c_tmat.Cp[ph[i]];
        }
        const T rhoq = rq * (T(1) - aq * (Tq - a.Tref) + bq * Pq);
        const T dtrc = a.dt / (rhoq * cq);
        T gT[DIM];
        for (int k = 0; k < DIM; ++k) gT[k] = T(0);
        T dn[NV][DIM];
        for (int i = 0; i < NV; ++i)
            for (int k = 0; k < DIM; ++k) {
                T s = T(0);
                for (int j = 0; j < DIM; ++j) s += (T)TB::dN(q, i, j) * (T)g[j + DIM * k];
                dn[i][k] = s;
                gT[k] += s * Tl[i];
            }
        const T Phi = a.src_ip ? ld(a.src_ip + e * NQ + q) : T(0);
        const T Hq = a.src_ip ? dtrc * Phi : T(0);
        const T rate = T0q - Tq + dtrc * sq + Hq;
        for (int i = 0; i < NV; ++i) {
            T KT = T(0);
            for (int k = 0; k < DIM; ++k) KT += dn[i][k] * gT[k];
            KT = kq * KT;
            R[i] += rate * (T)TB::N(q, i) * dO - dtrc * KT * dO;
        }
    }
    for (int i = 0; i < NV; ++i) {
        if (a.group) a.R[node[i]] += R[i];
        else atomic_add(a.R + node[i], R[i]);
    }
    if (!a.jac) return;
    // Jacobian rows: J[i][b] = Σ_q dΩ [ (−N_b + ∂dtrc_b (s_q + Φ_q)) N_i − ∂dtrc_b KT_i − dtrc k ∇N_i·∇N_b ]
    // with ∂dtrc/∂T_b = dtrc·αq·ρ0q·N_b/ρq (EOS dependence of the density).
    for (int i = 0; i < NV; ++i) {
        T Jrow[NV];
        for (int b = 0; b < NV; ++b) Jrow[b] = T(0);
        for (int q = 0; q < NQ; ++q) {
            const TG* g = G + q * S;
            const T dO = (T)g[DIM * DIM];
            T Tq = T(0), Pq = T(0), sq = T(0), kq = T(0), aq = T(0), bq = T(0), rq = T(0), cq = T(0);
            T gT[DIM];
            for (int k = 0; k < DIM; ++k) gT[k] = T(0);
            for (int m = 0; m < NV; ++m) {
                const T N = (T)TB::N(q, m);
                Tq += N * Tl[m];
                Pq += N * (a.P ? ld(a.P + node[m]) : T(0));
                sq += N * (a.src ? ld(a.src + node[m]) : T(0));
                kq += N * (T)c_tmat.k[ph[m]]; aq += N * (T)c_tmat.alpha[ph[m]]; bq += N * (T)c_tmat.beta[ph[m]];
                rq += N * (T)c_tmat.rho0[ph[m]]; cq += N * (T)c_tmat.Cp[ph[m]];
                for (int k = 0; k < DIM; ++k) {
                    T s = T(0);
                    for (int jj = 0; jj < DIM; ++jj) s += (T)TB::dN(q, m, jj) * (T)g[jj + DIM * k];
                    gT[k] += s * Tl[m];
                }
            }
            const T rhoq = rq * (T(1) - aq * (Tq - a.Tref) + bq * Pq);
            const T dtrc = a.dt / (rhoq * cq);
            const T Ni = (T)TB::N(q, i);
            const T Phi = a.src_ip ? ld(a.src_ip + e * NQ + q) : T(0);
            T dni[DIM];
            for (int k = 0; k < DIM; ++k) {
                dni[k] = T(0);
                for (int jj = 0; jj < DIM; ++jj) dni[k] += (T)TB::dN(q, i, jj) * (T)g[jj + DIM * k];
            }
            T KTi = T(0);
            for (int k = 0; k < DIM; ++k) KTi += dni[k] * gT[k];
            const T cfac = dtrc * aq * rq / rhoq;   // ∂dtrc/∂T_b = cfac·N_b
            for (int b = 0; b < NV; ++b) {
                const T Nb = (T)TB::N(q, b);
                const T ddt = cfac * Nb;
                T KK = T(0);
                for (int k = 0; k < DIM; ++k) {
                    T dnb = T(0);
                    for (int jj = 0; jj < DIM; ++jj) dnb += (T)TB::dN(q, b, jj) * (T)g[jj + DIM * k];
                    KK += dni[k] * dnb;
                }
                Jrow[b] += ((-Nb + ddt * (sq + Phi)) * Ni - ddt * kq * KTi - dtrc * kq * KK) * dO;
            }
        }
        T row = T(0);
        for (int b = 0; b < NV; ++b) row += fabs(Jrow[b]);
        if (a.group) {
            a.dRdT[node[i]] += row;
            a.PC[node[i]] += fabs(Jrow[i]);
        } else {
            atomic_add(a.dRdT + node[i], row);
            atomic_add(a.PC + node[i], fabs(Jrow[i]));
        }
    }
}

// Lithostatic-pressure element residual (lp_integrate_residual,
// src/lithostatic_pressure/assembly/residual.jl:48-63): R_i = Σ_q (ρ_q ∇N_i·g − ∇N_i·∇P) dΩ
// with ρ_q = ρ0_q (1 − α_q (T_q − Tref) + β_q P_q), and the row sums and diagonal of its
// Jacobian (the ForwardDiff diagnostics of lp_element_jacobian, :22-36), in closed form:
// ∂R_i/∂P_b = Σ_q (ρ0_q β_q N_b ∇N_i·g − ∇N_i·∇N_b) dΩ.
template <int DIM>
__global__ void lithostatic_kernel(LithoArgs a) {
    using TB = Tabs<DIM>;
    constexpr int NV = TB::NV, NQ = TB::NQ, S = DIM * DIM + 1;
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= a.nels) return;
    int node[NV], ph[NV];
    double Pl[NV], Tl[NV];
    for (int i = 0; i < NV; ++i) {
        node[i] = __ldg(a.el2n + NV * e + i) - 1;
        Pl[i] = a.P[node[i]];
        Tl[i] = a.Tn ? __ldg(a.Tn + node[i]) : 0.0;
        ph[i] = phase_of(a.ph, a.ph_layout, (int64_t)node[i] + 1, i, e, NV);
    }
    const double* G = a.geo + e * NQ * S;
    double R[NV];
    for (int i = 0; i < NV; ++i) R[i] = 0.0;
    for (int q = 0; q < NQ; ++q) {
        const double* g = G + q * S;
        const double dO = g[DIM * DIM];
        double Tq = 0, Pq = 0, aq = 0, bq = 0, rq = 0;
        for (int i = 0; i < NV; ++i) {
            const double N = TB::N(q, i);
            Tq += N * Tl[i]; Pq += N * Pl[i];
            aq += N * a.alpha[ph[i]]; bq += N * a.beta[ph[i]]; rq += N * a.rho0[ph[i]];
        }
        const double rho = rq * (1.0 - aq * (Tq - a.Tref) + bq * Pq);
        double dn[NV][DIM], gP[DIM];
        for (int k = 0; k < DIM; ++k) gP[k] = 0.0;
        for (int i = 0; i < NV; ++i)
            for (int k = 0; k < DIM; ++k) {
                double s = 0;
                for (int j = 0; j < DIM; ++j) s += TB::dN(q, i, j) * g[j + DIM * k];
                dn[i][k] = s;
                gP[k] += s * Pl[i];
            }
        for (int i = 0; i < NV; ++i) {
            double ng = 0, np = 0;
            for (int k = 0; k < DIM; ++k) { ng += dn[i][k] * a.g[k]; np += dn[i][k] * gP[k]; }
            R[i] += (rho * ng - np) * dO;
        }
    }
    for (int i = 0; i < NV; ++i) atomicAdd(a.R + node[i], R[i]);
    if (!a.jac) return;
    for (int i = 0; i < NV; ++i) {
        double Jrow[NV];
        for (int b = 0; b < NV; ++b) Jrow[b] = 0.0;
        for (int q = 0; q < NQ; ++q) {
            const double* g = G + q * S;
            const double dO = g[DIM * DIM];
            double bq = 0, rq = 0;
            for (int m = 0; m < NV; ++m) {
                const double N = TB::N(q, m);
                bq += N * a.beta[ph[m]]; rq += N * a.rho0[ph[m]];
            }
            double dni[DIM], ng = 0;
            for (int k = 0; k < DIM; ++k) {
                double s = 0;
                for (int j = 0; j < DIM; ++j) s += TB::dN(q, i, j) * g[j + DIM * k];
                dni[k] = s;
                ng += s * a.g[k];
            }
            const double cf = rq * bq * ng;
            for (int b = 0; b < NV; ++b) {
                double kk = 0;
                for (int k = 0; k < DIM; ++k) {
                    double s = 0;
                    for (int j = 0; j < DIM; ++j) s += TB::dN(q, b, j) * g[j + DIM * k];
                    kk += dni[k] * s;
                }
                Jrow[b] += (cf * TB::N(q, b) - kk) * dO;
            }
        }
        double row = 0;
        for (int b = 0; b < NV; ++b) row += fabs(Jrow[b]);
        atomicAdd(a.dRdP + node[i], row);
        atomicAdd(a.PC + node[i], fabs(Jrow[i]));
    }
}

inline unsigned nb(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }

}  // namespace

cudaError_t launch_lithostatic(const LithoArgs& a, cudaStream_t st) {
    if (a.nels <= 0) return cudaSuccess;
    count_launch();
    if (a.dim == 3) lithostatic_kernel<3><<<nb(a.nels, 64), 64, 0, st>>>(a);
    else lithostatic_kernel<2><<<nb(a.nels, 128), 128, 0, st>>>(a);
    return cudaGetLastError();
}

template <class T, class TG>
cudaError_t launch_pressure_scaling(int dim, const int32_t* el2n, const int32_t* dofsP, const TG* geo_P,
                                    const int32_t* phv, int phv_layout, const T* eta_ip, int use_eta_ip, T* MP, T* gP,
                                    int64_t nels, int64_t nnodesP, T gfact, T dt, cudaStream_t st) {
    count_launch();
    if (dim == 3)
        pressure_scaling_kernel<3, T, TG><<<nb(nels, 128), 128, 0, st>>>(el2n, dofsP, geo_P, phv, phv_layout, eta_ip,
                                                                         use_eta_ip, MP, gP, nels, gfact, dt);
    else
        pressure_scaling_kernel<2, T, TG><<<nb(nels, 128), 128, 0, st>>>(el2n, dofsP, geo_P, phv, phv_layout, eta_ip,
                                                                         use_eta_ip, MP, gP, nels, gfact, dt);
    count_launch();
    scaling_finalize_kernel<T><<<nb(nnodesP, 256), 256, 0, st>>>(gP, MP, nnodesP);
    return cudaGetLastError();
}

template <class T, class TG>
cudaError_t launch_thermal(const ThermalArgs<T, TG>& a, int num_sms, cudaStream_t st, bool pdl) {
    const int64_t n = a.group ? a.ngroup : a.nels;
    if (n <= 0) return cudaSuccess;
    count_launch();
    if (a.dim == 3) return launch_thermal3d<T, TG>(a, num_sms, st, pdl);
    thermal_kernel<2, T, TG><<<nb(n, 128), 128, 0, st>>>(a);
    return cudaGetLastError();
}

#define FEMB_INST2(T, TG)                                                                                            \
    template cudaError_t launch_pressure_scaling<T, TG>(int, const int32_t*, const int32_t*, const TG*,             \
                                                        const int32_t*, int, const T*, int, T*, T*, int64_t,       \
                                                        int64_t, T, T, cudaStream_t);                              \
    template cudaError_t launch_thermal<T, TG>(const ThermalArgs<T, TG>&, int, cudaStream_t, bool);
FEMB_INST2(double, double)
FEMB_INST2(float, float)
FEMB_INST2(double, float)
FEMB_INST2(float, double)
#undef FEMB_INST2

}  // namespace femb
