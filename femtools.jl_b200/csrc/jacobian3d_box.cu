// jacobian3d_box.cu — augmented momentum-Jacobian diagnostics in FP64 on axis-aligned Hex27 boxes with
// one phase per cell (momentum_residuals.jl:998-1117; jacobian3d.cu takes every other mesh and
// FP32). Tiles of 32 elements, nine warps, lane = element (hex27_tile.cuh), two kernels:
//
// * Where no point of a tile yields, an element's tangent is one viscosity and its J⁻¹ (its centre's: the
//   points agree to rounding, GEO_NOT_BOX) times integrals of products of one-dimensional basis functions:
//   the 81×81 entries come from nine products per node pair, with no quadrature and no exchange. Warp = node
//   line, whose three nodes' rows it sums. Bound by FP64 issue (87 operations per pair; 74 % of the pipe).
//   169 us at 32³ with a viscosity per point, where 81 columns an element took 1 382. Error against 64-bit
//   sums at the points 1.8e-15 at 32×31×33 (1.3e-15 by 81 columns).
// * A tile with a yielding point is marked and taken by the second kernel: 81 columns through the
//   transposed contraction, warp = line of points and nodes. The exchange buffers are double, so that
//   two barriers of 96 threads per column suffice: writing a buffer again needs the barriers
//   of the column between. The tangents and the gradients of the columns take each point's geometry. Bound
//   by shared-memory bandwidth (90 accesses of 256 B per warp and column).
//   1 019 us at 32×31×33 with every tile yielding (59 % of the shared-memory cycles, 40 % of FP64's; 894 with
//   the centre's J⁻¹, half as far again from 64 bits; three elements to a warp took 1 736).
#include <cstddef>
#include <type_traits>
#include "hex27_tile.cuh"
#include "kernels.cuh"
#include "rheology.cuh"

namespace femb {
namespace {

// integrals of two and points' values of one of the basis functions (L) and their derivatives (D)
FEMB_HD constexpr double jb_int(int da, int db, int i, int j) {
    double s = 0;
    for (int q = 0; q < 3; ++q) s += ht_w(q) * (da ? ht_D(q, i) : ht_L(q, i)) * (db ? ht_D(q, j) : ht_L(q, j));
    return s;
}
// Σ_q w_q N^P_p ∂N_a/∂ξ_c in one entry: products of the moments of order m of L or D
FEMB_HD constexpr double jb_mom(int m, int d, int i) {
    double s = 0;
    for (int q = 0; q < 3; ++q) s += ht_w(q) * (m ? ht_x(q) : 1.0) * (d ? ht_D(q, i) : ht_L(q, i));
    return s;
}

struct JbTab {
    double K[4][3][27];       // Σ_q w_q N^P_p(q) ∂N_a/∂ξ_c(q), a in tensor order
    // η- and ζ-factors of ∫ ∂_kN_a ∂_lN_b, pairs (k, l) xx yy zz xy yx xz zx yz zy: [pair][i + 3j of a][of b]
    double YZ[9][9][9];
};

__device__ void jb_tables(JbTab& t, bool yz) {
    __shared__ double I[4][3][3], M[4][3];   // [2·da + db], [2·m + d]
    if (threadIdx.x < 36) {
        const int k = threadIdx.x / 9, i = threadIdx.x % 9 / 3, j = threadIdx.x % 3;
        I[k][i][j] = jb_int(k / 2, k % 2, i, j);
    } else if (threadIdx.x < 48) {
        const int k = (threadIdx.x - 36) / 3;
        M[k][threadIdx.x % 3] = jb_mom(k / 2, k % 2, threadIdx.x % 3);
    }
    __syncthreads();
    for (int n = threadIdx.x; n < 324; n += HT_THREADS) {
        const int p = n / 81, c = n / 27 % 3, a = n % 27, ia[3] = {a % 3, a / 3 % 3, a / 9};
        auto mom = [&](int r) {   // the moment along direction r (−1: none)
            double x = 1;
            for (int d = 0; d < 3; ++d) x *= M[2 * (d == r) + (d == c)][ia[d]];
            return x;
        };
        (&t.K[0][0][0])[n] = p == 0 ? mom(-1) - mom(0) - mom(1) - mom(2) : mom(p - 1);
    }
    if (yz)
        for (int n = threadIdx.x; n < 729; n += HT_THREADS) {
            constexpr int KL[9][2] = {{0, 0}, {1, 1}, {2, 2}, {0, 1}, {1, 0}, {0, 2}, {2, 0}, {1, 2}, {2, 1}};
            const int r = n / 81, a = n / 9 % 9, b = n % 9, k = KL[r][0], l = KL[r][1];
            (&t.YZ[0][0][0])[n] = I[2 * (k == 1) + (l == 1)][a % 3][b % 3] * I[2 * (k == 2) + (l == 2)][a / 3][b / 3];
        }
}

struct JbElastic {
    JbTab tab;
    double mx[9][HT_E];
    double S1[HT_S1], S2[HT_S2];   // plastic materials only (the trial stress)
};
struct JbGeneral {
    double S1[2][HT_S1], S2[2][HT_S2];
    JbTab tab;
    double mx[9][HT_E];
};
static_assert(sizeof(JbGeneral) <= 227 * 1024 - 1024 && 2 * (sizeof(JbElastic) + 2048) <= 228 * 1024, "shared memory");

// What both kernels load of the thread's element.
struct JbElem {
    int64_t e0, e;
    int ne, lane, w, la, lb, node[3], p0;
    bool act;
    double J[3], detJ, G[4];   // G: γP/M_P
    double eta;                // the element's largest viscosity
};
template <class TG>
FEMB_D JbElem jb_load(const H27JacArgs<double, TG>& a, const double* geo_c, double (&mx)[9][HT_E]) {
    JbElem t;
    t.lane = threadIdx.x & 31; t.w = ht_warp(); t.la = t.w % 3; t.lb = t.w / 3;
    t.e0 = (int64_t)blockIdx.x * HT_E;
    t.ne = (int)(a.nels - t.e0 < HT_E ? a.nels - t.e0 : HT_E);
    t.act = t.lane < t.ne;
    t.e = t.e0 + (t.act ? t.lane : t.ne - 1);   // lanes past the end repeat the last element
#pragma unroll
    for (int i = 0; i < 3; ++i) t.node[i] = __ldg(a.el2n + 27 * t.e + c_tab.tn3[i + 3 * t.w]) - 1;
#pragma unroll
    for (int d = 0; d < 3; ++d) t.J[d] = ld(geo_c + t.e * 10 + 4 * d);
    t.detJ = ld(geo_c + t.e * 10 + 9);
    t.p0 = a.phv ? __ldg(a.phv + t.e) - 1 : 0;
#pragma unroll
    for (int p = 0; p < 4; ++p) {
        const int dof = __ldg(a.dofsP + 4 * t.e + p) - 1;
        t.G[p] = ld(a.gammaP + dof) / ld(a.MP + dof);
    }
    // element-max viscosity η_pc (_element_max_phase_property, momentum_residuals.jl:36-44)
    if (a.eta_ip) {
        double m = -INFINITY;
#pragma unroll
        for (int q = 0; q < 3; ++q) m = fmax(m, ld(a.eta_ip + t.e * 27 + t.w + 9 * q));
        mx[t.w][t.lane] = m;
        __syncthreads();
#pragma unroll
        for (int l = 0; l < 9; ++l) m = fmax(m, mx[l][t.lane]);
        t.eta = m;
    } else t.eta = c_mat.eta[t.p0];
    return t;
}

// The geometry of the line's point qz: J⁻¹'s diagonal at 0, 4, 8 and dΩ at 9.
template <class TG>
FEMB_D const TG* jb_point(const H27JacArgs<double, TG>& a, const JbElem& t, int q) { return a.geo_v + (t.e * 27 + t.w + 9 * q) * 10; }

// Trial stress, yield value and its norm at the line's points.
struct JbTrial {
    double t[6], tII, Fy;
};
template <class TG, class Fn>
FEMB_D void jb_trial(const H27JacArgs<double, TG>& a, const JbElem& t, double etave, double* S1, double* S2, Fn point) {
    double g[3][3][3];
    {
        double v[3][3];
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int c = 0; c < 3; ++c) v[c][i] = ld(a.v[c] + t.node[i]);
        ht_gradient<double, 3>(v, S1, S2, t.la, t.lb, t.lane, g);
    }
    double P[4];
#pragma unroll
    for (int p = 0; p < 4; ++p) {
        const int dof = __ldg(a.dofsP + 4 * t.e + p) - 1;
        P[p] = ld(a.P + dof);
        if (a.Pf) P[p] -= ld(a.Pf + dof);
    }
    const double xi = ht_xr<double>(t.la), et = ht_xr<double>(t.lb);
    const double twoe = 2.0 * etave, inv2Gdt = c_mat.invG[t.p0] / (2.0 * a.dt);
    const double cC = c_mat.cos_phi[t.p0] * c_mat.C[t.p0], sphi = c_mat.sin_phi[t.p0];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        const TG* G = jb_point(a, t, q);
        const double Jq[3] = {(double)ld(G), (double)ld(G + 4), (double)ld(G + 8)};
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int k = 0; k < 3; ++k) g[c][k][q] *= Jq[k];
        const double tr = (g[0][0][q] + g[1][1][q] + g[2][2][q]) * (1.0 / 3.0);
        JbTrial r;
        const double ep[6] = {g[0][0][q] - tr, g[1][1][q] - tr, g[2][2][q] - tr, 0.5 * (g[0][1][q] + g[1][0][q]),
                              0.5 * (g[0][2][q] + g[2][0][q]), 0.5 * (g[1][2][q] + g[2][1][q])};
#pragma unroll
        for (int c = 0; c < 6; ++c)
            r.t[c] = twoe * (ep[c] + (a.told[c] ? ld(a.told[c] + t.e * 27 + t.w + 9 * q) * inv2Gdt : 0.0));
        r.tII = sqrt(0.5 * (r.t[0] * r.t[0] + r.t[1] * r.t[1] + r.t[2] * r.t[2]) + r.t[3] * r.t[3] + r.t[4] * r.t[4] +
                     r.t[5] * r.t[5] + eps2<double>());
        const double Peq = P[0] + xi * (P[1] - P[0]) + et * (P[2] - P[0]) + ht_x(q) * (P[3] - P[0]);
        r.Fy = r.tII - cC - sphi * Peq;
        point(q, r);
    }
}

template <class TG, bool PLASTIC>
__global__ void __launch_bounds__(HT_THREADS, 2) jac_box_elastic_kernel(const H27JacArgs<double, TG> a,
                                                                       const double* __restrict__ geo_c, uint8_t* general) {
    extern __shared__ __align__(16) unsigned char jb_smem[];
    JbElastic& S = *reinterpret_cast<JbElastic*>(jb_smem);
    jb_tables(S.tab, true);
    const JbElem t = jb_load(a, geo_c, S.mx);
    const double etave = 1.0 / (1.0 / t.eta + c_mat.invG[t.p0] / a.dt);
    if constexpr (PLASTIC) {
        bool yields = false;
        jb_trial(a, t, etave, S.S1, S.S2, [&](int, const JbTrial& r) { yields = yields || r.Fy > 0.0; });
        const bool any = __syncthreads_or(t.act && yields) != 0;
        if (threadIdx.x == 0) general[blockIdx.x] = any ? 1 : 0;
        if (any) return;
    } else {
        __syncthreads();
    }
    const double E = 2.0 * etave * t.detJ;
    const double e00 = E * t.J[0] * t.J[0], e11 = E * t.J[1] * t.J[1], e22 = E * t.J[2] * t.J[2], e01 = E * t.J[0] * t.J[1],
                 e02 = E * t.J[0] * t.J[2], e12 = E * t.J[1] * t.J[2];
    const double hJ[3] = {t.detJ * t.J[0], t.detJ * t.J[1], t.detJ * t.J[2]};
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        // γP/M_P ∂RP/∂v of the row's node, the element's own factors taken out
        double RA[3][4];
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int p = 0; p < 4; ++p) RA[c][p] = t.G[p] * S.tab.K[p][c][i + 3 * t.w];
        double rows[3] = {0, 0, 0}, diag[3] = {0, 0, 0};
#pragma unroll 1
        for (int b2 = 0; b2 < 9; ++b2) {
            auto yz = [&](int r) { return S.tab.YZ[r][t.w][b2]; };
            const double xx = e00 * yz(0), yy = e11 * yz(1), zz = e22 * yz(2), xy = e01 * yz(3), yx = e01 * yz(4),
                         xz = e02 * yz(5), zx = e02 * yz(6), yzf = e12 * yz(7), zyf = e12 * yz(8);
#pragma unroll
            for (int bx = 0; bx < 3; ++bx) {
                constexpr double third = 1.0 / 3.0, sixth = 1.0 / 6.0;
                const double LL = jb_int(0, 0, i, bx), LD = jb_int(0, 1, i, bx), DL = jb_int(1, 0, i, bx), DD = jb_int(1, 1, i, bx);
                // G[k][l] = 2ηve ∫ ∂_kN_a ∂_lN_b
                const double G[3][3] = {{DD * xx, DL * xy, DL * xz}, {LD * yx, LL * yy, LL * yzf}, {LD * zx, LL * zyf, LL * zz}};
                const double half = 0.5 * (G[0][0] + G[1][1] + G[2][2]);
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    double kb[4];
#pragma unroll
                    for (int p = 0; p < 4; ++p) kb[p] = S.tab.K[p][j][bx + 3 * b2];
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        const double pn = RA[c][0] * kb[0] + RA[c][1] * kb[1] + RA[c][2] * kb[2] + RA[c][3] * kb[3];
                        const double k = fabs((c == j ? half + sixth * G[c][c] : 0.5 * G[j][c] - third * G[c][j]) + hJ[c] * hJ[j] * pn);
                        rows[c] += k;
                        if (c == j && bx == i && b2 == t.w) diag[c] = k;
                    }
                }
            }
        }
        if (t.act) {
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                atomic_add(a.dRdv[c] + t.node[i], rows[c]);
                atomic_add(a.PC[c] + t.node[i], diag[c]);
            }
        }
    }
}

// The ζ stage of the transposed contraction (ht_scatter_z without a value density).
FEMB_D void jb_scatter_z(const double (&F)[3][3][3], double* S2, int w, int lane) {
    double* o = S2 + w * HT_E + lane;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        double z0[3], z1[3], z2[3];
        ht_val_t(F[c][0], z0);
        ht_val_t(F[c][1], z1);
        ht_der_t(F[c][2], z2);
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            o[((i * 3 + c) * 3 + 0) * 9 * HT_E] = z0[i];
            o[((i * 3 + c) * 3 + 1) * 9 * HT_E] = z1[i];
            o[((i * 3 + c) * 3 + 2) * 9 * HT_E] = z2[i];
        }
    }
}

template <class TG>
__global__ void __launch_bounds__(HT_THREADS, 1) jac_box_general_kernel(const H27JacArgs<double, TG> a,
                                                                       const double* __restrict__ geo_c, const uint8_t* general) {
    extern __shared__ __align__(16) unsigned char jb_smem[];
    JbGeneral& S = *reinterpret_cast<JbGeneral*>(jb_smem);
    if (!__ldg(general + blockIdx.x)) return;
    jb_tables(S.tab, false);
    const JbElem t = jb_load(a, geo_c, S.mx);
    const double etave = 1.0 / (1.0 / t.eta + c_mat.invG[t.p0] / a.dt);
    const double xi = ht_xr<double>(t.la), et = ht_xr<double>(t.lb);
    // A point's tangent: δτ_c = e_c δε_c + κ h_c (h·δε), e the normal or shear value, h = (½τ, τ) of
    // the trial stress; dΩ is in e and κ. Linearised radial return (rheology.jl:441-472).
    double en[3], es[3], kap[3], h[3][6], wJ[3], Jp[3][3];
    {
        const double rest = c_mat.eta_reg[t.p0] + c_mat.Kb[t.p0] * a.dt * (-c_mat.sin_psi[t.p0]) * (-c_mat.sin_phi[t.p0]);
        const double iden = 1.0 / (etave + rest), twoe = 2.0 * etave;
        jb_trial(a, t, etave, S.S1[0], S.S2[0], [&](int q, const JbTrial& r) {
            const TG* G = jb_point(a, t, q);
#pragma unroll
            for (int k = 0; k < 3; ++k) Jp[q][k] = (double)ld(G + 4 * k);
            wJ[q] = (double)ld(G + 9);
            const double lam = r.Fy > 0.0 ? r.Fy * iden : 0.0;
            const double its = 1.0 / (r.tII + eps2<double>());
            const bool y = lam > 0.0;
            en[q] = wJ[q] * twoe * (y ? 1.0 - twoe * lam * 0.5 * its : 1.0);
            es[q] = wJ[q] * twoe * (y ? 1.0 - twoe * lam * its : 1.0);
            kap[q] = y ? wJ[q] * twoe * twoe * (its / r.tII) * (lam * its - iden) : 0.0;
#pragma unroll
            for (int c = 0; c < 6; ++c) h[q][c] = y ? (c < 3 ? 0.5 * r.t[c] : r.t[c]) : 0.0;
        });
    }
    double rows[3][3];
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int i = 0; i < 3; ++i) rows[c][i] = 0.0;
    __syncthreads();
    int buf = 0;
#pragma unroll 1
    for (int b = 0; b < 27; ++b) {
        const int bx = b % 3, by = b / 3 % 3, bz = b / 9;
        const double Lx = c_tab.B[t.la][bx], Ly = c_tab.B[t.lb][by];
        const double s0 = c_tab.Dd[t.la][bx] * Ly, s1 = Lx * c_tab.Dd[t.lb][by], s2 = Lx * Ly;
        double dn[3][3];   // [point][direction]
#pragma unroll
        for (int q = 0; q < 3; ++q) { dn[q][0] = Jp[q][0] * (s0 * c_tab.B[q][bz]); dn[q][1] = Jp[q][1] * (s1 * c_tab.B[q][bz]); dn[q][2] = Jp[q][2] * (s2 * c_tab.Dd[q][bz]); }
        auto column = [&](auto jc) {
            constexpr int j = decltype(jc)::value, m = (j + 1) % 3, l = (j + 2) % 3;
            // Voigt places of the pairs (j, m), (j, l), (m, l)
            constexpr int V[3][3] = {{0, 3, 4}, {3, 1, 5}, {4, 5, 2}};
            // −δPnum at the points: γP/M_P ∂RP/∂v through N^P
            double bp[4];
#pragma unroll
            for (int p = 0; p < 4; ++p) bp[p] = t.G[p] * (S.tab.K[p][j][b] * (t.detJ * t.J[j]));
            const double c0 = bp[0] + xi * (bp[1] - bp[0]) + et * (bp[2] - bp[0]), c1 = bp[3] - bp[0];
            double F[3][3][3];
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                const double d = dn[q][j], th = d * (1.0 / 3.0), np = wJ[q] * (c0 + c1 * ht_x(q));
                const double (&hq)[6] = h[q];
                const double wv = kap[q] * ((hq[j] - (hq[0] + hq[1] + hq[2]) * (1.0 / 3.0)) * d +
                                            0.5 * (hq[V[j][m]] * dn[q][m] + hq[V[j][l]] * dn[q][l]));
                double sg[6];
                sg[j] = en[q] * (d - th) + hq[j] * wv + np;
                sg[m] = hq[m] * wv - en[q] * th + np;
                sg[l] = hq[l] * wv - en[q] * th + np;
                sg[V[j][m]] = es[q] * (0.5 * dn[q][m]) + hq[V[j][m]] * wv;
                sg[V[j][l]] = es[q] * (0.5 * dn[q][l]) + hq[V[j][l]] * wv;
                sg[V[m][l]] = hq[V[m][l]] * wv;
#pragma unroll
                for (int c = 0; c < 3; ++c)
#pragma unroll
                    for (int k = 0; k < 3; ++k) F[c][k][q] = Jp[q][k] * sg[V[c][k]];
            }
            jb_scatter_z(F, S.S2[buf], t.w, t.lane);
            ht_bar_a(t.la);
            double R[3][3];
            ht_scatter_yx<double, 3>(S.S1[buf], S.S2[buf], t.la, t.lb, t.lane, R);
            buf ^= 1;
#pragma unroll
            for (int c = 0; c < 3; ++c)
#pragma unroll
                for (int i = 0; i < 3; ++i) rows[c][i] += fabs(R[c][i]);
            if (b / 3 == t.w) {
#pragma unroll
                for (int i = 0; i < 3; ++i)
                    if (bx == i && t.act) atomic_add(a.PC[j] + t.node[i], fabs(R[j][i]));
            }
        };
        column(std::integral_constant<int, 0>{});
        column(std::integral_constant<int, 1>{});
        column(std::integral_constant<int, 2>{});
    }
    if (t.act) {
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int i = 0; i < 3; ++i) atomic_add(a.dRdv[c] + t.node[i], rows[c][i]);
    }
}

}  // namespace

template <class TG>
cudaError_t launch_hex27_jacobian_box(const H27JacArgs<double, TG>& a, const double* geo_c, bool plastic, uint8_t* general,
                                      cudaStream_t st) {
    const int64_t tiles = (a.nels + HT_E - 1) / HT_E;
    if (tiles < 1) return cudaSuccess;
    const auto fn = plastic ? jac_box_elastic_kernel<TG, true> : jac_box_elastic_kernel<TG, false>;
    const size_t smem = plastic ? sizeof(JbElastic) : offsetof(JbElastic, S1);
    cudaError_t err = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (err != cudaSuccess) return err;
    count_launch();
    fn<<<(unsigned)tiles, HT_THREADS, smem, st>>>(a, geo_c, general);
    err = cudaGetLastError();
    if (err != cudaSuccess || !plastic) return err;
    err = cudaFuncSetAttribute(jac_box_general_kernel<TG>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(JbGeneral));
    if (err != cudaSuccess) return err;
    count_launch();
    jac_box_general_kernel<TG><<<(unsigned)tiles, HT_THREADS, sizeof(JbGeneral), st>>>(a, geo_c, general);
    return cudaGetLastError();
}
template cudaError_t launch_hex27_jacobian_box<double>(const H27JacArgs<double, double>&, const double*, bool, uint8_t*, cudaStream_t);
template cudaError_t launch_hex27_jacobian_box<float>(const H27JacArgs<double, float>&, const double*, bool, uint8_t*, cudaStream_t);

}  // namespace femb
