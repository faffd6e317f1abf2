// cellpressure.cu — the viscous Hex27 Stokes operator with four cell-local pressure
// modes (1, ξ, η, ζ) (CellPressureStokesDR): preconditioner and pressure mass
// (stokes_preconditioner_3d!, src/stokes/assemblers/momentum_residuals.jl:703-745),
// pressure residual (assemble_stokes_pressure_residual_3d!, pressure_residual.jl:330-364),
// momentum residual (assemble_stokes_momentum_residual_3d!, momentum_residuals.jl:644-700)
// and the node/cell updates of the Arrow–Hurwicz relaxation (DR.jl:1004-1057).
//
// The residuals and the pressure step of an iteration are one kernel on tiles of 32 elements
// (hex27_tile.cuh; the shared buffers' strides replace the LY::SLOT stages of three elements to a
// warp). The velocity is the same in both residuals, so its gradient is taken once; the mean of the
// constant pressure mode, which the reference removes between them, is only known when every element
// has stepped: the momentum residual is linear in it, so the velocity step adds mean·∫∇N (one vector
// per solve) and takes the mean off the pressure. The preconditioner, once per solve, is one warp per
// element: lane a < 27 owns node a and lane q < 27 point q, with the Hex27 tables staged once per
// block in shared memory because the lanes index them by their own point or node.
#include <algorithm>
#include "hex27_tile.cuh"
#include "kernels.cuh"

namespace femb {
namespace {

constexpr int CP_WARPS = 4;
constexpr int CP_THREADS = CP_WARPS * 32;

struct CpTabs {
    double dN[27][27][3];   // ∂N_a/∂ξ_j at q
    double N[27][27];       // N_a at q
    double sumN[27];
    double x[27][3];        // reference coordinates of q (the pressure modes ξ, η, ζ)
};

FEMB_D void stage_tables(CpTabs& T) {
    for (int i = threadIdx.x; i < 27 * 27 * 3; i += blockDim.x) (&T.dN[0][0][0])[i] = (&c_tab.dN3[0][0][0])[i];
    for (int i = threadIdx.x; i < 27 * 27; i += blockDim.x) (&T.N[0][0])[i] = (&c_tab.N3[0][0])[i];
    for (int q = threadIdx.x; q < 27; q += blockDim.x) {
        T.sumN[q] = c_tab.sumN3[q];
        T.x[q][0] = c_tab.qx[q % 3];
        T.x[q][1] = c_tab.qx[(q / 3) % 3];
        T.x[q][2] = c_tab.qx[q / 9];
    }
    __syncthreads();
}

FEMB_D double warp_sum_d(double x) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}

struct CpSmem {
    double S1[HT_S1], S2[HT_S2];
    double part[4][9][HT_E];     // pressure-mode parts of the lines
    double P[4][HT_E];
    double eta[MAXPH], rho[MAXPH];
};
static_assert(2 * (sizeof(CpSmem) + 1024) <= 228 * 1024, "two blocks per SM");

// RP(m, e) = −Σ_q mode_m ∇·v dΩ, P += step·RP/M (with a.mass), and the momentum residual: the viscous
// stress 2ηε̇′ − P·I and the body force −ρg. With a.mass the last block to finish reduces the
// tiles' Σ P(1,e)·M(1,e) and Σ M(1,e), in tile order, to *a.mean. Bound by the latency between its
// barriers and the atomics (18 warps per SM). An iteration at 32³, this kernel and the velocity step,
// 45 us (51 before dependent launches); two residual kernels with three elements to a warp, two for the
// pressure and the step took 97.
// AFF: every cell is affine and a.geo_c holds one J⁻¹ and |det J| per cell (dΩ_q = |det J|·ω_q).
// MINB: blocks per SM the registers are cut for.
template <bool AFF, int MINB>
__global__ void __launch_bounds__(HT_THREADS, MINB) cp_tile_kernel(const CpArgs a) {
    extern __shared__ __align__(16) unsigned char cp_smem[];
    CpSmem& S = *reinterpret_cast<CpSmem*>(cp_smem);
    __shared__ bool last;
    const int lane = threadIdx.x & 31, w = ht_warp(), la = w % 3, lb = w / 3;
    const int64_t e0 = (int64_t)blockIdx.x * HT_E;
    const int ne = (int)(a.nels - e0 < HT_E ? a.nels - e0 : HT_E);
    const bool act = lane < ne;
    const int64_t e = e0 + (act ? lane : ne - 1);   // lanes past the end repeat the last element

    int node[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) node[i] = __ldg(a.el2n + 27 * e + c_tab.tn3[i + 3 * w]) - 1;
    double Ja[10];
    if constexpr (AFF) {
#pragma unroll
        for (int r = 0; r < 10; ++r) Ja[r] = ld(a.geo_c + e * 10 + r);
    }
    double P = 0, M = 1;
    if (w < 4) {   // warp w brings pressure mode w of every element
        if (a.mass) M = ld(a.mass + 4 * e + w);
    }
    const int ph = __ldg(a.phases + e) - 1;
    if (threadIdx.x < MAXPH) { S.eta[threadIdx.x] = a.eta[threadIdx.x]; S.rho[threadIdx.x] = a.rho[threadIdx.x]; }
    pdl_enter();   // everything so far is constant over the iterations
    if (w < 4) P = a.P[4 * e + w];
    double g[3][3][3];
    {
        double v[3][3];
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int c = 0; c < 3; ++c) v[c][i] = a.v[c][node[i]];
        ht_gradient<double, 3>(v, S.S1, S.S2, la, lb, lane, g);
    }
    const double xi = ht_xr<double>(la), et = ht_xr<double>(lb);
    const double wxy = ht_wr<double>(la) * ht_wr<double>(lb);
    const double* Gp = a.geo_v + e * 270 + w * 10;   // point qz at Gp + 90·qz
    {
        double f[3];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            double J[10];
#pragma unroll
            for (int r = 0; r < 10; ++r) J[r] = AFF ? Ja[r] : ld(Gp + 90 * q + r);
            if constexpr (AFF) J[9] *= wxy * ht_w(q);
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const double r0 = g[c][0][q], r1 = g[c][1][q], r2 = g[c][2][q];
#pragma unroll
                for (int k = 0; k < 3; ++k) g[c][k][q] = r0 * J[3 * k] + r1 * J[1 + 3 * k] + r2 * J[2 + 3 * k];
            }
            f[q] = -(g[0][0][q] + g[1][1][q] + g[2][2][q]) * J[9];
        }
        const double s = f[0] + f[1] + f[2], sz = HT_GA * (f[2] - f[0]);
        S.part[0][w][lane] = s;
        S.part[1][w][lane] = xi * s;
        S.part[2][w][lane] = et * s;
        S.part[3][w][lane] = sz;
    }
    __syncthreads();
    double sPM = 0, sM = 0;
    if (w < 4) {
        if (a.RP) {
            double rp = S.part[w][0][lane];
#pragma unroll
            for (int l = 1; l < 9; ++l) rp += S.part[w][l][lane];
            if (act) a.RP[4 * e + w] = rp;
            if (a.mass) {
                P += a.step * rp / M;
                if (act) a.Pnew[4 * e + w] = P;
                if (w == 0 && act) { sPM = P * M; sM = M; }
            }
        }
        S.P[w][lane] = P;
    }
    if (!a.Rv[0]) return;
    __syncthreads();

    const double eta2 = 2.0 * S.eta[ph], rho = S.rho[ph];
    const double Pc = S.P[0][lane] + S.P[1][lane] * xi + S.P[2][lane] * et, Pz = S.P[3][lane];
    double bq[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        double J[10];
#pragma unroll
        for (int r = 0; r < 10; ++r) J[r] = AFF ? Ja[r] : ld(Gp + 90 * q + r);
        if constexpr (AFF) J[9] *= wxy * ht_w(q);
        // η and ρ interpolated over the cell's single phase (interp2ip_phase)
        const double sN = c_tab.sumN3[w + 9 * q];
        bq[q] = rho * sN * J[9];
        const double et2 = eta2 * sN * J[9], pq = (Pc + Pz * ht_x(q)) * J[9];
        const double tr = (g[0][0][q] + g[1][1][q] + g[2][2][q]) * (1.0 / 3.0);
        const double xy = et2 * (0.5 * (g[0][1][q] + g[1][0][q])), xz = et2 * (0.5 * (g[0][2][q] + g[2][0][q])),
                     yz = et2 * (0.5 * (g[1][2][q] + g[2][1][q]));
        const double sg[3][3] = {{et2 * (g[0][0][q] - tr) - pq, xy, xz}, {xy, et2 * (g[1][1][q] - tr) - pq, yz},
                                 {xz, yz, et2 * (g[2][2][q] - tr) - pq}};
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int d = 0; d < 3; ++d) g[c][d][q] = J[d] * sg[c][0] + J[d + 3] * sg[c][1] + J[d + 6] * sg[c][2];
    }
    ht_scatter_z<double, 3>(g, [&](int c, int q) { return -a.g[c] * bq[q]; }, S.S2, la, lb, lane);
    __syncthreads();
    double R[3][3];
    ht_scatter_yx<double, 3>(S.S1, S.S2, la, lb, lane, R);
    // the next lane's ξ = −1 node, when it is this lane's ξ = +1 node, is added here (stokes3d.cu)
    const int n0n = __shfl_down_sync(0xffffffffu, node[0], 1);
    const bool fold = lane + 1 < ne && n0n == node[2];
    const bool folded = __shfl_up_sync(0xffffffffu, (int)fold, 1) && lane > 0;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const double r0n = __shfl_down_sync(0xffffffffu, R[c][0], 1);
        if (fold) R[c][2] += r0n;
        if (act) {
            if (!folded) atomicAdd(a.Rv[c] + node[0], R[c][0]);
            atomicAdd(a.Rv[c] + node[1], R[c][1]);
            atomicAdd(a.Rv[c] + node[2], R[c][2]);
        }
    }
    if (!a.mass) return;
    if (w == 0) {
        sPM = warp_sum_d(sPM);
        sM = warp_sum_d(sM);
        if (lane == 0) {
            a.partials[2 * blockIdx.x] = sPM;
            a.partials[2 * blockIdx.x + 1] = sM;
            __threadfence();
            last = atomicAdd(a.done, 1u) == gridDim.x - 1;
        }
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double t0 = 0, t1 = 0;
    for (unsigned k = threadIdx.x; k < gridDim.x; k += HT_THREADS) { t0 += __ldcg(a.partials + 2 * k); t1 += __ldcg(a.partials + 2 * k + 1); }
    t0 = warp_sum_d(t0);
    t1 = warp_sum_d(t1);
    if (lane == 0) { S.part[0][w][0] = t0; S.part[1][w][0] = t1; }
    __syncthreads();
    if (threadIdx.x == 0) {
        t0 = t1 = 0;
        for (int l = 0; l < 9; ++l) { t0 += S.part[0][l][0]; t1 += S.part[1][l][0]; }
        *a.mean = t0 / t1;
        *a.done = 0;   // for the next launch
    }
}

__global__ void __launch_bounds__(CP_THREADS) cp_preconditioner_kernel(const CpArgs a) {
    __shared__ CpTabs T;
    stage_tables(T);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int64_t e = (int64_t)blockIdx.x * CP_WARPS + w; e < a.nels; e += (int64_t)gridDim.x * CP_WARPS) {
        const int ph = __ldg(a.phases + e) - 1;
        const double eta = a.eta[ph];
        double m[4] = {0, 0, 0, 0};
        if (lane < 27) {
            const int an = lane;
            const int node = __ldg(a.el2n + e * 27 + an) - 1;
            double dg[3] = {0, 0, 0}, gr[3] = {0, 0, 0};
            for (int q = 0; q < 27; ++q) {
                const double* g = a.geo_v + (e * 27 + q) * 10;
                double gN[3];
#pragma unroll
                for (int k = 0; k < 3; ++k)
                    gN[k] = T.dN[q][an][0] * __ldg(g + 3 * k) + T.dN[q][an][1] * __ldg(g + 1 + 3 * k) +
                            T.dN[q][an][2] * __ldg(g + 2 + 3 * k);
                const double dO = __ldg(g + 9);
                const double n2 = gN[0] * gN[0] + gN[1] * gN[1] + gN[2] * gN[2];
#pragma unroll
                for (int c = 0; c < 3; ++c) { dg[c] += eta * (n2 + gN[c] * gN[c] / 3.0) * dO; gr[c] += gN[c] * dO; }
            }
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                atomicAdd(a.diagonal[c] + node, dg[c]);
                if (a.grad[c]) atomicAdd(a.grad[c] + node, gr[c]);
            }
            // pressure mass: lane = point
            const int q = lane;
            const double dO = __ldg(a.geo_v + (e * 27 + q) * 10 + 9);
            m[0] = dO;
            m[1] = T.x[q][0] * T.x[q][0] * dO;
            m[2] = T.x[q][1] * T.x[q][1] * dO;
            m[3] = T.x[q][2] * T.x[q][2] * dO;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) m[k] = warp_sum_d(m[k]);
        if (lane < 4) a.pressure_mass[4 * e + lane] = lane == 0 ? m[0] : lane == 1 ? m[1] : lane == 2 ? m[2] : m[3];
    }
}

__global__ void cp_velocity_step_kernel(const CpVelArgs a) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x, t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    bool waited = false;
    double mean = 0;
    for (int64_t i = t; i < a.n; i += stride) {
        // v is the previous step's; the sweep between them only reads it
        const unsigned m = a.mask[i];
        double v[3], b[3], d[3], l[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            v[c] = a.v[c][i]; b[c] = __ldg(a.grad[c] + i); d[c] = __ldg(a.diag[c] + i);
            l[c] = a.load[c] ? __ldg(a.load[c] + i) : 0.0;
        }
        if (!waited) { pdl_enter(); waited = true; mean = *a.mean; }
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            double r = a.Rv[c][i] + mean * b[c];
            if (a.load[c]) r -= l[c];
            if ((m >> c) & 1u) r = 0.0;
            else a.v[c][i] = v[c] - a.step * r / d[c];
            a.Rv[c][i] = a.zero ? 0.0 : r;
        }
    }
    if (!waited) { pdl_enter(); mean = *a.mean; }
    for (int64_t e = t; e < a.nels; e += stride) a.P[4 * e] -= mean;
}

// Connectivity in 1..nnodes and phases in 1..nphases, before any kernel gathers by them.
__global__ void cp_validate_kernel(const int32_t* el2n, const int32_t* phases, int64_t nels, int64_t nnodes, int nphases,
                                   int* bad) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nels * 27; i += (int64_t)gridDim.x * blockDim.x) {
        const int32_t n = el2n[i];
        if (n < 1 || n > nnodes) atomicOr(bad, 1);
        if (i % 27 == 0) {
            const int32_t ph = phases[i / 27];
            if (ph < 1 || ph > nphases) atomicOr(bad, 2);
        }
    }
}

inline unsigned grid_for(int64_t n, int t, int cap) {
    return (unsigned)std::max<int64_t>(1, std::min<int64_t>((n + t - 1) / t, cap));
}

}  // namespace

cudaError_t launch_cp_tiles(const CpArgs& a, int num_sms, cudaStream_t st, bool pdl) {
    const int64_t tiles = (a.nels + HT_E - 1) / HT_E;
    auto fn = !a.geo_c ? cp_tile_kernel<false, 1> : tiles <= num_sms ? cp_tile_kernel<true, 1> : cp_tile_kernel<true, 2>;
    const cudaError_t err = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(CpSmem));
    if (err != cudaSuccess) return err;
    count_launch();
    return launch_pdl(pdl, fn, dim3((unsigned)tiles), dim3(HT_THREADS), sizeof(CpSmem), st, a);
}

namespace {
// One J⁻¹ and |det J| = dΩ_q/ω_q per cell from its centre point; *not_affine is set when
// any point of a cell differs from them by more than 1e-12 of their scale.
__global__ void cp_compress_geometry_kernel(const double* geo_v, int64_t nels, double* out, int* not_affine) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= nels) return;
    const double* G = geo_v + e * 270;
    double Jc[9], sc = 0;
    for (int r = 0; r < 9; ++r) { Jc[r] = G[13 * 10 + r]; sc = fmax(sc, fabs(Jc[r])); }
    const double dc = G[13 * 10 + 9] / c_tab.w3[13];
    bool ok = true;
    for (int q = 0; q < 27; ++q) {
        for (int r = 0; r < 9; ++r) ok = ok && fabs(G[q * 10 + r] - Jc[r]) <= 1e-12 * sc;
        ok = ok && fabs(G[q * 10 + 9] / c_tab.w3[q] - dc) <= 1e-12 * fabs(dc);
    }
    if (!ok) atomicOr(not_affine, 1);
    for (int r = 0; r < 9; ++r) out[e * 10 + r] = Jc[r];
    out[e * 10 + 9] = dc;
}
}  // namespace

cudaError_t launch_cp_compress_geometry(const double* geo_v, int64_t nels, double* out, int* not_affine, cudaStream_t st) {
    count_launch();
    cp_compress_geometry_kernel<<<grid_for(nels, 128, 1 << 30), 128, 0, st>>>(geo_v, nels, out, not_affine);
    return cudaGetLastError();
}

cudaError_t launch_cp_preconditioner(const CpArgs& a, int num_sms, cudaStream_t st) {
    count_launch();
    cp_preconditioner_kernel<<<grid_for(a.nels, CP_WARPS, num_sms * 8), CP_THREADS, 0, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_cp_validate(const int32_t* el2n, const int32_t* phases, int64_t nels, int64_t nnodes, int nphases,
                               int* bad, cudaStream_t st) {
    count_launch();
    cp_validate_kernel<<<grid_for(nels * 27, 256, 148 * 8), 256, 0, st>>>(el2n, phases, nels, nnodes, nphases, bad);
    return cudaGetLastError();
}

cudaError_t launch_cp_velocity_step(const CpVelArgs& a, cudaStream_t st, bool pdl) {
    count_launch();
    return launch_pdl(pdl, cp_velocity_step_kernel, dim3(grid_for(a.n, 256, 148 * 8)), dim3(256), 0, st, a);
}

}  // namespace femb
