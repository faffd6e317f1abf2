// geometry.cu — per-integration-point element geometry from the node coordinates:
// precompute_geometry_kernel! (src/mesh/mesh.jl:674-682) with the stored entry of
// _geometry_entry (mesh.jl:550-553), for Hex27 (3-D) and Q9 (2-D). Used at setup and
// by update_geometry! (mesh.jl:640-650, mixed_mesh.jl:337-345) after the nodes move.
#include <algorithm>
#include <cmath>
#include "kernels.cuh"

namespace femb {
namespace {

template <int DIM> struct GeoTabs;
template <> struct GeoTabs<3> {
    static constexpr int NV = 27;
    FEMB_D static double dN(int q, int a, int j) { return c_tab.dN3[q][a][j]; }
    FEMB_D static double w(int q) { return c_tab.w3[q]; }
};
template <> struct GeoTabs<2> {
    static constexpr int NV = 9;
    FEMB_D static double dN(int q, int a, int j) { return c_tab.dN2[q][a][j]; }
    FEMB_D static double w(int q) { return c_tab.w2[q]; }
};

// One thread per (element, integration point): J = Σ_a x_a ⊗ ∂N_a/∂ξ in FP64
// (J[i][j] = ∂x_i/∂ξ_j), the cofactor inverse and determinant, rounded once on store
// to TG. A connectivity entry outside [1, nnodes] sets *bad and the point's entries to
// NaN (no out-of-range read).
template <int DIM, class TG>
__global__ void geometry_kernel(const double* __restrict__ coords, const int32_t* __restrict__ el2n, int64_t nels,
                                int64_t nnodes, TG* geo_v, TG* geo_P, int* bad) {
    using G = GeoTabs<DIM>;
    constexpr int NV = G::NV, NQ = G::NV, NG = DIM * DIM + 1;
    // the derivatives in shared memory: a warp's threads stand at different points, and divergent
    // reads of constant memory go one by one (42 ms at 64³; 0.57 ms now). Points lie an odd stride apart: no conflicts.
    __shared__ double dN[NQ][NV][DIM];
    for (int i = threadIdx.x; i < NQ * NV * DIM; i += blockDim.x) {
        const int j = i % DIM, a = i / DIM % NV;
        dN[i / (DIM * NV)][a][j] = G::dN(i / (DIM * NV), a, j);
    }
    __syncthreads();
    const int64_t n = nels * NQ;
    for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < n; idx += (int64_t)gridDim.x * blockDim.x) {
        const int64_t e = idx / NQ;
        const int q = (int)(idx - e * NQ);
        double J[DIM][DIM];
#pragma unroll
        for (int i = 0; i < DIM; ++i)
#pragma unroll
            for (int j = 0; j < DIM; ++j) J[i][j] = 0.0;
        bool ok = true;
        for (int a = 0; a < NV; ++a) {
            const int64_t node = __ldg(el2n + e * NV + a);
            if (node < 1 || node > nnodes) { ok = false; break; }
            const double* x = coords + (node - 1) * DIM;
            double xa[DIM];
#pragma unroll
            for (int i = 0; i < DIM; ++i) xa[i] = __ldg(x + i);
#pragma unroll
            for (int j = 0; j < DIM; ++j) {
                const double d = dN[q][a][j];
#pragma unroll
                for (int i = 0; i < DIM; ++i) J[i][j] = fma(xa[i], d, J[i][j]);
            }
        }
        double inv[DIM][DIM], det;
        if constexpr (DIM == 3) {
            const double c00 = J[1][1] * J[2][2] - J[1][2] * J[2][1];
            const double c01 = J[1][2] * J[2][0] - J[1][0] * J[2][2];
            const double c02 = J[1][0] * J[2][1] - J[1][1] * J[2][0];
            det = J[0][0] * c00 + J[0][1] * c01 + J[0][2] * c02;
            const double r = 1.0 / det;
            inv[0][0] = c00 * r;
            inv[1][0] = c01 * r;
            inv[2][0] = c02 * r;
            inv[0][1] = (J[0][2] * J[2][1] - J[0][1] * J[2][2]) * r;
            inv[1][1] = (J[0][0] * J[2][2] - J[0][2] * J[2][0]) * r;
            inv[2][1] = (J[0][1] * J[2][0] - J[0][0] * J[2][1]) * r;
            inv[0][2] = (J[0][1] * J[1][2] - J[0][2] * J[1][1]) * r;
            inv[1][2] = (J[0][2] * J[1][0] - J[0][0] * J[1][2]) * r;
            inv[2][2] = (J[0][0] * J[1][1] - J[0][1] * J[1][0]) * r;
        } else {
            det = J[0][0] * J[1][1] - J[0][1] * J[1][0];
            const double r = 1.0 / det;
            inv[0][0] = J[1][1] * r;
            inv[0][1] = -J[0][1] * r;
            inv[1][0] = -J[1][0] * r;
            inv[1][1] = J[0][0] * r;
        }
        const double dO = fabs(det) * G::w(q);
        TG* g = geo_v + idx * NG;
        if (!ok) {
            atomicOr(bad, 1);
            for (int k = 0; k < NG; ++k) g[k] = (TG)NAN;
            if (geo_P) geo_P[idx] = (TG)NAN;
            continue;
        }
        // J⁻¹ column-major: entry (r, c) at r + DIM·c
#pragma unroll
        for (int c = 0; c < DIM; ++c)
#pragma unroll
            for (int r = 0; r < DIM; ++r) g[r + DIM * c] = (TG)inv[r][c];
        g[DIM * DIM] = (TG)dO;
        if (geo_P) geo_P[idx] = (TG)dO;
    }
}

}  // namespace

template <class TG>
cudaError_t launch_geometry(int dim, const double* coords, const int32_t* el2n, int64_t nels, int64_t nnodes, TG* geo_v,
                            TG* geo_P, int* bad, cudaStream_t st) {
    const int64_t n = nels * (dim == 3 ? 27 : 9);
    const int64_t blocks = std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, 148 * 16));
    count_launch();
    if (dim == 3) geometry_kernel<3, TG><<<(unsigned)blocks, 256, 0, st>>>(coords, el2n, nels, nnodes, geo_v, geo_P, bad);
    else geometry_kernel<2, TG><<<(unsigned)blocks, 256, 0, st>>>(coords, el2n, nels, nnodes, geo_v, geo_P, bad);
    return cudaGetLastError();
}
template cudaError_t launch_geometry<double>(int, const double*, const int32_t*, int64_t, int64_t, double*, double*,
                                             int*, cudaStream_t);
template cudaError_t launch_geometry<float>(int, const double*, const int32_t*, int64_t, int64_t, float*, float*, int*,
                                            cudaStream_t);

namespace {

// One J⁻¹ and |det J| per element when every quadrature point of the reference
// layout carries the same J⁻¹ and |det J|·ω/ω, and geo_P equals the velocity
// weights (Hex27 MixedMeshCache, src/mesh/mixed_mesh.jl:375-392). One warp per element reads its 270
// contiguous entries once, thirty lanes at a time: ten entries of three points, so that a lane
// compares one entry throughout and needs no shuffles (HBM-bound: 116 us at 64³ in
// FP64 against 95 for the bytes; a thread per element took 262).
template <class TG, class TC>
__global__ void __launch_bounds__(256) compress_geometry_kernel(const TG* __restrict__ geo_v, const TG* __restrict__ geo_P,
                                                               int64_t nels, double box_tol, TC* out, int* flags) {
    // one cell that is not affine settles it: the blocks that follow leave the rest unread
    if (*reinterpret_cast<volatile int*>(flags) & GEO_NOT_AFFINE) return;
    const int lane = threadIdx.x & 31, r = lane % 10;
    const int64_t nw = (int64_t)gridDim.x * (blockDim.x >> 5);
    const double tol = sizeof(TG) == 8 ? 1e-12 : 1e-5;
    const bool rd = lane < 30, dO = r == 9;
    // the weights ω of the lane's nine points: ω_x of its place among the three, times ω_yω_z
    const double w_x = lane < 30 ? c_tab.w3[12 + lane / 10] : 1.0;   // ω_xω_y(0)ω_z(0)
    const bool diag_lane = lane < 9 && lane % 4 == 0;
    for (int64_t e = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); e < nels; e += nw) {
        const TG* G = geo_v + e * 270;
        double x[9];
#pragma unroll
        for (int i = 0; i < 9; ++i) x[i] = rd ? (double)G[30 * i + lane] : 0.0;
        const double gv = lane < 27 ? (double)G[lane * 10 + 9] : 0.0, gp = lane < 27 ? (double)geo_P[e * 27 + lane] : 0.0;
        // the centre point's entry (lanes 10..19 of the fifth load); |det J| = dΩ·729/512
        double c = __shfl_sync(0xffffffffu, x[4], 10 + r);
        double sc = r < 9 ? fabs(c) : 0.0;
        sc = fmax(sc, __shfl_xor_sync(0xffffffffu, sc, 8));
        sc = fmax(sc, __shfl_xor_sync(0xffffffffu, sc, 4));
        sc = fmax(sc, __shfl_xor_sync(0xffffffffu, sc, 2));
        sc = fmax(sc, __shfl_xor_sync(0xffffffffu, sc, 1));
        sc = __shfl_sync(0xffffffffu, sc, 0);
        if (dO) c *= 729.0 / 512.0;
        const double ref = dO ? c * w_x : c, size = dO ? fabs(ref) : sc;
        bool ok = fabs(gp - gv) <= tol * fabs(gv), box = fabs(gp - gv) <= box_tol * fabs(gv);
#pragma unroll
        for (int i = 0; i < 9; ++i) {
            // ω_yω_z against the centre's 64/81
            const double f = dO ? (i % 3 == 1 ? 1.0 : 0.625) * (i / 3 == 1 ? 1.0 : 0.625) : 1.0;
            const double dev = fabs(x[i] - ref * f);
            ok = ok && (!rd || dev <= tol * size * f);
            box = box && (!rd || dev <= box_tol * size * f);
        }
        const bool diag = lane >= 9 || diag_lane || c == 0.0;
        const bool all_ok = __all_sync(0xffffffffu, ok), all_diag = __all_sync(0xffffffffu, diag), all_box = __all_sync(0xffffffffu, box && diag);
        if (lane == 0 && !(all_ok && all_box))
            atomicOr(flags, (all_ok ? 0 : GEO_NOT_AFFINE) | (all_diag ? 0 : GEO_NOT_DIAG) | (all_box ? 0 : GEO_NOT_BOX));
        if (lane < 10) out[e * 10 + lane] = (TC)c;
    }
}

}  // namespace

template <class TG, class TC>
cudaError_t launch_compress_geometry(const TG* geo_v, const TG* geo_P, int64_t nels, TC* out, int* flags, cudaStream_t st) {
    count_launch();
    const int64_t blocks = std::min<int64_t>((nels + 7) / 8, 148 * 32);
    // What forming J⁻¹ and |det J| from coordinates leaves on a box of n cells along an axis grows as the
    // cancellation in x_{i+1} − x_i does: up to 1.6e-15·n and 2.7e-15·n (measured for n from 2 to 256). Three times
    // that for a cube; a long box may fail and is then treated as any other mesh.
    const double box_tol = sizeof(TG) == 8 ? 8e-15 * std::max(8.0, std::cbrt((double)nels)) : 2.5e-7;
    compress_geometry_kernel<TG, TC><<<(unsigned)blocks, 256, 0, st>>>(geo_v, geo_P, nels, box_tol, out, flags);
    return cudaGetLastError();
}
template cudaError_t launch_compress_geometry<double, double>(const double*, const double*, int64_t, double*, int*, cudaStream_t);
template cudaError_t launch_compress_geometry<float, float>(const float*, const float*, int64_t, float*, int*, cudaStream_t);
template cudaError_t launch_compress_geometry<double, float>(const double*, const double*, int64_t, float*, int*, cudaStream_t);
template cudaError_t launch_compress_geometry<float, double>(const float*, const float*, int64_t, double*, int*, cudaStream_t);

}  // namespace femb
