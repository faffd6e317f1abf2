// stokes3d_incr.cu — FP32 incremental sweep of the mixed-precision solve.
//
// The sweep computes, for every Hex27/P1-disc element, the increments of the
// pressure residual, of the element-local Pnum and of the visco-elasto-plastic
// momentum residual between the FP64 base state x_k and x_k + δ
// (pressure_residual.jl:132-158, momentum_residuals.jl:209-258, rheology.jl:413-472),
// with the base trial stress and yield value of every integration point read
// from the tiled FP32 base data written by the FP64 base sweep.
//
// Mapping (hex27_tile.cuh): a block of nine warps owns a tile of 32 elements, lane = element,
// warp = line of the node and quadrature grids; every global read of a warp is one coalesced
// line of the tiled inputs and three blocks (27 warps) are resident per SM.
//
// Measured (64³ layered visco-elasto-plastic boxes, elastic first step): 163 -> 135 us a sweep
// against one thread per element with its 216 working values in shared memory (8 resident
// warps, 48 % issue); at 32³ with yielding points 36 -> 29 us. Issue 62 %, 1 220 instructions a
// thread (half of them FP32 arithmetic), 60 us of shared-memory wavefronts, DRAM 132 MB (20 us):
// bound by issue together with the latency of the gathers and barriers. Three warps per tile with
// a whole plane in registers (12 warps, 168 registers) took 192 us.
#include <algorithm>
#include "hex27_tile.cuh"
#include "kernels.cuh"
#include "rheology.cuh"

namespace femb {

// K[p][d][a] = Σ_q w_q N^P_p(q) ∂N_a/∂ξ_d(q), a in tensor order.
__constant__ float c_inc_K[4][3][27];

namespace {

void host_pnum_table(float K[4][3][27]) {
    for (int p = 0; p < 4; ++p)
        for (int d = 0; d < 3; ++d)
            for (int a = 0; a < 27; ++a) {
                const int ia[3] = {a % 3, (a / 3) % 3, a / 9};
                double s = 0;
                for (int q = 0; q < 27; ++q) {
                    const int iq[3] = {q % 3, (q / 3) % 3, q / 9};
                    const double np = p == 0 ? 1 - ht_x(iq[0]) - ht_x(iq[1]) - ht_x(iq[2]) : ht_x(iq[p - 1]);
                    double dn = 1;
                    for (int r = 0; r < 3; ++r) dn *= r == d ? ht_D(iq[r], ia[r]) : ht_L(iq[r], ia[r]);
                    s += ht_w(iq[0]) * ht_w(iq[1]) * ht_w(iq[2]) * np * dn;
                }
                K[p][d][a] = (float)s;
            }
}

// Phase of an element for the sweep: the common phase of its nodes (or DoFs) in
// any of the three layouts (src/utils.jl:70-74), 0-based; -1 when they differ.
__device__ int uniform_phase(const int32_t* ph, int layout, const int32_t* ids, int n, int64_t e) {
    if (!ph) return 0;
    if (layout == FEMB200_PHASE_CELL) return ph[e] - 1;
    int p0 = -2;
    for (int i = 0; i < n; ++i) {
        const int p = (layout == FEMB200_PHASE_ELEMENT_NODE ? ph[(int64_t)n * e + i] : ph[ids[(int64_t)n * e + i] - 1]) - 1;
        if (p0 == -2) p0 = p;
        else if (p != p0) return -1;
    }
    return p0;
}

__global__ void incr_tiles_kernel(const IncrTileSrc src, int64_t nels, int64_t nslots, IncrArgs dst, int* flags) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= nslots) return;
    const int64_t tile = e >> 5;
    const int lane = (int)(e & 31);
    const bool act = e < nels;
    int32_t* el2n_t = const_cast<int32_t*>(dst.el2n_t);
    int32_t* dofs_t = const_cast<int32_t*>(dst.dofs_t);
    float* geo_t = const_cast<float*>(dst.geo_t);
    float* pscale_t = const_cast<float*>(dst.pscale_t);
    for (int t = 0; t < 27; ++t) el2n_t[(tile * 27 + t) * 32 + lane] = act ? src.el2n[27 * e + c_tab.tn3[t]] - 1 : 0;
    bool linear = true;
    for (int p = 0; p < 4; ++p) {
        const int32_t d = act ? src.dofsP[4 * e + p] - 1 : 0;
        linear = linear && (!act || d == 4 * e + p);
        dofs_t[(tile * 4 + p) * 32 + lane] = d;
        pscale_t[(tile * 4 + p) * 32 + lane] = act ? src.gP[d] / src.MP[d] : 0.0f;
    }
    if (!linear) atomicOr(flags, INCR_DOFS_GENERAL);
    float J[9];
    for (int r = 0; r < 10; ++r) {
        const float gv = act ? src.geo_c[10 * e + r] : 0.0f;
        if (r < 9) J[r] = gv;
        geo_t[(tile * 10 + r) * 32 + lane] = gv;
    }
    // entries that vanish in the sweep's FP32 arithmetic (the structured generators leave
    // rounding residues of 1e-16 off the diagonal) count as zero
    bool offdiag = false;
    for (int r = 0; r < 9; ++r)
        if (r % 4 != 0) offdiag = offdiag || !(fabsf(J[r]) <= 1e-10f * fminf(fabsf(J[4 * (r % 3)]), fabsf(J[4 * (r / 3)])));
    if (offdiag) atomicOr(flags, INCR_GEOMETRY_FULL);
    if (src.eta) {
        float* eta_t = const_cast<float*>(dst.eta_t);
        for (int q = 0; q < 27; ++q) eta_t[(tile * 27 + q) * 32 + lane] = act ? src.eta[27 * e + q] : 1.0f;
    }
    int pv = 0, pp = 0;
    if (act) {
        pv = uniform_phase(src.phv, src.phv_layout, src.el2n, 27, e);
        pp = uniform_phase(src.php, src.php_layout, src.dofsP, 4, e);
        if (pv < 0 || pp < 0 || pv >= src.nphases || pp >= src.nphases) {
            atomicOr(flags, INCR_MIXED_PHASES);
            pv = pp = 0;
        }
    }
    int32_t* phase_t = const_cast<int32_t*>(dst.phase_t);
    phase_t[e] = pv;
    phase_t[nslots + e] = pp;
}

// Inputs and output of the FP64 return near the yield-surface apex, passed by value
// so that the caller's arrays stay in registers on the common (FP32) path.
struct ApexIn {
    float tb[6], dtt[6], Fk, Pq, twoe, sphi, inv_den;
};
struct ApexOut {
    float tau[6];
};
__device__ __noinline__ ApexOut apex_increment_f64(const ApexIn in) {
    double tbd[6], dtd[6], outd[6];
#pragma unroll
    for (int c = 0; c < 6; ++c) { tbd[c] = in.tb[c]; dtd[c] = in.dtt[c]; }
    dp_increment<double>(tbd, (double)in.Fk, dtd, (double)in.Pq, (double)in.twoe, (double)in.sphi, (double)in.inv_den,
                         eps2<double>(), outd);
    ApexOut o;
#pragma unroll
    for (int c = 0; c < 6; ++c) o.tau[c] = (float)outd[c];
    return o;
}

// The base data is read once per sweep and is larger than L2: it is loaded with an
// evict-first L2 policy so that the node arrays (δv gathers, residual atomics, the node
// update) stay resident across sweeps.
FEMB_D uint64_t l2_evict_first() {
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    return p;
}
FEMB_D float ldg_stream(const float* ptr, uint64_t pol) {
    float v;
    asm("ld.global.nc.L1::no_allocate.L2::cache_hint.f32 %0, [%1], %2;" : "=f"(v) : "l"(ptr), "l"(pol));
    return v;
}

FEMB_D int elem_dof(const IncrArgs& a, int64_t tile, int lane, int p) {
    // padding lanes (past the last element) read the first element's DoFs
    const int64_t e = tile * 32 + lane;
    return a.dofs_linear ? (int)(4 * (e < a.nels ? e : 0) + p) : __ldg(a.dofs_t + (tile * 4 + p) * 32 + lane);
}

struct IncrSmem {
    float S1[HT_S1], S2[HT_S2];
    float rp[9][4][HT_E];      // the lines' parts of the pressure residual
    float pn[3][4][HT_E];      // Pnum, one copy per group of warps that sums it
    IncrPhase PT[MAXPH];
};

// DIAG: every element's J⁻¹ is diagonal (axis-aligned boxes, the structured generators'
// meshes), so the gradient and flux transforms are one product per entry. APEX: the tiles
// with a base point near the yield-surface apex (a.apex_t), where the increment of such a point is
// formed in FP64 out of line; the other instantiations skip them, so that the rare call costs
// the common tiles no registers. The trial stress of a point is read where the elastic bound
// fails: with 27 warps resident its latency is hidden, and a variant that loaded every line's
// stresses ahead (96 registers, 18 warps) was slower also where a third of the points yield
// (35.0 us against 33.9 us at 32³).
template <bool DIAG, bool APEX>
__global__ void __launch_bounds__(HT_THREADS, (DIAG && !APEX) ? 3 : 2) hex27_incr_kernel(const IncrArgs a) {
    extern __shared__ __align__(16) unsigned char incr_smem[];
    IncrSmem& S = *reinterpret_cast<IncrSmem*>(incr_smem);
    const int lane = threadIdx.x & 31, w = ht_warp(), la = w % 3, lb = w / 3;
    const int64_t tile = a.tile_list ? __ldg(a.tile_list + blockIdx.x) : (int64_t)blockIdx.x;
    if (a.apex_t) {
        pdl_enter();   // before a block may leave: a grid that waits for nothing would release its successor
        if ((__ldg(a.apex_t + tile) != 0) != APEX) return;
    }
    const int64_t e = tile * 32 + lane;
    const bool act = e < a.nels;
    // the incremental sweep models the FP64 problem: its ε² is FP64's
    const float EPS2 = (float)eps2<double>();
    const bool plastic = a.plastic != 0;
    const uint64_t pol = l2_evict_first();
    // The stages run over (ξ, ζ, η): node line (j = lb, k = la), points (qx = la, ·, qz = lb). The
    // derivative taken last rounds at the scale of the whole increment instead of its own
    // direction's, and the vertical is the one that layered models vary along.
    // base data of the thread's three points q = la + 3qy + 9lb
    const float* base = a.base_t + (tile * 27 + la + 9 * lb) * BASE_FIELDS * 32 + lane;
    constexpr int QS = 3 * BASE_FIELDS * 32;
    const int t0 = 3 * lb + 9 * la;   // first node of the line, tensor order

    uint32_t n[3];   // byte offsets of the line's nodes
#pragma unroll
    for (int i = 0; i < 3; ++i) n[i] = 4u * (uint32_t)__ldg(a.el2n_t + (tile * 27 + t0 + i) * 32 + lane);
    const uint32_t nc = 4u * (uint32_t)__ldg(a.el2n_t + (tile * 27 + 13) * 32 + lane);   // the element's centre node
    float F[3] = {0.0f, 0.0f, 0.0f};
    if (plastic) {
#pragma unroll
        for (int q = 0; q < 3; ++q) F[q] = ldg_stream(base + q * QS + 6 * 32, pol);
    }
    const float* gt = a.geo_t + tile * 10 * 32 + lane;
    float Ji[9];
#pragma unroll
    for (int r = 0; r < 9; ++r) Ji[r] = (!DIAG || r % 4 == 0) ? __ldg(gt + r * 32) : 0.0f;
    const float detJ = __ldg(gt + 9 * 32);   // 0 on padding lanes
    const int ph = __ldg(a.phase_t + e), phP = __ldg(a.phase_t + ((a.nels + 31) / 32) * 32 + e);
    if (threadIdx.x < MAXPH) S.PT[threadIdx.x] = a.ph[threadIdx.x];
    if (!a.apex_t) pdl_enter();   // everything so far is constant over the iterations
    float dP[4];
    if (a.dofs_linear) {
        const float4 p4 = ld_coherent(reinterpret_cast<const float4*>(a.dP) + (act ? e : 0));
        dP[0] = p4.x; dP[1] = p4.y; dP[2] = p4.z; dP[3] = p4.w;
    } else {
#pragma unroll
        for (int p = 0; p < 4; ++p) dP[p] = ld_coherent(a.dP + elem_dof(a, tile, lane, p));
    }
    float g[3][3][3];
    {
        // only gradients are taken: the increments relative to the centre node's, so that the
        // interpolations before a derivative round at the scale of the differences
        float v[3][3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const float vc = ld_coherent(ht_at(a.dv[c], nc));
#pragma unroll
            for (int i = 0; i < 3; ++i) v[c][i] = ld_coherent(ht_at(a.dv[c], n[i])) - vc;
        }
        ht_gradient<float, 3>(v, S.S1, S.S2, la, lb, lane, g);
    }
    const float xi = ht_xr<float>(la), ze = ht_xr<float>(lb);
    const float wxz = detJ * ht_wr<float>(la) * ht_wr<float>(lb);

    // physical gradients ∂δv_c/∂x_k = Σ_d g[c][d] ∂ξ_d/∂x_k, in place (d = ξ, ζ, η on the way in)
#pragma unroll
    for (int q = 0; q < 3; ++q)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const float r0 = g[c][0][q], r1 = g[c][2][q], r2 = g[c][1][q];
#pragma unroll
            for (int k = 0; k < 3; ++k)
                g[c][k][q] = DIAG ? (k == 0 ? r0 : k == 1 ? r1 : r2) * Ji[4 * k]
                                  : fmaf(r0, Ji[3 * k], fmaf(r1, Ji[1 + 3 * k], r2 * Ji[2 + 3 * k]));
        }
    // δP along the η line, Pc + Py·η, from the centre value and the slopes (the four DoFs are
    // near one another: the slopes round little)
    const float Pc = fmaf(xi, dP[1] - dP[0], fmaf(ze, dP[3] - dP[0], dP[0])), Py = dP[2] - dP[0];
    // (S.PT: written before the gradient's barriers by warps 0, read after them by all: the block
    // barrier below orders it)
    __syncthreads();
    const IncrPhase M = S.PT[ph];
    {
        // continuity: −∇·δv − δP/(bulk·Δt) (pressure_residual.jl:132-158); the storage term's
        // phase is that of the pressure DoFs
        const float invbulkdt = S.PT[phP].invbulkdt;
        float f[3];
#pragma unroll
        for (int q = 0; q < 3; ++q)
            f[q] = -(g[0][0][q] + g[1][1][q] + g[2][2][q] + fmaf((float)ht_x(q), Py, Pc) * invbulkdt) * (wxz * (float)ht_w(q));
        const float s = f[0] + f[1] + f[2], sy = (float)HT_GA * (f[2] - f[0]);
        S.rp[w][0][lane] = fmaf(1.0f - xi - ze, s, -sy);
        S.rp[w][1][lane] = xi * s;
        S.rp[w][2][lane] = sy;
        S.rp[w][3][lane] = ze * s;
    }
    unsigned reads = 0;
    float bq[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        const float Pq = fmaf((float)ht_x(q), Py, Pc);
        const float dO = wxz * (float)ht_w(q);
        // deviatoric strain-rate increment and the stress increment
        const float tr = (g[0][0][q] + g[1][1][q] + g[2][2][q]) * (1.0f / 3.0f);
        const float ed[6] = {g[0][0][q] - tr, g[1][1][q] - tr, g[2][2][q] - tr, 0.5f * (g[0][1][q] + g[1][0][q]),
                             0.5f * (g[0][2][q] + g[2][0][q]), 0.5f * (g[1][2][q] + g[2][1][q])};
        float twoe = M.twoe, inv_den = M.inv_den;
        if (a.eta_t) {
            const float eq = act ? __ldg(a.eta_t + (tile * 27 + la + 3 * q + 9 * lb) * 32 + lane) : 1.0f;
            const float etave = 1.0f / (1.0f / eq + M.invG_dt);
            twoe = 2.0f * etave;
            inv_den = 1.0f / (etave + M.den_rest);
        }
        float tau[6];
#pragma unroll
        for (int c = 0; c < 6; ++c) tau[c] = twoe * ed[c];
        if (plastic) {
            // Elastic bound: τII = sqrt(‖τ‖² + ε²) is 1-Lipschitz in the J2 norm
            // ‖τ‖² = ½Σ τ_ii² + Σ_{i<j} τ_ij², so the trial yield value satisfies
            // F(τb + δτ) ≤ F_k + ‖δτ‖ + sinϕ·|δP|. Where that bound (with a 1e-3
            // relative margin over the rounding of either path) stays negative,
            // base and trial are both elastic, the return leaves the increment
            // unchanged (dp_increment gives δτ exactly), and the base trial
            // stress is not needed.
            const float dd = 0.5f * (tau[0] * tau[0] + tau[1] * tau[1] + tau[2] * tau[2]) + tau[3] * tau[3] +
                             tau[4] * tau[4] + tau[5] * tau[5];
            // (sqrt(dd) + |sinϕ·δP|)·1.001 + 1e-20 < −F_k, compared on squares
            const float lim = -(F[q] + 1e-20f) * 0.999000999f - fabsf(M.sphi * Pq);
            if (!(lim > 0.0f && dd < lim * lim)) {
                reads += act ? 1u : 0u;
                float t[6];
#pragma unroll
                for (int c = 0; c < 6; ++c) t[c] = ldg_stream(base + q * QS + c * 32, pol);
                const float Jk = 0.5f * (t[0] * t[0] + t[1] * t[1] + t[2] * t[2]) + t[3] * t[3] + t[4] * t[4] + t[5] * t[5];
                if (APEX && Jk < 1e-6f * M.cC * M.cC) {
                    // within 1e-3·C·cosϕ of the yield-surface apex the return direction
                    // is ill-conditioned: this point's increment is formed in FP64
                    ApexIn in;
#pragma unroll
                    for (int c = 0; c < 6; ++c) { in.tb[c] = t[c]; in.dtt[c] = tau[c]; }
                    in.Fk = F[q]; in.Pq = Pq; in.twoe = twoe; in.sphi = M.sphi; in.inv_den = inv_den;
                    const ApexOut o = apex_increment_f64(in);
#pragma unroll
                    for (int c = 0; c < 6; ++c) tau[c] = o.tau[c];
                } else {
                    float out[6];
                    dp_increment<float, true>(t, F[q], tau, Pq, twoe, M.sphi, inv_den, EPS2, out);
#pragma unroll
                    for (int c = 0; c < 6; ++c) tau[c] = out[c];
                }
            }
        }
        // reference-frame fluxes g[c][d] = dΩ Σ_k ∂ξ_d/∂x_k σ_kc, σ = δτ − δP·I; d = ξ, ζ, η
        const float sg[3][3] = {{tau[0] - Pq, tau[3], tau[4]}, {tau[3], tau[1] - Pq, tau[5]}, {tau[4], tau[5], tau[2] - Pq}};
#pragma unroll
        for (int f = 0; f < 3; ++f) {
            const int d = f == 0 ? 0 : 3 - f;
            const float k0 = dO * Ji[DIAG ? 4 * d : d];
#pragma unroll
            for (int c = 0; c < 3; ++c)
                g[c][f][q] = DIAG ? k0 * sg[d][c]
                                  : fmaf(k0, sg[0][c], dO * fmaf(Ji[d + 3], sg[1][c], Ji[d + 6] * sg[2][c]));
        }
        // EOS density increment ρ0·δP/K (momentum_residuals.jl:11-16)
        bq[q] = M.rho0beta * Pq * dO;
    }
    ht_scatter_z<float, 3>(g, [&](int c, int q) { return -a.g[c] * bq[q]; }, S.S2, la, lb, lane);
    __syncthreads();   // the point lines' fluxes and their parts of the pressure residual
    // the three warps of one b sum the pressure residual for themselves (their barrier inside
    // ht_scatter_yx orders it); b = 0 stores it
#pragma unroll
    for (int p = 0; p < 4; ++p)
        if (p % 3 == la) {
            float rp = S.rp[0][p][lane];
#pragma unroll
            for (int l = 1; l < 9; ++l) rp += S.rp[l][p][lane];
            if (act && lb == 0) a.RPinc[elem_dof(a, tile, lane, p)] = rp;
            S.pn[lb][p][lane] = __ldg(a.pscale_t + (tile * 4 + p) * 32 + lane) * rp;
        }
    float R[3][3];
    ht_scatter_yx<float, 3>(S.S1, S.S2, la, lb, lane, R);
    {
        // Pnum = γP/M_P·RP is affine in the element, so its term −|det J| Σ_d ∂ξ_d/∂x_c ∫ ∂_d N_a Pnum
        // is a table of the element: exact to one rounding, which a sum over the points is not
        // (Pnum is large against δP)
        const float Pn[4] = {S.pn[lb][0][lane], S.pn[lb][1][lane], S.pn[lb][2][lane], S.pn[lb][3][lane]};
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            float s[3];
#pragma unroll
            for (int d = 0; d < 3; ++d)
                s[d] = fmaf(Pn[0], c_inc_K[0][d][t0 + i], fmaf(Pn[1], c_inc_K[1][d][t0 + i],
                            fmaf(Pn[2], c_inc_K[2][d][t0 + i], Pn[3] * c_inc_K[3][d][t0 + i])));
#pragma unroll
            for (int c = 0; c < 3; ++c)
                R[c][i] -= detJ * (DIAG ? Ji[4 * c] * s[c] : fmaf(Ji[3 * c], s[0], fmaf(Ji[3 * c + 1], s[1], Ji[3 * c + 2] * s[2])));
        }
    }
    // when the next lane's element shares this line's ξ = +1 node as its ξ = −1 node (tiles that
    // run along ξ), its contribution is added here and one atomic per component is saved; any
    // shared node folds correctly
    const uint32_t n0n = __shfl_down_sync(0xffffffffu, n[0], 1);
    const int actn = __shfl_down_sync(0xffffffffu, (int)act, 1);
    const bool fold = lane < 31 && actn && n0n == n[2];
    const bool folded = __shfl_up_sync(0xffffffffu, (int)fold, 1) && lane > 0;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const float r0n = __shfl_down_sync(0xffffffffu, R[c][0], 1);
        if (fold) R[c][2] += r0n;
    }
    if (act) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            if (!folded) atomicAdd(ht_at(a.R[c], n[0]), R[c][0]);
            atomicAdd(ht_at(a.R[c], n[1]), R[c][1]);
            atomicAdd(ht_at(a.R[c], n[2]), R[c][2]);
        }
    }
    if (a.stress_reads) {
        const unsigned r = __reduce_add_sync(0xffffffffu, reads);
        if (lane == 0 && r) atomicAdd(a.stress_reads, (unsigned long long)r);
    }
}

}  // namespace

cudaError_t launch_incr_tiles(const IncrTileSrc& src, int64_t nels, const IncrArgs& dst, int32_t* flags,
                              cudaStream_t st) {
    // the Pnum table and the sweep's shared-memory limit, for the solve's device
    static const struct PnumTable {
        float K[4][3][27];
        PnumTable() { host_pnum_table(K); }
    } table;
    cudaError_t terr = cudaMemcpyToSymbolAsync(c_inc_K, table.K, sizeof(table.K), 0, cudaMemcpyHostToDevice, st);
    if (terr != cudaSuccess) return terr;
    for (auto fn : {hex27_incr_kernel<false, false>, hex27_incr_kernel<true, false>, hex27_incr_kernel<false, true>,
                    hex27_incr_kernel<true, true>}) {
        const cudaError_t err = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(IncrSmem));
        if (err != cudaSuccess) return err;
    }
    const int64_t nslots = (nels + 31) / 32 * 32;
    count_launch();
    incr_tiles_kernel<<<(unsigned)((nslots + 255) / 256), 256, 0, st>>>(src, nels, nslots, dst, flags);
    return cudaGetLastError();
}

namespace {
__global__ void add_f32_kernel(float* out, const float* x, const float* y, int64_t n) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = x[i] + y[i];
}
}  // namespace

cudaError_t launch_add_f32(float* out, const float* x, const float* y, int64_t n, cudaStream_t st) {
    count_launch();
    const int64_t blocks = std::min<int64_t>((n + 255) / 256, 148 * 8);
    add_f32_kernel<<<(unsigned)std::max<int64_t>(blocks, 1), 256, 0, st>>>(out, x, y, n);
    return cudaGetLastError();
}

int64_t incr_tile_slots(int num_sms) {
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, hex27_incr_kernel<true, false>, HT_THREADS, sizeof(IncrSmem));
    return (int64_t)num_sms * std::max(per_sm, 1);
}

namespace {
template <bool APEX>
cudaError_t launch_incr_tiles_of(const IncrArgs& a, int64_t ntiles, cudaStream_t st, bool pdl) {
    auto fn = a.diag_geometry ? hex27_incr_kernel<true, APEX> : hex27_incr_kernel<false, APEX>;
    count_launch();
    return launch_pdl(pdl, fn, dim3((unsigned)ntiles), dim3(HT_THREADS), sizeof(IncrSmem), st, a);
}
}  // namespace

cudaError_t launch_hex27_incr(const IncrArgs& a, cudaStream_t st, bool pdl) {
    const int64_t ntiles = a.tile_list ? a.tile_count : (a.nels + 31) / 32;
    if (ntiles < 1) return cudaSuccess;
    const cudaError_t err = launch_incr_tiles_of<false>(a, ntiles, st, pdl);
    if (err != cudaSuccess || !a.apex_t) return err;
    return launch_incr_tiles_of<true>(a, ntiles, st, pdl);
}

}  // namespace femb
