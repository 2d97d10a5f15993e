// Newton assembly of the P1 grad-grad (scalar potential / Laplace) operator.
//
// Element arithmetic of compute_K_dK (fem_c/ctools.c:730-919), one thread per element,
// scattered into a fixed CSR pattern through the slot map:
//   Jm = sum_i X_i (x) dphi_i, H = Jm^-T sum_i dphi_i x_i        (ctools.c:506-547)
//   mu, mu' = B-spline in log10|H| or constant                   (ctools.c:317-346)
//   K_ab  = sum_q mu det w_q (Jm^-T dphi_a . Jm^-T dphi_b)
//   dK_ab = sum_q [|H| >= 1e-14] mu' det w_q (g_a . H)(g_b . H) / |H|
// For linear tetrahedra the gradients are constant per element, so mu is evaluated once
// and the sums over q factor through sum_q w_q.
//
// By default the values are added deterministically: one launch over all materials' elements stores
// each element's 10 upper-triangle values (of one matrix, or pairs of two), then one thread per CSR
// entry sums the entry's couplings in element order from the pattern's sorted coupling list and
// writes (or adds) the outputs, so the result does not depend on the launch.  SNP_ASSEMBLY=atomic,
// or a pattern without coupling lists, adds each element's contributions with float64 atomics.
#include <cstdlib>
#include <cstring>
#include <vector>

#include "snp_common.cuh"
#include "snp_internal.cuh"

namespace snp {

namespace {

constexpr int kBlock = 128;

constexpr int kGgBatch = 4;     // contributions an entry requests together
constexpr int kGradMats = 16;  // materials of one launch (its parameters hold their tables)

struct GradMat {
    int64_t e0, n;             // first element in the stored values, number of elements
    const int32_t *cells;
    const double *knots, *ctrl;
    double H_min, mu_H_min;
    double wj;                 // J gets dK + wj K
    int32_t type, degree, n_ctrl;
    int32_t block0;            // first block of this material
};

struct GradArgs {
    GradMat m[kGradMats];
    int32_t n_mats;
    const double *nodes, *dphi0, *w, *x;
    int32_t nq;
    int32_t table;             // doubles of shared memory before the tile
    // packed store: T[e * 10 + q] is the K, dK or J value (one matrix) or a pair of them
    double *T;
    // atomic mode
    const int32_t *slots;      // of element 0 of the stored values
    double *K, *dK, *J;
};

// Which values the element kernel hands on, by the outputs that are wanted.
enum GradStore {
    kGradAtomic = 0,
    kGradK = 1,   // K
    kGradD = 2,   // dK
    kGradJ = 3,   // J
    kGradKD = 4,  // K, dK (J is their sum)
    kGradKJ = 5,  // K, J
    kGradDJ = 6,  // dK, J
};

// index of the pair (i, k), i <= k, in the upper triangle's rows
__device__ __forceinline__ int tri4(int i, int k) { return i * 4 - (i * (i - 1)) / 2 + (k - i); }

// Element values, one thread per element, staged in shared memory so that a block writes one run.
// Two materials of 150k elements with K and J: 23 us in one launch (2 x 13.7 us before, one launch
// per material); it writes 48 MB, and waits on the dependent chain of an element's inverse, root,
// logarithm and spline at the 20 warps an SM that 92 registers allow.
template <int STORE>
__global__ void __launch_bounds__(kBlock) k_gradgrad(const __grid_constant__ GradArgs a) {
    constexpr int kVals = STORE >= kGradKD ? 2 : 1;
    extern __shared__ double sm[];
    int im = 0;
    while (im + 1 < a.n_mats && (int)blockIdx.x >= a.m[im + 1].block0) ++im;
    const GradMat &M = a.m[im];
    const int n_t = M.type == 1 ? M.n_ctrl + M.degree + 1 : 0;
    double *s_dphi = sm;
    double *s_t = sm + 12;
    double *s_c = s_t + n_t;
    double *tile = sm + a.table;
    for (int t = threadIdx.x; t < 12; t += blockDim.x) s_dphi[t] = __ldg(a.dphi0 + t);
    for (int t = threadIdx.x; t < n_t; t += blockDim.x) s_t[t] = __ldg(M.knots + t);
    for (int t = threadIdx.x; t < (M.type == 1 ? M.n_ctrl : 0); t += blockDim.x) s_c[t] = __ldg(M.ctrl + t);
    __syncthreads();
    double wsum = 0.0;
    for (int q = 0; q < a.nq; ++q) wsum += __ldg(a.w + q);

    const int64_t base = (int64_t)((int)blockIdx.x - M.block0) * kBlock;
    const int cnt = (int)min(M.n - base, (int64_t)kBlock);
    if ((int)threadIdx.x < cnt) {
        const int64_t e = base + threadIdx.x;
        const int4 cv = __ldg(reinterpret_cast<const int4 *>(M.cells) + e);
        const int cidx[4] = {cv.x, cv.y, cv.z, cv.w};
        double Jm[9];
#pragma unroll
        for (int r = 0; r < 9; ++r) Jm[r] = 0.0;
        double gr[3] = {0.0, 0.0, 0.0};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const double X0 = __ldg(a.nodes + 3 * (int64_t)cidx[i]);
            const double X1 = __ldg(a.nodes + 3 * (int64_t)cidx[i] + 1);
            const double X2 = __ldg(a.nodes + 3 * (int64_t)cidx[i] + 2);
            const double xi = __ldg(a.x + cidx[i]);
#pragma unroll
            for (int l = 0; l < 3; ++l) {
                const double d = s_dphi[3 * i + l];
                Jm[0 + l] += X0 * d;
                Jm[3 + l] += X1 * d;
                Jm[6 + l] += X2 * d;
                gr[l] += d * xi;
            }
        }
        const double det = Jm[0] * (Jm[4] * Jm[8] - Jm[7] * Jm[5]) - Jm[1] * (Jm[3] * Jm[8] - Jm[5] * Jm[6]) +
                           Jm[2] * (Jm[3] * Jm[7] - Jm[4] * Jm[6]);
        const double id = 1.0 / det;
        double Ji[9];
        Ji[0] = (Jm[4] * Jm[8] - Jm[7] * Jm[5]) * id;
        Ji[1] = (Jm[2] * Jm[7] - Jm[1] * Jm[8]) * id;
        Ji[2] = (Jm[1] * Jm[5] - Jm[2] * Jm[4]) * id;
        Ji[3] = (Jm[5] * Jm[6] - Jm[3] * Jm[8]) * id;
        Ji[4] = (Jm[0] * Jm[8] - Jm[2] * Jm[6]) * id;
        Ji[5] = (Jm[3] * Jm[2] - Jm[0] * Jm[5]) * id;
        Ji[6] = (Jm[3] * Jm[7] - Jm[6] * Jm[4]) * id;
        Ji[7] = (Jm[6] * Jm[1] - Jm[0] * Jm[7]) * id;
        Ji[8] = (Jm[0] * Jm[4] - Jm[3] * Jm[1]) * id;
        // transposed map (mat_vec with transpose = 1, ctools.c:415-438)
        double H[3];
        H[0] = Ji[0] * gr[0] + Ji[3] * gr[1] + Ji[6] * gr[2];
        H[1] = Ji[1] * gr[0] + Ji[4] * gr[1] + Ji[7] * gr[2];
        H[2] = Ji[2] * gr[0] + Ji[5] * gr[1] + Ji[8] * gr[2];
        double gphi[4][3];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const double d0 = s_dphi[3 * i], d1 = s_dphi[3 * i + 1], d2 = s_dphi[3 * i + 2];
            gphi[i][0] = Ji[0] * d0 + Ji[3] * d1 + Ji[6] * d2;
            gphi[i][1] = Ji[1] * d0 + Ji[4] * d1 + Ji[7] * d2;
            gphi[i][2] = Ji[2] * d0 + Ji[5] * d1 + Ji[8] * d2;
        }
        const double hm = sqrt(H[0] * H[0] + H[1] * H[1] + H[2] * H[2]);
        double dmu;
        const double mu = bspline_mu(M.type, M.degree, M.n_ctrl, s_t, s_c, M.H_min, M.mu_H_min, hm, dmu);
        const double kf = mu * det * wsum;
        const double df = (hm >= 1e-14) ? dmu * det * wsum / hm : 0.0;
        double p[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) p[i] = gphi[i][0] * H[0] + gphi[i][1] * H[1] + gphi[i][2] * H[2];
        const int32_t *sl = STORE == kGradAtomic ? a.slots + 16 * (M.e0 + e) : nullptr;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
#pragma unroll
            for (int k = i; k < 4; ++k) {
                const double kv = kf * (gphi[i][0] * gphi[k][0] + gphi[i][1] * gphi[k][1] + gphi[i][2] * gphi[k][2]);
                const double dv = df * p[i] * p[k];
                const double jv = dv + M.wj * kv;
                if constexpr (STORE == kGradAtomic) {
                    const int s1 = __ldg(sl + 4 * i + k);
                    if (a.K) atomicAdd(a.K + s1, kv);
                    if (a.dK) atomicAdd(a.dK + s1, dv);
                    if (a.J) atomicAdd(a.J + s1, jv);
                    if (k != i) {
                        const int s2 = __ldg(sl + 4 * k + i);
                        if (a.K) atomicAdd(a.K + s2, kv);
                        if (a.dK) atomicAdd(a.dK + s2, dv);
                        if (a.J) atomicAdd(a.J + s2, jv);
                    }
                } else {
                    const int at = (int)threadIdx.x * kPackPairs4 + tri4(i, k);
                    if constexpr (kVals == 1)
                        tile[at] = STORE == kGradK ? kv : STORE == kGradD ? dv : jv;
                    else
                        reinterpret_cast<double2 *>(tile)[at] =
                            make_double2(STORE == kGradDJ ? dv : kv, STORE == kGradKD ? dv : jv);
                }
            }
        }
    }
    if constexpr (STORE != kGradAtomic) {
        __syncthreads();
        double2 *dst = reinterpret_cast<double2 *>(a.T + (M.e0 + base) * kPackPairs4 * kVals);
        for (int t = threadIdx.x; t < cnt * kPackPairs4 * kVals / 2; t += kBlock)
            dst[t] = reinterpret_cast<const double2 *>(tile)[t];
    }
}

struct GradEntryArgs {
    int64_t nnz;
    const int32_t *cptr, *cid;
    const double *T;
    uint32_t t0, n_t;          // value indices [t0, t0 + n_t) are stored
    double *first, *second, *sum;  // of the stored pair; first alone for one matrix
    int add;                   // add to the outputs, and leave entries without a coupling alone
};

// One thread per CSR entry; the pattern's coupling words are the value indices.
// Bound by L1: 4.8M gathers of a pair at 300k elements, each in a sector of its own and one
// sector per SM and cycle (17 us); batches of 2, 4, 6 or 8 measure alike.  27 us for K and J of both
// materials together; a launch per material that decoded (element, pair) and read the two matrices
// from separate blocks took 2 x 37.8 us, and torch added their sums in another 16 us.
template <int VALS>
__global__ void __launch_bounds__(256) k_gg_entries(GradEntryArgs r) {
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < r.nnz; p += (int64_t)gridDim.x * blockDim.x) {
        const int c0 = __ldg(r.cptr + p), c1 = __ldg(r.cptr + p + 1);
        double s0 = 0.0, s1 = 0.0;
        bool any = false;
        for (int c = c0; c < c1; c += kGgBatch) {
            uint32_t t[kGgBatch];
            double v0[kGgBatch], v1[kGgBatch];
#pragma unroll
            for (int u = 0; u < kGgBatch; ++u)
                t[u] = c + u < c1 ? (uint32_t)__ldg(r.cid + c + u) - r.t0 : 0xffffffffu;
#pragma unroll
            for (int u = 0; u < kGgBatch; ++u) {
                v0[u] = v1[u] = 0.0;
                if (t[u] < r.n_t) {
                    if constexpr (VALS == 2) {
                        const double2 v = __ldg(reinterpret_cast<const double2 *>(r.T) + t[u]);
                        v0[u] = v.x;
                        v1[u] = v.y;
                    } else {
                        v0[u] = __ldg(r.T + t[u]);
                    }
                }
            }
#pragma unroll
            for (int u = 0; u < kGgBatch; ++u)
                if (t[u] < r.n_t) {
                    any = true;
                    s0 += v0[u];
                    s1 += v1[u];
                }
        }
        if (r.add) {
            if (!any) continue;
            if (r.first) r.first[p] += s0;
            if (VALS == 2 && r.second) r.second[p] += s1;
            if (VALS == 2 && r.sum) r.sum[p] += s0 + s1;
        } else {
            if (r.first) r.first[p] = s0;
            if (VALS == 2 && r.second) r.second[p] = s1;
            if (VALS == 2 && r.sum) r.sum[p] = s0 + s1;
        }
    }
}

struct GradOut {
    double *K, *dK, *J;
    bool add;
};

template <int STORE>
int launch_elements(const GradArgs &a, int blocks, size_t tile_bytes, cudaStream_t st) {
    const size_t smem = sizeof(double) * (size_t)a.table + tile_bytes;
    auto kern = k_gradgrad<STORE>;
    if (smem > 48 * 1024)
        SNP_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    kern<<<blocks, kBlock, smem, st>>>(a);
    SNP_LAUNCH_CHECK();
    return SNP_OK;
}

// All materials' elements (consecutive elements of the pattern from e_first on), then the entries.
int gradgrad_run(const snp_pattern *pat, int64_t e_first, const GradMat *mats, int n_mats, const double *nodes,
                 const double *d_phi, const double *w, int32_t nq, const double *x, const GradOut &o, cudaStream_t st) {
    const char *env = getenv("SNP_ASSEMBLY");
    const bool atomic = (env && std::strcmp(env, "atomic") == 0) || !pat->has_contrib;
    int64_t n = 0;
    for (int m = 0; m < n_mats; ++m) n += mats[m].n;
    int store = kGradAtomic, vals = 1;
    if (!atomic) {
        if (o.K && o.dK) store = kGradKD;
        else if (o.K && o.J) store = kGradKJ;
        else if (o.dK && o.J) store = kGradDJ;
        else store = o.K ? kGradK : o.dK ? kGradD : kGradJ;
        vals = store >= kGradKD ? 2 : 1;
        const size_t need = (size_t)(kPackPairs4 * vals) * (size_t)n;
        if (pat->gg_terms.n < need) SNP_TRY(pat->gg_terms.alloc(need));
    } else if (!o.add) {
        for (double *out : {o.K, o.dK, o.J})
            if (out) SNP_CUDA_TRY(cudaMemsetAsync(out, 0, sizeof(double) * (size_t)pat->nnz, st));
    }
    if (!o.K && !o.dK && !o.J) return SNP_OK;
    int64_t e0 = 0;
    for (int m = 0; m < n_mats;) {
        GradArgs a{};
        a.nodes = nodes;
        a.dphi0 = d_phi;
        a.w = w;
        a.nq = nq;
        a.x = x;
        a.T = pat->gg_terms.p;
        a.slots = pat->slots.p + 16 * e_first;
        a.K = o.K;
        a.dK = o.dK;
        a.J = o.J;
        int64_t blocks = 0;
        for (; m < n_mats && a.n_mats < kGradMats; ++m) {
            const int64_t nb = (mats[m].n + kBlock - 1) / kBlock;
            if (nb == 0) continue;
            GradMat &M = a.m[a.n_mats++];
            M = mats[m];
            M.e0 = e0;
            M.block0 = (int32_t)blocks;
            blocks += nb;
            e0 += M.n;
            const int tab = 12 + (M.type == 1 ? 2 * M.n_ctrl + M.degree + 1 : 0);
            if (tab + tab % 2 > a.table) a.table = tab + tab % 2;
        }
        if (blocks == 0) continue;
        const size_t tile = sizeof(double) * kPackPairs4 * kBlock;
        switch (store) {
            case kGradAtomic: SNP_TRY(launch_elements<kGradAtomic>(a, (int)blocks, 0, st)); break;
            case kGradK: SNP_TRY(launch_elements<kGradK>(a, (int)blocks, tile, st)); break;
            case kGradD: SNP_TRY(launch_elements<kGradD>(a, (int)blocks, tile, st)); break;
            case kGradJ: SNP_TRY(launch_elements<kGradJ>(a, (int)blocks, tile, st)); break;
            case kGradKD: SNP_TRY(launch_elements<kGradKD>(a, (int)blocks, 2 * tile, st)); break;
            case kGradKJ: SNP_TRY(launch_elements<kGradKJ>(a, (int)blocks, 2 * tile, st)); break;
            default: SNP_TRY(launch_elements<kGradDJ>(a, (int)blocks, 2 * tile, st)); break;
        }
    }
    if (atomic || pat->nnz == 0) return SNP_OK;
    GradEntryArgs r{};
    r.nnz = pat->nnz;
    r.cptr = pat->cptr.p;
    r.cid = pat->cid.p;
    r.T = pat->gg_terms.p;
    r.t0 = (uint32_t)(e_first * kPackPairs4);
    r.n_t = (uint32_t)(n * kPackPairs4);
    r.add = o.add ? 1 : 0;
    r.first = store == kGradDJ ? o.dK : o.K ? o.K : o.dK ? o.dK : o.J;
    r.second = store == kGradKD ? o.dK : store == kGradKJ || store == kGradDJ ? o.J : nullptr;
    r.sum = store == kGradKD ? o.J : nullptr;
    if (vals == 2)
        k_gg_entries<2><<<wave_grid(k_gg_entries<2>, r.nnz, 256), 256, 0, st>>>(r);
    else
        k_gg_entries<1><<<wave_grid(k_gg_entries<1>, r.nnz, 256), 256, 0, st>>>(r);
    SNP_LAUNCH_CHECK();
    return SNP_OK;
}

int gradgrad_material(const char *who, GradMat &M, int64_t n_elems, const int32_t *cells, int32_t type, int32_t degree,
                      int32_t n_ctrl, const double *knots, const double *ctrl, double H_min, double mu_H_min,
                      double wj) {
    SNP_REQUIRE(type == 0 || type == 1, "%s: permeability type must be 0 or 1", who);
    if (type == 1) {
        SNP_REQUIRE(degree >= 0 && degree <= kMaxSplineDegree, "%s: spline degree %d unsupported", who, degree);
        SNP_REQUIRE(n_ctrl >= 1 && knots && ctrl, "%s: spline tables missing", who);
        SNP_REQUIRE(sizeof(double) * (12 + 2 * (size_t)n_ctrl + degree + 1) <= 200 * 1024,
                    "%s: spline tables too large", who);
    }
    SNP_REQUIRE(n_elems == 0 || cells, "%s: NULL input", who);
    SNP_REQUIRE(((uintptr_t)cells & 15) == 0, "cells must be 16-byte aligned");
    M = GradMat{0, n_elems, cells, knots, ctrl, H_min, mu_H_min, wj, type, degree, n_ctrl, 0};
    return SNP_OK;
}

}  // namespace
}  // namespace snp

extern "C" int snp_gradgrad_assemble(const snp_pattern *pat, int64_t elem_offset, int64_t n_elems, const double *nodes,
                                     const int32_t *cells, const double *d_phi, const double *w, int32_t n_quad,
                                     const double *x, int32_t perm_type, int32_t degree, int32_t n_ctrl,
                                     const double *knots, const double *ctrl, double H_min, double mu_H_min,
                                     double *K_vals, double *dK_vals, double *J_vals, void *stream) {
    snp::clear_error();
    SNP_REQUIRE(pat != nullptr && pat->dpe == 4, "snp_gradgrad_assemble: pattern with 4 DoFs per element required");
    SNP_REQUIRE(n_elems >= 0 && elem_offset >= 0 && elem_offset + n_elems <= pat->n_elems,
                "snp_gradgrad_assemble: element range outside the pattern");
    SNP_REQUIRE(n_quad >= 1, "snp_gradgrad_assemble: n_quad must be >= 1");
    SNP_REQUIRE(n_elems == 0 || (nodes && d_phi && w && x), "snp_gradgrad_assemble: NULL input");
    snp::GradMat M;
    SNP_TRY(snp::gradgrad_material("snp_gradgrad_assemble", M, n_elems, cells, perm_type, degree, n_ctrl, knots, ctrl,
                                   H_min, mu_H_min, 1.0));
    if (n_elems == 0) return SNP_OK;
    return snp::gradgrad_run(pat, elem_offset, &M, 1, nodes, d_phi, w, n_quad, x,
                             snp::GradOut{K_vals, dK_vals, J_vals, true}, snp::as_stream(stream));
}

extern "C" int snp_gradgrad_system(const snp_pattern *pat, int32_t n_mats, const snp_gradgrad_material *mats,
                                   const double *nodes, const double *d_phi, const double *w, int32_t n_quad,
                                   const double *x, double *K_vals, double *dK_vals, double *J_vals, void *stream) {
    snp::clear_error();
    SNP_REQUIRE(pat != nullptr && pat->dpe == 4, "snp_gradgrad_system: pattern with 4 DoFs per element required");
    SNP_REQUIRE(n_mats >= 0 && (n_mats == 0 || mats), "snp_gradgrad_system: NULL argument");
    SNP_REQUIRE(n_quad >= 1, "snp_gradgrad_system: n_quad must be >= 1");
    std::vector<snp::GradMat> m((size_t)n_mats);
    int64_t n = 0;
    for (int i = 0; i < n_mats; ++i) {
        const snp_gradgrad_material &P = mats[i];
        SNP_REQUIRE(P.n_elems >= 0 && n + P.n_elems <= pat->n_elems,
                    "snp_gradgrad_system: more elements than the pattern's");
        SNP_REQUIRE(P.J_weight == 1.0 || !(K_vals && dK_vals && J_vals),
                    "snp_gradgrad_system: with K, dK and J the weights must be 1");
        SNP_TRY(snp::gradgrad_material("snp_gradgrad_system", m[i], P.n_elems, P.cells, P.perm_type, P.degree, P.n_ctrl,
                                       P.knots, P.ctrl, P.H_min, P.mu_H_min, P.J_weight));
        n += P.n_elems;
    }
    SNP_REQUIRE(n == 0 || (nodes && d_phi && w && x), "snp_gradgrad_system: NULL input");
    return snp::gradgrad_run(pat, 0, m.data(), n_mats, nodes, d_phi, w, n_quad, x,
                             snp::GradOut{K_vals, dK_vals, J_vals, false}, snp::as_stream(stream));
}
