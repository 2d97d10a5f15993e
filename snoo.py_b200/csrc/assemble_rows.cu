// Deterministic two-phase assembly of the curl-curl Newton system into a fixed CSR pattern.
//
// The reference sums its element matrices into the global matrix in scipy's COO->CSR
// conversion (fem_c/interface_c.pyx:365-368, csr_array((v, (i, j))) sums duplicates) and adds
// the materials' matrices with K += this_K (curl_curl_assembler.py:900-932).  Here phase 1 is
// the single-launch element kernel (k_curlcurl, assemble_curlcurl.cu) storing each element's
// values instead of adding them into the CSR: the 21 values of the upper triangle of K, dK or
// J = K + dK (the reference kernels' arithmetic) and the six residual and reduced-rhs terms, as
// structure-of-arrays blocks over the pattern's elements.  Phase 2 (this file) forms
//
//   A_p = sum over the couplings (e, a, b) of CSR position p, in element order, of A_e,ab
//   F_i = sum over the incidences (e, a) of DoF i, in element order, of F_e,a
//
// from the pattern's sorted coupling list (cid / cptr) and incidence lists (inc / inc_ptr): one
// thread per CSR entry and one per DoF, no atomics, every output written exactly once.  Each
// entry is the same sum whatever the launch shape, so the results are bitwise repeatable.
#include <vector>

#include "snp_common.cuh"
#include "snp_internal.cuh"

namespace snp {

namespace {

constexpr int kEntryBlock = 256;

// What the entry kernel writes, from which blocks.
enum EntryMode {
    kEntJ = 1,   // J from the J block
    kEntK = 2,   // K from the K block
    kEntKD = 3,  // K and dK from their blocks, J = K + dK
    kEntD = 4,   // dK alone
};

struct EntryArgs {
    int64_t nnz, n_elems;
    const int32_t *cptr, *cid;
    const double *terms;
    int b0, b1;  // block offsets of the first (and second) matrix read
    double *K, *dK, *J;
    float *J32;
};

// value index of coupling word t = e * 21 + q (the pattern's cid) in the block layout: q * n_elems + e
__device__ __forceinline__ int64_t coupling_index(uint32_t t, int64_t S) {
    const uint32_t e = t / (uint32_t)kPackPairs;
    return (int64_t)(t - e * (uint32_t)kPackPairs) * S + (int64_t)e;
}

// Each thread sums kEntU consecutive entries.  The entries' first two contributions are
// requested together before any is added (a CSR entry has 1.9 on average), so a thread keeps
// up to 2 kEntU independent gathers in flight; longer entries finish in a loop.  Every entry's
// sum runs over its contributions in order.
constexpr int kEntU = 4;

template <int MODE>
__global__ void __launch_bounds__(kEntryBlock) k_cc_entries(EntryArgs r) {
    const int64_t S = r.n_elems;
    const double *m0 = r.terms + (int64_t)r.b0 * S;
    const double *m1 = r.terms + (int64_t)r.b1 * S;
    const int64_t n_groups = (r.nnz + kEntU - 1) / kEntU;
    for (int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; g < n_groups; g += (int64_t)gridDim.x * blockDim.x) {
        const int64_t p0 = g * kEntU;
        int c[kEntU + 1];
#pragma unroll
        for (int u = 0; u <= kEntU; ++u) c[u] = __ldg(r.cptr + (p0 + u < r.nnz ? p0 + u : r.nnz));
        uint32_t t0[kEntU], t1[kEntU];
#pragma unroll
        for (int u = 0; u < kEntU; ++u) {
            t0[u] = c[u + 1] > c[u] ? (uint32_t)__ldg(r.cid + c[u]) : 0u;
            t1[u] = c[u + 1] > c[u] + 1 ? (uint32_t)__ldg(r.cid + c[u] + 1) : 0u;
        }
        double a0[kEntU], a1[kEntU], d0[kEntU], d1[kEntU];
#pragma unroll
        for (int u = 0; u < kEntU; ++u) {
            const int64_t i0 = coupling_index(t0[u], S), i1 = coupling_index(t1[u], S);
            a0[u] = c[u + 1] > c[u] ? __ldg(m0 + i0) : 0.0;
            a1[u] = c[u + 1] > c[u] + 1 ? __ldg(m0 + i1) : 0.0;
            d0[u] = 0.0;
            d1[u] = 0.0;
            if constexpr (MODE == kEntKD) {
                d0[u] = c[u + 1] > c[u] ? __ldg(m1 + i0) : 0.0;
                d1[u] = c[u + 1] > c[u] + 1 ? __ldg(m1 + i1) : 0.0;
            }
        }
#pragma unroll
        for (int u = 0; u < kEntU; ++u) {
            const int64_t p = p0 + u;
            if (p >= r.nnz) break;
            double s0 = a0[u], s1 = d0[u];
            if (c[u + 1] > c[u] + 1) {
                s0 += a1[u];
                s1 += d1[u];
            }
            for (int k = c[u] + 2; k < c[u + 1]; ++k) {
                const int64_t ik = coupling_index((uint32_t)__ldg(r.cid + k), S);
                s0 += __ldg(m0 + ik);
                if constexpr (MODE == kEntKD) s1 += __ldg(m1 + ik);
            }
            if constexpr (MODE == kEntJ) {
                if (r.J) r.J[p] = s0;
                if (r.J32) r.J32[p] = (float)s0;
            } else if constexpr (MODE == kEntK) {
                r.K[p] = s0;
            } else if constexpr (MODE == kEntD) {
                r.dK[p] = s0;
            } else {
                if (r.K) r.K[p] = s0;
                if (r.dK) r.dK[p] = s1;
                if (r.J) r.J[p] = s0 + s1;
                if (r.J32) r.J32[p] = (float)(s0 + s1);
            }
        }
    }
}

// F_i and rhs_i from the six-term blocks over DoF i's incidences (e * 8 + a, element order)
__global__ void __launch_bounds__(kEntryBlock)
    k_cc_dofvec(int32_t n, int64_t n_elems, const int32_t *__restrict__ inc_ptr, const int32_t *__restrict__ inc,
                const double *__restrict__ Fe, const double *__restrict__ Re, double *__restrict__ F,
                double *__restrict__ rhs) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        double f = 0.0, rr = 0.0;
        for (int t = __ldg(inc_ptr + i); t < __ldg(inc_ptr + i + 1); ++t) {
            const uint32_t u = (uint32_t)__ldg(inc + t);
            const int64_t idx = (int64_t)(u & 7u) * n_elems + (int64_t)(u >> 3);
            if (F) f += __ldg(Fe + idx);
            if (rhs) rr += __ldg(Re + idx);
        }
        if (F) F[i] = f;
        if (rhs) rhs[i] = rr;
    }
}

// ---------------------------------------------------------------- packed element values

// Element ranges whose reduced-rhs terms (no source field) are zero, or whose dK is unless x holds an
// infinity or a NaN (constant reluctance): phase 1 does not store the zeros and phase 2 does not read
// them.
constexpr int kMaxRanges = 16;
struct ZeroRanges {
    int n = 0;
    int32_t lo[kMaxRanges], hi[kMaxRanges];
    bool add(int64_t l, int64_t h) {
        if (n > 0 && hi[n - 1] == l) {
            hi[n - 1] = (int32_t)h;
            return true;
        }
        if (n == kMaxRanges) return false;
        lo[n] = (int32_t)l;
        hi[n] = (int32_t)h;
        ++n;
        return true;
    }
};

__device__ __forceinline__ bool in_ranges(const ZeroRanges &z, int32_t e) {
    bool in = false;
    for (int i = 0; i < z.n; ++i) in |= e >= z.lo[i] && e < z.hi[i];
    return in;
}

struct PackedEntryArgs {
    int64_t nnz;
    const int32_t *cptr, *cid;
    const double *m0, *m1;  // K (or J) and dK values
    double *K, *dK, *J;
    float *J32;
    // value indices [lo, hi) whose dK is zero and not stored (up to two ranges), but for the elements
    // that kept[] lists where one of any[] is set
    uint32_t lo[2], hi[2];
    const uint8_t *kept, *any;
    int32_t n_any;  // a multiple of 16
};

// One thread per CSR entry: its contributions' values (the pattern's coupling words are the value
// indices) summed in element order, the first two requested together (an entry has 1.9 on
// average; a diagonal about five).  Bound by the gathers' sectors and the streams of the outputs and
// words, about 1.0 GB a call at 1.16M tets; a warp's 32 consecutive entries are two rows, whose
// elements' values are runs of doubles, so most of each sector is used.  Decoding element and
// pair from a coupling id and four entries a thread took 1600 instructions per 128 entries
// (422 us at 1.16M tets); from the block layout the sums took 571 us, this way 205 us.
//
// KEPT: elements of the ranges may have values (an infinity or a NaN in x).  The ordinary call's loop does
// not look at kept[]: with one loop for both a call at 1.16M tets took 457 us instead of 445.
template <int MODE, bool KEPT>
__device__ __forceinline__ void packed_entries(const PackedEntryArgs &r) {
    auto stored = [&](uint32_t t) {
        if constexpr (MODE == kEntKD || MODE == kEntD) {
            const bool zero = (t >= r.lo[0] && t < r.hi[0]) || (t >= r.lo[1] && t < r.hi[1]);
            if constexpr (KEPT) return !zero || __ldg(r.kept + t / (uint32_t)kPackPairs) != 0;
            else return !zero;
        } else {
            return true;
        }
    };
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < r.nnz; p += (int64_t)gridDim.x * blockDim.x) {
        const int c0 = __ldcs(r.cptr + p), c1 = __ldg(r.cptr + p + 1);
        double s0 = 0.0, s1 = 0.0;
        if (c1 > c0) {  // every entry of a pattern has a contribution
            const bool two = c1 > c0 + 1;
            const uint32_t t0 = (uint32_t)__ldg(r.cid + c0), t1 = two ? (uint32_t)__ldg(r.cid + c0 + 1) : t0;
            const bool n0 = stored(t0), n1 = stored(t1) && two;
            double b0 = 0.0, b1 = 0.0, e0 = 0.0, e1 = 0.0;
            if constexpr (MODE == kEntD) {
                if (n0) b0 = __ldg(r.m0 + t0);
                if (n1) b1 = __ldg(r.m0 + t1);
            } else {
                b0 = __ldg(r.m0 + t0);
                if (two) b1 = __ldg(r.m0 + t1);
                if constexpr (MODE == kEntKD) {
                    if (n0) e0 = __ldg(r.m1 + t0);
                    if (n1) e1 = __ldg(r.m1 + t1);
                }
            }
            s0 = two ? b0 + b1 : b0;
            s1 = two ? e0 + e1 : e0;
            for (int k = c0 + 2; k < c1; ++k) {
                const uint32_t t = (uint32_t)__ldg(r.cid + k);
                if constexpr (MODE == kEntD) {
                    if (stored(t)) s0 += __ldg(r.m0 + t);
                } else {
                    s0 += __ldg(r.m0 + t);
                    if constexpr (MODE == kEntKD)
                        if (stored(t)) s1 += __ldg(r.m1 + t);
                }
            }
        }
        if constexpr (MODE == kEntKD) {
            if (r.K) __stcs(r.K + p, s0);
            if (r.dK) __stcs(r.dK + p, s1);
            if (r.J) __stcs(r.J + p, s0 + s1);
            if (r.J32) r.J32[p] = (float)(s0 + s1);
        } else if constexpr (MODE == kEntJ) {
            if (r.J) __stcs(r.J + p, s0);
            if (r.J32) r.J32[p] = (float)s0;
        } else if constexpr (MODE == kEntK) {
            __stcs(r.K + p, s0);
        } else {
            __stcs(r.dK + p, s0);
        }
    }
}

template <int MODE>
__global__ void __launch_bounds__(kEntryBlock) k_cc_entries_packed(PackedEntryArgs r) {
    if constexpr (MODE == kEntKD || MODE == kEntD) {
        bool any = false;
        for (int i = threadIdx.x & 31; i < r.n_any / 16; i += 32) {
            const uint4 v = __ldg(reinterpret_cast<const uint4 *>(r.any) + i);
            any |= (v.x | v.y | v.z | v.w) != 0u;
        }
        if (__any_sync(0xffffffffu, any)) return packed_entries<MODE, true>(r);
    }
    packed_entries<MODE, false>(r);
}

// F_i and rhs_i from the packed six-term values over DoF i's incidences, in element order
__global__ void __launch_bounds__(kEntryBlock)
    k_cc_dofvec_packed(int32_t n, const int32_t *__restrict__ inc_ptr, const int32_t *__restrict__ inc,
                       const double *__restrict__ Fe, const double *__restrict__ Re, double *__restrict__ F,
                       double *__restrict__ rhs, ZeroRanges no_source) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        double f = 0.0, rr = 0.0;
        for (int t = __ldg(inc_ptr + i); t < __ldg(inc_ptr + i + 1); ++t) {
            const uint32_t u = (uint32_t)__ldg(inc + t);
            const int64_t idx = (int64_t)(u >> 3) * 6 + (int64_t)(u & 7u);
            if (F) f += __ldg(Fe + idx);
            if (rhs && !in_ranges(no_source, (int32_t)(u >> 3))) rr += __ldg(Re + idx);
        }
        if (F) F[i] = f;
        if (rhs) rhs[i] = rr;
    }
}

template <int MODE>
int launch_packed_entries(const PackedEntryArgs &r, cudaStream_t st) {
    auto kern = k_cc_entries_packed<MODE>;
    kern<<<wave_grid(kern, r.nnz, kEntryBlock), kEntryBlock, 0, st>>>(r);
    SNP_LAUNCH_CHECK();
    return SNP_OK;
}

// Which element matrices an output set needs.
struct PackedNeeds {
    bool k, d, j;
};
PackedNeeds packed_needs(const SystemOut &o) {
    const bool wj = o.J != nullptr || o.J32 != nullptr;
    const bool only_j = o.fused_j && wj && !o.K && !o.dK;
    return {!only_j && (o.K || wj), !only_j && (o.dK || wj), only_j};
}

template <int MODE>
int launch_entries(const EntryArgs &r, cudaStream_t st) {
    auto kern = k_cc_entries<MODE>;
    kern<<<wave_grid(kern, (r.nnz + kEntU - 1) / kEntU, kEntryBlock), kEntryBlock, 0, st>>>(r);
    SNP_LAUNCH_CHECK();
    return SNP_OK;
}

}  // namespace

bool rows_supported(const snp_pattern *pat) {
    return pat != nullptr && pat->dpe == 6 && pat->has_incidence && pat->has_contrib;
}

int launch_curlcurl_rows(const snp_pattern *pat, const double *terms, const TermLayout &L, double *K, double *dK,
                         double *J, float *J32, double *rhs, double *F, cudaStream_t st) {
    SNP_REQUIRE(rows_supported(pat), "row assembly: the pattern has no contribution or incidence lists");
    SNP_REQUIRE(pat->n_elems == 0 || terms != nullptr, "row assembly: terms is NULL");
    SNP_REQUIRE(F == nullptr || L.f >= 0, "row assembly: F needs SNP_TERMS_F blocks");
    SNP_REQUIRE(rhs == nullptr || L.r >= 0, "row assembly: rhs needs SNP_TERMS_RHS blocks");
    const bool wj = J != nullptr || J32 != nullptr;
    EntryArgs r{};
    r.nnz = pat->nnz;
    r.n_elems = pat->n_elems;
    r.cptr = pat->cptr.p;
    r.cid = pat->cid.p;
    r.terms = terms;
    r.K = K;
    r.dK = dK;
    r.J = J;
    r.J32 = J32;
    if (r.nnz > 0 && (K || dK || wj)) {
        if (wj && L.k >= 0 && L.d >= 0) {
            r.b0 = L.k;
            r.b1 = L.d;
            SNP_TRY(launch_entries<kEntKD>(r, st));
        } else if (wj) {
            SNP_REQUIRE(L.j >= 0, "row assembly: J needs SNP_TERMS_J or SNP_TERMS_K | SNP_TERMS_DK blocks");
            SNP_REQUIRE(K == nullptr || L.k >= 0, "row assembly: K needs SNP_TERMS_K blocks");
            SNP_REQUIRE(dK == nullptr, "row assembly: dK needs SNP_TERMS_DK blocks");
            r.b0 = L.j;
            SNP_TRY(launch_entries<kEntJ>(r, st));
            if (K) {
                EntryArgs rk = r;
                rk.J = nullptr;
                rk.J32 = nullptr;
                rk.b0 = L.k;
                SNP_TRY(launch_entries<kEntK>(rk, st));
            }
        } else if (K && dK) {
            SNP_REQUIRE(L.k >= 0 && L.d >= 0, "row assembly: K and dK need SNP_TERMS_K | SNP_TERMS_DK blocks");
            r.b0 = L.k;
            r.b1 = L.d;
            SNP_TRY(launch_entries<kEntKD>(r, st));
        } else if (K) {
            SNP_REQUIRE(L.k >= 0, "row assembly: K needs SNP_TERMS_K blocks");
            r.b0 = L.k;
            SNP_TRY(launch_entries<kEntK>(r, st));
        } else {
            SNP_REQUIRE(L.d >= 0, "row assembly: dK needs SNP_TERMS_DK blocks");
            r.b0 = L.d;
            SNP_TRY(launch_entries<kEntD>(r, st));
        }
    }
    if ((F || rhs) && pat->n_rows > 0) {
        const double *Fe = L.f >= 0 ? terms + (int64_t)L.f * pat->n_elems : nullptr;
        const double *Re = L.r >= 0 ? terms + (int64_t)L.r * pat->n_elems : nullptr;
        k_cc_dofvec<<<wave_grid(k_cc_dofvec, pat->n_rows, kEntryBlock), kEntryBlock, 0, st>>>(
            pat->n_rows, pat->n_elems, pat->inc_ptr.p, pat->inc.p, Fe, Re, F, rhs);
        SNP_LAUNCH_CHECK();
    }
    return SNP_OK;
}

// PackedTerms::any of all launches; a material that finds no room left stores its dK
static size_t any_bytes(const snp_pattern *pat) { return ((size_t)pat->n_elems / kPackBlock + 256) / 16 * 16; }

size_t curlcurl_system_work(const snp_pattern *pat, const SystemOut &o) {
    const PackedNeeds nd = packed_needs(o);
    const size_t zeros = nd.d ? (any_bytes(pat) + (size_t)pat->n_elems + 15) / 16 * 2 + 2 : 0;
    return (size_t)pat->n_elems * ((nd.k + nd.d + nd.j) * kPackPairs + (o.F ? 6 : 0) + (o.rhs ? 6 : 0)) + zeros;
}

int launch_curlcurl_system(const snp_pattern *pat, const CurlArgs *mats, int n_mats, double *work, const SystemOut &o,
                           cudaStream_t st) {
    SNP_REQUIRE(rows_supported(pat), "curl-curl system: the pattern has no contribution or incidence lists");
    SNP_REQUIRE(pat->n_elems == 0 || work != nullptr || curlcurl_system_work(pat, o) == 0,
                "curl-curl system: work is NULL");
    const PackedNeeds nd = packed_needs(o);
    const size_t E = (size_t)pat->n_elems;
    PackedEntryArgs r{};
    ZeroRanges no_source, zero_dk;
    bool packed = true;
    int64_t at = 0;
    for (int m = 0; m < n_mats; ++m) {
        const CurlArgs &a = mats[m];
        SNP_REQUIRE(a.t_offset == at, "curl-curl system: material %d starts at element %lld, expected %lld", m,
                    (long long)a.t_offset, (long long)at);
        at += a.n_elems;
        packed = packed && packed_fits(a.n_orient, a.nq, a.n_int);
        if (o.rhs && a.n_elems > 0 && a.Bs == nullptr) packed = packed && no_source.add(a.t_offset, at);
    }
    SNP_REQUIRE(at == pat->n_elems, "curl-curl system: the materials hold %lld of the pattern's %lld elements",
                (long long)at, (long long)pat->n_elems);
    if (!packed) {
        const TermLayout L = term_layout((nd.k ? SNP_TERMS_K : 0) | (nd.d ? SNP_TERMS_DK : 0) | (nd.j ? SNP_TERMS_J : 0) |
                                         (o.F ? SNP_TERMS_F : 0) | (o.rhs ? SNP_TERMS_RHS : 0));
        for (int m = 0; m < n_mats; ++m) SNP_TRY(launch_curlcurl_terms(mats[m], L, work, pat->n_elems, st));
        return launch_curlcurl_rows(pat, work, L, o.K, o.dK, o.J, o.J32, o.rhs, o.F, st);
    }
    PackedTerms all;
    double *p = work;
    auto take = [&](bool want, size_t per) {
        double *q = want ? p : nullptr;
        if (want) p += per * E;
        return q;
    };
    all.K = take(nd.k, kPackPairs);
    all.D = take(nd.d, kPackPairs);
    all.J = take(nd.j, kPackPairs);
    all.F = take(o.F != nullptr, 6);
    all.R = take(o.rhs != nullptr, 6);
    // read 16 bytes at a time
    uint8_t *const any = nd.d ? reinterpret_cast<uint8_t *>(((uintptr_t)p + 15) / 16 * 16) : nullptr;
    uint8_t *const kept = nd.d ? any + any_bytes(pat) : nullptr;
    bool beside = false;
    for (int m = 0; m < n_mats; ++m) {
        CurlArgs a = mats[m];
        if (a.n_elems == 0) continue;
        a.beside = beside;
        PackedTerms out = all;
        // constant reluctance: nu' = 0, and with it dK unless B is not finite
        const size_t most = (size_t)(a.n_elems / kPackBlock) + 16;
        if (out.D && a.n_int < 0 && (size_t)r.n_any + most <= any_bytes(pat) && zero_dk.n < 2 &&
            zero_dk.add(a.t_offset, a.t_offset + a.n_elems)) {
            out.D = nullptr;
            out.Dz = all.D;
            out.kept = kept;
            out.any = any + r.n_any;
        }
        if (a.Bs == nullptr) out.R = nullptr;
        if (out.K || out.D || out.J || out.F || out.R || out.any) {
            int blocks = 0;
            SNP_TRY(launch_curlcurl_packed(a, out, st, &blocks));
            if (out.any) r.n_any += (blocks + 15) / 16 * 16;
            // the next material's element kernel starts while this one's points are bound by
            // latency (183 -> 175 us a call at 150k tets diluted, 250 -> 235 at 300k); beside a kernel
            // bound by its streams it gains nothing (485 -> 485-510 us at 1.16M tets, 4 points)
            beside = a.Bs != nullptr && a.nq >= kManyPoints;
        }
    }
    r.nnz = pat->nnz;
    r.cptr = pat->cptr.p;
    r.cid = pat->cid.p;
    r.K = o.K;
    r.dK = o.dK;
    r.J = o.J;
    r.J32 = o.J32;
    for (int i = 0; i < zero_dk.n; ++i) {
        r.lo[i] = (uint32_t)zero_dk.lo[i] * kPackPairs;
        r.hi[i] = (uint32_t)zero_dk.hi[i] * kPackPairs;
    }
    r.kept = kept;
    r.any = any;
    if (r.nnz > 0) {
        if (nd.j) {
            r.m0 = all.J;
            SNP_TRY(launch_packed_entries<kEntJ>(r, st));
        } else if (nd.k && nd.d) {
            r.m0 = all.K;
            r.m1 = all.D;
            SNP_TRY(launch_packed_entries<kEntKD>(r, st));
        } else if (nd.k) {
            r.m0 = all.K;
            SNP_TRY(launch_packed_entries<kEntK>(r, st));
        } else if (nd.d) {
            r.m0 = all.D;
            SNP_TRY(launch_packed_entries<kEntD>(r, st));
        }
    }
    if ((o.F || o.rhs) && pat->n_rows > 0) {
        k_cc_dofvec_packed<<<wave_grid(k_cc_dofvec_packed, pat->n_rows, kEntryBlock), kEntryBlock, 0, st>>>(
            pat->n_rows, pat->inc_ptr.p, pat->inc.p, all.F, all.R, o.F, o.rhs, no_source);
        SNP_LAUNCH_CHECK();
    }
    return SNP_OK;
}

}  // namespace snp

extern "C" {

int snp_curlcurl_system_work(const snp_pattern *pat, int32_t want_K, int32_t want_dK, int32_t want_J, int32_t want_rhs,
                             int32_t want_F, int64_t *n_doubles) {
    snp::clear_error();
    SNP_REQUIRE(pat != nullptr && n_doubles != nullptr, "snp_curlcurl_system_work: NULL argument");
    snp::SystemOut o;
    double d = 0.0;
    if (want_K) o.K = &d;
    if (want_dK) o.dK = &d;
    if (want_J) o.J = &d;
    if (want_rhs) o.rhs = &d;
    if (want_F) o.F = &d;
    *n_doubles = (int64_t)snp::curlcurl_system_work(pat, o);
    return SNP_OK;
}

int snp_curlcurl_system(const snp_pattern *pat, int32_t n_mats, const snp_curlcurl_material *mats, const double *nodes,
                        const double *curls, int32_t n_orient, const double *d_phi, const double *w, int32_t n_quad,
                        const double *x, double *work, double *K_vals, double *dK_vals, double *J_vals, double *rhs,
                        double *F, void *stream) {
    snp::clear_error();
    SNP_REQUIRE(pat != nullptr && n_mats >= 0 && (n_mats == 0 || mats), "snp_curlcurl_system: NULL argument");
    std::vector<snp::CurlArgs> args((size_t)n_mats);
    for (int m = 0; m < n_mats; ++m) {
        const snp_curlcurl_material &M = mats[m];
        SNP_TRY(snp::fill_args(args[m], pat, M.elem_offset, M.n_elems, nodes, M.cells, M.glob_ids, M.orientations,
                               curls, n_orient, d_phi, w, n_quad, x, M.B_s, M.n_int, M.rel_c, M.rel_x));
        args[m].slots = nullptr;
        args[m].t_offset = M.elem_offset;
        if (M.B_s != nullptr && M.phi != nullptr) {
            args[m].phi = M.phi;
            for (int i = 0; i < 4; ++i) args[m].dil[i] = M.dilution[i];
        }
    }
    snp::SystemOut o;
    o.K = K_vals;
    o.dK = dK_vals;
    o.J = J_vals;
    o.rhs = rhs;
    o.F = F;
    return snp::launch_curlcurl_system(pat, args.data(), n_mats, work, o, snp::as_stream(stream));
}

int snp_curlcurl_terms_stride(int32_t parts, int32_t *stride) {
    snp::clear_error();
    SNP_REQUIRE(stride != nullptr, "snp_curlcurl_terms_stride: stride is NULL");
    SNP_REQUIRE((parts & ~31) == 0, "snp_curlcurl_terms_stride: unknown bits in parts (0x%x)", (unsigned)parts);
    *stride = snp::term_layout(parts).stride;
    return SNP_OK;
}

int snp_curlcurl_rows_supported(const snp_pattern *pat, int32_t *supported) {
    snp::clear_error();
    SNP_REQUIRE(pat != nullptr && supported != nullptr, "snp_curlcurl_rows_supported: NULL argument");
    *supported = snp::rows_supported(pat) ? 1 : 0;
    return SNP_OK;
}

int snp_curlcurl_terms(const snp_pattern *pat, int64_t elem_offset, int64_t n_elems, const double *nodes,
                       const int32_t *cells, const int32_t *glob_ids, const int32_t *orientations, const double *curls,
                       int32_t n_orient, const double *phi, const double *d_phi, const double *w, int32_t n_quad,
                       const double *x, const double *B_s, int32_t n_int, const double *rel_c, const double *rel_x,
                       const double *dilution, int32_t parts, double *terms, void *stream) {
    snp::clear_error();
    SNP_REQUIRE(pat != nullptr, "snp_curlcurl_terms: pattern is NULL");
    SNP_REQUIRE((parts & ~31) == 0, "snp_curlcurl_terms: unknown bits in parts (0x%x)", (unsigned)parts);
    SNP_REQUIRE((phi == nullptr) == (dilution == nullptr), "snp_curlcurl_terms: give both phi and dilution, or neither");
    snp::CurlArgs a;
    SNP_TRY(snp::fill_args(a, pat, elem_offset, n_elems, nodes, cells, glob_ids, orientations, curls, n_orient, d_phi,
                           w, n_quad, x, B_s, n_int, rel_c, rel_x));
    if (B_s != nullptr && phi != nullptr) {
        a.phi = phi;
        for (int i = 0; i < 4; ++i) a.dil[i] = dilution[i];
    }
    a.t_offset = elem_offset;
    return snp::launch_curlcurl_terms(a, snp::term_layout(parts), terms, pat->n_elems, snp::as_stream(stream));
}

int snp_curlcurl_rows(const snp_pattern *pat, const double *terms, int32_t parts, double *K_vals, double *dK_vals,
                      double *J_vals, float *J32_vals, double *rhs, double *F, void *stream) {
    snp::clear_error();
    SNP_REQUIRE(pat != nullptr, "snp_curlcurl_rows: pattern is NULL");
    SNP_REQUIRE((parts & ~31) == 0, "snp_curlcurl_rows: unknown bits in parts (0x%x)", (unsigned)parts);
    return snp::launch_curlcurl_rows(pat, terms, snp::term_layout(parts), K_vals, dK_vals, J_vals, J32_vals, rhs, F,
                                     snp::as_stream(stream));
}

}  // extern "C"
