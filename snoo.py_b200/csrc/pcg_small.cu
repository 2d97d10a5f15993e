// Jacobi-PCG (float64) of small masked systems in one thread-block cluster.
//
// A coil's potential problem has one or two thousand free nodes in a mesh of tens of thousands
// (snoopy/laplace_subdomain_solver.py:117-158), and its CG about 130 iterations.  Three launches
// over the whole mesh and their reductions took 19 us per iteration, all of it latency.  Here the
// free rows are listed once, their columns renumbered, and eight blocks of one cluster keep the
// whole solve in shared memory: p and z in every block, the matrix and the other vectors by rows.
// Partial sums and z travel through distributed shared memory, two cluster barriers per iteration:
//
//   q = A p (own rows), p.q           | barrier | r -= alpha q, z = D^-1 r to every block, r.z, r.r
//   x += alpha p                      | barrier | p = z + beta p (whole, in every block)
//
// Measured at 1.1k free rows of 36k, 136 iterations: 2.55 ms -> 0.43 ms, and 12 us for the list
// (3.2 us per iteration, a chain of two barriers, four reductions and the row sums: latency; with
// the matrix left in L2 4.1 us, with four lanes per row 3.6, with 1024 threads 4.8).
//
// The path is taken where the vectors (at most 8192 free rows) and every block's entries fit into
// shared memory: 5700 rows of 15 entries.  8192 rows of 4 entries take 14 us per iteration here and
// 19 us in the general path over 36k rows; a matrix that had to be streamed from L2 took 20 us.
// The list is one block's work, so meshes above 262144 rows go to the general path unasked.  A masked
// system below that whose free rows turn out not to fit pays the list and an empty launch: 3.2 ms
// per call of 40k rows as before there was this path (3.8 ms while the list had an allocation and a
// synchronisation of its own).
#include <cooperative_groups.h>

#include "snp_common.cuh"
#include "snp_internal.cuh"
#include "snp_krylov.cuh"
#include "snp_reduce.cuh"

namespace cg = cooperative_groups;

namespace snp {
namespace {

constexpr int kCta = 8;        // blocks of the cluster
constexpr int kThreads = 512;
constexpr int kTpr = 2;        // lanes per row
constexpr int kWarps = kThreads / 32;
constexpr int kListBlock = 1024;
constexpr size_t kSmem = 222 * 1024;  // what a block can have beside its slots

struct SmallHead {
    int32_t run, bad, nf, done, nnz;  // nnz: entries of the whole matrix
    long long iter;
    double rr;
};

// what a block keeps in shared memory: p and z whole; r, x, q, 1/diag and the rows' places of its
// own rows; then its entries (value, renumbered column)
__host__ __device__ constexpr size_t vector_doubles(int32_t nf) {
    return 2 * ((size_t)nf + 1) + 5 * (((size_t)nf + kCta - 1) / kCta) + 1;
}

// rows[]: the free rows in order, loff[]: number of entries in the rows before each (and in all),
// local_of[i]: place of row i in rows, or -1.  Each warp takes a contiguous range of the mask, 32
// rows per step, once to count and once to write.  run = 0 when the system does not fit.
__global__ void __launch_bounds__(kListBlock)
    k_small_rows(int32_t n, const uint8_t *__restrict__ fm, const int32_t *__restrict__ rp,
                 int32_t *__restrict__ rows, int32_t *__restrict__ loff, int32_t *__restrict__ local_of,
                 SmallHead *head) {
    constexpr int kListWarps = kListBlock / 32;
    constexpr int kStep = 4;
    __shared__ int32_t s_rows[kListWarps];
    __shared__ int64_t s_nnz[kListWarps];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (threadIdx.x == 0) head->nnz = rp[n];
    const int32_t span = (n + kListBlock - 1) / kListBlock * 32;
    const int32_t i0 = min(wid * span, n), i1 = min(i0 + span, n);
    int32_t cnt = 0;
    for (int32_t i = i0; i < i1; i += 32 * kStep) {
        bool f[kStep];
#pragma unroll
        for (int u = 0; u < kStep; ++u) f[u] = i + 32 * u + lane < i1 && is_free(fm, i + 32 * u + lane);
#pragma unroll
        for (int u = 0; u < kStep; ++u) cnt += __popc(__ballot_sync(0xffffffffu, f[u]));
    }
    if (lane == 0) s_rows[wid] = cnt;
    __syncthreads();
    int32_t at = 0, nf = 0;
    for (int w = 0; w < kListWarps; ++w) {
        if (w < wid) at += s_rows[w];
        nf += s_rows[w];
    }
    if (nf == 0 || nf > kPcgSmallRows) {
        if (threadIdx.x == 0) head->run = 0;
        return;
    }
    int64_t len = 0;
    int32_t j = at;
    for (int32_t i = i0; i < i1; i += 32 * kStep) {
        bool f[kStep];
#pragma unroll
        for (int u = 0; u < kStep; ++u) f[u] = i + 32 * u + lane < i1 && is_free(fm, i + 32 * u + lane);
#pragma unroll
        for (int u = 0; u < kStep; ++u) {
            const int32_t k = i + 32 * u + lane;
            const unsigned m = __ballot_sync(0xffffffffu, f[u]);
            const int32_t mine = j + __popc(m & ((1u << lane) - 1u));
            if (f[u]) {
                rows[mine] = k;
                len += rp[k + 1] - rp[k];
            }
            if (k < i1) local_of[k] = f[u] ? mine : -1;
            j += __popc(m);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) len += __shfl_xor_sync(0xffffffffu, len, o);
    if (lane == 0) s_nnz[wid] = len;
    __syncthreads();  // also makes this warp's rows[] visible to its other lanes
    int64_t off = 0, nnz = 0;
    for (int w = 0; w < kListWarps; ++w) {
        if (w < wid) off += s_nnz[w];
        nnz += s_nnz[w];
    }
    if (nnz > kCta * (int64_t)(kSmem / 10)) {
        if (threadIdx.x == 0) head->run = 0;
        return;
    }
    if (threadIdx.x == 0) {
        head->bad = 0;
        head->nf = nf;
        loff[nf] = (int32_t)nnz;
    }
    for (int32_t t = at; t < at + cnt; t += 32) {
        const bool in = t + lane < at + cnt;
        int32_t l = 0;
        if (in) {
            const int32_t k = rows[t + lane];
            l = rp[k + 1] - rp[k];
        }
        int32_t incl = l;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int32_t y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        if (in) loff[t + lane] = (int32_t)off + incl - l;
        off += __shfl_sync(0xffffffffu, incl, 31);
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        const int32_t R = (nf + kCta - 1) / kCta, c = threadIdx.x % kCta;
        const int32_t own = loff[min((c + 1) * R, nf)] - loff[min(c * R, nf)];
        const bool fits = 8 * vector_doubles(nf) + 10 * (size_t)own <= kSmem;
        const bool all = __all_sync(0xffffffffu, fits);
        if (threadIdx.x == 0) head->run = all;
    }
}

struct SmallArgs {
    int32_t n;
    const int32_t *rp, *ci;
    const double *v;
    const uint8_t *fm;
    const double *b;
    double *x;
    double rtol, atol;
    long long maxit;
    const int32_t *rows, *loff, *local_of;
    SmallHead *head;
};

// Sums over the cluster: every warp writes its W sums into all blocks' slots, and after the
// cluster's barrier every warp adds all of them in the same order.  `between` runs while the
// other blocks arrive.  A slot array may be used again once another barrier has passed.
template <int W, typename F>
__device__ __forceinline__ void cluster_sums(cg::cluster_group &cl, double (&v)[W], double (*slot)[kWarps * kCta],
                                             F between) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int w = 0; w < W; ++w) {
        const double t = warp_sum(v[w]);
        if (lane / kCta == w) cl.map_shared_rank(&slot[w][0], lane % kCta)[cl.block_rank() * kWarps + wid] = t;
    }
    cl.barrier_arrive();
    between();
    cl.barrier_wait();
#pragma unroll
    for (int w = 0; w < W; ++w) {
        double t = 0.0;
#pragma unroll
        for (int i = 0; i < kWarps * kCta / 32; ++i) t += slot[w][i * 32 + lane];
        v[w] = warp_sum(t);
    }
}

__global__ void __cluster_dims__(kCta, 1, 1) __launch_bounds__(kThreads, 1) k_pcg_small(const SmallArgs a) {
    extern __shared__ double sm[];
    __shared__ double slot_a[1][kWarps * kCta], slot_b[3][kWarps * kCta];
    cg::cluster_group cl = cg::this_cluster();
    if (!a.head->run) return;  // the same in every block, before any cluster barrier
    const int32_t nf = a.head->nf, R = (nf + kCta - 1) / kCta;
    const int32_t lo = min((int32_t)cl.block_rank() * R, nf), m = min(nf - lo, R);
    double *p = sm, *z = p + nf + 1, *r = z + nf + 1, *x = r + R, *q = x + R, *dinv = q + R;
    int32_t *off = reinterpret_cast<int32_t *>(dinv + R);
    double *val = sm + vector_doubles(nf);
    const int32_t o0 = a.loff[lo], own = a.loff[lo + m] - o0;
    uint16_t *lc = reinterpret_cast<uint16_t *>(val + own);  // constrained columns point at entry nf (0)
    const int sub = threadIdx.x % kTpr, grp = threadIdx.x / kTpr;
    constexpr int kGroups = kThreads / kTpr;
    if (threadIdx.x == 0) p[nf] = z[nf] = 0.0;
    double s[3] = {0.0, 0.0, 0.0};
    cl.sync();  // every block runs before its shared memory is written from outside
    auto spread = [&](double *vec, int32_t j, double v) {  // all lanes of a row's group, v from the first
        v = __shfl_sync(0xffffffffu, v, 0, kTpr);
        if (j < m)
            for (int c = sub; c < kCta; c += kTpr) cl.map_shared_rank(vec, c)[lo + j] = v;
    };
    for (int32_t j0 = 0; j0 < m; j0 += kGroups) {
        const int32_t j = j0 + grp;
        double ax = 0.0, d = 0.0, zi = 0.0;
        int32_t row = 0;
        if (j < m) {
            row = a.rows[lo + j];
            const int32_t b = a.rp[row], o = a.loff[lo + j] - o0, end = a.loff[lo + j + 1] - o0;
            if (sub == 0) {
                off[j] = o;
                if (j == m - 1) off[m] = end;
            }
            for (int32_t k = sub; k < end - o; k += kTpr) {
                const int32_t c = a.ci[b + k], l = a.local_of[c];
                const double v = a.v[b + k];
                val[o + k] = v;
                lc[o + k] = (uint16_t)(l >= 0 ? l : nf);
                if (l >= 0) ax += v * a.x[c];
                if (l == lo + j) d = v;
            }
        }
#pragma unroll
        for (int o = 1; o < kTpr; o <<= 1) {
            ax += __shfl_xor_sync(0xffffffffu, ax, o);
            d += __shfl_xor_sync(0xffffffffu, d, o);
        }
        if (j < m && sub == 0) {
            if (d == 0.0 || !(d == d)) atomicExch(&a.head->bad, 1);
            const double bi = a.b[row], ri = bi - ax, di = 1.0 / d;
            zi = di * ri;
            r[j] = ri;
            x[j] = a.x[row];
            dinv[j] = di;
            s[0] += ri * zi;
            s[1] += ri * ri;
            s[2] += bi * bi;
        }
        spread(p, j, zi);
    }
    __threadfence();
    cluster_sums<3>(cl, s, slot_b, [] {});
    double rz = s[0], rr = s[1];
    const double bnorm = sqrt(s[2]), atol_eff = fmax(a.atol, a.rtol * bnorm);
    long long iter = 0;
    int done = 0;
    if (*(volatile int32_t *)&a.head->bad) return;  // zero pivot: x untouched
    if (s[2] == 0.0) done = 4;
    else if (!(rr == rr) || isinf(rr)) done = 3;
    else if (sqrt(rr) < atol_eff) done = 1;
    else if (a.maxit <= 0) done = 2;
    while (!done) {
        // a row's first lane keeps the row: it alone reads and writes r, x, q and dinv there
        double t[1] = {0.0};
        for (int32_t j0 = 0; j0 < m; j0 += kGroups) {
            const int32_t j = j0 + grp;
            double sum = 0.0;
            if (j < m) {
                const int32_t o = off[j], end = off[j + 1];
#pragma unroll 4
                for (int32_t k = o + sub; k < end; k += kTpr) sum += val[k] * p[lc[k]];
            }
#pragma unroll
            for (int o = 1; o < kTpr; o <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            if (j < m && sub == 0) {
                q[j] = sum;
                t[0] += p[lo + j] * sum;
            }
        }
        cluster_sums<1>(cl, t, slot_a, [] {});
        const double alpha = rz / t[0];
        double u[2] = {0.0, 0.0};
        for (int32_t j0 = 0; j0 < m; j0 += kGroups) {
            const int32_t j = j0 + grp;
            double zi = 0.0;
            if (j < m && sub == 0) {
                const double ri = r[j] - alpha * q[j];
                zi = dinv[j] * ri;
                r[j] = ri;
                u[0] += ri * zi;
                u[1] += ri * ri;
            }
            spread(z, j, zi);
        }
        cluster_sums<2>(cl, u, slot_b, [&] {
            if (sub == 0)
                for (int32_t j = grp; j < m; j += kGroups) x[j] += alpha * p[lo + j];
            __syncthreads();  // p changes next
        });
        const double beta = u[0] / rz;
        rz = u[0];
        rr = u[1];
        ++iter;
        for (int32_t i = threadIdx.x; i < nf; i += kThreads) p[i] = z[i] + beta * p[i];
        if (!(rr == rr) || isinf(rr)) done = 3;
        else if (sqrt(rr) < atol_eff) done = 1;
        else if (iter >= a.maxit) done = 2;
        __syncthreads();
    }
    if (sub == 0)
        for (int32_t j = grp; j < m; j += kGroups) a.x[a.rows[lo + j]] = x[j];
    for (int64_t i = (int64_t)cl.block_rank() * kThreads + threadIdx.x; i < a.n; i += kCta * kThreads)
        if (!is_free(a.fm, i)) a.x[i] = 0.0;
    if (cl.block_rank() == 0 && threadIdx.x == 0) {
        a.head->rr = rr;
        a.head->iter = iter;
        a.head->done = done;
    }
}

constexpr size_t align16(size_t v) { return (v + 15) / 16 * 16; }

}  // namespace

size_t pcg_small_scratch(int32_t n) {
    return align16(sizeof(SmallHead)) + align16(sizeof(int32_t) * (kPcgSmallRows + 1)) * 2 +
           align16(sizeof(int32_t) * (size_t)n);
}

int pcg_small(int32_t n, const int32_t *rp, const int32_t *ci, const double *v, const uint8_t *fm, const double *b,
              double *x, double rtol, double atol, int64_t maxit, void *scratch, cudaStream_t s, bool *ran,
              int32_t *nnz, int64_t *its, double *res, int *status) {
    *ran = false;
    unsigned char *at = static_cast<unsigned char *>(scratch);
    auto take = [&](size_t count) {
        int32_t *p = reinterpret_cast<int32_t *>(at);
        at += align16(sizeof(int32_t) * count);
        return p;
    };
    SmallHead *head = reinterpret_cast<SmallHead *>(at);
    at += align16(sizeof(SmallHead));
    int32_t *rows = take(kPcgSmallRows + 1), *loff = take(kPcgSmallRows + 1);
    int32_t *local_of = take((size_t)n);
    if (maxit < 0) maxit = 10 * (int64_t)n;
    // per device, so it is set on every call
    SNP_CUDA_TRY(cudaFuncSetAttribute(k_pcg_small, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem));
    k_small_rows<<<1, kListBlock, 0, s>>>(n, fm, rp, rows, loff, local_of, head);
    SNP_LAUNCH_CHECK();
    k_pcg_small<<<kCta, kThreads, kSmem, s>>>(
        SmallArgs{n, rp, ci, v, fm, b, x, rtol, atol, (long long)maxit, rows, loff, local_of, head});
    SNP_LAUNCH_CHECK();
    SmallHead h;
    SNP_CUDA_TRY(cudaMemcpyAsync(&h, head, sizeof(h), cudaMemcpyDeviceToHost, s));
    SNP_CUDA_TRY(cudaStreamSynchronize(s));
    *nnz = h.nnz;
    if (!h.run) return SNP_OK;
    *ran = true;
    if (h.bad) {
        *status = SNP_ZERO_PIVOT;
        return SNP_OK;
    }
    if (its) *its = h.iter;
    if (res) *res = sqrt(h.rr);
    *status = h.done == 2 ? SNP_NOT_CONVERGED : h.done == 3 ? SNP_NAN_DETECTED : SNP_OK;
    return SNP_OK;
}

}  // namespace snp
