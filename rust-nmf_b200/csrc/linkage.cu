// linkage.cu -- consensus statistics on the device: Brunet's cophenetic
// correlation (average-linkage tree on the distances 1 - C) and Kim & Park's
// dispersion coefficient of a p x p consensus matrix C.
//
// The consensus workflow these summarise is examples/build_scaling_notebook.py
// :121-141 of the reference (connectivity -> consensus -> average linkage on
// 1 - C via scipy -> cophenetic correlation; dispersion = mean 4 (C - 0.5)^2).
//
// Average linkage (UPGMA) is built by the nearest-neighbour chain
// (Murtagh 1983; Muellner, "Modern hierarchical, agglomerative clustering
// algorithms", 2011): grow a chain of nearest neighbours from the first
// active cluster until its last two elements are reciprocal nearest
// neighbours, merge them (the merged cluster keeps the larger index), and
// update its distances with the Lance-Williams average rule
//   d(i, a u b) = (n_a d(i, a) + n_b d(i, b)) / (n_a + n_b).
// A nearest neighbour is the strictly smallest distance in index order,
// the chain's previous element winning ties -- the same choices (and the
// same f64 update, no FMA) as scipy.cluster.hierarchy.linkage's chain, so
// the tree is the same one even where consensus distances tie.
//
// The cophenetic distance of a pair is the height of the merge that joins
// it.  In an average-linkage tree a merge of clusters A and B happens at the
// mean original distance over A x B, so the sums the correlation needs come
// from the merges alone:  sum over A x B of d = |A||B| h, hence with
// N = p (p - 1) / 2 pairs, mean distance m_d and mean cophenetic distance
// m_c = sum_k n_k h_k / N (n_k = |A_k||B_k|),
//   cov = sum_k n_k (h_k - m_c)(h_k - m_d),  var_c = sum_k n_k (h_k - m_c)^2,
// and var_d from one pass over the pairs.  Nothing of size p^2 beyond D.
#include <cooperative_groups.h>

#include <cfloat>
#include <climits>
#include <cmath>
#include <vector>
#include <algorithm>

#include "internal.h"

namespace {

constexpr int kR = 256;  // threads of the reduction kernels

__device__ double block_sum(double v, double *red) {
    red[threadIdx.x] = v;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
        if ((int)threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
        __syncthreads();
    }
    const double out = red[0];
    __syncthreads();
    return out;
}

// One matrix of a batch: block (b, m) takes rows b, b + gridDim.x, ... of
// matrix m and, from one read of C, writes D = 1 - C in f64 (p x p, pitch p,
// zero diagonal: the reference fills the consensus diagonal with 1 before
// taking distances) and sums d over its pairs i < j and 4 (C - 0.5)^2 over
// all its entries (diagonal read as 1).  Bound: HBM, 12 bytes an entry; a
// matrix of p = 5000 took 140 us when the three were kernels of their own.
__global__ void __launch_bounds__(kR)
    distances_and_sums(const float *__restrict__ C, int64_t ldc, int64_t cstride, int p,
                       double *__restrict__ D, double *__restrict__ part, int64_t pstride) {
    __shared__ double red[kR];
    C += blockIdx.y * cstride;
    D += (size_t)blockIdx.y * p * p;
    part += blockIdx.y * pstride;
    double sd = 0.0, sc = 0.0;
    for (int i = blockIdx.x; i < p; i += gridDim.x) {
        const float *row = C + (size_t)i * ldc;
        double *out = D + (size_t)i * p;
#pragma unroll 4
        for (int j = threadIdx.x; j < p; j += kR) {
            const double c = (i == j) ? 1.0 : (double)row[j];
            const double d = 1.0 - c;
            out[j] = d;
            if (j > i) sd += d;
            sc += 4.0 * (c - 0.5) * (c - 0.5);
        }
    }
    const double a = block_sum(sd, red), b = block_sum(sc, red);
    if (threadIdx.x == 0) {
        part[blockIdx.x] = a;
        part[gridDim.x + blockIdx.x] = b;
    }
}

// Per-block sums over the pairs i < j of (d - mean)^2, mean = stat[1].
__global__ void __launch_bounds__(kR)
    deviation_sums(const double *__restrict__ D, int p, double *__restrict__ part,
                   int64_t pstride, const double *__restrict__ stat) {
    __shared__ double red[kR];
    D += (size_t)blockIdx.y * p * p;
    const double m = stat[blockIdx.y * pstride + 1];
    double acc = 0.0;
    for (int i = blockIdx.x; i < p; i += gridDim.x)
#pragma unroll 4
        for (int j = i + 1 + threadIdx.x; j < p; j += kR) {
            const double d = D[(size_t)i * p + j];
            acc += (d - m) * (d - m);
        }
    const double s = block_sum(acc, red);
    if (threadIdx.x == 0) part[blockIdx.y * pstride + blockIdx.x] = s;
}

// The B partials of matrix blockIdx.x in a fixed tree order: stat[0], stat[1]
// = the sum of the distances and their mean, stat[3] = the dispersion.
__global__ void __launch_bounds__(kR) finish_sums(const double *__restrict__ part, int B,
                                                  double inv_pairs, double inv_all,
                                                  double *__restrict__ stat, int64_t pstride) {
    __shared__ double red[kR];
    part += blockIdx.x * pstride;
    stat += blockIdx.x * pstride;
    double sd = 0.0, sc = 0.0;
    for (int b = threadIdx.x; b < B; b += kR) {
        sd += part[b];
        sc += part[B + b];
    }
    const double a = block_sum(sd, red), c = block_sum(sc, red);
    if (threadIdx.x == 0) {
        stat[0] = a;
        stat[1] = a * inv_pairs;
        stat[3] = c * inv_all;
    }
}

// ---------------------------------------------------------------------------
// The tree: one cluster of kCl blocks per matrix.
//
// A chain step is an argmin over the tip's row.  It is bound by latency, not
// by bandwidth: the row's read, the reduction, and the way back to every
// thread.  One block of 1024 threads a matrix took 4.3 us a step (64 ms for
// nine matrices of p = 5000, 2.95 p steps each); this takes 1.7 us (25 ms),
// 1.2 us at p = 1000.  Index i belongs to thread i mod kTc of block
// (i / kTc) mod kCl, so a thread holds E = ceil(p / 2048) entries of the row
// in registers; a warp reduces with redux.sync and sends its candidate to all
// kCl blocks by st.async, which counts it in on the receiver's mbarrier; when
// all kCl * kTc / 32 are there, every warp reduces them and knows the step's
// outcome.  All blocks decide from the same candidates, so they take the same
// steps.  Eight blocks a cluster: at one block a multiprocessor sixteen such
// clusters are resident at once, of clusters of 16 only eight; sizes and chain
// of up to p = 13000 or so leave shared memory for a second block.  Blocks of
// 128 / 512 threads took 28.0 / 26.5 ms.
//
// Two candidate buffers in turn: a warp sends step t + 2 after it has all of
// step t + 1, which holds every warp's candidate, sent after that warp had
// read step t's.
//
// A step reads the tip's row alone: the predecessor's was the tip's of the
// step before, still in registers, except after a merge.  While its candidate
// travels, a warp computes the merge it may have to write.
//
// A merge of a < b writes row and column b (reading each entry from the row
// of whichever of the two was merged last, with row b alone written, gathers
// sectors in every step, which took longer).  The step after a merge, which may
// start before those writes are visible, reads only rows c1 and c2 (the
// chain's next two), where entry b alone is new: the thread that owns index b
// has computed d(c1, b) and d(c2, b) itself.  Each thread fences its writes
// before its warp sends that step's candidate, so the steps after it see them.
//
// The hardware barriers stand before and after the steps alone, so that a
// thread whose wait has run out meets the others at the last one.
// ---------------------------------------------------------------------------
namespace cg = cooperative_groups;

constexpr int kCl = 8;    // blocks of a cluster
constexpr int kTc = 256;  // threads of a block
constexpr int kCand = kCl * kTc / 32;
constexpr unsigned kWaitLimit = 1u << 22;  // try_waits (each may suspend) of a bounded wait
// Cluster sizes and chain live in shared memory up to this many bytes.
constexpr size_t kTreeSmem = 160 * 1024;

// Distances as unsigned keys of the same order; NaN after everything else.
__device__ __forceinline__ unsigned long long dist_key(double v) {
    if (v != v) return ~0ull;
    const long long b = __double_as_longlong(v + 0.0);
    return (unsigned long long)b ^ (b < 0 ? ~0ull : 0x8000000000000000ull);
}
__device__ __forceinline__ double key_dist(unsigned long long k) {
    return __longlong_as_double((long long)(k ^ ((k >> 63) ? 0x8000000000000000ull : ~0ull)));
}
// The warp's smallest (key, index), in every lane.
__device__ __forceinline__ void warp_argmin(unsigned long long &key, unsigned &idx) {
    const unsigned hi = (unsigned)(key >> 32), lo = (unsigned)key;
    const unsigned mh = __reduce_min_sync(0xffffffffu, hi);
    const unsigned ml = __reduce_min_sync(0xffffffffu, hi == mh ? lo : ~0u);
    idx = __reduce_min_sync(0xffffffffu, (hi == mh && lo == ml) ? idx : ~0u);
    key = ((unsigned long long)mh << 32) | ml;
}
__device__ __forceinline__ unsigned smem_addr(const void *p) {
    return (unsigned)__cvta_generic_to_shared(p);
}
// {a, b} into block `to` of the cluster at this block's address `dst`, counted
// in (16 bytes) on that block's barrier at `bar`.
__device__ __forceinline__ void send_async(unsigned dst, unsigned bar, int to,
                                           unsigned long long a, unsigned long long b) {
    asm volatile(
        "{\n .reg .b32 d, m;\n mapa.shared::cluster.u32 d, %0, %2;\n"
        " mapa.shared::cluster.u32 m, %1, %2;\n"
        " st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.b64 [d], {%3, %4}, [m];\n}"
        ::"r"(dst), "r"(bar), "r"(to), "l"(a), "l"(b)
        : "memory");
}
__device__ __forceinline__ void bar_expect(unsigned bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
                 : "memory");
}
// A warp's lanes leave a wait together, with one answer: what follows votes and
// reduces over all of them.  (A lane that has seen the phase end goes on seeing
// it: the next one of that barrier needs this warp.  The vote in the loop costs
// 0.3 % of a step; behind it, 7 %.)
__device__ __forceinline__ bool bar_wait(unsigned bar, unsigned parity) {
    for (unsigned i = 0; i < kWaitLimit; i++) {
        unsigned ok;
        asm volatile(
            "{\n .reg .pred p;\n"
            " mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
            " selp.u32 %0, 1, 0, p;\n}"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (__all_sync(0xffffffffu, ok)) return true;
    }
    return false;
}
// x / y, correctly rounded, for y = n_a + n_b with r = RN(1 / y): two steps of
// the residual correction q <- RN(q + RN(x - q y) r) (Markstein, "Computation
// of elementary functions on the IBM RISC System/6000 processor", 1990), the
// first of which makes q faithful and the second correctly rounded.
__device__ __forceinline__ double quotient(double x, double y, double r) {
    const double ax = fabs(x);
    if (!(ax < 0x1p900) || (ax < 0x1p-900 && x != 0.0)) return __ddiv_rn(x, y);
    double q = __dmul_rn(x, r);
    q = __fma_rn(__fma_rn(-q, y, x), r, q);
    return __fma_rn(__fma_rn(-q, y, x), r, q);
}
// Lance-Williams average of the distances to a and b; r = 1 / fs.
__device__ __forceinline__ double average(double fa, double da, double fb, double db, double fs,
                                          double r) {
    return quotient(__dadd_rn(__dmul_rn(fa, da), __dmul_rn(fb, db)), fs, r);
}

// E: a thread's entries of a row (0: any number, read when needed, with a
// meeting of the cluster after a merge).  Writes each merge's height and pair
// count n_a n_b.  Every loop ends: a chain of a symmetric D holds distinct
// clusters; a chain that would exceed p (an asymmetric or NaN D) ends the
// tree with the remaining heights NaN.
template <int E>
__global__ void __cluster_dims__(kCl, 1, 1) __launch_bounds__(kTc)
    nn_chain_average(double *__restrict__ D, int p, int *__restrict__ scratch,
                     double *__restrict__ height, double *__restrict__ npair, int64_t hstride,
                     int *__restrict__ gave_up) {
    cg::cluster_group cl = cg::this_cluster();
    const int rank = (int)cl.block_rank();
    const int m = blockIdx.x / kCl;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    D += (size_t)m * p * p;
    height += m * hstride;
    npair += m * hstride;
    __shared__ __align__(16) ulonglong2 cand[2][kCand];
    __shared__ __align__(8) unsigned long long bars[2];
    extern __shared__ int tree_smem[];
    int *size = scratch ? scratch + (size_t)blockIdx.x * 2 * p : tree_smem;
    int *chain = size + p;
    for (int i = tid; i < p; i += kTc) size[i] = 1;
    if (tid == 0) {
        chain[0] = 0;
        for (int q = 0; q < 2; q++)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&bars[q])));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    cl.sync();

    const auto row = [&](int i) { return D + (size_t)i * p; };
    constexpr int EN = E > 0 ? E : 1;
    const int entries = E > 0 ? E : (p + kCl * kTc - 1) / (kCl * kTc);
    const auto index = [&](int e) { return (rank + kCl * e) * kTc + tid; };
    double vx[EN], vp[EN], vm[EN];  // the rows of x and prev; their merge
    bool live[EN];
#pragma unroll
    for (int e = 0; e < EN; e++) {
        live[e] = index(e) < p;
        vx[e] = vp[e] = vm[e] = 0.0;
    }
    int len = 1, x = 0, prev = -1, first = 0;
    unsigned par = 0, phase = 0;
    bool wrote = false;      // global writes of a merge not fenced yet
    bool have_prev = false;  // vp holds prev's row
    int fresh = -1;                 // the index merged in the step before
    double new1 = 0.0, new2 = 0.0;  // its distances to x and prev (its owner)
    bool late = false;              // this thread's wait ran out
    // A step without candidates: every thread's writes before it are visible
    // to the cluster's threads after it.
    const auto meet = [&] {
        asm volatile("fence.acq_rel.cluster;" ::: "memory");
        __syncwarp();
        const unsigned bar = smem_addr(&bars[par]);
        if (tid == 0) bar_expect(bar, kCand * sizeof(ulonglong2));
        if (lane < kCl)
            send_async(smem_addr(&cand[par][rank * (kTc / 32) + warp]), bar, lane, ~0ull, ~0ull);
        const bool ok = bar_wait(bar, phase);
        if (ok) {
            par ^= 1;
            phase ^= (par == 0);
        }
        return ok;
    };
    int k = 0;
    while (k < p - 1) {
        if (E > 0) {
            // every load before the first comparison
#pragma unroll
            for (int e = 0; e < EN; e++)
                if (live[e]) vx[e] = __ldcg(row(x) + index(e));
            if (!have_prev && prev >= 0) {
#pragma unroll
                for (int e = 0; e < EN; e++)
                    if (live[e]) vp[e] = __ldcg(row(prev) + index(e));
            }
        }
        const int c1 = len >= 3 ? chain[len - 3] : -1, c2 = len >= 4 ? chain[len - 4] : -1;
        const int nx = size[x], np = prev >= 0 ? size[prev] : 0;
        // If x and prev merge, the smaller, a, goes and b keeps the cluster.
        const bool xa = x < prev;
        const int a = xa ? x : prev, b = xa ? prev : x;
        const bool own_b = E > 0 && prev >= 0 && b % kTc == tid && (b / kTc) % kCl == rank;
        double dx1 = 0.0, dp1 = 0.0, dx2 = 0.0, dp2 = 0.0;
        if (own_b && c1 >= 0) {
            dx1 = __ldcg(row(x) + c1);
            dp1 = __ldcg(row(prev) + c1);
            if (c2 >= 0) {
                dx2 = __ldcg(row(x) + c2);
                dp2 = __ldcg(row(prev) + c2);
            }
        }
        unsigned long long key = ~0ull;
        unsigned idx = ~0u;
#pragma unroll
        for (int e = 0; e < entries; e++) {
            const int i = index(e);
            double v;
            if (E > 0) {
                if (i == fresh) {
                    vx[e % EN] = new1;
                    vp[e % EN] = new2;
                }
                v = vx[e % EN];
                if (!live[e % EN] || i == x) continue;
            } else {
                if (i >= p || i == x || size[i] == 0) continue;
                v = __ldcg(row(x) + i);
            }
            // the chain's previous element wins ties, then the smaller index
            const unsigned long long kv = dist_key(v);
            const unsigned iv = i == prev ? 0u : (unsigned)i + 1u;
            if (kv < key || (kv == key && iv < idx)) {
                key = kv;
                idx = iv;
            }
        }
        warp_argmin(key, idx);
        if (wrote)
            asm volatile("fence.acq_rel.cluster;" ::: "memory");
        else
            __threadfence_block();  // sizes and chain, for the block's other warps
        wrote = false;
        __syncwarp();
        const unsigned bar = smem_addr(&bars[par]);
        if (tid == 0) bar_expect(bar, kCand * sizeof(ulonglong2));
        if (lane < kCl)
            send_async(smem_addr(&cand[par][rank * (kTc / 32) + warp]), bar, lane, key, idx);
        const double fa = (double)(xa ? nx : np), fb = (double)(xa ? np : nx), fs = (double)(nx + np);
        const double rs = __drcp_rn(fs);
        if (E > 0 && prev >= 0) {
#pragma unroll
            for (int e = 0; e < EN; e++)
                vm[e] = xa ? average(fa, vx[e], fb, vp[e], fs, rs)
                           : average(fa, vp[e], fb, vx[e], fs, rs);
            if (own_b) {
                new1 = xa ? average(fa, dx1, fb, dp1, fs, rs) : average(fa, dp1, fb, dx1, fs, rs);
                new2 = xa ? average(fa, dx2, fb, dp2, fs, rs) : average(fa, dp2, fb, dx2, fs, rs);
            }
        }
        if (!bar_wait(bar, phase)) {
            late = true;
            break;
        }
        key = ~0ull;
        idx = ~0u;
#pragma unroll
        for (int q = 0; q < kCand / 32; q++) {
            const ulonglong2 c = cand[par][q * 32 + lane];
            if (c.x < key || (c.x == key && (unsigned)c.y < idx)) {
                key = c.x;
                idx = (unsigned)c.y;
            }
        }
        warp_argmin(key, idx);
        par ^= 1;
        phase ^= (par == 0);
        fresh = -1;
        if (idx == ~0u || (idx != 0u && len >= p)) break;
        if (idx != 0u) {  // the chain grows
            const int y = (int)idx - 1;
            if (tid == 0) chain[len] = y;
#pragma unroll
            for (int e = 0; e < EN; e++) vp[e] = vx[e];
            have_prev = true;
            prev = x;
            x = y;
            len++;
            continue;
        }
        // Reciprocal nearest neighbours: write the merged row and column.
#pragma unroll
        for (int e = 0; e < entries; e++) {
            const int i = index(e);
            if (E > 0 && i == a) live[e % EN] = false;
            if (E > 0 ? !live[e % EN] : (i >= p || size[i] == 0)) continue;
            if (i == a || i == b) continue;
            const double d = E > 0 ? vm[e % EN]
                                   : average(fa, __ldcg(row(a) + i), fb, __ldcg(row(b) + i), fs, rs);
            __stcg(row(b) + i, d);
            __stcg(row(i) + b, d);
            wrote = true;
        }
        if (a % kTc == tid) size[a] = 0;
        if (b % kTc == tid) size[b] = nx + np;
        if (rank == 0 && tid == 0) {
            height[k] = key_dist(key);
            npair[k] = fa * fb;
        }
        k++;
        len -= 2;
        fresh = b;
        x = c1;
        prev = c2;
        have_prev = false;
        if (E == 0 || len == 0) {
            if (!meet()) {  // the merge's writes, for whichever row comes next
                late = true;
                break;
            }
            fresh = -1;
            wrote = false;
        }
        if (len == 0 && k < p - 1) {  // start a chain at the first active cluster
            while (size[first] == 0) first++;
            x = first;
            prev = -1;
            len = 1;
            if (tid == 0) chain[0] = x;
        }
    }
    for (; k < p - 1; k++)
        if (rank == 0 && tid == 0) {
            height[k] = NAN;
            npair[k] = 0.0;
        }
    if (late) atomicExch(gave_up, 1);
    // No block leaves while another may still write its candidates.  Every
    // thread gets here, late or not: it waits for nothing but its own bounded
    // waits, and a warp that is late sends no more, so the others are late in
    // the step after at most.
    cl.sync();
    if (late) {  // what is on its way here, of this step and the next, has as long again
        bar_wait(smem_addr(&bars[par]), phase);
        par ^= 1;
        phase ^= (par == 0);
        bar_wait(smem_addr(&bars[par]), phase);
    }
}

// stat[4] = the cophenetic correlation of matrix blockIdx.x from its merges
// (height, npair), the sum of its distances (stat[0]) and of their squared
// deviations (the B partials); 1 when either side has no spread (the
// reference's convention).
__global__ void __launch_bounds__(kR) cophenetic_from_merges(
    const double *__restrict__ height, const double *__restrict__ npair, int m,
    const double *__restrict__ part, int B, double npairs, double *__restrict__ stat,
    int64_t stride) {
    __shared__ double red[kR];
    height += blockIdx.x * stride;
    npair += blockIdx.x * stride;
    part += blockIdx.x * stride;
    stat += blockIdx.x * stride;
    double dv = 0.0;
    for (int b = threadIdx.x; b < B; b += kR) dv += part[b];
    const double var_d = block_sum(dv, red);
    double a = 0.0;
    for (int k = threadIdx.x; k < m; k += kR) a += npair[k] * height[k];
    const double mc = block_sum(a, red) / npairs;
    const double md = stat[0] / npairs;
    double cv = 0.0, vc = 0.0;
    for (int k = threadIdx.x; k < m; k += kR) {
        cv += npair[k] * (height[k] - mc) * (height[k] - md);
        vc += npair[k] * (height[k] - mc) * (height[k] - mc);
    }
    const double cov = block_sum(cv, red);
    const double var_c = block_sum(vc, red);
    if (threadIdx.x == 0) {
        stat[4] = (var_d > 0.0 && var_c > 0.0) ? cov / sqrt(var_d * var_c) : 1.0;
    }
}

// Launches the trees of `count` matrices with E entries a thread.
template <int E>
cudaError_t launch_trees(int count, double *D, int p, int *scratch, double *height, double *npair,
                         int64_t stride, int *gave_up, cudaStream_t s) {
    const size_t sm = scratch ? 0 : 2 * sizeof(int) * (size_t)p;
    cudaError_t e = cudaFuncSetAttribute(nn_chain_average<E>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)kTreeSmem);
    if (e != cudaSuccess) return e;
    nn_chain_average<E><<<count * kCl, kTc, sm, s>>>(D, p, scratch, height, npair, stride, gave_up);
    return cudaGetLastError();
}

// The statistics of `count` consensus matrices (matrix m at dC + m * stride):
// two streaming passes over all of them and their trees in one launch, a
// cluster of blocks each.
nmfcu_status consensus_stats(nmfcu_context *ctx, int count, int64_t p, const float *dC,
                             int64_t ldc, int64_t stride, double *cophenetic, double *dispersion,
                             cudaStream_t s) {
    const int sms = nmfcu_internal::context_sms(ctx);
    const int B = sms * 8;
    const size_t pp = (size_t)p * (size_t)p;
    // doubles of one matrix: height, npair, two sums' partials, stat
    const size_t nd = 2 * (size_t)p + 2 * (size_t)B + 8;
    void *pD = nullptr, *pi = nullptr, *pd = nullptr;
    NMFCU_TRY(nmfcu_internal::context_buffer(ctx, 13, sizeof(double) * pp * count, &pD));
    const bool smem_tree = 2 * sizeof(int) * (size_t)p <= kTreeSmem;
    if (!smem_tree)  // sizes and chain of every block
        NMFCU_TRY(nmfcu_internal::context_buffer(ctx, 14,
                                                 sizeof(int) * 2 * (size_t)p * count * kCl, &pi));
    NMFCU_TRY(nmfcu_internal::context_buffer(ctx, 15, sizeof(double) * (nd * count + 1), &pd));
    int *gave_up = reinterpret_cast<int *>(static_cast<double *>(pd) + nd * count);
    NMFCU_CUDA_TRY(cudaMemsetAsync(gave_up, 0, sizeof(int), s));
    double *D = static_cast<double *>(pD);
    double *height = static_cast<double *>(pd), *npair = height + p;
    double *part = npair + p;
    double *stat = part + 2 * B;  // [sum d, mean d, -, dispersion, cophenetic]
    const double npairs = (double)p * (double)(p - 1) / 2.0;
    int launches = 0;
    for (int m0 = 0; m0 < count; m0 += 65535) {  // grid.y's limit
        const int mc = std::min(count - m0, 65535);
        const float *C = dC + (size_t)m0 * stride;
        double *Dm = D + pp * m0, *pm = part + nd * m0, *sm = stat + nd * m0;
        distances_and_sums<<<dim3(B, mc), kR, 0, s>>>(C, ldc, stride, (int)p, Dm, pm, (int64_t)nd);
        finish_sums<<<mc, kR, 0, s>>>(pm, B, npairs > 0 ? 1.0 / npairs : 0.0,
                                      1.0 / ((double)p * (double)p), sm, (int64_t)nd);
        launches += 2;
        if (p < 2) continue;
        deviation_sums<<<dim3(B, mc), kR, 0, s>>>(Dm, (int)p, pm, (int64_t)nd, sm);
        launches += 1;
    }
    if (p >= 2) {
        int *scratch = static_cast<int *>(pi);
        const int64_t st = (int64_t)nd;
        const int64_t span = (int64_t)kCl * kTc;
        const int64_t per = (p + span - 1) / span;
        const auto go = [&](auto launch) {
            return launch(count, D, (int)p, scratch, height, npair, st, gave_up, s);
        };
        const cudaError_t e = per <= 1    ? go(launch_trees<1>)
                              : per <= 2  ? go(launch_trees<2>)
                              : per <= 3  ? go(launch_trees<3>)
                              : per <= 4  ? go(launch_trees<4>)
                              : per <= 5  ? go(launch_trees<5>)
                              : per <= 6  ? go(launch_trees<6>)
                              : per <= 8  ? go(launch_trees<8>)
                                          : go(launch_trees<0>);
        NMFCU_CUDA_TRY(e);
        cophenetic_from_merges<<<count, kR, 0, s>>>(height, npair, (int)p - 1, part, B, npairs,
                                                    stat, st);
        launches += 2;
    }
    NMFCU_CUDA_TRY(cudaGetLastError());
    nmfcu_internal::count_launches(ctx, launches);
    std::vector<double> host(5 * (size_t)count, 0.0);
    for (int m = 0; m < count; m++) {
        NMFCU_CUDA_TRY(cudaMemcpyAsync(host.data() + 5 * m, stat + nd * m,
                                       sizeof(double) * (p >= 2 ? 5 : 4),
                                       cudaMemcpyDeviceToHost, s));
    }
    int late = 0;
    NMFCU_CUDA_TRY(cudaMemcpyAsync(&late, gave_up, sizeof(int), cudaMemcpyDeviceToHost, s));
    NMFCU_CUDA_TRY(cudaStreamSynchronize(s));
    if (late)
        return nmfcu_internal::fail(NMFCU_ERR_TIMEOUT, "a wait between a tree's blocks ran out");
    for (int m = 0; m < count; m++) {
        dispersion[m] = host[5 * m + 3];
        cophenetic[m] = p >= 2 ? host[5 * m + 4] : 1.0;
    }
    return NMFCU_OK;
}

}  // namespace

extern "C" nmfcu_status nmfcu_consensus_stats_device(nmfcu_context *ctx, int64_t p,
                                                     const float *dC, int64_t ldc,
                                                     double *cophenetic, double *dispersion,
                                                     void *stream) {
    using nmfcu_internal::fail;
    if (!ctx || !dC || !cophenetic || !dispersion)
        return fail(NMFCU_ERR_INVALID_ARG, "NULL pointer");
    if (p < 1 || p > 200000) return fail(NMFCU_ERR_INVALID_ARG, "p must be in [1, 200000]");
    if (ldc < p) return fail(NMFCU_ERR_INVALID_ARG, "ldc must be >= p");
    std::lock_guard<std::mutex> lk(nmfcu_internal::context_mutex(ctx));
    nmfcu_internal::DeviceScope dg(nmfcu_internal::context_device(ctx));
    return consensus_stats(ctx, 1, p, dC, ldc, 0, cophenetic, dispersion,
                           static_cast<cudaStream_t>(stream));
}

extern "C" nmfcu_status nmfcu_consensus_stats_batch_device(nmfcu_context *ctx, int32_t count,
                                                           int64_t p, const float *dC,
                                                           int64_t ldc, int64_t stride,
                                                           double *cophenetic,
                                                           double *dispersion, void *stream) {
    using nmfcu_internal::fail;
    if (!ctx || !dC || !cophenetic || !dispersion)
        return fail(NMFCU_ERR_INVALID_ARG, "NULL pointer");
    if (count < 1) return fail(NMFCU_ERR_INVALID_ARG, "count must be >= 1");
    if (p < 1 || p > 200000) return fail(NMFCU_ERR_INVALID_ARG, "p must be in [1, 200000]");
    if (ldc < p) return fail(NMFCU_ERR_INVALID_ARG, "ldc must be >= p");
    if (count > 1 && stride < ldc * p)
        return fail(NMFCU_ERR_INVALID_ARG, "stride must be >= ldc * p");
    std::lock_guard<std::mutex> lk(nmfcu_internal::context_mutex(ctx));
    nmfcu_internal::DeviceScope dg(nmfcu_internal::context_device(ctx));
    return consensus_stats(ctx, count, p, dC, ldc, stride, cophenetic, dispersion,
                           static_cast<cudaStream_t>(stream));
}
