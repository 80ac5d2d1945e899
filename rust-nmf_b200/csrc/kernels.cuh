// kernels.cuh -- device code of the B200 NMF engine.
//
// One iteration of every built method is two streaming passes over V plus
// small O(r^2 (n + p)) work:
//
//   H step  (reduce over the n rows of V, one output column per thread):
//     plain : A[k][j] = sum_u W[u][k] V[u][j]                 lee, hals, dnmf
//     ratio : A[k][j] = sum_u W[u][k] V[u][j] / (W H)[u][j]    brunet (WH never stored)
//   W step  (reduce over the p columns of V, one output row per thread):
//     plain : B[i][k] = sum_j V[i][j] H'[k][j]
//     ratio : B[i][k] = sum_j H'[k][j] V[i][j] / (W H')[i][j]
//
// followed by a per-column (H) / per-row (W) epilogue that applies the
// method's update exactly as the reference writes it (multiplicative update
// or a Gauss-Seidel sweep).  Partial sums are written per split and summed
// in a fixed order, so every result is bit-reproducible run to run.
//
// Layouts (device): V row-major n x p with leading dimension ldv; W n x RP
// and H RP x p f64 with the rank padded to the compile-time bucket RP by
// zero columns / rows (a zero pad contributes exact zeros to every sum).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace nmfcu {

// Method ids, same values as include/nmfcu.h.
enum : int { M_BRUNET = 0, M_LEE = 1, M_OFFSET = 2, M_NSNMF = 3, M_HALS = 4, M_EHALS = 5,
             M_DNMF = 6, M_LSNMF = 7 };
// Not a method: the epilogues store the contraction itself (the products of
// the randomized range finder behind the NNDSVD start).
constexpr int M_PRODUCT = 100;

// Device-side state of the stationary stop (lib.rs:1336-1401) and of the
// run: written by single-thread kernels, read by every kernel of an
// iteration so that the iterations after a stop do no work.
struct RunState {
    double last_max;
    double last_min;
    long long n_collected;
    long long n_iter;  // iteration at which the stop fired
    int stopped;       // 1 once the loop has stopped
    int error;         // 1: `iter % check_interval` with check_interval == 0
    int timeout;       // a bounded mbarrier wait gave up (stream.cuh codes)
    // Tickets of the running epilogue or Gram launch: [0] the blocks (or
    // groups of blocks) whose Gram partials are out, [1 + g] group g's blocks.
    unsigned gram_ticket[1 + 32];
};

// Fixed constants of the streaming kernels.
constexpr int kThreads = 256;
constexpr int kWarps = 8;

// (A kernel bound by latency reads it first and acts on it after its loads.)
__device__ __forceinline__ bool run_stopped(const RunState *st) {
    return st != nullptr && st->stopped != 0;
}

// ---------------------------------------------------------------------------
// Arithmetic helpers
// ---------------------------------------------------------------------------

// x / y for the ratio V / (WH), y != 0.  f64: x (1 / y) with the reciprocal
// r from the hardware approximation (rcp.approx.ftz.f64): with e = 1 - y r,
// 1 / y = r / (1 - e) = r (1 + e + e^2 + ...).  |e| is at most 2^-19.9 (2^28
// random y), so the terms left out are below 2^-59.8, a 110th of an ulp.
// The same 2^28 quotients are at most 1.487 ulp from the exact one and 0.353372
// on average; with two Newton steps in place of the series 1.487 and 0.353371.
// (The tests hold the loop to 1e-10 of the oracle's IEEE divisions.)  |y|
// outside [2^-1000, 2^1000) and NaN take the IEEE division; an integer test of
// the exponent, since comparisons of doubles share the pipe the passes are
// bound by.  f32: the fast reciprocal-multiply
// form (the FP32 form is tolerance-checked).
__device__ __forceinline__ bool ratio_plain(double y) {
    return ((unsigned)__double2hiint(y) & 0x7fffffffu) - (23u << 20) < (2000u << 20);
}
__device__ __forceinline__ double ratio_fast(double x, double y) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(y));
    const double e = fma(-y, r, 1.0);
    return x * fma(r, fma(e, e, e), r);
}
// The IEEE division, kept in the branch it stands in: the compiler takes a
// plain one for cheap enough to do ahead of the branch, for every element
// (20000 x 20000 at rank 20: 2.7 ms a pass; 1.52 with comparisons of doubles
// and two Newton steps, 1.35 as it is).
__device__ __forceinline__ double ratio_ieee(double x, double y) {
    asm volatile("" : "+d"(y));
    return x / y;
}
__device__ __forceinline__ double ratio_div(double x, double y) {
    return ratio_plain(y) ? ratio_fast(x, y) : ratio_ieee(x, y);
}
// q[i] = x[i] / y[i], 0 where y[i] is: the fast form of all of them side by
// side, then at most one branch, taken where a y is 0 or at the ends of the
// range.
template <int N>
__device__ __forceinline__ void ratios_or_zero(const double (&x)[N], const double (&y)[N],
                                               double (&q)[N]) {
    bool plain = true;
#pragma unroll
    for (int i = 0; i < N; i++) {
        plain = plain && ratio_plain(y[i]);
        q[i] = ratio_fast(x[i], y[i]);
    }
    if (plain) return;
#pragma unroll
    for (int i = 0; i < N; i++)
        if (!ratio_plain(y[i])) q[i] = y[i] != 0.0 ? ratio_ieee(x[i], y[i]) : 0.0;
}
__device__ __forceinline__ float ratio_div(float x, float y) { return __fdividef(x, y); }

// Epilogue arithmetic without FMA contraction, so that the update formulas
// round exactly as the reference's scalar Rust code does.
__device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }

// ---------------------------------------------------------------------------
// nsNMF and offset helpers
// ---------------------------------------------------------------------------
// Smoothing matrix entry S[k][j] = (1 - theta) I + (theta / r) (lib.rs:458-466).
__device__ __forceinline__ double smooth_at(int k, int j, int r, double theta) {
    const double off = theta / (double)r;
    return (k == j) ? (1.0 - theta) + off : off;
}
// out = X S for X (rows x RP, row-major; columns >= r zero), forward k
// (W S of nmf_run_nsnmf, lib.rs:1811).
template <int RP>
__global__ void __launch_bounds__(kThreads)
    ns_right_s(const double *__restrict__ X, int rows, int r, double theta,
               double *__restrict__ out, const RunState *st) {
    if (run_stopped(st)) return;
    const int i = blockIdx.x * kThreads + threadIdx.x;
    if (i >= rows) return;
    double x[RP];
#pragma unroll
    for (int k = 0; k < RP; k++) x[k] = X[(size_t)i * RP + k];
#pragma unroll
    for (int j = 0; j < RP; j++) {
        double acc = 0.0;
#pragma unroll
        for (int k = 0; k < RP; k++)
            if (k < r && j < r) acc = add(acc, mul(x[k], smooth_at(k, j, r, theta)));
        out[(size_t)i * RP + j] = acc;
    }
}
// out = S H for H (RP x p; rows >= r zero), forward l (S H, lib.rs:1819).
template <int RP>
__global__ void __launch_bounds__(kThreads)
    ns_left_s(const double *__restrict__ H, int p, int r, double theta, double *__restrict__ out,
              const RunState *st) {
    if (run_stopped(st)) return;
    const int j = blockIdx.x * kThreads + threadIdx.x;
    if (j >= p) return;
    double h[RP];
#pragma unroll
    for (int l = 0; l < RP; l++) h[l] = H[(size_t)l * p + j];
#pragma unroll
    for (int k = 0; k < RP; k++) {
        double acc = 0.0;
#pragma unroll
        for (int l = 0; l < RP; l++)
            if (k < r && l < r) acc = add(acc, mul(smooth_at(k, l, r, theta), h[l]));
        out[(size_t)k * p + j] = acc;
    }
}
// addon[k] = sum_u W[u][k] off[u] (den_addon, lib.rs:1705-1709); one block a
// component, a fixed-order tree over the rows.
template <int RP>
__global__ void __launch_bounds__(kThreads)
    off_addon(const double *__restrict__ W, int n, int r, const double *__restrict__ off,
              double *__restrict__ addon, const RunState *st) {
    if (run_stopped(st)) return;
    const int k = blockIdx.x;
    __shared__ double red[kThreads];
    double acc = 0.0;
    if (k < r)
        for (int u = threadIdx.x; u < n; u += kThreads) acc = add(acc, mul(W[(size_t)u * RP + k], off[u]));
    red[threadIdx.x] = acc;
    __syncthreads();
    for (int s = kThreads / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0) addon[k] = (k < r) ? red[0] : 0.0;
}
// lsNMF objective partials (lib.rs:1024-1035): sum_ij (Vs_ij - (W H)_ij S_ij)^2
// with Vs = V o S precomputed, i.e. ((V - W H) o S)^2.  Block b takes rows
// b, b + nblocks, ... one warp a row (lanes over columns in a fixed order, a
// xor butterfly), and writes its sum to part[b].
template <int RP>
__global__ void __launch_bounds__(kThreads)
    ls_objective(const double *__restrict__ Vs, const double *__restrict__ S, int64_t ld, int n,
                 int p, const double *__restrict__ W, const double *__restrict__ H,
                 double *__restrict__ part, const RunState *st) {
    if (run_stopped(st)) return;
    constexpr int kWarps = kThreads / 32;
    __shared__ double red[kWarps];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double acc = 0.0;
    for (int i = blockIdx.x * kWarps + warp; i < n; i += gridDim.x * kWarps) {
        double w[RP];
#pragma unroll
        for (int k = 0; k < RP; k++) w[k] = W[(size_t)i * RP + k];
        for (int j = lane; j < p; j += 32) {
            double wh = 0.0;
#pragma unroll
            for (int k = 0; k < RP; k++) wh = fma(w[k], H[(size_t)k * p + j], wh);
            const double d = Vs[(size_t)i * ld + j] - wh * S[(size_t)i * ld + j];
            acc = fma(d, d, acc);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) red[warp] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int q = 0; q < kWarps; q++) s += red[q];
        part[blockIdx.x] = s;
    }
}
// Vs <- V o S in place (the weighted target of lsNMF, lib.rs:961).
static __global__ void mul_weight(double *__restrict__ V, const double *__restrict__ S,
                                  int64_t ld, int n, int p) {
    const int64_t total = (int64_t)n * p;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total;
         t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = t / p, at = i * ld + (t - i * p);
        V[at] = mul(V[at], S[at]);
    }
}

// E-HALS extrapolation (nmf_run_ehals, lib.rs:755-767) of the first `cols`
// entries of each of `rows` rows (leading dimension ld):
//   x <- max(eps, x + beta (x - prev)),  prev <- the old x.
static __global__ void ehals_extrapolate(double *__restrict__ X, double *__restrict__ prev,
                                         int64_t rows, int ld, int cols, double beta, double eps,
                                         const RunState *st) {
    if (run_stopped(st)) return;
    const int64_t total = rows * cols;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total;
         t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = t / cols;
        const int64_t at = i * ld + (t - i * cols);
        const double x = X[at];
        const double ext = add(x, mul(beta, sub(x, prev[at])));
        X[at] = ext > eps ? ext : eps;
        prev[at] = x;
    }
}

// Row sums of V (one warp a row, fixed-order lanes + butterfly).
static __global__ void __launch_bounds__(kThreads)
    v_row_sums(const double *__restrict__ V, int64_t ldv, int n, int p, double *__restrict__ out) {
    const int i = (int)(((size_t)blockIdx.x * kThreads + threadIdx.x) >> 5);
    const int lane = threadIdx.x & 31;
    if (i >= n) return;
    double acc = 0.0;
    for (int j = lane; j < p; j += 32) acc += V[(size_t)i * ldv + j];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) out[i] = acc;
}
// Default offset: rowMeans(V) (lib.rs:1667-1679).
static __global__ void off_init(const double *__restrict__ rsv, int n, int p,
                                double *__restrict__ off) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) off[i] = rsv[i] / (double)p;
}
// off_i <- off_i max(rowSums(V)_i, eps) / (rowSums(W H + off)_i + eps)
// (lib.rs:1729-1742), with rowSums(W H)_i = sum_k W[i][k] rowSums(H)_k.
template <int RP>
__global__ void __launch_bounds__(kThreads)
    off_update(const double *__restrict__ W, int n, int r, const double *__restrict__ rsh,
               const double *__restrict__ rsv, int p, double eps, double *__restrict__ off,
               const RunState *st) {
    if (run_stopped(st)) return;
    const int i = blockIdx.x * kThreads + threadIdx.x;
    if (i >= n) return;
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < RP; k++)
        if (k < r) s = add(s, mul(W[(size_t)i * RP + k], rsh[k]));
    const double o = off[i];
    const double rsw = add(s, mul((double)p, o));
    const double num = rsv[i] > eps ? rsv[i] : eps;
    off[i] = mul(o, num) / add(rsw, eps);
}

// ---------------------------------------------------------------------------
// Epilogues.  Parameters shared by the H and W epilogues.
// ---------------------------------------------------------------------------
struct EpiParams {
    int method;
    int r;
    double eps;
    double lambda;  // dnmf L1 (sparsity)
    double gamma;   // dnmf L2 (smoothness)
    const double *G;    // RP x RP Gram (W^T W for H, H H^T for W)
    const double *sums; // colsum(W) for the brunet H step, rowsum(H) for the W step
    const double *addon = nullptr;  // offset, H step: (W^T off)[k] added to the denominator
    const double *roff = nullptr;   // offset, W step: the row offsets off[i]
    // lsNMF: the numerator contraction (W^T (V o S) as RP x p for the H step,
    // (V o S) H^T as n x RP for the W step); the pass supplies the denominator.
    const double *aux = nullptr;
};

// Per-column H update from the reduced contraction num[] (old column hc[]).
//   lee    : euclidean_update_h_inner  lib.rs:227-241
//   brunet : divergence_update_h_inner lib.rs:105-111
//   hals   : hals_update_h             lib.rs:595-605
//   dnmf   : hals_update_h_reg         lib.rs:1079-1089
template <int RP>
__device__ __forceinline__ void h_update(const EpiParams &e, const double *num, double *hc,
                                         const double *ax = nullptr) {
    const int r = e.r;
    if (e.method == M_LSNMF) {
        // nmf_run_lsnmf lib.rs:990-999: max(eps, H numer) / (denom + eps)
#pragma unroll
        for (int i = 0; i < RP; i++)
            if (i < r) {
                const double temp = mul(hc[i], ax[i]);
                hc[i] = (temp > e.eps ? temp : e.eps) / add(num[i], e.eps);
            }
    } else if (e.method == M_PRODUCT) {
#pragma unroll
        for (int i = 0; i < RP; i++)
            if (i < r) hc[i] = num[i];
    } else if (e.method == M_LEE || e.method == M_OFFSET) {
        // offset (offset_update_h_inner, lib.rs:330-361): + (W^T off)[i]
        double out[RP];
#pragma unroll
        for (int i = 0; i < RP; i++) {
            if (i < r) {
                double den = 0.0;
#pragma unroll
                for (int l = RP - 1; l >= 0; l--)
                    if (l < r) den = add(den, mul(e.G[i * RP + l], hc[l]));
                if (e.addon) den = add(den, e.addon[i]);
                const double temp = mul(hc[i], num[i]);
                out[i] = (temp > e.eps ? temp : e.eps) / add(den, e.eps);
            }
        }
#pragma unroll
        for (int i = 0; i < RP; i++)
            if (i < r) hc[i] = out[i];
    } else if (e.method == M_BRUNET || e.method == M_NSNMF) {
#pragma unroll
        for (int i = 0; i < RP; i++)
            if (i < r) hc[i] = mul(hc[i], num[i]) / e.sums[i];
    } else {
        const bool reg = (e.method == M_DNMF);
#pragma unroll
        for (int k = 0; k < RP; k++) {
            if (k < r) {
                double s = reg ? sub(num[k], e.lambda) : num[k];
#pragma unroll
                for (int jj = 0; jj < RP; jj++)
                    if (jj < r && jj != k) s = sub(s, mul(e.G[k * RP + jj], hc[jj]));
                const double d = reg ? fmax(add(e.G[k * RP + k], e.gamma), e.eps)
                                     : fmax(e.G[k * RP + k], e.eps);
                const double val = s / d;
                hc[k] = val > e.eps ? val : e.eps;
            }
        }
    }
}

// Per-row W update from the reduced contraction num[] (old row wr[]).
//   lee    : euclidean_update_w_impl lib.rs:307-318
//   brunet : divergence_update_w_impl lib.rs:194-200
//   hals   : hals_update_w           lib.rs:622-632
//   dnmf   : hals_update_w_reg       lib.rs:1106-1116
// ro: the row's offset (offset method; lib.rs:441-446), else unused.
template <int RP>
__device__ __forceinline__ void w_update(const EpiParams &e, const double *num, double *wr,
                                         double ro = 0.0, const double *ax = nullptr) {
    const int r = e.r;
    if (e.method == M_LSNMF) {
        // nmf_run_lsnmf lib.rs:1011-1018
#pragma unroll
        for (int j = 0; j < RP; j++)
            if (j < r) {
                const double temp = mul(wr[j], ax[j]);
                wr[j] = (temp > e.eps ? temp : e.eps) / add(num[j], e.eps);
            }
    } else if (e.method == M_PRODUCT) {
#pragma unroll
        for (int j = 0; j < RP; j++)
            if (j < r) wr[j] = num[j];
    } else if (e.method == M_LEE || e.method == M_OFFSET) {
        double out[RP];
#pragma unroll
        for (int j = 0; j < RP; j++) {
            if (j < r) {
                double den = 0.0;
#pragma unroll
                for (int l = RP - 1; l >= 0; l--)
                    if (l < r) den = add(den, mul(wr[l], e.G[l * RP + j]));
                if (e.method == M_OFFSET) den = add(den, mul(ro, e.sums[j]));
                const double temp = mul(wr[j], num[j]);
                out[j] = (temp < e.eps ? e.eps : temp) / add(den, e.eps);
            }
        }
#pragma unroll
        for (int j = 0; j < RP; j++)
            if (j < r) wr[j] = out[j];
    } else if (e.method == M_BRUNET || e.method == M_NSNMF) {
#pragma unroll
        for (int j = 0; j < RP; j++)
            if (j < r) wr[j] = mul(wr[j], num[j]) / e.sums[j];
    } else {
        const bool reg = (e.method == M_DNMF);
#pragma unroll
        for (int k = 0; k < RP; k++) {
            if (k < r) {
                double s = reg ? sub(num[k], e.lambda) : num[k];
#pragma unroll
                for (int jj = 0; jj < RP; jj++)
                    if (jj < r && jj != k) s = sub(s, mul(e.G[k * RP + jj], wr[jj]));
                const double d = reg ? fmax(add(e.G[k * RP + k], e.gamma), e.eps)
                                     : fmax(e.G[k * RP + k], e.eps);
                const double val = s / d;
                wr[k] = val > e.eps ? val : e.eps;
            }
        }
    }
}

// Whether w_update's new W[i][j] depends on row i's old values and num only
// through column j's own formula (every method but the sequential HALS /
// dnmf sweeps), so that its columns can be computed by different threads.
__device__ __forceinline__ bool w_update_by_column(int method) {
    return method == M_LEE || method == M_OFFSET || method == M_BRUNET ||
           method == M_NSNMF || method == M_LSNMF || method == M_PRODUCT;
}
// Column j (< e.r) of w_update for those methods, with the same operations
// in the same order (so the same bits).  numj = num[j]; wr: the row's old
// values.
template <int RP>
__device__ __forceinline__ double w_update_column(const EpiParams &e, double numj,
                                                  const double *wr, int j, double ro,
                                                  const double *ax) {
    const double wrj = wr[j];
    if (e.method == M_LSNMF) {
        const double temp = mul(wrj, ax[j]);
        return (temp > e.eps ? temp : e.eps) / add(numj, e.eps);
    }
    if (e.method == M_PRODUCT) return numj;
    if (e.method == M_LEE || e.method == M_OFFSET) {
        double den = 0.0;
#pragma unroll
        for (int l = RP - 1; l >= 0; l--)
            if (l < e.r) den = add(den, mul(wr[l], e.G[l * RP + j]));
        if (e.method == M_OFFSET) den = add(den, mul(ro, e.sums[j]));
        const double temp = mul(wrj, numj);
        return (temp < e.eps ? e.eps : temp) / add(den, e.eps);
    }
    return mul(wrj, numj) / e.sums[j];  // M_BRUNET, M_NSNMF
}
// Row i (< e.r) of h_update for the same methods.  hc(l): the column's old
// values; ax: lsNMF's numerator of this row and column.
template <int RP, typename Col>
__device__ __forceinline__ double h_update_row(const EpiParams &e, double numi, Col &&hc, int i,
                                               double ax) {
    if (e.method == M_LSNMF) {
        const double temp = mul(hc(i), ax);
        return (temp > e.eps ? temp : e.eps) / add(numi, e.eps);
    }
    if (e.method == M_PRODUCT) return numi;
    if (e.method == M_LEE || e.method == M_OFFSET) {
        double den = 0.0;
#pragma unroll
        for (int l = RP - 1; l >= 0; l--)
            if (l < e.r) den = add(den, mul(e.G[i * RP + l], hc(l)));
        if (e.addon) den = add(den, e.addon[i]);
        const double temp = mul(hc(i), numi);
        return (temp > e.eps ? temp : e.eps) / add(den, e.eps);
    }
    return mul(hc(i), numi) / e.sums[i];  // M_BRUNET, M_NSNMF
}

// ---------------------------------------------------------------------------
// Gram matrices and sums.
// ---------------------------------------------------------------------------
// X^T X and the column sums of X (W, or H^T).  A launch runs in one of two
// ways (GramPlan):
//   few tiles   a block a tile of kTileRows rows of W / kTileCols columns of
//               H, its warps sharing the tile;
//   many tiles  a warp a tile of 32 rows / columns: tile t goes to block
//               t mod B, whose warps take its tiles in turn, so that a
//               launch has a warp on every multiprocessor before it has two.
// A warp adds four rows (columns) of its tile at a time on the FP64 tensor
// cores (mma.sync.m8n8k4: a fragment of X is both operands), a block adds its
// warps in a fixed tree, publishes its entries and takes a ticket; the last
// block sums the blocks' partials.  Where that is more than 32 loads a thread
// (a round trip to L2 per eight, and a second ticket costs two), the last
// block of each group of 16 sums the group's and the last group the groups'.
// No block waits on another.  The update epilogues (stream.cuh)
// form the same sums over the same tiles from the values they have just
// written, so a Gram has the same bits wherever it is formed.
//
// For brunet, which needs the sums alone, only those are formed.
//
// (One thread an entry walking all rows of a block, and the last block alone
// summing 148 partials, took 31 us for H at 20 x 40000 and 9.1 us at 8 x 3000.)
constexpr int kEpiThreads = 512;   // threads of a block, few tiles
constexpr int kWideThreads = 256;  // threads of a block, many tiles
constexpr int kTileCols = 32;      // columns of H a tile
constexpr int kTileRows = 16;      // rows of W a tile (few tiles)
constexpr int kGramGroup = 16;     // blocks of a group
enum : int { GRAM_NONE = 0, GRAM_SUMS = 1, GRAM_FULL = 2 };

// Tiles of `len` rows or columns, up to 2^31 - 1 of them.
__host__ __device__ inline int tile_count(int len, int tile) {
    return (int)(((unsigned)len + (unsigned)tile - 1u) / (unsigned)tile);
}

// How an epilogue or Gram launch over `len` rows of W / columns of H runs: a
// block a tile up to two blocks a multiprocessor, beyond that a warp a tile.
// At 296 tiles the first still fits the chip at once; the second has every
// warp at work, which the sequential HALS sweeps need.
struct GramPlan {
    bool few;
    int blocks;
};
inline GramPlan gram_plan(int64_t len, int tile, int sms) {
    GramPlan g;
    const int64_t tiles = (len + tile - 1) / tile, cap = 2 * (int64_t)sms;
    g.few = tiles <= cap;
    if (g.few) {
        g.blocks = (int)(tiles < 1 ? 1 : tiles);
    } else {
        const int64_t b = (len + 31) / 32;
        g.blocks = (int)(b < sms ? b : sms);  // its registers leave room for one
    }
    // the tickets count at most 32 groups
    const int most = 32 * kGramGroup;
    if (g.blocks > most) {
        g.few = false;
        g.blocks = most;
    }
    return g;
}

struct GramOut {
    int want = GRAM_NONE;
    // lee, whose W columns are divided by their sums right after: write the
    // Gram of the divided columns (sums stay those of W itself).
    int rescaled = 0;
    double *part = nullptr;  // (blocks + 32) x gram_entries(RP)
    double *G = nullptr;     // RP x RP
    double *sums = nullptr;  // RP
    unsigned *ticket = nullptr;  // RunState::gram_ticket
};

__host__ __device__ constexpr int gram_entries(int RP) { return RP * (RP + 1) / 2 + RP; }

// Entry e of the list [column sums | pairs k <= l]: k, and l (-1: a sum).
template <int RP>
__device__ __forceinline__ void gram_entry(int e, int &k, int &l) {
    if (e < RP) {
        k = e;
        l = -1;
        return;
    }
    e -= RP;
    k = 0;
    while (e >= RP - k) {
        e -= RP - k;
        k++;
    }
    l = k + e;
}

// mma.sync.m8n8k4 with f64 operands: D (8 x 8) += A (8 x 4) B (4 x 8), one
// A and one B element and two D elements a thread (A[g][q], B[q][g],
// D[g][2q + e] with g = lane / 4, q = lane % 4).  The asm has no side effects
// beyond its operands (not volatile), so independent MMAs may be scheduled
// across one another; each accumulator's chain keeps its order.
__device__ __forceinline__ void dmma_8x8x4(double (&d)[2], double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
        : "+d"(d[0]), "+d"(d[1])
        : "d"(a), "d"(b));
}

// a + src[0] + src[step] + ... (count of them, in order), up to eight loads in
// flight at a time: left to itself the remainder of an unrolled loop waits for
// its loads in ever smaller groups.
template <int N, bool ALL, typename Load>
__device__ __forceinline__ double sum_batch(double a, const double *&src, size_t step, int count,
                                            Load &&load) {
    double v[N];
#pragma unroll
    for (int u = 0; u < N; u++) {
        v[u] = ALL || u < count ? load(src) : 0.0;
        src += step;
    }
#pragma unroll
    for (int u = 0; u < N; u++) a += v[u];
    return a;
}
template <typename Load>
__device__ __forceinline__ double sum_strided(double a, const double *src, size_t step, int count,
                                              Load &&load) {
    for (; count >= 8; count -= 8) a = sum_batch<8, true>(a, src, step, 8, load);
    if (count > 4)
        a = sum_batch<7, false>(a, src, step, count, load);
    else if (count > 0)
        a = sum_batch<4, false>(a, src, step, count, load);
    return a;
}

// One more block's partials are out: its ticket.  Orders the block's earlier
// writes before it and the other blocks' before what follows.
__device__ __forceinline__ unsigned take_ticket(unsigned *t) {
    unsigned old;
    asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(old) : "l"(t) : "memory");
    return old;
}

// ACTIVE: the block's warps that add rows (the first ones).
template <int RP, int THREADS, int ACTIVE>
struct GramAcc {
    static constexpr int E = gram_entries(RP);
    static constexpr int MT = (RP + 7) / 8;
    static constexpr int NP = MT * (MT + 1) / 2;  // tiles mt <= nt
    static constexpr int RAW = 2 * NP + MT;       // a lane's values
    static constexpr int WARPS = THREADS / 32;
    // Shared memory of finish(), in doubles.
    static constexpr int SCRATCH_TREE = ACTIVE / 2 * RAW * 32;
    static constexpr int SCRATCH = SCRATCH_TREE > 2 * THREADS + RP ? SCRATCH_TREE : 2 * THREADS + RP;
    double d[NP][2], sm[MT];
    __device__ __forceinline__ void init() {
#pragma unroll
        for (int i = 0; i < NP; i++) d[i][0] = d[i][1] = 0.0;
#pragma unroll
        for (int i = 0; i < MT; i++) sm[i] = 0.0;
    }
    // Adds four rows: at(k, q) is the value of row q (0..3) in column k < RP.
    template <typename At>
    __device__ __forceinline__ void add4(int want, At &&at) {
        const int g = (threadIdx.x & 31) >> 2, q = threadIdx.x & 3;
        double f[MT];
#pragma unroll
        for (int mt = 0; mt < MT; mt++) {
            const int k = mt * 8 + g;
            f[mt] = k < RP ? at(k, q) : 0.0;
            sm[mt] += f[mt];
        }
        if (want != GRAM_FULL) return;
        int i = 0;
#pragma unroll
        for (int mt = 0; mt < MT; mt++)
#pragma unroll
            for (int nt = mt; nt < MT; nt++) dmma_8x8x4(d[i++], f[mt], f[nt]);
    }
    // Where entry (k, l) is in the warps' sum `raw`.
    __device__ __forceinline__ static int raw_index(int k, int l) {
        const int mt = k >> 3, g = k & 7;
        if (l < 0) return (2 * NP + mt) * 32 + g * 4;
        const int nt = l >> 3, c = l & 7;
        const int pair = mt * MT - mt * (mt - 1) / 2 + (nt - mt);
        return (2 * pair + (c & 1)) * 32 + g * 4 + (c >> 1);
    }
    // Sum of `count` partials of entry e (stride E from src) by the whole
    // block: `split` threads an entry, each every split-th.  Valid in threads
    // tid < cnt where split > 1, else in thread e - base.
    __device__ __forceinline__ static double sum_parts(const double *src, int count, int e,
                                                       bool on, int first, int step) {
        if (!on || first >= count) return 0.0;
        return sum_strided(0.0, src + (size_t)first * E + e, (size_t)step * E,
                           (count - first + step - 1) / step,
                           [](const double *q) { return __ldcg(q); });
    }
    // `count` partials at src into dst (E entries each), or, with the last
    // group done, the finished Gram and sums.
    __device__ __forceinline__ static void reduce(const double *src, int count, int limit,
                                                  double *dst, const GramOut &g, double *scratch) {
        const int tid = threadIdx.x;
        double *red = scratch, *val = scratch + THREADS;  // val: THREADS + RP
        const int split = limit < THREADS ? min(THREADS / limit, 16) : 1;
        for (int base = 0; base < limit; base += THREADS) {
            const int q = split > 1 ? tid / limit : 0;
            const int e = split > 1 ? tid - q * limit : base + tid;
            double a = sum_parts(src, count, e, e < limit && q < split, q, split);
            if (split > 1) {
                red[tid] = a;
                __syncthreads();
                if (tid < limit)
                    for (int s = 1; s < split; s++) a += red[s * limit + tid];
            }
            const bool mine = split > 1 ? tid < limit : e < limit;
            if (dst != nullptr) {
                if (mine) dst[e] = a;
                continue;
            }
            // The sums are the first entries, so the first round has them all.
            if (base == 0) {
                if (mine && e < RP) {
                    val[e] = a;
                    g.sums[e] = a;
                }
                __syncthreads();
            }
            if (!mine || e < RP) continue;
            int k, l;
            gram_entry<RP>(e, k, l);
            if (g.rescaled) {
                if (val[k] > 0.0) a /= val[k];
                if (val[l] > 0.0) a /= val[l];
            }
            g.G[k * RP + l] = a;
            g.G[l * RP + k] = a;
        }
    }
    // Adds up the block's warps, publishes, and finishes where this block is
    // the last.  scratch: SCRATCH doubles of shared memory, free to overwrite
    // once every thread of the block has called this.
    __device__ __forceinline__ void finish(const GramOut &g, double *scratch) {
        if (g.want == GRAM_NONE) return;
        const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
        const int limit = g.want == GRAM_FULL ? E : RP;
#pragma unroll
        for (int mt = 0; mt < MT; mt++) {  // over the four rows of a step
            sm[mt] += __shfl_xor_sync(0xffffffffu, sm[mt], 1);
            sm[mt] += __shfl_xor_sync(0xffffffffu, sm[mt], 2);
        }
        for (int half = ACTIVE / 2; half >= 1; half >>= 1) {
            __syncthreads();
            if (warp >= half && warp < 2 * half) {
                double *w = scratch + (size_t)(warp - half) * RAW * 32 + lane;
#pragma unroll
                for (int i = 0; i < NP; i++) {
                    w[(2 * i) * 32] = d[i][0];
                    w[(2 * i + 1) * 32] = d[i][1];
                }
#pragma unroll
                for (int i = 0; i < MT; i++) w[(2 * NP + i) * 32] = sm[i];
            }
            __syncthreads();
            if (warp < half) {
                const double *w = scratch + (size_t)warp * RAW * 32 + lane;
#pragma unroll
                for (int i = 0; i < NP; i++) {
                    d[i][0] += w[(2 * i) * 32];
                    d[i][1] += w[(2 * i + 1) * 32];
                }
#pragma unroll
                for (int i = 0; i < MT; i++) sm[i] += w[(2 * NP + i) * 32];
            }
        }
        __syncthreads();
        if (warp == 0) {
            double *w = scratch + lane;
#pragma unroll
            for (int i = 0; i < NP; i++) {
                w[(2 * i) * 32] = d[i][0];
                w[(2 * i + 1) * 32] = d[i][1];
            }
#pragma unroll
            for (int i = 0; i < MT; i++) w[(2 * NP + i) * 32] = sm[i];
        }
        __syncthreads();
        const int B = (int)gridDim.x;
        for (int e = tid; e < limit; e += THREADS) {
            int k, l;
            gram_entry<RP>(e, k, l);
            g.part[(size_t)blockIdx.x * E + e] = scratch[raw_index(k, l)];
        }
        __shared__ bool last;
        __syncthreads();
        const double *src = g.part;
        int count = B;
        if (B > 2 * kGramGroup && (int64_t)B * limit > 32 * THREADS) {
            const int group = (int)blockIdx.x / kGramGroup;
            const int groups = (B + kGramGroup - 1) / kGramGroup;
            const int members = min(kGramGroup, B - group * kGramGroup);
            if (tid == 0) last = (take_ticket(g.ticket + 1 + group) == (unsigned)members - 1u);
            __syncthreads();
            if (!last) return;
            double *dst = g.part + (size_t)(B + group) * E;
            reduce(g.part + (size_t)group * kGramGroup * E, members, limit, dst, g, scratch);
            if (tid == 0) g.ticket[1 + group] = 0u;
            __syncthreads();
            src = g.part + (size_t)B * E;
            count = groups;
        }
        if (tid == 0) last = (take_ticket(g.ticket) == (unsigned)count - 1u);
        __syncthreads();
        if (!last) return;
        reduce(src, count, limit, nullptr, g, scratch);
        if (tid == 0) *g.ticket = 0u;
    }
};

// W^T W and colsum(W) on their own (a W no epilogue has just written).
template <int RP, int THREADS>
__global__ void __launch_bounds__(THREADS)
    gram_w_tiles(const double *__restrict__ W, int n, GramOut g, const RunState *st) {
    if (run_stopped(st)) return;
    constexpr bool FEW = THREADS == kEpiThreads;
    using GA = GramAcc<RP, THREADS, FEW ? kTileRows / 4 : THREADS / 32>;
    extern __shared__ double scratch[];
    const int warp = threadIdx.x >> 5;
    GA ga;
    ga.init();
    const auto steps = [&](int i0, int rows, int s0, int s1) {
        for (int s = s0; s < s1; s++)
            ga.add4(g.want, [&](int k, int q) {
                const int u = 4 * s + q;
                return u < rows ? W[(size_t)(i0 + u) * RP + k] : 0.0;
            });
    };
    if (FEW) {
        const int i0 = blockIdx.x * kTileRows;
        if (warp < kTileRows / 4) steps(i0, min(kTileRows, n - i0), warp, warp + 1);
    } else {
        const int tiles = tile_count(n, 32);
        for (int t = blockIdx.x + gridDim.x * warp; t < tiles; t += gridDim.x * GA::WARPS)
            steps(t * 32, min(32, n - t * 32), 0, 8);
    }
    ga.finish(g, scratch);
}

// H H^T and rowsum(H) on their own.
template <int RP, int THREADS>
__global__ void __launch_bounds__(THREADS)
    gram_h_tiles(const double *__restrict__ H, int p, GramOut g, const RunState *st) {
    if (run_stopped(st)) return;
    constexpr bool FEW = THREADS == kEpiThreads;
    using GA = GramAcc<RP, THREADS, FEW ? kTileCols / 4 : THREADS / 32>;
    extern __shared__ double scratch[];
    const int warp = threadIdx.x >> 5;
    GA ga;
    ga.init();
    const auto steps = [&](int j0, int s0, int s1) {
        for (int s = s0; s < s1; s++)
            ga.add4(g.want, [&](int k, int q) {
                const int j = j0 + 4 * s + q;
                return j < p ? H[(size_t)k * p + j] : 0.0;
            });
    };
    if (FEW) {
        if (warp < kTileCols / 4) steps(blockIdx.x * kTileCols, warp, warp + 1);
    } else {
        const int tiles = tile_count(p, kTileCols);
        for (int t = blockIdx.x + gridDim.x * warp; t < tiles; t += gridDim.x * GA::WARPS)
            steps(t * kTileCols, 0, kTileCols / 4);
    }
    ga.finish(g, scratch);
}

// lee's col_rescale (lib.rs:1461-1470): W[:, k] /= sums[k] when sums[k] > 0.
template <int RP>
__global__ void col_rescale(double *__restrict__ W, int n, int r, const double *__restrict__ sums,
                            const RunState *st) {
    if (run_stopped(st)) return;
    __shared__ double s[RP];
    if (threadIdx.x < RP) s[threadIdx.x] = sums[threadIdx.x];
    __syncthreads();
    const int64_t total = (int64_t)n * RP;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total;
         t += (int64_t)gridDim.x * blockDim.x) {
        const int k = (int)(t % RP);
        if (k < r && s[k] > 0.0) W[t] = W[t] / s[k];
    }
}

// dnmf's extract_diagonal (lib.rs:808-824) followed by H *= d (lib.rs:880-884).
// Gw / Gh are the Grams of the current W and H; their diagonals are the
// squared norms of W's columns and H's rows.
template <int RP>
__global__ void dnmf_rescale(double *__restrict__ W, double *__restrict__ H, int n, int p, int r,
                             const double *__restrict__ Gw, const double *__restrict__ Gh,
                             const RunState *st) {
    if (run_stopped(st)) return;
    __shared__ double nw[RP], nh[RP], dk[RP];
    if (threadIdx.x < RP) {
        const int k = threadIdx.x;
        const double a = sqrt(Gw[k * RP + k]);
        const double b = sqrt(Gh[k * RP + k]);
        nw[k] = a;
        nh[k] = b;
        dk[k] = a * b;
    }
    __syncthreads();
    const int64_t tw = (int64_t)n * RP;
    const int64_t th = (int64_t)r * p;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < tw; t += stride) {
        const int k = (int)(t % RP);
        if (k < r && nw[k] > 0.0) W[t] = W[t] / nw[k];
    }
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < th; t += stride) {
        const int k = (int)(t / p);
        double h = H[t];
        if (nh[k] > 0.0) h = h / nh[k];
        H[t] = h * dk[k];
    }
}

// brunet's every-10-iterations clamp (pmax_inplace, lib.rs:1452-1458):
// x < eps -> eps (NaN stays NaN), on the r real columns / rows only.
template <int RP>
__global__ void clamp_wh(double *__restrict__ W, double *__restrict__ H, int n, int p, int r,
                         double eps, const RunState *st) {
    if (run_stopped(st)) return;
    const int64_t tw = (int64_t)n * RP;
    const int64_t th = (int64_t)r * p;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < tw; t += stride) {
        const int k = (int)(t % RP);
        if (k < r && W[t] < eps) W[t] = eps;
    }
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < th; t += stride)
        if (H[t] < eps) H[t] = eps;
}

// ---------------------------------------------------------------------------
// Objective finalisation + stationary stop (one block).
// ---------------------------------------------------------------------------
struct StopParams {
    int stationary;       // 1: run StationaryStop::should_stop
    long long iter;       // 0 for the initial objective
    long long check_interval;
    long long check_niter;
    double threshold;
    double scale;         // 0.5 for the Frobenius objective, 1 for KL
};

// Sum of B partials in objective_finalize's order, into out[0] (a column
// shard's objective term, before the sum over shards).
static __global__ void sum_partials(const double *__restrict__ part, int B,
                                    double *__restrict__ out) {
    __shared__ double red[kThreads];
    const int tid = threadIdx.x;
    double a = 0.0;
    for (int b = tid; b < B; b += kThreads) a += part[b];
    red[tid] = a;
    __syncthreads();
    for (int s = kThreads / 2; s > 0; s >>= 1) {
        if (tid < s) red[tid] += red[tid + s];
        __syncthreads();
    }
    if (tid == 0) out[0] = red[0];
}

// W update from a dense contraction num (n x RP) summed over column shards:
// one thread a row, the update of w_update.
template <int RP>
__global__ void __launch_bounds__(kThreads)
    w_apply_dense(double *__restrict__ W, int n, const double *__restrict__ num, EpiParams e,
                  const RunState *st) {
    if (run_stopped(st)) return;
    const int i = blockIdx.x * kThreads + threadIdx.x;
    if (i >= n) return;
    double nm[RP], wr[RP];
#pragma unroll
    for (int k = 0; k < RP; k++) {
        nm[k] = num[(size_t)i * RP + k];
        wr[k] = W[(size_t)i * RP + k];
    }
    w_update<RP>(e, nm, wr);
#pragma unroll
    for (int k = 0; k < RP; k++)
        if (k < e.r) W[(size_t)i * RP + k] = wr[k];
}

static __global__ void objective_finalize(const double *__restrict__ part, int B, double *__restrict__ dev,
                                   StopParams sp, RunState *st) {
    if (st->stopped) return;
    __shared__ double red[kThreads];
    const int tid = threadIdx.x;
    double a = 0.0;
    for (int b = tid; b < B; b += kThreads) a += part[b];
    red[tid] = a;
    __syncthreads();
    for (int s = kThreads / 2; s > 0; s >>= 1) {
        if (tid < s) red[tid] += red[tid + s];
        __syncthreads();
    }
    if (tid != 0) return;
    const double d = red[0] * sp.scale;
    if (dev) dev[sp.iter] = d;
    if (!sp.stationary) return;
    // StationaryStop::should_stop, lib.rs:1378-1400.
    bool stop = false;
    if (isnan(d)) {
        stop = true;
    } else if (sp.iter == 0) {
        st->last_max = d;  // reset() then record(d)
        st->last_min = d;
        st->n_collected = 1;
    } else {
        bool sample = true;
        if (st->n_collected == 0) {
            if (sp.check_interval == 0) {
                st->error = 1;  // the reference panics on `i % 0`
                stop = true;
                sample = false;
            } else if (sp.iter % sp.check_interval != 0) {
                sample = false;
            }
        }
        if (sample) {
            if (d > st->last_max) st->last_max = d;
            if (d < st->last_min) st->last_min = d;
            st->n_collected += 1;
            if (st->n_collected == sp.check_niter + 1) {
                const double crit = fabs(st->last_max - st->last_min) / (double)sp.check_niter;
                if (crit <= sp.threshold) {
                    stop = true;
                } else {
                    st->last_max = -INFINITY;
                    st->last_min = INFINITY;
                    st->n_collected = 0;
                }
            }
        }
    }
    if (stop) {
        st->stopped = 1;
        st->n_iter = sp.iter;
    }
}

// ---------------------------------------------------------------------------
// Layout helpers.
// ---------------------------------------------------------------------------

// H (RP x p f64) -> H^T (p x rps, type TH), zero past the first r entries.
template <typename TH>
__global__ void h_transpose(const double *__restrict__ H, TH *__restrict__ Ht, int p, int r,
                            int rps) {
    const int64_t total = (int64_t)p * rps;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total;
         t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t j = t / rps;
        const int k = (int)(t - j * rps);
        Ht[t] = (k < r) ? (TH)H[(int64_t)k * p + j] : (TH)0;
    }
}

// dst = (float)src, four columns a thread, rows over grid.y.  ldd is a multiple
// of 4 and dst 16-byte aligned; `aligned`: src's rows are too.  Bound: HBM, 12
// bytes an element (3.7 ms at 20000 x 60000 with one element a thread and a
// 64-bit division for its place, 2.1 this way).
static __global__ void __launch_bounds__(kThreads)
    convert_f64_f32(const double *__restrict__ src, int64_t lds, float *__restrict__ dst,
                    int64_t ldd, int n, int p, bool aligned) {
    const int64_t j = ((int64_t)blockIdx.x * kThreads + threadIdx.x) * 4;
    if (j >= p) return;
    for (int64_t i = blockIdx.y; i < n; i += gridDim.y) {
        const double *a = src + i * lds + j;
        float *d = dst + i * ldd + j;
        if (aligned && j + 3 < p) {
            const double2 x = __ldcs(reinterpret_cast<const double2 *>(a));
            const double2 y = __ldcs(reinterpret_cast<const double2 *>(a) + 1);
            *reinterpret_cast<float4 *>(d) =
                make_float4((float)x.x, (float)x.y, (float)y.x, (float)y.y);
        } else {
            for (int c = 0; c < 4 && j + c < p; c++) d[c] = (float)a[c];
        }
    }
}

}  // namespace nmfcu
