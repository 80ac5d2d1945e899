// wide.cu -- the FP64 loop for ranks above the streaming passes' largest
// bucket (NMFCU_MAX_RANK = 32): lee, brunet, hals and dnmf at any rank up to
// NMFCU_MAX_WIDE_RANK.  The reference has no rank limit (nmf_run_lee
// rust/src/lib.rs:1589-1647, nmf_run_brunet :1529-1586, nmf_run_hals
// :638-688, nmf_run_dnmf :827-906).
//
// The V contractions are the FP64 tensor-core streaming passes run in rank
// chunks of at most 32 (nmfcu_internal::v_product_locked, one pass over V a
// chunk):
//   lee / hals / dnmf   W^T V and V H'^T  -> the H and W numerators
//   brunet              the ratio Q = V / (W H) (0 where W H is 0,
//                       lib.rs:89-97 / 181-189) is written out by a tiled
//                       kernel, then W^T Q and Q H'^T by the same passes.
// Everything rank-dependent (Grams, updates, rescaling, objective) runs in
// the kernels below with the rank as a run-time value; the updates follow the
// formulas of the dense engine's epilogues (kernels.cuh h_update / w_update).  The stop state is the context's run state, so
// every pass and kernel of an iteration after a stationary stop does no work.
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <climits>
#include <string>
#include <vector>

#include "../../include/nmfcu.h"
#include "internal.h"
#include "kernels.cuh"

using nmfcu_internal::fail;

namespace {

using nmfcu::RunState;
using nmfcu::add;
using nmfcu::mul;
using nmfcu::sub;
constexpr int kT = 256;

// Context scratch slots of this file.
constexpr int kSlotQ = 24;    // brunet: the ratio V / (W H), n x ldq
constexpr int kSlotBuf = 25;  // factors, contractions, Grams, partials

inline unsigned cdiv(int64_t a, int64_t b) { return (unsigned)((a + b - 1) / b); }
inline size_t align256(size_t x) { return (x + 255) / 256 * 256; }

// ---------------------------------------------------------------------------
// Grams: G[k][l] = sum_u X(u, k) X(u, l) and sums[k] = sum_u X(u, k) for
// X(u, k) = X[u * sr + k * sc] (W: sr = r, sc = 1; H^T: sr = 1, sc = p), on the
// FP64 tensor cores (mma.sync.m8n8k4, kernels.cuh dmma_8x8x4) over X with a
// column of ones behind it, whose products are the sums.
// Stage 1: block (b, y) takes rows [b * rpb, (b + 1) * rpb), kRowsChunk at a
// time through shared memory, and the 8 x 8 tiles (mt <= nt) y * 64 .. + 63 of
// the product, eight a warp.  Stage 2 adds the blocks in order.
// One thread eight entries on the CUDA cores took 94 us for H at 50 x 20000,
// this 20.
// ---------------------------------------------------------------------------
constexpr int kRowsChunk = 32;
constexpr int kGramLd = 36;  // a warp's fragment loads meet every bank once
constexpr int kWarpPairs = 8;
constexpr int kBlockPairs = kWarpPairs * (kT / 32);

__host__ __device__ inline int wide_mt(int r) { return (r + 1 + 7) / 8; }
__host__ __device__ inline int wide_pairs(int r) { return wide_mt(r) * (wide_mt(r) + 1) / 2; }
// Tile number -> (mt, nt), mt <= nt.
__device__ __forceinline__ void wide_pair(int t, int MT, int &mt, int &nt) {
    mt = 0;
    while (t >= MT - mt) {
        t -= MT - mt;
        mt++;
    }
    nt = mt + t;
}

__global__ void __launch_bounds__(kT)
    wide_gram_partial(const double *__restrict__ X, int64_t m, int r, int64_t sr, int64_t sc,
                      int64_t rpb, double *__restrict__ part, const RunState *st) {
    if (nmfcu::run_stopped(st)) return;
    extern __shared__ double chunk[];  // [8 MT columns][kGramLd]
    const int MT = wide_mt(r), pairs = wide_pairs(r);
    const int64_t u0 = blockIdx.x * rpb, u1 = min(m, u0 + rpb);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane >> 2, q = lane & 3;
    const int t0 = blockIdx.y * kBlockPairs + warp * kWarpPairs;
    int am[kWarpPairs], an[kWarpPairs];  // the tiles' fragments in chunk
    double acc[kWarpPairs][2];
#pragma unroll
    for (int i = 0; i < kWarpPairs; i++) {
        int mt = 0, nt = 0;
        if (t0 + i < pairs) wide_pair(t0 + i, MT, mt, nt);
        am[i] = (mt * 8 + g) * kGramLd + q;
        an[i] = (nt * 8 + g) * kGramLd + q;
        acc[i][0] = acc[i][1] = 0.0;
    }
    for (int64_t c0 = u0; c0 < u1; c0 += kRowsChunk) {
        const int nr = (int)min((int64_t)kRowsChunk, u1 - c0);
        __syncthreads();
        for (int e = threadIdx.x; e < MT * 8 * kRowsChunk; e += kT) {
            int uu, k;
            if (sr == 1) {  // neighbours along the rows
                k = e / kRowsChunk;
                uu = e - k * kRowsChunk;
            } else {
                uu = e / (MT * 8);
                k = e - uu * (MT * 8);
            }
            double v = 0.0;
            if (uu < nr) v = k < r ? X[(c0 + uu) * sr + (int64_t)k * sc] : k == r ? 1.0 : 0.0;
            chunk[k * kGramLd + uu] = v;
        }
        __syncthreads();
        if (t0 < pairs)
#pragma unroll 2
            for (int s = 0; s < kRowsChunk; s += 4)
#pragma unroll
                for (int i = 0; i < kWarpPairs; i++)
                    if (t0 + i < pairs)
                        nmfcu::dmma_8x8x4(acc[i], chunk[am[i] + s], chunk[an[i] + s]);
    }
#pragma unroll
    for (int i = 0; i < kWarpPairs; i++)
        if (t0 + i < pairs) {
            double *d = part + ((size_t)blockIdx.x * pairs + t0 + i) * 64 + g * 8 + 2 * q;
            d[0] = acc[i][0];
            d[1] = acc[i][1];
        }
}

__global__ void wide_gram_final(const double *__restrict__ part, int B, int r,
                                double *__restrict__ G, double *__restrict__ sums,
                                const RunState *st) {
    if (nmfcu::run_stopped(st)) return;
    const int MT = wide_mt(r), pairs = wide_pairs(r);
    const int x = blockIdx.x * kT + threadIdx.x;
    if (x >= pairs * 64) return;
    int mt, nt;
    wide_pair(x >> 6, MT, mt, nt);
    const int k = mt * 8 + ((x >> 3) & 7), l = nt * 8 + (x & 7);
    if (k >= r || l > r || l < k) return;
    const double a = nmfcu::sum_strided(0.0, part + x, (size_t)pairs * 64, B,
                                        [](const double *p) { return *p; });
    if (l == r) {
        sums[k] = a;
    } else {
        G[k * r + l] = a;
        G[l * r + k] = a;
    }
}

// Ht (p x r) = H (r x p)^T through 32 x 32 shared-memory tiles.
__global__ void wide_transpose(const double *__restrict__ H, int r, int64_t p,
                               double *__restrict__ Ht, const RunState *st) {
    if (nmfcu::run_stopped(st)) return;
    __shared__ double t[32][33];
    const int64_t j0 = (int64_t)blockIdx.x * 32;
    const int k0 = blockIdx.y * 32;
    for (int y = threadIdx.y; y < 32; y += 8) {
        const int k = k0 + y;
        const int64_t j = j0 + threadIdx.x;
        if (k < r && j < p) t[y][threadIdx.x] = H[(int64_t)k * p + j];
    }
    __syncthreads();
    for (int y = threadIdx.y; y < 32; y += 8) {
        const int64_t j = j0 + y;
        const int k = k0 + threadIdx.x;
        if (k < r && j < p) Ht[j * r + k] = t[threadIdx.x][y];
    }
}

// ---------------------------------------------------------------------------
// W H in 128 x 64 tiles on the FP64 tensor cores (eight warps of 32 x 32, the
// rank in chunks of 16 through shared memory, the next chunk in registers),
// and what each use makes of it:
//   MODE 0  Q[i][j] = V[i][j] / (W H)[i][j], 0 where W H is 0 (brunet's ratio)
//   MODE 1  per-block partial of the KL objective (kl_divergence lib.rs:1418-1427)
//   MODE 2  per-block partial of sum (V - W H)^2 (euclidean_distance :1440-1441)
// Bound: FP64.  5000 x 20000 rank 50, MODE 0: 1062 us on the CUDA cores, 797
// here (two blocks a multiprocessor; 983 with one).
// ---------------------------------------------------------------------------
// v / w: the refined reciprocal of the dense passes (ratio_div) and one residual
// correction (Markstein 1990), so the quotient is as good as a division's,
// which takes its slow way out for every v of 0.
__device__ __forceinline__ double quotient(double v, double w) {
    const double q = nmfcu::ratio_div(v, w);
    const double a = fabs(w);
    if (!(a > 0x1p-500 && a < 0x1p500 && fabs(q) < 0x1p500)) return q;
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(w));
    return fma(fma(-q, w, v), r, q);
}
constexpr int kWhRows = 128, kWhCols = 64, kWhK = 16;
constexpr int kWhLdW = 20, kWhLdH = 68;  // fragment loads meet every bank once

template <int MODE>
__global__ void __launch_bounds__(kT, 2)
    wide_wh(const double *__restrict__ V, int64_t ldv, const double *__restrict__ W,
            const double *__restrict__ H, int n, int64_t p, int r, double *__restrict__ Q,
            int64_t ldq, double *__restrict__ part, const RunState *st) {
    if (nmfcu::run_stopped(st)) return;
    __shared__ double sW[kWhRows][kWhLdW];
    __shared__ double sH[kWhK][kWhLdH];
    constexpr int PW = kWhRows * kWhK / kT, PH = kWhK * kWhCols / kT;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane >> 2, q = lane & 3;
    const int wr = (warp >> 1) * 32, wc = (warp & 1) * 32;  // the warp's tile
    const int i0 = blockIdx.y * kWhRows;
    const int64_t j0 = (int64_t)blockIdx.x * kWhCols;
    double acc[4][4][2];
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
        for (int b = 0; b < 4; b++) acc[a][b][0] = acc[a][b][1] = 0.0;
    double vw[PW], vh[PH];
    const auto fetch = [&](int k0) {
#pragma unroll
        for (int t = 0; t < PW; t++) {
            const int e = threadIdx.x + t * kT;
            const int i = i0 + e / kWhK, k = k0 + e % kWhK;
            vw[t] = (i < n && k < r) ? W[(int64_t)i * r + k] : 0.0;
        }
#pragma unroll
        for (int t = 0; t < PH; t++) {
            const int e = threadIdx.x + t * kT;
            const int k = k0 + e / kWhCols;
            const int64_t j = j0 + e % kWhCols;
            vh[t] = (k < r && j < p) ? H[(int64_t)k * p + j] : 0.0;
        }
    };
    fetch(0);
    for (int k0 = 0; k0 < r; k0 += kWhK) {
        __syncthreads();
#pragma unroll
        for (int t = 0; t < PW; t++) {
            const int e = threadIdx.x + t * kT;
            sW[e / kWhK][e % kWhK] = vw[t];
        }
#pragma unroll
        for (int t = 0; t < PH; t++) {
            const int e = threadIdx.x + t * kT;
            sH[e / kWhCols][e % kWhCols] = vh[t];
        }
        __syncthreads();
        if (k0 + kWhK < r) fetch(k0 + kWhK);
#pragma unroll
        for (int ks = 0; ks < kWhK; ks += 4) {
            if (k0 + ks >= r) break;
            double a[4], b[4];
#pragma unroll
            for (int t = 0; t < 4; t++) {
                a[t] = sW[wr + t * 8 + g][ks + q];
                b[t] = sH[ks + q][wc + t * 8 + g];
            }
#pragma unroll
            for (int x = 0; x < 4; x++)
#pragma unroll
                for (int y = 0; y < 4; y++) nmfcu::dmma_8x8x4(acc[x][y], a[x], b[y]);
        }
    }
    // Past V's edge one operand is 0, the other a factor's entry: 0 also where
    // that is infinite.
    if (MODE != 0 && (n - i0 < kWhRows || p - j0 < kWhCols))
#pragma unroll
        for (int x = 0; x < 4; x++)
#pragma unroll
            for (int y = 0; y < 4; y++)
#pragma unroll
                for (int e = 0; e < 2; e++)
                    if (i0 + wr + x * 8 + g >= n || j0 + wc + y * 8 + 2 * q + e >= p)
                        acc[x][y][e] = 0.0;
    // A row's eight elements a thread are loaded together, the next row's while
    // this one's are divided (or their logarithms taken).
    double term = 0.0;
    const auto load_row = [&](int x, double (&v)[8]) {
        const int i = i0 + wr + x * 8 + g;
#pragma unroll
        for (int y = 0; y < 4; y++) {
            const int64_t j = j0 + wc + y * 8 + 2 * q;
            const double *src = V + (int64_t)i * ldv + j;  // 16-byte aligned
            double2 d = make_double2(0.0, 0.0);
            if (i < n && j + 1 < p)
                d = *reinterpret_cast<const double2 *>(src);
            else if (i < n && j < p)
                d.x = *src;
            v[2 * y] = d.x;
            v[2 * y + 1] = d.y;
        }
    };
    double vn[8];
    load_row(0, vn);
#pragma unroll
    for (int x = 0; x < 4; x++) {
        const int i = i0 + wr + x * 8 + g;
        double v[8];
#pragma unroll
        for (int t = 0; t < 8; t++) v[t] = vn[t];
        if (x < 3) load_row(x + 1, vn);
#pragma unroll
        for (int y = 0; y < 4; y++) {
            const int64_t j = j0 + wc + y * 8 + 2 * q;
            double o[2];
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const double ve = v[2 * y + e], wh = acc[x][y][e];
                // past V's edge v and W H are 0: no term
                if (MODE == 0) {
                    o[e] = (wh != 0.0) ? quotient(ve, wh) : 0.0;
                } else if (MODE == 1) {
                    if (ve > 0.0) {
                        if (wh > 0.0) term = add(term, add(sub(mul(ve, log(ve / wh)), ve), wh));
                    } else {
                        term = add(term, wh);
                    }
                } else {
                    const double d = sub(ve, wh);
                    term = add(term, mul(d, d));
                }
            }
            if (MODE == 0 && i < n) {
                double *dst = Q + (int64_t)i * ldq + j;
                if (j + 1 < p)
                    *reinterpret_cast<double2 *>(dst) = make_double2(o[0], o[1]);
                else if (j < p)
                    *dst = o[0];
            }
        }
    }
    if (MODE != 0) {
        __shared__ double red[kT];
        red[threadIdx.x] = term;
        __syncthreads();
        for (int s = kT / 2; s > 0; s >>= 1) {
            if ((int)threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
            __syncthreads();
        }
        if (threadIdx.x == 0) part[(int64_t)blockIdx.y * gridDim.x + blockIdx.x] = red[0];
    }
}

// ---------------------------------------------------------------------------
// Updates, in the dense epilogues' operation order (kernels.cuh h_update /
// w_update).  A block takes kUpd columns of H / rows of W, their old values
// in shared memory, a lane a column / row; lee's and brunet's entries are
// independent and go to the warps in turn, four at a time; so do the old
// values' terms of the HALS / dnmf sweeps, which then go eight entries at a time.  (One
// thread a column, reading H from L2 for every term, took 124 us for H at 50 x
// 20000 and 188 us for W at 5000 x 50 with lee; now 47 and 17.)
// ---------------------------------------------------------------------------
constexpr int kUpd = 32;
struct WideEpi {
    int method;
    int r;
    double eps, lambda, gamma;
    const double *G;     // r x r, symmetric
    const double *sums;  // r
};

// The Gauss-Seidel sweeps (hals_update_{h,w} lib.rs:595-605, :622-632; their
// regularised forms :1079-1089, :1106-1116): entry k becomes
//   max(eps, (num_k [- lambda] - sum_{j != k} G_kj x_j) / max(G_kk [+ gamma], eps))
// with x_j new for j < k.  Written as one sum it is a chain of r dependent
// subtractions an entry, r^2 a line: 357 us for H at 90 x 10000, 132 this way.  x_j is old for
// j > k, so those terms go first, for all entries at once, and a new value's
// term goes to every later entry as soon as it is there.  The same terms in
// another order, by FMA: the rounding of a sum differs by an ulp or so of its
// largest term.
struct SweepDiv {
    double d, r;  // the divisor and RN(1 / d)
    bool plain;   // r and 1 / r are far from the ends of the range
};
__device__ __forceinline__ SweepDiv sweep_div(const WideEpi &e, double gkk) {
    const double d = e.method == nmfcu::M_DNMF ? fmax(add(gkk, e.gamma), e.eps) : fmax(gkk, e.eps);
    return {d, __drcp_rn(d), d > 0x1p-900 && d < 0x1p900};
}
// max(eps, s / d): the quotient from the reciprocal with one residual
// correction (Markstein 1990), three dependent operations.  The IEEE division
// at the ends of the range: with eps = 0 a component that has all but vanished
// has a divisor whose reciprocal is infinite.
__device__ __forceinline__ double sweep_value(double s, SweepDiv v, double eps) {
    double q = __dmul_rn(s, v.r);
    if (v.plain && fabs(s) < 0x1p900)
        q = fma(fma(-q, v.d, s), v.r, q);
    else
        q = nmfcu::ratio_ieee(s, v.d);
    return q > eps ? q : eps;
}

// The new values of one line (a column of H or a row of W): line x of the
// block's, its old values at old[k * (kUpd + 1) + x], its contraction at
// sum[k * (kUpd + 1) + x] (both may be overwritten); out(k, v) stores entry k.
template <bool HSIDE, typename Out>
__device__ __forceinline__ void wide_line(double *old, double *sum, int x, bool in,
                                          const WideEpi &e, int warp, int warps, Out &&out) {
    const int r = e.r;
    double *o = old + x;
    constexpr int LD = kUpd + 1;
    const auto num = [&](int k) { return sum[k * LD + x]; };
    if (e.method == nmfcu::M_LEE) {
        // euclidean_update_h_inner lib.rs:227-241, euclidean_update_w_impl :307-318
        for (int i = warp * 4; i < r; i += warps * 4) {
            double den[4] = {0.0, 0.0, 0.0, 0.0};
            const int m = min(4, r - i);
            if (m == 4) {
#pragma unroll 4
                for (int l = r - 1; l >= 0; l--) {
                    const double h = o[l * LD];
                    const double *gl = e.G + (int64_t)l * r + i;
#pragma unroll
                    for (int t = 0; t < 4; t++) den[t] = add(den[t], mul(gl[t], h));
                }
            } else {
                for (int l = r - 1; l >= 0; l--) {
                    const double h = o[l * LD];
#pragma unroll
                    for (int t = 0; t < 3; t++)
                        if (t < m) den[t] = add(den[t], mul(e.G[(int64_t)l * r + i + t], h));
                }
            }
#pragma unroll
            for (int t = 0; t < 4; t++) {
                if (t >= m || !in) continue;
                const double temp = mul(o[(i + t) * LD], num(i + t));
                // H keeps a NaN's clamp at eps, W the NaN (lib.rs:240, :317)
                const double top = HSIDE ? (temp > e.eps ? temp : e.eps)
                                         : (temp < e.eps ? e.eps : temp);
                out(i + t, top / add(den[t], e.eps));
            }
        }
    } else if (e.method == nmfcu::M_BRUNET) {
        // divergence_update_h_inner lib.rs:105-111, divergence_update_w_impl :194-200
        if (in)
            for (int i = warp; i < r; i += warps) out(i, mul(o[i * LD], num(i)) / e.sums[i]);
    } else {
        // The sweep: the old values' terms of every entry first, four entries
        // a warp at a time; then eight entries in order by one warp, and their
        // terms of every later entry by all.  Entry k's sum is in num(k)'s place.
        const bool reg = e.method == nmfcu::M_DNMF;
        double *sm = sum + x;
        for (int i = warp * 4; i < r; i += warps * 4) {
            const int m = min(4, r - i);
            double a[4];
#pragma unroll
            for (int t = 0; t < 4; t++)
                a[t] = t < m ? (reg ? sub(sm[(i + t) * LD], e.lambda) : sm[(i + t) * LD]) : 0.0;
#pragma unroll 4
            for (int l = i + 1; l < r; l++) {
                const double h = o[l * LD];
                const double *gl = e.G + (int64_t)l * r + i;
#pragma unroll
                for (int t = 0; t < 4; t++)
                    if (t < m && l > i + t) a[t] = fma(-gl[t], h, a[t]);
            }
#pragma unroll
            for (int t = 0; t < 4; t++)
                if (t < m) sm[(i + t) * LD] = a[t];
        }
        for (int k0 = 0; k0 < r; k0 += 8) {
            __syncthreads();
            const int m = min(8, r - k0);
            if (warp == 0) {
                double sv[8], g[8][8];
                SweepDiv dv[8];
#pragma unroll
                for (int a = 0; a < 8; a++) {
                    sv[a] = a < m ? sm[(k0 + a) * LD] : 0.0;
#pragma unroll
                    for (int b = a; b < 8; b++)
                        g[a][b] = b < m ? e.G[(int64_t)(k0 + a) * r + k0 + b] : 0.0;
                    dv[a] = sweep_div(e, g[a][a]);
                }
#pragma unroll
                for (int a = 0; a < 8; a++) {
                    if (a >= m) continue;
                    const double v = sweep_value(sv[a], dv[a], e.eps);
#pragma unroll
                    for (int b = a + 1; b < 8; b++) sv[b] = fma(-g[a][b], v, sv[b]);
                    o[(k0 + a) * LD] = v;
                    if (in) out(k0 + a, v);
                }
            }
            __syncthreads();
            for (int i = k0 + 8 + warp; i < r; i += warps) {
                const double *gi = e.G + (int64_t)i * r + k0;
                double a = sm[i * LD];
#pragma unroll
                for (int t = 0; t < 8; t++)  // (no later entry unless all eight are there)
                    a = fma(-gi[t], o[(k0 + t) * LD], a);
                sm[i * LD] = a;
            }
        }
    }
}

// H (r x p) in place; num: p x r (num[j * r + k]).
__global__ void __launch_bounds__(kT)
    wide_h_update(double *__restrict__ H, int64_t p, const double *__restrict__ num, WideEpi e,
                  const RunState *st) {
    if (nmfcu::run_stopped(st)) return;
    extern __shared__ double upd[];
    double *old = upd, *sn = upd + (size_t)e.r * (kUpd + 1);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const int64_t j0 = (int64_t)blockIdx.x * kUpd;
    const int cols = (int)min((int64_t)kUpd, p - j0), r = e.r;
    for (int k = warp; k < r; k += warps)
        old[k * (kUpd + 1) + lane] = lane < cols ? H[(int64_t)k * p + j0 + lane] : 0.0;
    for (int x = threadIdx.x; x < kUpd * r; x += blockDim.x)
        sn[(x % r) * (kUpd + 1) + x / r] = x < cols * r ? num[j0 * r + x] : 0.0;
    __syncthreads();
    wide_line<true>(old, sn, lane, lane < cols, e, warp, warps,
                    [&](int k, double v) { H[(int64_t)k * p + j0 + lane] = v; });
}

// W (n x r) in place; num: n x r.
__global__ void __launch_bounds__(kT)
    wide_w_update(double *__restrict__ W, int n, const double *__restrict__ num, WideEpi e,
                  const RunState *st) {
    if (nmfcu::run_stopped(st)) return;
    extern __shared__ double upd[];
    double *old = upd, *sn = upd + (size_t)e.r * (kUpd + 1);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const int64_t i0 = (int64_t)blockIdx.x * kUpd;
    const int rows = (int)min((int64_t)kUpd, n - i0), r = e.r;
    for (int x = threadIdx.x; x < kUpd * r; x += blockDim.x) {
        const int at = (x % r) * (kUpd + 1) + x / r;
        old[at] = x < rows * r ? W[i0 * r + x] : 0.0;
        sn[at] = x < rows * r ? num[i0 * r + x] : 0.0;
    }
    __syncthreads();
    // the new values take num's place, then go out contiguously
    wide_line<false>(old, sn, lane, lane < rows, e, warp, warps,
                     [&](int k, double v) { sn[k * (kUpd + 1) + lane] = v; });
    __syncthreads();
    for (int x = threadIdx.x; x < rows * r; x += blockDim.x)
        W[i0 * r + x] = sn[(x % r) * (kUpd + 1) + x / r];
}

// lee's col_rescale (lib.rs:1461-1470): W[:, k] /= colsum_k when > 0.
__global__ void wide_col_rescale(double *__restrict__ W, int64_t n, int r,
                                 const double *__restrict__ sums, const RunState *st) {
    if (nmfcu::run_stopped(st)) return;
    const int64_t total = n * r;
    for (int64_t t = blockIdx.x * (int64_t)kT + threadIdx.x; t < total;
         t += (int64_t)gridDim.x * kT) {
        const double s = sums[t % r];
        if (s > 0.0) W[t] = W[t] / s;
    }
}

// brunet's every-10-iterations clamp (pmax_inplace, lib.rs:1452-1458).
__global__ void wide_clamp(double *__restrict__ W, int64_t nw, double *__restrict__ H, int64_t nh,
                           double eps, const RunState *st) {
    if (nmfcu::run_stopped(st)) return;
    const int64_t stride = (int64_t)gridDim.x * kT;
    for (int64_t t = blockIdx.x * (int64_t)kT + threadIdx.x; t < nw; t += stride)
        if (W[t] < eps) W[t] = eps;
    for (int64_t t = blockIdx.x * (int64_t)kT + threadIdx.x; t < nh; t += stride)
        if (H[t] < eps) H[t] = eps;
}

// dnmf's extract_diagonal (lib.rs:808-824) and H *= d (lib.rs:880-884), as
// kernels.cuh dnmf_rescale.
__global__ void wide_dnmf_rescale(double *__restrict__ W, int64_t n, double *__restrict__ H,
                                  int64_t p, int r, const double *__restrict__ Gw,
                                  const double *__restrict__ Gh, const RunState *st) {
    if (nmfcu::run_stopped(st)) return;
    const int64_t stride = (int64_t)gridDim.x * kT;
    for (int64_t t = blockIdx.x * (int64_t)kT + threadIdx.x; t < n * r; t += stride) {
        const int k = (int)(t % r);
        const double a = sqrt(Gw[k * r + k]);
        if (a > 0.0) W[t] = W[t] / a;
    }
    for (int64_t t = blockIdx.x * (int64_t)kT + threadIdx.x; t < (int64_t)r * p; t += stride) {
        const int k = (int)(t / p);
        const double a = sqrt(Gw[k * r + k]), b = sqrt(Gh[k * r + k]);
        double h = H[t];
        if (b > 0.0) h = h / b;
        H[t] = h * (a * b);
    }
}

// ---------------------------------------------------------------------------
// Host loop
// ---------------------------------------------------------------------------

struct Bufs {
    double *W, *H, *Ht, *NW, *NH, *part, *Gw, *sw, *Gh, *sh, *Gw2, *sw2, *opart;
    double *Q;
    int64_t ldq;
    int Bw, Bh, gy;
    int64_t rpw, rph;
    int gx_obj, gy_obj;
};

struct Loop {
    nmfcu_context *c;
    const nmfcu_options *o;
    int64_t n, p;
    int r;
    const double *V;
    int64_t ldv;
    Bufs b;
    RunState *st;
    double *dev;
    cudaStream_t s;

    nmfcu_status gram(const double *X, int64_t m, int64_t sr, int64_t sc, int B, int64_t rpb,
                      double *G, double *sums) {
        nmfcu_internal::TimedScope sc_(c, s, NMFCU_KCLASS_OTHER, 2);
        const size_t sm = sizeof(double) * 8 * wide_mt(r) * kGramLd;
        NMFCU_CUDA_TRY(cudaFuncSetAttribute(
            wide_gram_partial, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
        wide_gram_partial<<<dim3(B, b.gy), kT, sm, s>>>(X, m, r, sr, sc, rpb, b.part, st);
        wide_gram_final<<<cdiv((int64_t)wide_pairs(r) * 64, kT), kT, 0, s>>>(b.part, B, r, G, sums,
                                                                            st);
        NMFCU_CUDA_TRY(cudaGetLastError());
        return NMFCU_OK;
    }
    nmfcu_status gram_w(double *G, double *sums) { return gram(b.W, n, r, 1, b.Bw, b.rpw, G, sums); }
    nmfcu_status gram_h(double *G, double *sums) { return gram(b.H, p, 1, p, b.Bh, b.rph, G, sums); }
    void transpose() {
        nmfcu_internal::TimedScope sc_(c, s, NMFCU_KCLASS_OTHER);
        wide_transpose<<<dim3(cdiv(p, 32), cdiv(r, 32)), dim3(32, 8), 0, s>>>(b.H, r, p, b.Ht, st);
    }
    void ratio() {
        nmfcu_internal::TimedScope sc_(c, s, NMFCU_KCLASS_OTHER);
        wide_wh<0><<<dim3(b.gx_obj, b.gy_obj), kT, 0, s>>>(V, ldv, b.W, b.H, (int)n, p, r, b.Q,
                                                          b.ldq, nullptr, st);
    }
    WideEpi epi(const double *G, const double *sums, bool hside) const {
        WideEpi e;
        e.method = o->method;
        e.r = r;
        e.eps = o->eps;
        e.lambda = hside ? o->sparsity_h : o->sparsity_w;
        e.gamma = hside ? o->smoothness_h : o->smoothness_w;
        e.G = G;
        e.sums = sums;
        return e;
    }
    // Old values and contraction of a block's lines: at most 135 KB.
    size_t update_smem() const { return sizeof(double) * 2 * (size_t)r * (kUpd + 1); }
    // The H step: numerator p x r (V^T W, or Q^T W for brunet), then the update.
    nmfcu_status h_step(const WideEpi &e) {
        const bool kl = o->method == NMFCU_BRUNET;
        if (kl) ratio();
        // (the passes time themselves as H-step launches)
        NMFCU_TRY(nmfcu_internal::v_product_locked(c, 1, n, p, r, kl ? b.Q : V, kl ? b.ldq : ldv,
                                                   b.W, r, b.NH, r, s, false, false));
        nmfcu_internal::TimedScope sc_(c, s, NMFCU_KCLASS_OTHER);
        const size_t sm = update_smem();
        NMFCU_CUDA_TRY(cudaFuncSetAttribute(
            wide_h_update, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
        if (p > 0) wide_h_update<<<cdiv(p, kUpd), kT, sm, s>>>(b.H, p, b.NH, e, st);
        NMFCU_CUDA_TRY(cudaGetLastError());
        return NMFCU_OK;
    }
    // The W step: numerator n x r (V H'^T, or Q H'^T for brunet), then the update.
    nmfcu_status w_step(const WideEpi &e) {
        const bool kl = o->method == NMFCU_BRUNET;
        if (kl) ratio();
        transpose();
        // (the passes time themselves as W-step launches)
        NMFCU_TRY(nmfcu_internal::v_product_locked(c, 0, n, p, r, kl ? b.Q : V, kl ? b.ldq : ldv,
                                                   b.Ht, r, b.NW, r, s, false, false));
        nmfcu_internal::TimedScope sc_(c, s, NMFCU_KCLASS_OTHER);
        const size_t sm = update_smem();
        NMFCU_CUDA_TRY(cudaFuncSetAttribute(
            wide_w_update, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
        if (n > 0)
            wide_w_update<<<cdiv(n, kUpd), kT, sm, s>>>(b.W, (int)n, b.NW, e, st);
        NMFCU_CUDA_TRY(cudaGetLastError());
        return NMFCU_OK;
    }
    nmfcu_status objective(long long iter) {
        const bool kl = o->method == NMFCU_BRUNET;
        {
            nmfcu_internal::TimedScope sc_(c, s, NMFCU_KCLASS_OBJECTIVE);
            if (kl)
                wide_wh<1><<<dim3(b.gx_obj, b.gy_obj), kT, 0, s>>>(V, ldv, b.W, b.H, (int)n, p, r,
                                                                  nullptr, 0, b.opart, st);
            else
                wide_wh<2><<<dim3(b.gx_obj, b.gy_obj), kT, 0, s>>>(V, ldv, b.W, b.H, (int)n, p, r,
                                                                  nullptr, 0, b.opart, st);
        }
        nmfcu::StopParams sp;
        sp.stationary = 1;
        sp.iter = iter;
        sp.check_interval = o->check_interval;
        sp.check_niter = o->check_niter;
        sp.threshold = o->stationary_th;
        sp.scale = kl ? 1.0 : 0.5;
        nmfcu_internal::TimedScope sc_(c, s, NMFCU_KCLASS_OTHER);
        nmfcu::objective_finalize<<<1, nmfcu::kThreads, 0, s>>>(
            b.opart, b.gx_obj * b.gy_obj, dev, sp, st);
        NMFCU_CUDA_TRY(cudaGetLastError());
        return NMFCU_OK;
    }
    nmfcu_status iteration(long long it) {
        switch (o->method) {
            case NMFCU_BRUNET:
                // nmf_run_brunet lib.rs:1558-1575
                NMFCU_TRY(gram_w(b.Gw, b.sw));
                NMFCU_TRY(h_step(epi(b.Gw, b.sw, true)));
                NMFCU_TRY(gram_h(b.Gh, b.sh));
                NMFCU_TRY(w_step(epi(b.Gh, b.sh, false)));
                if (it % 10 == 0) {
                    nmfcu_internal::TimedScope sc_(c, s, NMFCU_KCLASS_OTHER);
                    wide_clamp<<<std::min(4096u, std::max(1u, cdiv(std::max(n, p) * r, kT))), kT, 0, s>>>(
                        b.W, n * r, b.H, (int64_t)r * p, DBL_EPSILON, st);
                }
                break;
            case NMFCU_LEE:
                // nmf_run_lee lib.rs:1618-1636
                NMFCU_TRY(gram_w(b.Gw, b.sw));
                NMFCU_TRY(h_step(epi(b.Gw, b.sw, true)));
                NMFCU_TRY(gram_h(b.Gh, b.sh));
                NMFCU_TRY(w_step(epi(b.Gh, b.sh, false)));
                if (o->rescale) {
                    NMFCU_TRY(gram_w(b.Gw2, b.sw2));
                    nmfcu_internal::TimedScope sc_(c, s, NMFCU_KCLASS_OTHER);
                    wide_col_rescale<<<std::min(4096u, std::max(1u, cdiv(n * r, kT))), kT, 0, s>>>(
                        b.W, n, r, b.sw2, st);
                }
                break;
            default:
                // nmf_run_hals lib.rs:667-676; nmf_run_dnmf lib.rs:862-884
                NMFCU_TRY(gram_w(b.Gw, b.sw));
                NMFCU_TRY(h_step(epi(b.Gw, b.sw, true)));
                NMFCU_TRY(gram_h(b.Gh, b.sh));
                NMFCU_TRY(w_step(epi(b.Gh, b.sh, false)));
                if (o->method == NMFCU_DNMF) {
                    NMFCU_TRY(gram_w(b.Gw2, b.sw2));
                    nmfcu_internal::TimedScope sc_(c, s, NMFCU_KCLASS_OTHER);
                    wide_dnmf_rescale<<<std::min(4096u, std::max(1u, cdiv(std::max(n, p) * r, kT))), kT, 0, s>>>(
                        b.W, n, b.H, p, r, b.Gw2, b.Gh, st);
                }
                break;
        }
        NMFCU_CUDA_TRY(cudaGetLastError());
        return NMFCU_OK;
    }
};

nmfcu_status make_bufs(nmfcu_context *c, const nmfcu_options *o, int64_t n, int64_t p, int r,
                       Bufs &b) {
    const int sms = nmfcu_internal::context_sms(c);
    b.Bw = (int)std::max<int64_t>(1, std::min<int64_t>((n + 63) / 64, sms));
    b.rpw = std::max<int64_t>(1, (n + b.Bw - 1) / b.Bw);
    b.Bh = (int)std::max<int64_t>(1, std::min<int64_t>((p + 63) / 64, sms));
    b.rph = std::max<int64_t>(1, (p + b.Bh - 1) / b.Bh);
    b.gy = (int)cdiv(wide_pairs(r), kBlockPairs);
    b.gx_obj = (int)std::max<int64_t>(1, (p + kWhCols - 1) / kWhCols);
    b.gy_obj = (int)std::max<int64_t>(1, (n + kWhRows - 1) / kWhRows);
    const size_t d = sizeof(double);
    const size_t nr = (size_t)n * r, pr = (size_t)p * r;
    const std::vector<size_t> sizes = {
        d * nr, d * pr, d * pr, d * nr, d * pr,
        d * (size_t)std::max(b.Bw, b.Bh) * wide_pairs(r) * 64,
        d * r * r, d * r, d * r * r, d * r, d * r * r, d * r,
        d * (size_t)b.gx_obj * b.gy_obj};
    size_t total = 0;
    for (size_t z : sizes) total += align256(std::max<size_t>(z, 1));
    void *base = nullptr;
    NMFCU_TRY(nmfcu_internal::context_buffer(c, kSlotBuf, total, &base));
    double **dst[] = {&b.W, &b.H, &b.Ht, &b.NW, &b.NH, &b.part, &b.Gw, &b.sw,
                      &b.Gh, &b.sh, &b.Gw2, &b.sw2, &b.opart};
    char *q = static_cast<char *>(base);
    for (size_t i = 0; i < sizes.size(); i++) {
        *dst[i] = reinterpret_cast<double *>(q);
        q += align256(std::max<size_t>(sizes[i], 1));
    }
    b.Q = nullptr;
    b.ldq = std::max<int64_t>(16, (p + 15) / 16 * 16);
    if (o->method == NMFCU_BRUNET) {
        void *pq = nullptr;
        NMFCU_TRY(nmfcu_internal::context_buffer(c, kSlotQ, d * (size_t)n * b.ldq, &pq));
        b.Q = static_cast<double *>(pq);
    }
    return NMFCU_OK;
}

}  // namespace

namespace nmfcu_internal {

// The option checks for a rank above NMFCU_MAX_RANK.
nmfcu_status wide_validate(const nmfcu_options *o, int64_t n, int64_t p, int64_t r) {
    if (!o) return fail(NMFCU_ERR_INVALID_ARG, "options pointer is NULL");
    if (r > NMFCU_MAX_WIDE_RANK)
        return fail(NMFCU_ERR_UNSUPPORTED, "rank " + std::to_string(r) +
                                               " exceeds the largest supported rank (" +
                                               std::to_string(NMFCU_MAX_WIDE_RANK) + ")");
    if (o->method != NMFCU_LEE && o->method != NMFCU_BRUNET && o->method != NMFCU_HALS &&
        o->method != NMFCU_DNMF)
        return fail(NMFCU_ERR_UNSUPPORTED,
                    "ranks above " + std::to_string(NMFCU_MAX_RANK) +
                        " run lee, brunet, hals and dnmf");
    if (o->precision != NMFCU_PREC_FP64)
        return fail(NMFCU_ERR_UNSUPPORTED,
                    "ranks above " + std::to_string(NMFCU_MAX_RANK) + " run in FP64 only");
    return validate_options_rank(o, n, p, r, NMFCU_MAX_WIDE_RANK);
}

// The loop at a rank above NMFCU_MAX_RANK, V f64 n x p (pitch ldv, a
// 16-byte aligned base and pitch) on the device.  W0 (n x r) and H0 (r x p)
// are read with `in_kind`, W and H written with `out_kind` (host or device
// copies; they may alias W0 / H0); d_dev: device deviances (or NULL).  The
// caller holds the context's mutex with its device current and has checked
// the options (wide_validate).
nmfcu_status wide_run(nmfcu_context *c, const nmfcu_options *o, int64_t n, int64_t p, int64_t r,
                      const double *V, int64_t ldv, const double *W0, const double *H0,
                      double *W, double *H, cudaMemcpyKind in_kind, cudaMemcpyKind out_kind,
                      double *d_dev, cudaStream_t s, int64_t *n_dev, int64_t *n_iter) {
    const bool stat = o->stop == NMFCU_STOP_STATIONARY;
    // The passes' workspace (and the run state) for the largest chunk.
    NMFCU_TRY(context_prepare(c, n, p));
    RunState *st = static_cast<RunState *>(context_state(c));
    Bufs b;
    NMFCU_TRY(make_bufs(c, o, n, p, (int)r, b));
    NMFCU_CUDA_TRY(cudaMemcpyAsync(b.W, W0, sizeof(double) * (size_t)(n * r), in_kind, s));
    NMFCU_CUDA_TRY(cudaMemcpyAsync(b.H, H0, sizeof(double) * (size_t)(r * p), in_kind, s));
    NMFCU_CUDA_TRY(cudaMemsetAsync(st, 0, sizeof(RunState), s));
    Loop L{c, o, n, p, (int)r, V, ldv, b, st, d_dev, s};
    if (stat) NMFCU_TRY(L.objective(0));
    for (long long it = 1; it <= o->max_iter; it++) {
        NMFCU_TRY(L.iteration(it));
        if (stat) NMFCU_TRY(L.objective(it));
    }
    NMFCU_CUDA_TRY(cudaMemcpyAsync(W, b.W, sizeof(double) * (size_t)(n * r), out_kind, s));
    NMFCU_CUDA_TRY(cudaMemcpyAsync(H, b.H, sizeof(double) * (size_t)(r * p), out_kind, s));
    RunState hs;
    NMFCU_CUDA_TRY(cudaMemcpyAsync(&hs, st, sizeof(RunState), cudaMemcpyDeviceToHost, s));
    NMFCU_CUDA_TRY(cudaStreamSynchronize(s));
    drain_timing(c);
    if (hs.timeout != 0)
        return fail(NMFCU_ERR_TIMEOUT, "a streaming kernel gave up waiting for its copies (code " +
                                           std::to_string(hs.timeout) + ")");
    if (hs.error == 1)
        return fail(NMFCU_ERR_INVALID_ARG,
                    "check_interval must be > 0 (the stationary stop evaluates iter % check_interval)");
    const int64_t iters = hs.stopped ? hs.n_iter : o->max_iter;
    *n_iter = iters;
    *n_dev = stat ? iters + 1 : 0;
    return NMFCU_OK;
}

}  // namespace nmfcu_internal
