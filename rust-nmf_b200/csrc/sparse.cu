// sparse.cu -- the NMF loop on a sparse V given in compressed sparse row
// (CSR) form: lee, brunet, hals and dnmf in FP64, the same updates as the
// dense engine (rust/src/lib.rs nmf_run_lee :1589-1647, nmf_run_brunet
// :1529-1586, nmf_run_hals :638-688, nmf_run_dnmf :827-906).
//
// Single-cell matrices are mostly zeros (AnnData keeps them as CSR); the
// reference densifies V before its loop (python/nmf_rs/__init__.py:495).
// Every V term of the updates is zero at an unstored entry:
//   lee / hals / dnmf  W^T V and V H^T are sums over the stored entries;
//   brunet             V / (W H) is 0 where V is 0 (lib.rs:89-97, 181-189),
//                      so W H is formed only at the stored entries;
// the denominators (W^T W, H H^T, colsum(W), rowsum(H)) do not involve V.
// The objectives split into a stored-entry pass plus closed forms:
//   KL   sum_stored,v>0 [v ln(v/wh) - v + wh] + (sum_all wh - sum_stored,v>0 wh),
//        sum_all wh = sum_k colsum(W)_k rowsum(H)_k     (lib.rs:1410-1431)
//   Fro  sum_stored [(v - wh)^2 - wh^2] + ||W H||^2,
//        ||W H||^2 = sum_kl (W^T W)_kl (H H^T)_kl        (lib.rs:1434-1445)
//
// Passes (one warp a line, lanes across its stored entries, a fixed
// butterfly reduction, so results are bit-reproducible run to run):
//   W pass  rows of the CSR:     out[i][k] = sum_t f(v_t) H^T[j_t][k]
//   H pass  columns of a CSC copy made once a run (each column lists its
//           rows in order: by tiles, or a stable sort of the column indices):
//                                out[k][j] = sum_t f(v_t) W[i_t][k]
// with f(v) = v, or v / (W H)_ij for brunet (0 where W H is 0).  The outputs
// have the layouts of the dense engine's one-split epilogue partials, so its
// update epilogues (h_epilogue / w_epilogue), Grams, rescaling, clamp and
// stationary stop run unchanged.  Bytes per pass: nnz x 12 (value + index)
// plus the factor rows, read from shared memory a block at a time where lines
// have enough entries in each block, else gathered from L2 (W: n x RP, H^T:
// p x RP f64).
#include <cuda_runtime.h>

#include <cub/cub.cuh>

#include <algorithm>
#include <cfloat>
#include <string>
#include <vector>

#include "../../include/nmfcu.h"
#include "internal.h"
#include "kernels.cuh"
#include "launch.h"
#include "stream.cuh"

using nmfcu_internal::fail;

namespace {

using nmfcu::RunState;
using nmfcu::EpiParams;
constexpr int kT = nmfcu::kThreads;  // 256

// Context scratch slots of this file.
constexpr int kSlotCsr = 18;    // host entry: the uploaded CSR
constexpr int kSlotCsc = 19;    // the CSC copy
constexpr int kSlotSort = 20;   // the radix sort's buffers (CSC build only)
constexpr int kSlotFac = 21;    // padded W, H, H^T and the two contractions
constexpr int kSlotSmall = 22;  // Grams, sums, objective partials, state, deviances
constexpr int kSlotSeg = 26;    // the blocked passes' segments and line ranges
constexpr int kSlotCheck = 23;  // validation flags of the device entry

inline unsigned cdiv(int64_t a, int64_t b) { return (unsigned)((a + b - 1) / b); }
inline size_t align256(size_t x) { return (x + 255) / 256 * 256; }

int bucket_for(int64_t r) {
    static const int b[] = {2, 4, 6, 8, 10, 12, 14, 16, 20, 24, 28, 32};
    for (int v : b)
        if (r <= v) return v;
    return -1;
}

// ---------------------------------------------------------------------------
// Kernels
// ---------------------------------------------------------------------------

// rows_of[t] = the row of stored entry t.
__global__ void csr_rows_of(const int64_t *__restrict__ indptr, int n, int32_t *__restrict__ rows) {
    const int lane = threadIdx.x & 31;
    const int gw = (int)((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5);
    const int nw = (int)(((int64_t)gridDim.x * blockDim.x) >> 5);
    for (int i = gw; i < n; i += nw)
        for (int64_t t = indptr[i] + lane; t < indptr[i + 1]; t += 32) rows[t] = i;
}

__global__ void iota32(int32_t *__restrict__ x, int64_t nnz) {
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < nnz;
         t += (int64_t)gridDim.x * blockDim.x)
        x[t] = (int32_t)t;
}

// The CSC copy from the sorted column keys and the permutation of the sort.
__global__ void csc_gather(const int32_t *__restrict__ perm, const int32_t *__restrict__ rows_of,
                           const double *__restrict__ data, int32_t *__restrict__ rows,
                           double *__restrict__ vals, int64_t nnz) {
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < nnz;
         t += (int64_t)gridDim.x * blockDim.x) {
        const int32_t src = perm[t];
        rows[t] = rows_of[src];
        vals[t] = data[src];
    }
}

// colptr[c] = first position of column c in the sorted keys (empty columns
// included); thread t = nnz closes the columns after the last key.
__global__ void csc_colptr(const int32_t *__restrict__ keys, int64_t nnz, int p,
                           int64_t *__restrict__ colptr) {
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t <= nnz;
         t += (int64_t)gridDim.x * blockDim.x) {
        const int prev = (t == 0) ? -1 : keys[t - 1];
        const int cur = (t == nnz) ? p : keys[t];
        for (int c = prev + 1; c <= cur; c++) colptr[c] = t;
    }
}

// The CSC copy of a CSR whose rows are in strict column order, without a sort:
// the matrix in tiles of kCscRows rows x kCscCols columns, a block each.  A
// tile marks its entries in a bit mask a column (a bit a row); the bits below
// an entry's row count the tile's entries before it in its column.
//   tile_counts    table[tile row][column] = entries of the column in the tile
//   column_counts  table -> entries of the column in the tile rows above; total
//   tile_scatter   each entry to colptr + table + its rank in the tile
constexpr int kCscRows = 128, kCscCols = 2048;
// Marks a tile's entries: mask[c][row / 32].
__device__ __forceinline__ void tile_mask(const int64_t *ptr, const int32_t *idx,
                                          const int32_t *seg, int n, unsigned (*mask)[4]) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    const int r0 = blockIdx.y * kCscRows, c0 = blockIdx.x * kCscCols;
    for (int e = threadIdx.x; e < kCscCols * 4; e += blockDim.x) (&mask[0][0])[e] = 0u;
    __syncthreads();
    const int32_t *s0 = seg + (size_t)blockIdx.x * n, *s1 = s0 + n;
    for (int i = warp; i < kCscRows && r0 + i < n; i += warps) {
        const int64_t base = ptr[r0 + i], t1 = base + s1[r0 + i];
        for (int64_t t = base + s0[r0 + i] + lane; t < t1; t += 32)
            atomicOr(&mask[idx[t] - c0][i >> 5], 1u << (i & 31));
    }
    __syncthreads();
}
__global__ void __launch_bounds__(512)
    tile_counts(const int64_t *__restrict__ ptr, const int32_t *__restrict__ idx,
                const int32_t *__restrict__ seg, int n, int p, int32_t *__restrict__ table) {
    __shared__ unsigned mask[kCscCols][4];
    tile_mask(ptr, idx, seg, n, mask);
    const int c0 = blockIdx.x * kCscCols;
    for (int c = threadIdx.x; c < kCscCols && c0 + c < p; c += blockDim.x)
        table[(size_t)blockIdx.y * p + c0 + c] =
            __popc(mask[c][0]) + __popc(mask[c][1]) + __popc(mask[c][2]) + __popc(mask[c][3]);
}
__global__ void column_counts(int32_t *__restrict__ table, int rows, int p,
                              int64_t *__restrict__ total) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c > p) return;
    int64_t sum = 0;
    if (c < p) {
        for (int r0 = 0; r0 < rows; r0 += 8) {
            int32_t v[8];
#pragma unroll
            for (int u = 0; u < 8; u++) v[u] = r0 + u < rows ? table[(size_t)(r0 + u) * p + c] : 0;
#pragma unroll
            for (int u = 0; u < 8; u++) {
                if (r0 + u < rows) table[(size_t)(r0 + u) * p + c] = (int32_t)sum;
                sum += v[u];
            }
        }
    }
    total[c] = sum;  // total[p] = 0 closes the scan
}
// The tile's columns kCscSub at a time: their entries are put in column order
// in shared memory and leave in runs (8 bytes here and there, straight from the
// rows, took 5.6 ms at 10^8 entries).  Entries past kCscList of a sub-tile (more
// than a ninth of it stored) go out directly.
constexpr int kCscSub = 256, kCscList = 3840;
__global__ void __launch_bounds__(512)
    tile_scatter(const int64_t *__restrict__ ptr, const int32_t *__restrict__ idx,
                 const double *__restrict__ val, const int32_t *__restrict__ seg, int n, int p,
                 const int32_t *__restrict__ table, const int64_t *__restrict__ colptr,
                 int32_t *__restrict__ rows, double *__restrict__ vals) {
    __shared__ double lval[kCscList];
    __shared__ unsigned char lrow[kCscList], lcol[kCscList];
    __shared__ unsigned mask[kCscSub][4];
    __shared__ int start[kCscSub + 1], wsum[kCscSub / 32];
    __shared__ int64_t dest[kCscSub];  // where the sub-tile's part of a column goes
    __shared__ int64_t at[kCscRows], upto[kCscRows];  // the rows' entries of the sub-tile
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, warps = blockDim.x >> 5;
    const int r0 = blockIdx.y * kCscRows, c0 = blockIdx.x * kCscCols;
    const int nr = min(kCscRows, n - r0);
    const int32_t *s0 = seg + (size_t)blockIdx.x * n, *s1 = s0 + n;
    if (tid < nr) at[tid] = ptr[r0 + tid] + s0[r0 + tid];
    for (int sub = c0; sub < min(c0 + kCscCols, p); sub += kCscSub) {
        for (int e = tid; e < kCscSub * 4; e += blockDim.x) (&mask[0][0])[e] = 0u;
        if (tid < kCscSub && sub + tid < p)
            dest[tid] = colptr[sub + tid] + table[(size_t)blockIdx.y * p + sub + tid];
        __syncthreads();
        for (int i = warp; i < nr; i += warps) {
            const int64_t end = ptr[r0 + i] + s1[r0 + i];
            int64_t t = at[i];
            for (;; t += 32) {
                const int c = t + lane < end ? idx[t + lane] - sub : kCscSub;
                const bool in = c < kCscSub;
                if (in) atomicOr(&mask[c][i >> 5], 1u << (i & 31));
                const unsigned all = __ballot_sync(0xffffffffu, in);
                if (all != 0xffffffffu) {  // (sorted: the row's entries here are a prefix)
                    t += __popc(all);
                    break;
                }
            }
            if (lane == 0) upto[i] = t;
        }
        __syncthreads();
        // Exclusive sums of the columns' counts.
        int cnt = 0, incl = 0;
        if (tid < kCscSub) {
            cnt = __popc(mask[tid][0]) + __popc(mask[tid][1]) + __popc(mask[tid][2]) +
                  __popc(mask[tid][3]);
            incl = cnt;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += y;
            }
            if (lane == 31) wsum[warp] = incl;
        }
        __syncthreads();
        if (tid < kCscSub) {
            int before = 0;
            for (int w = 0; w < warp; w++) before += wsum[w];
            start[tid] = before + incl - cnt;
            if (tid == kCscSub - 1) start[kCscSub] = before + incl;
        }
        __syncthreads();
        for (int i = warp; i < nr; i += warps) {
            const int w = i >> 5;
            const unsigned below = (1u << (i & 31)) - 1u;
            for (int64_t t = at[i] + lane; t < upto[i]; t += 32) {
                const int c = idx[t] - sub;
                int rank = __popc(mask[c][w] & below);
                for (int q = 0; q < w; q++) rank += __popc(mask[c][q]);
                const int l = start[c] + rank;
                if (l < kCscList) {
                    lval[l] = val[t];
                    lrow[l] = (unsigned char)i;
                    lcol[l] = (unsigned char)c;
                } else {
                    rows[dest[c] + rank] = r0 + i;
                    vals[dest[c] + rank] = val[t];
                }
            }
        }
        __syncthreads();
        for (int l = tid; l < min(start[kCscSub], kCscList); l += blockDim.x) {
            const int c = lcol[l];
            const int64_t to = dest[c] + (l - start[c]);
            rows[to] = r0 + lrow[l];
            vals[to] = lval[l];
        }
        if (tid < nr) at[tid] = upto[tid];
        __syncthreads();
    }
}

// Checks a device CSR: indptr[0] == 0, non-decreasing, indptr[n] == nnz, and
// every column index in [0, p).  flags[0] = 1 on a bad indptr, flags[1] = 1
// on a bad index (flags cleared by the caller).
__global__ void csr_check(const int64_t *__restrict__ indptr, int n, const int32_t *__restrict__ idx,
                          int64_t nnz, int p, int *__restrict__ flags) {
    const int64_t tid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = tid; i <= n; i += stride) {
        const int64_t v = indptr[i];
        if ((i == 0 && v != 0) || (i == n && v != nnz) || v < 0 || v > nnz ||
            (i > 0 && indptr[i - 1] > v))
            flags[0] = 1;
    }
    for (int64_t t = tid; t < nnz; t += stride) {
        const int32_t j = idx[t];
        if (j < 0 || j >= p) flags[1] = 1;
    }
}

// The contraction over the stored entries of each line (a CSR row for the W
// pass, a CSC column for the H pass), one warp a line:
//   out[m][k] = sum_t f(v_t) F[x_t][k],  f(v) = v, or v / (sum_k G[m][k] F[x_t][k])
// (0 where that is 0) when RATIO.  G: the line's own factor rows (lines x
// RP), F: the rows the stored entries index.  OUT_KM writes out[k * ldo + m]
// (the H epilogue's [RP][p] layout), else out[m * RP + k].
template <int RP, bool RATIO, bool OUT_KM>
__global__ void __launch_bounds__(kT)
    sparse_pass(const int64_t *__restrict__ ptr, const int32_t *__restrict__ idx,
                const double *__restrict__ val, int lines, int64_t ldo,
                const double *__restrict__ G, const double *__restrict__ F,
                double *__restrict__ out, const RunState *st) {
    if (nmfcu::run_stopped(st)) return;
    const int lane = threadIdx.x & 31;
    const int gw = (int)((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5);
    const int nw = (int)(((int64_t)gridDim.x * blockDim.x) >> 5);
    for (int m = gw; m < lines; m += nw) {
        double g[RATIO ? RP : 1];
        if (RATIO) {
            const double2 *g2 = reinterpret_cast<const double2 *>(G + (int64_t)m * RP);
#pragma unroll
            for (int k = 0; k < RP / 2; k++) {
                const double2 x = g2[k];
                g[2 * k] = x.x;
                g[2 * k + 1] = x.y;
            }
        }
        double acc[RP];
#pragma unroll
        for (int k = 0; k < RP; k++) acc[k] = 0.0;
        const int64_t t1 = ptr[m + 1];
        for (int64_t t = ptr[m] + lane; t < t1; t += 32) {
            const int x = idx[t];
            const double v = val[t];
            const double2 *f2 = reinterpret_cast<const double2 *>(F + (int64_t)x * RP);
            double f[RP];
#pragma unroll
            for (int k = 0; k < RP / 2; k++) {
                const double2 y = __ldg(f2 + k);
                f[2 * k] = y.x;
                f[2 * k + 1] = y.y;
            }
            double q = v;
            if (RATIO) {
                double wh = 0.0;
#pragma unroll
                for (int k = 0; k < RP; k++) wh = fma(g[k], f[k], wh);
                q = (wh != 0.0) ? nmfcu::ratio_div(v, wh) : 0.0;
            }
#pragma unroll
            for (int k = 0; k < RP; k++) acc[k] = fma(q, f[k], acc[k]);
        }
        double mine = 0.0;
#pragma unroll
        for (int k = 0; k < RP; k++) {
            double a = acc[k];
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) a += __shfl_xor_sync(0xffffffffu, a, off);
            if (lane == k) mine = a;
        }
        if (lane < RP) {
            if (OUT_KM)
                out[(int64_t)lane * ldo + m] = mine;
            else
                out[(int64_t)m * RP + lane] = mine;
        }
    }
}

// ---------------------------------------------------------------------------
// The same contraction with the gathered factor rows in shared memory.
// ---------------------------------------------------------------------------
// sparse_pass pulls an RP x 8-byte factor row from L2 for every stored entry:
// 16 GB a pass at 10^8 entries and rank 20, 2.4 ms (plain) and 4.0 ms (ratio).
// Here a block keeps B consecutive rows of F in shared memory (one bulk copy)
// and its warps run over the entries that index them, line by line; a line's
// entries are sorted, so those of one block of F are a segment of it
// (line_segments).  A block owns a range of lines with about the same number
// of entries, goes through the blocks of F in order, and adds each segment's
// sum to the line's (always the same warp, in block order: the same bits from
// run to run).
//
// A warp takes 32 entries at a time, one a lane.  A group of GL lanes goes
// through its GL entries, each lane with every GL-th pair of the entry's row;
// W H comes together so that each lane ends with its own entry's, and divides
// it once.  A fixed butterfly adds the groups at the segment's end.  Bound:
// latency.  The shared-memory reads of factor rows, at random bank phases about
// 2.6 cycles an entry, are half of a pass (0.93 of 1.83 ms with the ratio, of
// 1.54 without, at 10^8 entries and rank 20); a warp has one chunk of 32
// entries in flight, whose shuffles (and FP64 chain at the ratio) follow one
// another, and a segment ends in a butterfly and a sum in global memory.
constexpr int kBlkBytes = 200 * 1024;  // of F in shared memory
constexpr int blk_rows(int RP) { return kBlkBytes / (RP * 8) / 32 * 32; }  // rows of F a block
template <int RP>
struct BlkCfg {
    static constexpr int PAIRS = RP / 2;
    static constexpr int GL = 4;                       // lanes of an entry
    static constexpr int UPL = (PAIRS + GL - 1) / GL;  // pairs of a lane
    // Warps: as many as the registers of GL rows' pairs leave room for.
    static constexpr int WARPS = UPL >= 4 ? 12 : 16;
    static constexpr int ROWS = blk_rows(RP);
    static constexpr int SMEM = ROWS * RP * 8 + 16;
};

// seg[b * lines + m] = entries of line m that index rows below b * rows of F
// (b = 0 .. blocks).
__global__ void line_segments(const int64_t *__restrict__ ptr, const int32_t *__restrict__ idx,
                              int lines, int rows, int blocks, int32_t *__restrict__ seg) {
    const int64_t total = (int64_t)lines * (blocks + 1);
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
         t += (int64_t)gridDim.x * blockDim.x) {
        const int b = (int)(t / lines), m = (int)(t - (int64_t)b * lines);
        const int64_t t0 = ptr[m], t1 = ptr[m + 1];
        const int64_t key = (int64_t)b * rows;
        int64_t lo = t0, hi = t1;
        while (lo < hi) {
            const int64_t mid = (lo + hi) >> 1;
            if (idx[mid] < key)
                lo = mid + 1;
            else
                hi = mid;
        }
        seg[t] = (int32_t)(lo - t0);
    }
}
// order[0] = 1 if a line's indices ever decrease, order[1] = 1 if one repeats.
__global__ void lines_order(const int64_t *__restrict__ ptr, const int32_t *__restrict__ idx,
                            int lines, int *__restrict__ order) {
    const int lane = threadIdx.x & 31;
    const int gw = (int)((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5);
    const int nw = (int)(((int64_t)gridDim.x * blockDim.x) >> 5);
    bool down = false, same = false;
    for (int m = gw; m < lines; m += nw)
        for (int64_t t = ptr[m] + lane; t + 1 < ptr[m + 1]; t += 32) {
            const int a = idx[t], b = idx[t + 1];
            down |= a > b;
            same |= a == b;
        }
    if (down) order[0] = 1;
    if (same) order[1] = 1;
}
// bound[g] = the first line of block g's range: ranges of equal entries.
__global__ void line_bounds(const int64_t *__restrict__ ptr, int lines, int64_t nnz, int G,
                            int *__restrict__ bound) {
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g > G) return;
    const int64_t key = nnz * g / G;
    int lo = 0, hi = lines;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (ptr[mid] < key)
            lo = mid + 1;
        else
            hi = mid;
    }
    bound[g] = g == G ? lines : lo;
}

// acc: lines x RP; OUT_KM writes the finished sums to out[k * ldo + m]
// (otherwise acc is the output).
template <int RP, bool RATIO, bool OUT_KM>
__global__ void __launch_bounds__(32 * BlkCfg<RP>::WARPS, 1)
    sparse_pass_blocked(const int64_t *__restrict__ ptr, const int32_t *__restrict__ idx,
                        const double *__restrict__ val, const int32_t *__restrict__ seg,
                        const int *__restrict__ bound, int lines, int64_t ldo,
                        const double *__restrict__ G, const double *__restrict__ F, int frows,
                        double *__restrict__ acc_out, double *__restrict__ out, RunState *st) {
    using C = BlkCfg<RP>;
    if (nmfcu::run_stopped(st)) return;
    extern __shared__ __align__(16) unsigned char blk_smem[];
    double *sF = reinterpret_cast<double *>(blk_smem);
    uint64_t *bar = reinterpret_cast<uint64_t *>(blk_smem + (size_t)C::ROWS * RP * 8);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int gl = lane % C::GL, slot = lane / C::GL, first = lane - gl;
    const int m0 = bound[blockIdx.x], m1 = bound[blockIdx.x + 1];
    const int blocks = (frows + C::ROWS - 1) / C::ROWS;
    if (threadIdx.x == 0) {
        nmfcu::mbar_init(bar, 1);
        nmfcu::fence_mbar_init();
    }
    for (int b = 0; b < blocks; b++) {
        __syncthreads();  // everyone is done with the last block of F (and sees the barrier)
        const int x0 = b * C::ROWS, nx = min(C::ROWS, frows - x0);
        if (threadIdx.x == 0) {
            nmfcu::fence_proxy_async_smem();
            const uint32_t bytes = (uint32_t)nx * RP * 8;
            nmfcu::mbar_expect_tx(bar, bytes);
            asm volatile(
                "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, "
                "[%3];" ::"r"(nmfcu::smem_u32(sF)),
                "l"(F + (size_t)x0 * RP), "r"(bytes), "r"(nmfcu::smem_u32(bar))
                : "memory");
        }
        if (!nmfcu::mbar_wait(bar, (uint32_t)(b & 1))) {
            nmfcu::record_timeout(st, nmfcu::TIMEOUT_FULL);
            return;
        }
        const int32_t *s0 = seg + (size_t)b * lines, *s1 = s0 + lines;
        // The next line's segment is read while this one is worked on.
        int m = m0 + warp;
        int64_t nt0 = 0, nt1 = 0;
        const auto segment = [&](int l) {
            nt0 = nt1 = 0;
            if (l < m1) {
                const int64_t base = ptr[l];
                nt0 = base + s0[l];
                nt1 = base + s1[l];
            }
        };
        segment(m);
        for (; m < m1; m += C::WARPS) {
            const int64_t t0 = nt0, t1 = nt1;
            double2 g[RATIO ? C::UPL : 1], a[C::UPL];
            int xo;
            double vo;
            const auto entry = [&](int64_t t) {
                xo = t + lane < t1 ? idx[t + lane] - x0 : -1;
                vo = t + lane < t1 ? val[t + lane] : 0.0;
            };
            entry(t0);
#pragma unroll
            for (int u = 0; u < C::UPL; u++) {
                const int pr = gl + C::GL * u;
                a[u] = make_double2(0.0, 0.0);
                if (RATIO)
                    g[u] = pr < C::PAIRS
                               ? reinterpret_cast<const double2 *>(G + (int64_t)m * RP)[pr]
                               : make_double2(0.0, 0.0);
            }
            segment(m + C::WARPS);
            for (int64_t t = t0; t < t1; t += 32) {
                // The group's entries side by side.
                double2 f[C::GL][C::UPL];
#pragma unroll
                for (int q = 0; q < C::GL; q++) {
                    const int x = __shfl_sync(0xffffffffu, xo, first + q);
                    const double2 *row =
                        reinterpret_cast<const double2 *>(sF + (size_t)max(x, 0) * RP);
#pragma unroll
                    for (int u = 0; u < C::UPL; u++) {
                        const int pr = gl + C::GL * u;
                        f[q][u] = pr < C::PAIRS && x >= 0 ? row[pr] : make_double2(0.0, 0.0);
                    }
                }
                double w = vo;
                if (t + 32 < t1) entry(t + 32);
                if (RATIO) {
                    double wh[C::GL];
#pragma unroll
                    for (int q = 0; q < C::GL; q++) wh[q] = 0.0;
#pragma unroll
                    for (int u = 0; u < C::UPL; u++)
#pragma unroll
                        for (int q = 0; q < C::GL; q++)
                            wh[q] = fma(g[u].y, f[q][u].y, fma(g[u].x, f[q][u].x, wh[q]));
                    // Each lane ends with the sum of its own entry: halves of
                    // the list change places with the other half of the group.
#pragma unroll
                    for (int o = C::GL / 2; o >= 1; o >>= 1) {
                        const bool hi = (gl & o) != 0;
#pragma unroll
                        for (int q = 0; q < o; q++) {
                            const double keep = hi ? wh[q + o] : wh[q];
                            const double give = hi ? wh[q] : wh[q + o];
                            wh[q] = keep + __shfl_xor_sync(0xffffffffu, give, o);
                        }
                    }
                    // 0 where W H is, and in a lane past the entries, whose W H
                    // is 0 times the line's factor row: NaN where that is
                    // infinite.
                    if (nmfcu::ratio_plain(wh[0]))
                        w = nmfcu::ratio_fast(w, wh[0]);
                    else if (wh[0] == 0.0 || (t + 32 >= t1 && xo < 0))
                        w = 0.0;
                    else
                        w = nmfcu::ratio_ieee(w, wh[0]);
                }
#pragma unroll
                for (int q = 0; q < C::GL; q++) {
                    const double wq = __shfl_sync(0xffffffffu, w, first + q);
#pragma unroll
                    for (int u = 0; u < C::UPL; u++) {
                        a[u].x = fma(wq, f[q][u].x, a[u].x);
                        a[u].y = fma(wq, f[q][u].y, a[u].y);
                    }
                }
            }
            double2 old[C::UPL];
#pragma unroll
            for (int u = 0; u < C::UPL; u++) {
                const int pr = gl + C::GL * u;
                old[u] = b > 0 && slot == 0 && pr < C::PAIRS
                             ? reinterpret_cast<const double2 *>(acc_out + (int64_t)m * RP)[pr]
                             : make_double2(0.0, 0.0);
            }
#pragma unroll
            for (int u = 0; u < C::UPL; u++)
#pragma unroll
                for (int o = C::GL; o < 32; o <<= 1) {
                    a[u].x += __shfl_xor_sync(0xffffffffu, a[u].x, o);
                    a[u].y += __shfl_xor_sync(0xffffffffu, a[u].y, o);
                }
            if (slot == 0) {
                double2 *dst = reinterpret_cast<double2 *>(acc_out + (int64_t)m * RP);
#pragma unroll
                for (int u = 0; u < C::UPL; u++) {
                    const int pr = gl + C::GL * u;
                    if (pr >= C::PAIRS) continue;
                    a[u].x += old[u].x;
                    a[u].y += old[u].y;
                    if (OUT_KM && b == blocks - 1) {
                        out[(int64_t)(2 * pr) * ldo + m] = a[u].x;
                        out[(int64_t)(2 * pr + 1) * ldo + m] = a[u].y;
                    } else {
                        dst[pr] = a[u];
                    }
                }
            }
        }
    }
}

// Stored-entry part of the objective, one warp a CSR row; per block two
// partials: part[2 b] the stored terms, part[2 b + 1] (KL) the sum of W H
// over the stored entries with v > 0.
template <int RP, bool KL>
__global__ void __launch_bounds__(kT)
    sparse_objective(const int64_t *__restrict__ ptr, const int32_t *__restrict__ idx,
                     const double *__restrict__ val, int n, const double *__restrict__ W,
                     const double *__restrict__ Ht, double *__restrict__ part,
                     const RunState *st) {
    if (nmfcu::run_stopped(st)) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int gw = (int)((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5);
    const int nw = (int)(((int64_t)gridDim.x * blockDim.x) >> 5);
    double a = 0.0, b = 0.0;
    for (int i = gw; i < n; i += nw) {
        double w[RP];
        const double2 *w2 = reinterpret_cast<const double2 *>(W + (int64_t)i * RP);
#pragma unroll
        for (int k = 0; k < RP / 2; k++) {
            const double2 x = w2[k];
            w[2 * k] = x.x;
            w[2 * k + 1] = x.y;
        }
        const int64_t t1 = ptr[i + 1];
        for (int64_t t = ptr[i] + lane; t < t1; t += 32) {
            const double2 *h2 = reinterpret_cast<const double2 *>(Ht + (int64_t)idx[t] * RP);
            double wh = 0.0;
#pragma unroll
            for (int k = 0; k < RP / 2; k++) {
                const double2 y = __ldg(h2 + k);
                wh = fma(w[2 * k], y.x, wh);
                wh = fma(w[2 * k + 1], y.y, wh);
            }
            const double v = val[t];
            if (KL) {
                if (v > 0.0) {
                    if (wh > 0.0) a += v * log(v / wh) - v + wh;
                    b += wh;
                }
            } else {
                const double d = v - wh;
                a += d * d - wh * wh;
            }
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, off);
        b += __shfl_xor_sync(0xffffffffu, b, off);
    }
    __shared__ double ra[kT / 32], rb[kT / 32];
    if (lane == 0) {
        ra[warp] = a;
        rb[warp] = b;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double sa = 0.0, sb = 0.0;
        for (int w = 0; w < kT / 32; w++) {
            sa += ra[w];
            sb += rb[w];
        }
        part[2 * blockIdx.x] = sa;
        part[2 * blockIdx.x + 1] = sb;
    }
}

// obj[0] = the objective before its scale: the stored-entry partials (in
// block order) plus the closed-form part over all entries.
template <int RP, bool KL>
__global__ void sparse_objective_combine(const double *__restrict__ part, int B, int r,
                                         const double *__restrict__ Gw, const double *__restrict__ sw,
                                         const double *__restrict__ Gh, const double *__restrict__ sh,
                                         double *__restrict__ obj, const RunState *st) {
    if (nmfcu::run_stopped(st)) return;
    __shared__ double ra[kT], rb[kT];
    double a = 0.0, b = 0.0;
    for (int i = threadIdx.x; i < B; i += kT) {
        a += part[2 * i];
        b += part[2 * i + 1];
    }
    ra[threadIdx.x] = a;
    rb[threadIdx.x] = b;
    __syncthreads();
    for (int s = kT / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) {
            ra[threadIdx.x] += ra[threadIdx.x + s];
            rb[threadIdx.x] += rb[threadIdx.x + s];
        }
        __syncthreads();
    }
    if (threadIdx.x != 0) return;
    double dense = 0.0;
    if (KL) {
        for (int k = 0; k < r; k++) dense += sw[k] * sh[k];  // sum of W H over all entries
        obj[0] = ra[0] + (dense - rb[0]);
    } else {
        for (int k = 0; k < r; k++)
            for (int l = 0; l < r; l++) dense += Gw[k * RP + l] * Gh[k * RP + l];  // ||W H||^2
        obj[0] = ra[0] + dense;
    }
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------

// Device views of one run.
struct SparseV {
    const int64_t *rptr;   // CSR
    const int32_t *ridx;
    const double *rval;
    int64_t *cptr;         // CSC copy
    int32_t *cidx;
    double *cval;
    int64_t nnz;
    bool sorted = false, strict = false;  // the CSR's rows: no decrease, no repeat
    // The blocked passes' segments and line ranges (null: the pass gathers
    // from L2): rows against blocks of H^T, columns against blocks of W.
    int32_t *rseg = nullptr, *cseg = nullptr;
    int *rbound = nullptr, *cbound = nullptr;
};

struct Work {
    double *W, *H, *Ht, *numW, *numH, *accH;   // padded factors, contractions
    double *pg, *Gw, *sw, *Gh, *sh, *Gw2, *sw2;
    double *opart, *obj, *dev;
    RunState *st;
    nmfcu::GramPlan gw, gh;
    int Bo;
};

// Carves `sizes` (bytes) out of one context slot, 256-byte aligned.
nmfcu_status carve(nmfcu_context *c, int slot, const std::vector<size_t> &sizes,
                   std::vector<void *> &out) {
    size_t total = 0;
    for (size_t b : sizes) total += align256(std::max<size_t>(b, 1));
    void *base = nullptr;
    NMFCU_TRY(nmfcu_internal::context_buffer(c, slot, total, &base));
    out.clear();
    char *p = static_cast<char *>(base);
    for (size_t b : sizes) {
        out.push_back(p);
        p += align256(std::max<size_t>(b, 1));
    }
    return NMFCU_OK;
}

// Entries of an average segment from which the blocked passes run (0: never): a
// segment costs a warp its line's pointers, factor row and sum, which a few
// entries do not pay for, and the gathering passes lose by the length of a
// factor row: up to rank 6, and at ranks 9 and 10 without the ratio, which leave
// three eighths of a group's lanes idle, the blocked ones never win.  The lines
// are where both are about equally fast at 10000 x 50000 and at 8000 x 16000
// (10000 x 50000 with the ratio, gathering / blocked, us an iteration: rank 20 at
// 16 entries 724 / 735, at 24 987 / 782; rank 10 at 32 339 / 447, at 96 828 /
// 812; rank 4 at 128 257 / 337).
constexpr int64_t blk_entries(int RP, bool ratio) {
    switch (RP) {
        case 8: return ratio ? 192 : 80;
        case 10: return ratio ? 90 : 0;
        case 12: return ratio ? 56 : 80;
        case 14: return ratio ? 54 : 72;
        case 16: return ratio ? 28 : 20;
        case 20: return ratio ? 18 : 36;
        case 24: return ratio ? 15 : 18;
        case 28: return ratio ? 19 : 24;
        case 32: return 15;
        default: return 0;
    }
}
// Whether the pass over `lines` against `len` factor rows runs blocked.
inline bool blk_pass(int64_t lines, int64_t len, int RP, bool ratio, int64_t nnz) {
    const int64_t least = blk_entries(RP, ratio);
    return least > 0 && nnz >= least * lines * (int64_t)cdiv(len, blk_rows(RP));
}

// Whether the rows of the CSR are in (strict) column order.
nmfcu_status check_order(nmfcu_context *c, int64_t n, SparseV &sv, cudaStream_t s) {
    void *fl = nullptr;
    NMFCU_TRY(nmfcu_internal::context_buffer(c, kSlotCheck, 2 * sizeof(int), &fl));
    NMFCU_CUDA_TRY(cudaMemsetAsync(fl, 0, 2 * sizeof(int), s));
    {
        nmfcu_internal::TimedScope sc(c, s, NMFCU_KCLASS_OTHER);
        lines_order<<<(unsigned)nmfcu_internal::context_sms(c) * 16, kT, 0, s>>>(
            sv.rptr, sv.ridx, (int)n, static_cast<int *>(fl));
    }
    int hf[2] = {0, 0};
    NMFCU_CUDA_TRY(cudaMemcpyAsync(hf, fl, sizeof(hf), cudaMemcpyDeviceToHost, s));
    NMFCU_CUDA_TRY(cudaStreamSynchronize(s));
    sv.sorted = !hf[0];
    sv.strict = !hf[0] && !hf[1];
    return NMFCU_OK;
}

// The CSC copy by tiles (rows in strict order).
nmfcu_status build_csc_tiles(nmfcu_context *c, int64_t n, int64_t p, SparseV &sv, cudaStream_t s) {
    const int rows = (int)cdiv(n, kCscRows), cols = (int)cdiv(p, kCscCols);
    const int sms = nmfcu_internal::context_sms(c);
    size_t temp = 0;
    NMFCU_CUDA_TRY(cub::DeviceScan::ExclusiveSum(nullptr, temp, (const int64_t *)nullptr,
                                                 (int64_t *)nullptr, (int)(p + 1), s));
    std::vector<void *> b;
    NMFCU_TRY(carve(c, kSlotSort,
                    {sizeof(int32_t) * (size_t)n * (cols + 1), sizeof(int32_t) * (size_t)rows * p,
                     sizeof(int64_t) * (size_t)(p + 1), temp},
                    b));
    int32_t *seg = static_cast<int32_t *>(b[0]), *table = static_cast<int32_t *>(b[1]);
    int64_t *total = static_cast<int64_t *>(b[2]);
    nmfcu_internal::TimedScope sc(c, s, NMFCU_KCLASS_OTHER, 5);
    line_segments<<<std::min<unsigned>(cdiv(n * (cols + 1), kT), (unsigned)sms * 32), kT, 0, s>>>(
        sv.rptr, sv.ridx, (int)n, kCscCols, cols, seg);
    const dim3 grid((unsigned)cols, (unsigned)rows);
    tile_counts<<<grid, 512, 0, s>>>(sv.rptr, sv.ridx, seg, (int)n, (int)p, table);
    column_counts<<<cdiv(p + 1, 64), 64, 0, s>>>(table, rows, (int)p, total);
    NMFCU_CUDA_TRY(cub::DeviceScan::ExclusiveSum(b[3], temp, (const int64_t *)total, sv.cptr,
                                                 (int)(p + 1), s));
    tile_scatter<<<grid, 512, 0, s>>>(sv.rptr, sv.ridx, sv.rval, seg, (int)n, (int)p, table,
                                      sv.cptr, sv.cidx, sv.cval);
    NMFCU_CUDA_TRY(cudaGetLastError());
    return NMFCU_OK;
}

// The CSC copy of the CSR: by tiles, or (few entries, fewer than four a column
// of a tile, rows out of order or with repeats) by a stable radix sort of the
// column indices.  The tiles cost their table and a pass over the order first.
// A run of no iterations at rank 2, sort / tiles, us: 20000 x 50000, 94 10^6
// entries (12 a tile's column) 5161 / 2009, 31 10^6 (4) 1570 / 1459, 24 10^6 (3)
// 1159 / 1380; 10000 x 20000, 12.6 10^6 545 / 496, 6.3 10^6 376 / 454; 5000 x
// 4000, 5.1 10^6 332 / 456.
constexpr int64_t kCscTileEntries = 1 << 23;
constexpr int64_t kCscColumnEntries = 4;
nmfcu_status build_csc(nmfcu_context *c, int64_t n, int64_t p, int RP, bool ratio, SparseV &sv,
                       cudaStream_t s) {
    const int64_t nnz = sv.nnz;
    std::vector<void *> cb;
    NMFCU_TRY(carve(c, kSlotCsc,
                    {sizeof(int64_t) * (size_t)(p + 1), sizeof(int32_t) * (size_t)nnz,
                     sizeof(double) * (size_t)nnz},
                    cb));
    sv.cptr = static_cast<int64_t *>(cb[0]);
    sv.cidx = static_cast<int32_t *>(cb[1]);
    sv.cval = static_cast<double *>(cb[2]);
    const int64_t tile_rows = (n + kCscRows - 1) / kCscRows;
    const bool tiles = nnz >= kCscTileEntries && p <= INT32_MAX - kCscCols && tile_rows <= 65535 &&
                       kCscColumnEntries * tile_rows * p <= nnz;
    // (a pass over the indices and a wait for its answer, for those who ask)
    if (nnz > 0 && (tiles || blk_pass(n, p, RP, ratio, nnz) || blk_pass(p, n, RP, ratio, nnz)))
        NMFCU_TRY(check_order(c, n, sv, s));
    if (tiles && sv.strict) return build_csc_tiles(c, n, p, sv, s);
    int bits = 1;
    while (bits < 31 && ((int64_t)1 << bits) < p) bits++;
    size_t temp = 0;
    NMFCU_CUDA_TRY(cub::DeviceRadixSort::SortPairs(nullptr, temp, (const int32_t *)nullptr,
                                                   (int32_t *)nullptr, (const int32_t *)nullptr,
                                                   (int32_t *)nullptr, (int)std::max<int64_t>(nnz, 1),
                                                   0, bits, s));
    std::vector<void *> b;
    const size_t i4 = sizeof(int32_t) * (size_t)nnz;
    NMFCU_TRY(carve(c, kSlotSort, {i4, i4, i4, i4, temp}, b));
    int32_t *keys_out = static_cast<int32_t *>(b[0]);
    int32_t *perm_in = static_cast<int32_t *>(b[1]);
    int32_t *perm = static_cast<int32_t *>(b[2]);
    int32_t *rows_of = static_cast<int32_t *>(b[3]);
    const int sms = nmfcu_internal::context_sms(c);
    const unsigned gb = std::max(1u, std::min<unsigned>(cdiv(std::max<int64_t>(nnz, 1), kT), (unsigned)sms * 16));
    nmfcu_internal::TimedScope sc(c, s, NMFCU_KCLASS_OTHER, 5);
    if (nnz > 0) {
        iota32<<<gb, kT, 0, s>>>(perm_in, nnz);
        NMFCU_CUDA_TRY(cub::DeviceRadixSort::SortPairs(b[4], temp, sv.ridx, keys_out, perm_in, perm,
                                                       (int)nnz, 0, bits, s));
        if (n > 0)
            csr_rows_of<<<std::max(1u, std::min<unsigned>(cdiv(n, kT / 32), (unsigned)sms * 16)), kT, 0, s>>>(
                sv.rptr, (int)n, rows_of);
        csc_gather<<<gb, kT, 0, s>>>(perm, rows_of, sv.rval, sv.cidx, sv.cval, nnz);
    }
    csc_colptr<<<std::max(1u, std::min<unsigned>(cdiv(nnz + 1, kT), (unsigned)sms * 16)), kT, 0, s>>>(
        keys_out, nnz, (int)p, sv.cptr);
    NMFCU_CUDA_TRY(cudaGetLastError());
    return NMFCU_OK;
}

unsigned line_grid(int64_t lines, int sms) {
    return std::max(1u, std::min<unsigned>(cdiv(lines, kT / 32), (unsigned)sms * 8));
}

template <int RP>
struct Loop {
    nmfcu_context *c;
    const nmfcu_options *o;
    int n, p, r;
    SparseV sv;
    Work w;
    cudaStream_t s;
    int sms;

    template <bool RATIO, bool OUT_KM>
    void blocked(const int64_t *ptr, const int32_t *idx, const double *val, const int32_t *seg,
                 const int *bound, int lines, const double *G, const double *F, int frows,
                 double *acc, double *out) {
        if constexpr (blk_entries(RP, RATIO) > 0) {
            auto *k = sparse_pass_blocked<RP, RATIO, OUT_KM>;
            cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, BlkCfg<RP>::SMEM);
            k<<<sms, 32 * BlkCfg<RP>::WARPS, BlkCfg<RP>::SMEM, s>>>(
                ptr, idx, val, seg, bound, lines, lines, G, F, frows, acc, out, w.st);
        }
    }
    // H^T of an H the last epilogue did not write.
    void transpose_h() {
        if (p <= 0) return;
        nmfcu_internal::TimedScope sc(c, s, NMFCU_KCLASS_OTHER);
        const unsigned blocks =
            std::max(1u, std::min<unsigned>(cdiv((int64_t)p * RP, kT), 4096u));
        nmfcu::h_transpose<double><<<blocks, kT, 0, s>>>(w.H, w.Ht, p, r, RP);
    }
    nmfcu::GramOut gram_out(int want, double *G, double *sums, bool rescaled = false) const {
        nmfcu::GramOut g;
        g.want = want;
        g.rescaled = rescaled ? 1 : 0;
        g.part = w.pg;
        g.G = G;
        g.sums = sums;
        g.ticket = w.st->gram_ticket;
        return g;
    }
    void gram_w(double *G, double *sums) {
        nmfcu_internal::TimedScope sc(c, s, NMFCU_KCLASS_OTHER);
        nmfcu::launch_gram_w<RP>(w.W, n, gram_out(nmfcu::GRAM_FULL, G, sums), w.gw, w.st, s);
    }
    void gram_h(double *G, double *sums) {
        nmfcu_internal::TimedScope sc(c, s, NMFCU_KCLASS_OTHER);
        nmfcu::launch_gram_h<RP>(w.H, p, gram_out(nmfcu::GRAM_FULL, G, sums), w.gh, w.st, s);
    }
    // The contractions as partials of one CTA's one slot.
    static nmfcu::StreamK one_slot() {
        nmfcu::StreamK sk;
        sk.U = 1;
        sk.G = sk.UPT = sk.slots = sk.nseg = sk.fold = sk.valid = 1;
        return sk;
    }
    EpiParams epi(const double *G, const double *sums, bool hside) const {
        EpiParams e;
        e.method = o->method;
        e.r = r;
        e.eps = o->eps;
        e.lambda = hside ? o->sparsity_h : o->sparsity_w;
        e.gamma = hside ? o->smoothness_h : o->smoothness_w;
        e.G = G;
        e.sums = sums;
        return e;
    }
    void h_step(bool ratio, const EpiParams &e, const nmfcu::GramOut &g) {
        {
            nmfcu_internal::TimedScope sc(c, s, NMFCU_KCLASS_HSTEP);
            if (sv.cseg) {
                if (ratio)
                    blocked<true, true>(sv.cptr, sv.cidx, sv.cval, sv.cseg, sv.cbound, p, w.Ht,
                                        w.W, n, w.accH, w.numH);
                else
                    blocked<false, true>(sv.cptr, sv.cidx, sv.cval, sv.cseg, sv.cbound, p, nullptr,
                                         w.W, n, w.accH, w.numH);
            } else {
                const unsigned grid = line_grid(p, sms);
                if (ratio)
                    sparse_pass<RP, true, true><<<grid, kT, 0, s>>>(sv.cptr, sv.cidx, sv.cval, p, p,
                                                                    w.Ht, w.W, w.numH, w.st);
                else
                    sparse_pass<RP, false, true><<<grid, kT, 0, s>>>(
                        sv.cptr, sv.cidx, sv.cval, p, p, nullptr, w.W, w.numH, w.st);
            }
        }
        nmfcu_internal::TimedScope sc(c, s, NMFCU_KCLASS_OTHER);
        nmfcu::launch_h_epilogue<RP, double, RP>(w.H, w.Ht, p, w.numH, one_slot(), std::max(p, 1),
                                                 e, g, w.gh, w.st, s);
    }
    void w_step(bool ratio, const EpiParams &e, const nmfcu::GramOut &g) {
        {
            nmfcu_internal::TimedScope sc(c, s, NMFCU_KCLASS_WSTEP);
            if (sv.rseg) {
                if (ratio)
                    blocked<true, false>(sv.rptr, sv.ridx, sv.rval, sv.rseg, sv.rbound, n, w.W,
                                         w.Ht, p, w.numW, nullptr);
                else
                    blocked<false, false>(sv.rptr, sv.ridx, sv.rval, sv.rseg, sv.rbound, n,
                                          nullptr, w.Ht, p, w.numW, nullptr);
            } else {
                const unsigned grid = line_grid(n, sms);
                if (ratio)
                    sparse_pass<RP, true, false><<<grid, kT, 0, s>>>(
                        sv.rptr, sv.ridx, sv.rval, n, 0, w.W, w.Ht, w.numW, w.st);
                else
                    sparse_pass<RP, false, false><<<grid, kT, 0, s>>>(
                        sv.rptr, sv.ridx, sv.rval, n, 0, nullptr, w.Ht, w.numW, w.st);
            }
        }
        nmfcu_internal::TimedScope sc(c, s, NMFCU_KCLASS_OTHER);
        nmfcu::launch_w_epilogue<RP>(w.W, n, w.numW, one_slot(), std::max(n, 1), e, g, w.gw, w.st,
                                     s);
    }
    void objective(long long iter) {
        const bool kl = (o->method == NMFCU_BRUNET);
        gram_w(w.Gw2, w.sw2);
        gram_h(w.Gh, w.sh);
        {
            nmfcu_internal::TimedScope sc(c, s, NMFCU_KCLASS_OBJECTIVE, 2);
            if (kl) {
                sparse_objective<RP, true><<<w.Bo, kT, 0, s>>>(sv.rptr, sv.ridx, sv.rval, n, w.W,
                                                               w.Ht, w.opart, w.st);
                sparse_objective_combine<RP, true><<<1, kT, 0, s>>>(w.opart, w.Bo, r, w.Gw2, w.sw2,
                                                                    w.Gh, w.sh, w.obj, w.st);
            } else {
                sparse_objective<RP, false><<<w.Bo, kT, 0, s>>>(sv.rptr, sv.ridx, sv.rval, n, w.W,
                                                                w.Ht, w.opart, w.st);
                sparse_objective_combine<RP, false><<<1, kT, 0, s>>>(w.opart, w.Bo, r, w.Gw2,
                                                                     w.sw2, w.Gh, w.sh, w.obj, w.st);
            }
        }
        nmfcu::StopParams sp;
        sp.stationary = 1;
        sp.iter = iter;
        sp.check_interval = o->check_interval;
        sp.check_niter = o->check_niter;
        sp.threshold = o->stationary_th;
        sp.scale = kl ? 1.0 : 0.5;
        nmfcu_internal::TimedScope sc(c, s, NMFCU_KCLASS_OTHER);
        nmfcu::objective_finalize<<<1, kT, 0, s>>>(w.obj, 1, w.dev, sp, w.st);
    }
    void iteration(long long it) {
        switch (o->method) {
            case NMFCU_BRUNET:
                // nmf_run_brunet lib.rs:1558-1575
                if (it % 10 == 1) gram_w(w.Gw, w.sw);
                h_step(true, epi(nullptr, w.sw, true), gram_out(nmfcu::GRAM_SUMS, w.Gh, w.sh));
                w_step(true, epi(nullptr, w.sh, false),
                       gram_out(it % 10 == 0 ? nmfcu::GRAM_NONE : nmfcu::GRAM_SUMS, w.Gw, w.sw));
                if (it % 10 == 0) {
                    {
                        nmfcu_internal::TimedScope sc(c, s, NMFCU_KCLASS_OTHER);
                        const int64_t m = std::max<int64_t>((int64_t)n * RP, (int64_t)r * p);
                        nmfcu::clamp_wh<RP><<<std::max(1u, std::min<unsigned>(cdiv(m, kT), 1184u)), kT, 0, s>>>(
                            w.W, w.H, n, p, r, DBL_EPSILON, w.st);
                    }
                    transpose_h();
                }
                break;
            case NMFCU_LEE:
                // nmf_run_lee lib.rs:1618-1636
                if (it == 1) gram_w(w.Gw, w.sw);
                h_step(false, epi(w.Gw, w.sw, true), gram_out(nmfcu::GRAM_FULL, w.Gh, w.sh));
                w_step(false, epi(w.Gh, w.sh, false),
                       gram_out(nmfcu::GRAM_FULL, w.Gw, w.sw, o->rescale != 0));
                if (o->rescale && n > 0) {
                    nmfcu_internal::TimedScope sc(c, s, NMFCU_KCLASS_OTHER);
                    nmfcu::col_rescale<RP><<<std::min<unsigned>(cdiv((int64_t)n * RP, kT), 1184u), kT, 0, s>>>(
                        w.W, n, r, w.sw, w.st);
                }
                break;
            default: {
                // nmf_run_hals lib.rs:667-676; nmf_run_dnmf lib.rs:862-884
                const bool dnmf = o->method == NMFCU_DNMF;
                if (it == 1 || dnmf) gram_w(w.Gw, w.sw);
                h_step(false, epi(w.Gw, w.sw, true), gram_out(nmfcu::GRAM_FULL, w.Gh, w.sh));
                w_step(false, epi(w.Gh, w.sh, false),
                       dnmf ? gram_out(nmfcu::GRAM_FULL, w.Gw2, w.sw2)
                            : gram_out(nmfcu::GRAM_FULL, w.Gw, w.sw));
                if (dnmf) {
                    {
                        nmfcu_internal::TimedScope sc(c, s, NMFCU_KCLASS_OTHER);
                        const int64_t m = std::max<int64_t>((int64_t)n * RP, (int64_t)r * p);
                        nmfcu::dnmf_rescale<RP><<<std::max(1u, std::min<unsigned>(cdiv(m, kT), 1184u)), kT, 0, s>>>(
                            w.W, w.H, n, p, r, w.Gw2, w.Gh, w.st);
                    }
                    transpose_h();
                }
                break;
            }
        }
    }
};

// Workspace of a run: padded factors and contractions (slot kSlotFac), the
// small buffers (slot kSlotSmall).
nmfcu_status make_work(nmfcu_context *c, int64_t n, int64_t p, int RP, int64_t max_iter,
                       Work &w) {
    const int sms = nmfcu_internal::context_sms(c);
    std::vector<void *> b;
    const size_t d = sizeof(double);
    NMFCU_TRY(carve(c, kSlotFac,
                    {d * n * RP, d * RP * p, d * p * RP, d * n * RP, d * RP * p, d * RP * p}, b));
    w.W = static_cast<double *>(b[0]);
    w.H = static_cast<double *>(b[1]);
    w.Ht = static_cast<double *>(b[2]);
    w.numW = static_cast<double *>(b[3]);
    w.numH = static_cast<double *>(b[4]);
    w.accH = static_cast<double *>(b[5]);
    w.gw = nmfcu::gram_plan(n, nmfcu::kTileRows, sms);
    w.gh = nmfcu::gram_plan(p, nmfcu::kTileCols, sms);
    w.Bo = (int)line_grid(n, sms);
    const int B = std::max(w.gw.blocks, w.gh.blocks) + 32;
    const size_t g = d * RP * RP, v = d * RP;
    NMFCU_TRY(carve(c, kSlotSmall,
                    {d * B * nmfcu::gram_entries(RP), g, v, g, v, g, v, d * 2 * w.Bo, d * 8,
                     sizeof(RunState), d * (size_t)(max_iter + 1)},
                    b));
    w.pg = static_cast<double *>(b[0]);
    w.Gw = static_cast<double *>(b[1]);
    w.sw = static_cast<double *>(b[2]);
    w.Gh = static_cast<double *>(b[3]);
    w.sh = static_cast<double *>(b[4]);
    w.Gw2 = static_cast<double *>(b[5]);
    w.sw2 = static_cast<double *>(b[6]);
    w.opart = static_cast<double *>(b[7]);
    w.obj = static_cast<double *>(b[8]);
    w.st = static_cast<RunState *>(b[9]);
    w.dev = static_cast<double *>(b[10]);
    return NMFCU_OK;
}

// Segments and line ranges of the blocked passes, for the passes that take
// them (lines sorted, enough entries a segment).
template <int RP>
nmfcu_status plan_blocked(nmfcu_context *c, int64_t n, int64_t p, bool ratio, SparseV &sv,
                          cudaStream_t s) {
    if (n <= 0 || p <= 0 || sv.nnz <= 0 || !sv.sorted) return NMFCU_OK;
    const int rb = (int)cdiv(p, blk_rows(RP)), cb = (int)cdiv(n, blk_rows(RP));
    const bool rows = blk_pass(n, p, RP, ratio, sv.nnz), cols = blk_pass(p, n, RP, ratio, sv.nnz);
    if (!rows && !cols) return NMFCU_OK;
    const int sms = nmfcu_internal::context_sms(c);
    std::vector<void *> b;
    NMFCU_TRY(carve(c, kSlotSeg,
                    {rows ? sizeof(int32_t) * (size_t)n * (rb + 1) : 0,
                     cols ? sizeof(int32_t) * (size_t)p * (cb + 1) : 0, sizeof(int) * (sms + 1),
                     sizeof(int) * (sms + 1)},
                    b));
    nmfcu_internal::TimedScope sc(c, s, NMFCU_KCLASS_OTHER, 4);
    const auto plan = [&](const int64_t *ptr, const int32_t *idx, int64_t lines, int blocks,
                          int32_t *seg, int *bound) {
        line_segments<<<std::min<unsigned>(cdiv(lines * (blocks + 1), kT), (unsigned)sms * 32), kT,
                        0, s>>>(ptr, idx, (int)lines, blk_rows(RP), blocks, seg);
        line_bounds<<<cdiv(sms + 1, kT), kT, 0, s>>>(ptr, (int)lines, sv.nnz, sms, bound);
    };
    if (rows) {
        sv.rseg = static_cast<int32_t *>(b[0]);
        sv.rbound = static_cast<int *>(b[2]);
        plan(sv.rptr, sv.ridx, n, rb, sv.rseg, sv.rbound);
    }
    if (cols) {
        sv.cseg = static_cast<int32_t *>(b[1]);
        sv.cbound = static_cast<int *>(b[3]);
        plan(sv.cptr, sv.cidx, p, cb, sv.cseg, sv.cbound);
    }
    NMFCU_CUDA_TRY(cudaGetLastError());
    return NMFCU_OK;
}

template <int RP>
nmfcu_status run_loop_t(nmfcu_context *c, const nmfcu_options *o, int64_t n, int64_t p, int64_t r,
                        SparseV sv, Work w, cudaStream_t s, bool stat, int64_t *n_dev,
                        int64_t *n_iter) {
    NMFCU_TRY(plan_blocked<RP>(c, n, p, o->method == NMFCU_BRUNET, sv, s));
    Loop<RP> L{c, o, (int)n, (int)p, (int)r, sv, w, s, nmfcu_internal::context_sms(c)};
    NMFCU_CUDA_TRY(cudaMemsetAsync(w.st, 0, sizeof(RunState), s));
    L.transpose_h();
    if (stat) L.objective(0);
    for (long long it = 1; it <= o->max_iter; it++) {
        L.iteration(it);
        if (stat) L.objective(it);
    }
    NMFCU_CUDA_TRY(cudaGetLastError());
    RunState hs;
    NMFCU_CUDA_TRY(cudaMemcpyAsync(&hs, w.st, sizeof(RunState), cudaMemcpyDeviceToHost, s));
    NMFCU_CUDA_TRY(cudaStreamSynchronize(s));
    nmfcu_internal::drain_timing(c);
    if (hs.timeout != 0)
        return fail(NMFCU_ERR_TIMEOUT, "a sparse pass gave up waiting for its copies (code " +
                                           std::to_string(hs.timeout) + ")");
    if (hs.error == 1)
        return fail(NMFCU_ERR_INVALID_ARG,
                    "check_interval must be > 0 (the stationary stop evaluates iter % check_interval)");
    const int64_t iters = hs.stopped ? hs.n_iter : o->max_iter;
    *n_iter = iters;
    *n_dev = stat ? iters + 1 : 0;
    return NMFCU_OK;
}

nmfcu_status run_loop(int RP, nmfcu_context *c, const nmfcu_options *o, int64_t n, int64_t p,
                      int64_t r, const SparseV &sv, const Work &w, cudaStream_t s, bool stat,
                      int64_t *n_dev, int64_t *n_iter) {
    switch (RP) {
#define NMFCU_SPARSE_CASE(R) \
    case R: return run_loop_t<R>(c, o, n, p, r, sv, w, s, stat, n_dev, n_iter);
        NMFCU_SPARSE_CASE(2)
        NMFCU_SPARSE_CASE(4)
        NMFCU_SPARSE_CASE(6)
        NMFCU_SPARSE_CASE(8)
        NMFCU_SPARSE_CASE(10)
        NMFCU_SPARSE_CASE(12)
        NMFCU_SPARSE_CASE(14)
        NMFCU_SPARSE_CASE(16)
        NMFCU_SPARSE_CASE(20)
        NMFCU_SPARSE_CASE(24)
        NMFCU_SPARSE_CASE(28)
        NMFCU_SPARSE_CASE(32)
#undef NMFCU_SPARSE_CASE
        default: return fail(NMFCU_ERR_UNSUPPORTED, "rank bucket");
    }
}

nmfcu_status validate_csr_options(const nmfcu_options *o, int64_t n, int64_t p, int64_t r,
                                  int64_t nnz) {
    NMFCU_TRY(nmfcu_internal::validate_options(o, n, p, r));
    if (o->method != NMFCU_LEE && o->method != NMFCU_BRUNET && o->method != NMFCU_HALS &&
        o->method != NMFCU_DNMF)
        return fail(NMFCU_ERR_UNSUPPORTED,
                    "a sparse (CSR) V runs lee, brunet, hals and dnmf; densify V for the others");
    if (o->precision != NMFCU_PREC_FP64)
        return fail(NMFCU_ERR_UNSUPPORTED, "a sparse (CSR) V runs in FP64 only");
    if (nnz < 0) return fail(NMFCU_ERR_INVALID_ARG, "nnz must be >= 0");
    if (nnz > INT32_MAX)
        return fail(NMFCU_ERR_UNSUPPORTED, "nnz must fit in 31 bits (2147483647 stored entries)");
    return NMFCU_OK;
}

// Upload of the padded factors (W n x r -> n x RP, H r x p -> RP x p).
nmfcu_status put_factors(const Work &w, int64_t n, int64_t p, int64_t r, int RP, const double *W,
                         const double *H, cudaMemcpyKind kind, cudaStream_t s) {
    NMFCU_CUDA_TRY(cudaMemsetAsync(w.W, 0, sizeof(double) * (size_t)n * RP, s));
    NMFCU_CUDA_TRY(cudaMemsetAsync(w.H, 0, sizeof(double) * (size_t)RP * p, s));
    if (n > 0)
        NMFCU_CUDA_TRY(cudaMemcpy2DAsync(w.W, RP * sizeof(double), W, r * sizeof(double),
                                         r * sizeof(double), n, kind, s));
    if (p > 0) NMFCU_CUDA_TRY(cudaMemcpyAsync(w.H, H, sizeof(double) * (size_t)r * p, kind, s));
    return NMFCU_OK;
}
nmfcu_status get_factors(const Work &w, int64_t n, int64_t p, int64_t r, int RP, double *W,
                         double *H, cudaMemcpyKind kind, cudaStream_t s) {
    if (n > 0)
        NMFCU_CUDA_TRY(cudaMemcpy2DAsync(W, r * sizeof(double), w.W, RP * sizeof(double),
                                         r * sizeof(double), n, kind, s));
    if (p > 0) NMFCU_CUDA_TRY(cudaMemcpyAsync(H, w.H, sizeof(double) * (size_t)r * p, kind, s));
    return NMFCU_OK;
}

// The loop on a CSR already on the device; factors in/out through W, H
// (host or device per `kind`), deviances to `dev_out` (host or device).
nmfcu_status run_csr(nmfcu_context *c, const nmfcu_options *o, int64_t n, int64_t p, int64_t r,
                     SparseV sv, const double *W0, const double *H0, double *W, double *H,
                     double *dev_out, cudaMemcpyKind in_kind, cudaMemcpyKind out_kind,
                     cudaStream_t s, int64_t *n_dev, int64_t *n_iter) {
    const int RP = bucket_for(r);
    const bool stat = o->stop == NMFCU_STOP_STATIONARY;
    NMFCU_TRY(build_csc(c, n, p, RP, o->method == NMFCU_BRUNET, sv, s));
    Work w;
    NMFCU_TRY(make_work(c, n, p, RP, o->max_iter, w));
    NMFCU_TRY(put_factors(w, n, p, r, RP, W0, H0, in_kind, s));
    int64_t nd = 0, ni = 0;
    NMFCU_TRY(run_loop(RP, c, o, n, p, r, sv, w, s, stat, &nd, &ni));
    NMFCU_TRY(get_factors(w, n, p, r, RP, W, H, out_kind, s));
    if (stat && nd > 0 && dev_out)
        NMFCU_CUDA_TRY(cudaMemcpyAsync(dev_out, w.dev, sizeof(double) * (size_t)nd,
                                       out_kind == cudaMemcpyDeviceToHost ? cudaMemcpyDeviceToHost
                                                                          : cudaMemcpyDeviceToDevice,
                                       s));
    NMFCU_CUDA_TRY(cudaStreamSynchronize(s));
    *n_dev = nd;
    *n_iter = ni;
    return NMFCU_OK;
}

}  // namespace

extern "C" {

nmfcu_status nmfcu_run_csr(const nmfcu_options *opt, int64_t n, int64_t p, int64_t r, int64_t nnz,
                           const int64_t *indptr, const int32_t *indices, const double *data,
                           const double *W0, const double *H0, double *W, double *H,
                           double *deviances, int64_t deviances_cap, int64_t *n_deviances,
                           int64_t *n_iter) {
    NMFCU_TRY(validate_csr_options(opt, n, p, r, nnz));
    if (!indptr || (nnz > 0 && (!indices || !data)) || !W0 || !H0 || !W || !H || !n_deviances ||
        !n_iter)
        return fail(NMFCU_ERR_INVALID_ARG, "NULL pointer");
    const bool stat = opt->stop == NMFCU_STOP_STATIONARY;
    if (stat && (!deviances || deviances_cap < opt->max_iter + 1))
        return fail(NMFCU_ERR_INVALID_ARG, "deviances must hold max_iter + 1 values");
    // The CSR's structure, on the host (the kernels index with it).
    if (indptr[0] != 0 || indptr[n] != nnz)
        return fail(NMFCU_ERR_INVALID_ARG, "indptr must start at 0 and end at nnz");
    for (int64_t i = 0; i < n; i++)
        if (indptr[i + 1] < indptr[i])
            return fail(NMFCU_ERR_INVALID_ARG, "indptr must be non-decreasing");
    for (int64_t t = 0; t < nnz; t++)
        if (indices[t] < 0 || indices[t] >= p)
            return fail(NMFCU_ERR_INVALID_ARG,
                        "column index " + std::to_string(indices[t]) + " outside [0, p)");
    nmfcu_context *c = nullptr;
    NMFCU_TRY(nmfcu_internal::default_context(opt->device, &c));
    std::lock_guard<std::mutex> lk(nmfcu_internal::context_mutex(c));
    nmfcu_internal::DeviceScope dg(nmfcu_internal::context_device(c));
    cudaStream_t s = nmfcu_internal::context_stream(c);
    std::vector<void *> b;
    NMFCU_TRY(carve(c, kSlotCsr,
                    {sizeof(int64_t) * (size_t)(n + 1), sizeof(int32_t) * (size_t)nnz,
                     sizeof(double) * (size_t)nnz},
                    b));
    NMFCU_CUDA_TRY(cudaMemcpyAsync(b[0], indptr, sizeof(int64_t) * (size_t)(n + 1),
                                   cudaMemcpyHostToDevice, s));
    if (nnz > 0) {
        NMFCU_CUDA_TRY(cudaMemcpyAsync(b[1], indices, sizeof(int32_t) * (size_t)nnz,
                                       cudaMemcpyHostToDevice, s));
        NMFCU_CUDA_TRY(cudaMemcpyAsync(b[2], data, sizeof(double) * (size_t)nnz,
                                       cudaMemcpyHostToDevice, s));
    }
    SparseV sv{static_cast<const int64_t *>(b[0]), static_cast<const int32_t *>(b[1]),
               static_cast<const double *>(b[2]), nullptr, nullptr, nullptr, nnz};
    return run_csr(c, opt, n, p, r, sv, W0, H0, W, H, deviances, cudaMemcpyHostToDevice,
                   cudaMemcpyDeviceToHost, s, n_deviances, n_iter);
}

nmfcu_status nmfcu_run_csr_device(nmfcu_context *ctx, const nmfcu_options *opt, int64_t n,
                                  int64_t p, int64_t r, int64_t nnz, const int64_t *d_indptr,
                                  const int32_t *d_indices, const double *d_data, double *dW,
                                  double *dH, double *d_dev, int64_t *n_deviances,
                                  int64_t *n_iter, void *stream) {
    if (!ctx) return fail(NMFCU_ERR_INVALID_ARG, "context is NULL");
    NMFCU_TRY(validate_csr_options(opt, n, p, r, nnz));
    if (!d_indptr || (nnz > 0 && (!d_indices || !d_data)) || !dW || !dH || !n_deviances ||
        !n_iter)
        return fail(NMFCU_ERR_INVALID_ARG, "NULL pointer");
    std::lock_guard<std::mutex> lk(nmfcu_internal::context_mutex(ctx));
    nmfcu_internal::DeviceScope dg(nmfcu_internal::context_device(ctx));
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    // The CSR's structure is checked on the device before any kernel
    // indexes with it.
    void *fl = nullptr;
    NMFCU_TRY(nmfcu_internal::context_buffer(ctx, kSlotCheck, 2 * sizeof(int), &fl));
    NMFCU_CUDA_TRY(cudaMemsetAsync(fl, 0, 2 * sizeof(int), s));
    {
        nmfcu_internal::TimedScope sc(ctx, s, NMFCU_KCLASS_OTHER);
        const int sms = nmfcu_internal::context_sms(ctx);
        csr_check<<<std::max(1u, std::min<unsigned>(cdiv(std::max(n + 1, nnz), kT), (unsigned)sms * 8)), kT, 0, s>>>(
            d_indptr, (int)n, d_indices, nnz, (int)p, static_cast<int *>(fl));
    }
    int hf[2] = {0, 0};
    NMFCU_CUDA_TRY(cudaMemcpyAsync(hf, fl, sizeof(hf), cudaMemcpyDeviceToHost, s));
    NMFCU_CUDA_TRY(cudaStreamSynchronize(s));
    if (hf[0])
        return fail(NMFCU_ERR_INVALID_ARG,
                    "indptr must start at 0, be non-decreasing and end at nnz");
    if (hf[1]) return fail(NMFCU_ERR_INVALID_ARG, "a column index lies outside [0, p)");
    SparseV sv{d_indptr, d_indices, d_data, nullptr, nullptr, nullptr, nnz};
    return run_csr(ctx, opt, n, p, r, sv, dW, dH, dW, dH, d_dev, cudaMemcpyDeviceToDevice,
                   cudaMemcpyDeviceToDevice, s, n_deviances, n_iter);
}

}  // extern "C"
