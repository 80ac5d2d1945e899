// stream_tcr.cu -- launch of brunet's tensor-core passes (tcr.cuh) and the
// split of a factor into the two concatenated bf16 term layouts they read.
#include <atomic>
#include <algorithm>

#include "launch.h"
#include "tcr.cuh"

namespace nmfcu {
namespace tcr {

constexpr int kAttrDevices = 64;  // devices whose launch attributes are cached

// Three bf16 terms of f: h = bf16(f), m = bf16(f - h), l = bf16(f - h - m).
__device__ __forceinline__ void split3(double f, __nv_bfloat16 &h, __nv_bfloat16 &m,
                                       __nv_bfloat16 &l) {
    h = __double2bfloat16(f);
    const double r1 = f - (double)__bfloat162float(h);
    m = __double2bfloat16(r1);
    l = __double2bfloat16(r1 - (double)__bfloat162float(m));
}

// F (f64, logically R x K with F(k, x) = F[k * fk + x * fx]) -> rows x of
// KC bf16 in the two layouts of tcr.cuh: element b * R + k (block b < 6,
// k < R) holds term tile_term[b] of F(k, x) in `tile` and term unit_term[b]
// in `unit`; everything else (x >= K, positions >= 6 R) is zero.  Either
// output may be null.
//
// A block takes kSplitRows rows x: their R x kSplitRows values come in
// contiguously, are split once, and the rows go out 16 bytes a thread.  Bound:
// the rows' store.  (One thread an element, which read F strided by the
// rank's pitch and split it anew for each of its positions, took 42 us a
// launch, W and H on average, at 20000 x 60000 rank 20; this takes 10.)
constexpr int kSplitRows = 64;
constexpr int kSplitLd = kSplitRows + 2;
__global__ void __launch_bounds__(256)
    split_factor_concat(const double *__restrict__ F, int64_t fk, int64_t fx, int R, int K, int KC,
                        int64_t xpad, __nv_bfloat16 *__restrict__ tile,
                        __nv_bfloat16 *__restrict__ unit, const RunState *st) {
    if (run_stopped(st)) return;
    __shared__ __nv_bfloat16 terms[3][32][kSplitLd];
    // For the block's 8-position chunks: where each position's term is.
    __shared__ short from_tile[192], from_unit[192];
    const int64_t x0 = (int64_t)blockIdx.x * kSplitRows;
    if (threadIdx.x < KC) {
        // Products Th Fh, Th Fm, Th Fl, Tm Fh, Tm Fm, Tl Fh.
        constexpr int tile_term[6] = {0, 0, 0, 1, 1, 2};
        constexpr int unit_term[6] = {0, 1, 2, 0, 1, 0};
        const int p = threadIdx.x, blk = p / R, k = p - blk * R;
        const bool in = p < 6 * R;
        from_tile[p] = in ? (short)((tile_term[in ? blk : 0] * 32 + k) * kSplitLd) : (short)-1;
        from_unit[p] = in ? (short)((unit_term[in ? blk : 0] * 32 + k) * kSplitLd) : (short)-1;
    }
    for (int e = threadIdx.x; e < R * kSplitRows; e += 256) {
        int k, u;
        if (fx == 1) {  // H: neighbours along x
            k = e / kSplitRows;
            u = e - k * kSplitRows;
        } else {  // W: neighbours along k
            u = e / R;
            k = e - u * R;
        }
        const int64_t x = x0 + u;
        split3(x < K ? F[k * fk + x * fx] : 0.0, terms[0][k][u], terms[1][k][u], terms[2][k][u]);
    }
    __syncthreads();
    const __nv_bfloat16 *flat = &terms[0][0][0];
    const int chunks = KC / 8;
    for (int e = threadIdx.x; e < kSplitRows * chunks; e += 256) {
        const int u = e / chunks, c = e - u * chunks;
        if (x0 + u >= xpad) continue;
        __align__(16) __nv_bfloat16 v[8];
        const int64_t at = (x0 + u) * KC + 8 * c;
        if (tile) {
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const int f = from_tile[8 * c + i];
                v[i] = f >= 0 ? flat[f + u] : __float2bfloat16(0.f);
            }
            *reinterpret_cast<uint4 *>(tile + at) = *reinterpret_cast<const uint4 *>(v);
        }
        if (unit) {
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const int f = from_unit[8 * c + i];
                v[i] = f >= 0 ? flat[f + u] : __float2bfloat16(0.f);
            }
            *reinterpret_cast<uint4 *>(unit + at) = *reinterpret_cast<const uint4 *>(v);
        }
    }
}

template <bool HPASS, int KC>
cudaError_t launch_one(const CUtensorMap &v, const void *t, const CUtensorMap &f1, int kext,
                       int rank, int RP, const StreamK &sk, double *part, RunState *st,
                       cudaStream_t s) {
    // The attribute lives in each device's context: set it once per device
    // and instantiation.  Serving worker threads launch these passes
    // concurrently, so the flags are atomics (a repeated set is harmless).
    static std::atomic<bool> configured[kAttrDevices] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= kAttrDevices || !configured[dev].load(std::memory_order_acquire)) {
        e = cudaFuncSetAttribute(tcr_pass<HPASS, KC>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 Cfg<KC>::SMEM);
        if (e != cudaSuccess) return e;
        if (dev >= 0 && dev < kAttrDevices) configured[dev].store(true, std::memory_order_release);
    }
    tcr_pass<HPASS, KC><<<sk.G, kThreads, Cfg<KC>::SMEM, s>>>(
        v, static_cast<const __nv_bfloat16 *>(t), f1, kext, rank, RP, sk, part, st);
    return cudaGetLastError();
}

}  // namespace tcr

int tcr_concat_rank(int rank) { return rank <= 21 ? 128 : 192; }

cudaError_t tcr_pass_launch(bool hpass, const CUtensorMap &v, const void *t,
                            const CUtensorMap &f1, int kext, int rank, int RP, const StreamK &sk,
                            double *part, RunState *st, cudaStream_t s) {
    if (sk.G <= 0) return cudaSuccess;
    if (rank < 1 || rank > tcr::kMaxRank) return cudaErrorInvalidValue;
    if (tcr_concat_rank(rank) == 128)
        return hpass ? tcr::launch_one<true, 128>(v, t, f1, kext, rank, RP, sk, part, st, s)
                     : tcr::launch_one<false, 128>(v, t, f1, kext, rank, RP, sk, part, st, s);
    return hpass ? tcr::launch_one<true, 192>(v, t, f1, kext, rank, RP, sk, part, st, s)
                 : tcr::launch_one<false, 192>(v, t, f1, kext, rank, RP, sk, part, st, s);
}

void tcr_split_factor(const double *F, int64_t fk, int64_t fx, int R, int K, int64_t xpad,
                      void *tile, void *unit, const RunState *st, cudaStream_t s) {
    const int KC = tcr_concat_rank(R);
    const unsigned blocks = (unsigned)((xpad + tcr::kSplitRows - 1) / tcr::kSplitRows);
    tcr::split_factor_concat<<<blocks, 256, 0, s>>>(F, fk, fx, R, K, KC, xpad,
                                                    static_cast<__nv_bfloat16 *>(tile),
                                                    static_cast<__nv_bfloat16 *>(unit), st);
}

}  // namespace nmfcu
