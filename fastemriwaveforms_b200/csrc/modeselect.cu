// Mode selection by estimated power (the threshold branch of
// ModeSelector.__call__, src/few/utils/modeselector.py:393-486).
//
// k_mode_snr2: per mode j
//   p_n = |A_nj Y_j|^2 (+ |conj(A_nj) Y_j^-|^2 for m != 0),
//   snr2_j = sum_{n < N-1} (p_n / psd_nj) (t_{n+1} - t_n),
// accumulated in knot order, as numpy's reduction over the leading axis does
// (|z|^2 as hypot(re, im)^2, numpy's abs followed by its square).  A CTA takes 32
// modes (a lane each: the loads of a knot row coalesce): 24 warps form the terms
// of 72 knots in shared memory while one more adds the 72 before them in order, so
// only the additions are serial.
// k_mode_rank: the stable descending order (NaN first, as torch's sort places it):
// a mode's place is the number of modes before it, counted by one warp.
// k_mode_select: from the estimates in that order to the kept modes, in one CTA:
// the cumulative sum (one thread: numpy's cumsum is sequential), the keep rule
// keep_0 = true, keep_i = cumsum_{i-1} < cumsum_{K-1} (1 - threshold)^2, the kept
// modes in ascending order and each one's rank.
// k_mode_keep: the rule alone on an order formed elsewhere (lists longer than
// k_mode_select's shared memory).
#include <cuda_runtime.h>

#include <cmath>

#include "few_internal.h"

namespace few {
namespace msel {

constexpr int kFormWarps = 24;                        // warps forming terms; one more adds them
constexpr int kTile = 3 * kFormWarps;                 // knots per tile
constexpr int kSnrThreads = 32 * (kFormWarps + 1);

__global__ void __launch_bounds__(kSnrThreads) k_mode_snr2(const double2 *__restrict__ teuk, int N, int K,
                                                           const double2 *__restrict__ ylms,
                                                           const int *__restrict__ minus_index,
                                                           const double *__restrict__ psd,
                                                           const double *__restrict__ t, double *__restrict__ snr2) {
    __shared__ double s_term[2][kTile][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int j = blockIdx.x * 32 + lane;
    const int jc = j < K ? j : K - 1;
    const double2 yp = ylms[jc];
    const int mi = minus_index[jc];
    const double2 ym = mi >= 0 ? ylms[mi] : make_double2(0.0, 0.0);
    const int tiles = (N - 1 + kTile - 1) / kTile;
    double acc = 0.0;
    for (int tile = 0; tile <= tiles; ++tile) {
        if (w > 0 && tile < tiles) {
            for (int q = w - 1; q < kTile; q += kFormWarps) {
                const int n = tile * kTile + q;
                if (n >= N - 1) break;
                const double2 a = teuk[(long long)n * K + jc];
                double re = __dsub_rn(__dmul_rn(a.x, yp.x), __dmul_rn(a.y, yp.y));
                double im = __dadd_rn(__dmul_rn(a.x, yp.y), __dmul_rn(a.y, yp.x));
                double h = hypot(re, im);
                double p = __dmul_rn(h, h);
                if (mi >= 0) {  // conj(A) Y^-
                    double re2 = __dsub_rn(__dmul_rn(a.x, ym.x), __dmul_rn(-a.y, ym.y));
                    double im2 = __dadd_rn(__dmul_rn(a.x, ym.y), __dmul_rn(-a.y, ym.x));
                    double h2 = hypot(re2, im2);
                    p = __dadd_rn(p, __dmul_rn(h2, h2));
                }
                if (psd) p = __ddiv_rn(p, psd[(long long)n * K + jc]);
                s_term[tile & 1][q][lane] = __dmul_rn(p, __dsub_rn(t[n + 1], t[n]));
            }
        }
        if (w == 0 && tile > 0) {
            const int count = min(kTile, N - 1 - (tile - 1) * kTile);
            const double(*v)[32] = s_term[(tile - 1) & 1];
            int q = 0;
            for (; q + 8 <= count; q += 8)
#pragma unroll
                for (int r = 0; r < 8; ++r) acc = __dadd_rn(acc, v[q + r][lane]);
            for (; q < count; ++q) acc = __dadd_rn(acc, v[q][lane]);
        }
        __syncthreads();
    }
    if (w == 0 && j < K) snr2[j] = acc;
}

// An unsigned key that orders as the estimates do: NaN above infinity, -0 as +0.
__device__ __forceinline__ unsigned long long order_key(double v) {
    if (isnan(v)) return ~0ULL;
    const unsigned long long b = (unsigned long long)__double_as_longlong(v + 0.0);
    return (b >> 63) ? ~b : b | 0x8000000000000000ULL;
}

constexpr int kSelThreads = 1024;
constexpr int kSelMax = 8192;  // modes whose order fits shared memory (kSelBytes each)
constexpr int kSelBytes = 2 * sizeof(double) + 2 * sizeof(int);

// Exclusive prefix of flag[0..K) (0 or 1) by blocks of consecutive elements per
// thread: where the thread's first element stands; *total their number.
__device__ __forceinline__ int flag_offset(const int *flag, int f0, int f1, int *s_warp, int *total) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int mine = 0;
    for (int i = f0; i < f1; ++i) mine += flag[i];
    int x = mine;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, off);
        if (lane >= off) x += y;
    }
    __syncthreads();  // s_warp of an earlier call has been read
    if (lane == 31) s_warp[w] = x;
    __syncthreads();
    if (w == 0) {
        int y = s_warp[lane];
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int z = __shfl_up_sync(0xffffffffu, y, off);
            if (lane >= off) y += z;
        }
        s_warp[lane] = y;
    }
    __syncthreads();
    *total = s_warp[31];
    return (w > 0 ? s_warp[w - 1] : 0) + x - mine;
}

// order[r], sorted[r]: the mode at place r and its estimate.  K^2 comparisons over
// the whole chip (15 million at K = 3843), kRankModes modes a warp for each estimate
// read, instead of a sort's 78 dependent steps in one CTA (42 us).
constexpr int kRankModes = 4;

__global__ void __launch_bounds__(128) k_mode_rank(const double *__restrict__ snr2, int K,
                                                   double *__restrict__ sorted, int *__restrict__ order) {
    const int i0 = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * kRankModes, lane = threadIdx.x & 31;
    if (i0 >= K) return;
    unsigned long long key[kRankModes];
    int r[kRankModes];
#pragma unroll
    for (int q = 0; q < kRankModes; ++q) {
        key[q] = order_key(snr2[min(i0 + q, K - 1)]);
        r[q] = 0;
    }
#pragma unroll 4
    for (int j = lane; j < K; j += 32) {
        const unsigned long long kj = order_key(snr2[j]);
#pragma unroll
        for (int q = 0; q < kRankModes; ++q) r[q] += kj > key[q] || (kj == key[q] && j < i0 + q);
    }
#pragma unroll
    for (int q = 0; q < kRankModes; ++q) {
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) r[q] += __shfl_xor_sync(0xffffffffu, r[q], off);
        if (lane == q && i0 + q < K) {
            sorted[r[q]] = snr2[i0 + q];
            order[r[q]] = i0 + q;
        }
    }
}

// Bound by the serial sum, 10 cycles an estimate (20 us at K = 3843).
// out_keep: the kept modes ascending; out_ylm: their +m then their -m harmonic's
// index; out_rank: position in out_keep of the i-th kept mode of the descending
// order; out_count: how many.
__global__ void __launch_bounds__(kSelThreads) k_mode_select(const double *__restrict__ sorted,
                                                             const int *__restrict__ order, int K,
                                                             double threshold, int num_m0, int num_m_1_up,
                                                             long long *__restrict__ out_keep,
                                                             long long *__restrict__ out_ylm,
                                                             long long *__restrict__ out_rank,
                                                             int *__restrict__ out_count) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double *val = reinterpret_cast<double *>(smem_raw);
    double *before_sum = val + K;  // the sum of the estimates before each in the order
    int *idx = reinterpret_cast<int *>(before_sum + K), *flag = idx + K;
    __shared__ int s_warp[32];
    __shared__ double s_lim;
    const int tid = threadIdx.x;
    for (int i = tid; i < K; i += kSelThreads) {
        val[i] = sorted[i];
        idx[i] = order[i];
    }
    __syncthreads();
    if (tid == 0) {
        // eight estimates ahead of the additions, so that these alone are the chain
        double run = 0.0, v[8], ahead[8];
#pragma unroll
        for (int r = 0; r < 8; ++r) ahead[r] = val[r < K ? r : K - 1];
        int i = 0;
        for (; i + 8 <= K; i += 8) {
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                v[r] = ahead[r];
                ahead[r] = val[i + 8 + r < K ? i + 8 + r : K - 1];
            }
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                before_sum[i + r] = run;
                run = __dadd_rn(run, v[r]);
            }
        }
        for (; i < K; ++i) {
            before_sum[i] = run;
            run = __dadd_rn(run, val[i]);
        }
        const double one_m = __dsub_rn(1.0, threshold);
        s_lim = __dmul_rn(run, __dmul_rn(one_m, one_m));
    }
    __syncthreads();
    const double lim = s_lim;
    const int per = (K + kSelThreads - 1) / kSelThreads, f0 = min(tid * per, K), f1 = min(f0 + per, K);
    // kept modes, ascending
    for (int i = tid; i < K; i += kSelThreads) flag[idx[i]] = i == 0 || before_sum[i] < lim;
    __syncthreads();
    int count;
    int at = flag_offset(flag, f0, f1, s_warp, &count);
    for (int i = f0; i < f1; ++i) {
        if (!flag[i]) continue;
        out_keep[at] = i;
        out_ylm[at] = i;
        out_ylm[count + at] = i < num_m0 ? i : i + num_m_1_up;
        flag[i] = ++at;  // the mode's rank, from 1
    }
    if (tid == 0) *out_count = count;
    __syncthreads();
    // the kept modes' ranks in the descending order
    int *kept = reinterpret_cast<int *>(val);
    for (int i = tid; i < K; i += kSelThreads) kept[i] = flag[idx[i]] > 0;
    __syncthreads();
    int again;
    at = flag_offset(kept, f0, f1, s_warp, &again);
    for (int i = f0; i < f1; ++i)
        if (kept[i]) out_rank[at++] = flag[idx[i]] - 1;
}

__global__ void k_mode_keep(const double *__restrict__ sorted_desc, int K, double threshold, int *__restrict__ keep) {
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    double total = 0.0;
    for (int i = 0; i < K; ++i) total = __dadd_rn(total, sorted_desc[i]);
    const double one_m = __dsub_rn(1.0, threshold);
    const double lim = __dmul_rn(total, __dmul_rn(one_m, one_m));
    double run = 0.0;
    for (int i = 0; i < K; ++i) {
        keep[i] = (i == 0) ? 1 : (run < lim ? 1 : 0);
        run = __dadd_rn(run, sorted_desc[i]);
    }
}

}  // namespace msel
}  // namespace few

extern "C" FEW_API int few_mode_snr2(const void *teuk, int N, int K, const void *ylms, const int *minus_index,
                                     const double *psd, const double *t, double *snr2, void *stream) {
    few::clear_error();
    if (N < 1 || K < 0) return few::fail(FEW_ERR_SIZE, "few_mode_snr2: N=%d K=%d", N, K);
    if (K == 0) return FEW_OK;
    if (!teuk || !ylms || !minus_index || !t || !snr2) return few::fail(FEW_ERR_ARG, "few_mode_snr2: null pointer");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    few::msel::k_mode_snr2<<<(K + 31) / 32, few::msel::kSnrThreads, 0, st>>>(static_cast<const double2 *>(teuk), N, K,
                                                             static_cast<const double2 *>(ylms), minus_index, psd,
                                                             t, snr2);
    FEW_LAUNCH_CHECK("k_mode_snr2");
    return FEW_OK;
}

extern "C" FEW_API int few_mode_select_max(void) { return few::msel::kSelMax; }

extern "C" FEW_API int few_mode_select(const double *snr2, int K, double threshold, int num_m0, int num_m_1_up,
                                       void *scratch, long long *keep, long long *ylm_index, long long *rank,
                                       int *count, void *stream) {
    few::clear_error();
    if (K < 1 || K > few::msel::kSelMax)
        return few::fail(FEW_ERR_SIZE, "few_mode_select: K=%d out of 1..%d", K, few::msel::kSelMax);
    if (!snr2 || !scratch || !keep || !ylm_index || !rank || !count)
        return few::fail(FEW_ERR_ARG, "few_mode_select: null pointer");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    double *sorted = static_cast<double *>(scratch);
    int *order = reinterpret_cast<int *>(sorted + K);
    FEW_CUDA_TRY(few::ensure_smem_attr((const void *)few::msel::k_mode_select, few::msel::kSelMax * few::msel::kSelBytes));
    few::msel::k_mode_rank<<<(K + 4 * few::msel::kRankModes - 1) / (4 * few::msel::kRankModes), 128, 0, st>>>(snr2, K, sorted, order);
    FEW_LAUNCH_CHECK("k_mode_rank");
    few::msel::k_mode_select<<<1, few::msel::kSelThreads, K * few::msel::kSelBytes, st>>>(
        sorted, order, K, threshold, num_m0, num_m_1_up, keep, ylm_index, rank, count);
    FEW_LAUNCH_CHECK("k_mode_select");
    return FEW_OK;
}

extern "C" FEW_API int few_mode_keep(const double *sorted_desc, int K, double threshold, int *keep, void *stream) {
    few::clear_error();
    if (K < 0) return few::fail(FEW_ERR_SIZE, "few_mode_keep: K=%d", K);
    if (K == 0) return FEW_OK;
    if (!sorted_desc || !keep) return few::fail(FEW_ERR_ARG, "few_mode_keep: null pointer");
    few::msel::k_mode_keep<<<1, 32, 0, static_cast<cudaStream_t>(stream)>>>(sorted_desc, K, threshold, keep);
    FEW_LAUNCH_CHECK("k_mode_keep");
    return FEW_OK;
}
