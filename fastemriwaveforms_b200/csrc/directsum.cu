// Direct mode sum on dense inputs: amplitudes and phases given at every output
// sample, no splines.
//
// Reference: DirectModeSum.sum (src/few/summation/directmodesum.py:30-131):
//     h_i = sum_j Y_j A_ij exp(-i phi_ij)
//         + sum_{j: m_j > 0} (-1)^{l_j} Y_{K+j} conj(A_ij) exp(+i phi_ij),
//     phi_ij = (m_j Phi_phi,i + k_j Phi_theta,i) + n_j Phi_r,i,
// the phase rounded in numpy's order (explicitly rounded operations here).
// The large phases are reduced mod pi / 2 (Cody & Waite, sincos_phase).  FP64
// throughout.
#include <cuda_runtime.h>


#include "few_common.cuh"
#include "few_internal.h"

namespace few {
namespace direct {

// A phase that sincos_phase_core does not take: above kPhaseMax, or not finite.
__device__ __noinline__ double2 phasor_any(double ph) {
    double s, c;
    sincos(ph, &s, &c);
    return make_double2(c, s);
}

// |ph| >= 2^30 or not finite, from the high word (kPhaseMax)
__device__ __forceinline__ bool phase_too_large(double ph) {
    return (__double2hiint(ph) & 0x7fffffff) >= 0x41d00000;
}

// Terms of a lane that are added to each other before they go into its sum, so that the
// long chain of a large sum has K / (kFlush G) roundings only.
constexpr int kFlush = 4;

// G lanes share S neighbouring samples: a lane takes modes j = lane, lane + G, ... of
// each, so that the mode's numbers and harmonics are read once for S samples, the S
// phasors' chains interleave, and the G lanes read 16 G consecutive bytes of a row.
//
// Bound by instruction issue and FP64 together: about 50 FP64 operations per sample and
// mode (the phase 5, its reduction and both series 29, the products and sums 10).  B200,
// 100001 samples x 200 modes (324 MB, 50 us at the copy rate): one warp per sample with
// a full sincos each 179 us; 102 us at G = 8, S = 2 with 7 blocks per SM, and 70 us at
// 30000 x 400 (100 and 90 with 6 blocks; S = 1 118 and 87, S = 3 107 and 75, S = 4 102
// and 74; loading the next mode's amplitudes one turn ahead costs a fifth).  The two
// levels of sums cost 9 us and halve the error: against long double 1.8e-16 at 200
// modes and 2.1e-16 at 400, where one lane's plain chain gives 3.5e-16 and 4.8e-16 and
// the warp per sample gave 2.1e-16 and 2.3e-16.
template <int G, int S, int MB>
__global__ void __launch_bounds__(128, MB) k_direct_sum(const double2 *__restrict__ teuk,
                                                    const double2 *__restrict__ ylms,
                                                    const double *__restrict__ Pphi, const double *__restrict__ Pth,
                                                    const double *__restrict__ Pr, const int *__restrict__ l,
                                                    const int *__restrict__ m, const int *__restrict__ k,
                                                    const int *__restrict__ n, int N, int K,
                                                    double2 *__restrict__ out) {
    const int lane = threadIdx.x & (G - 1);
    const long long i0 = ((long long)blockIdx.x * (128 / G) + threadIdx.x / G) * S;
    double pp[S], pt[S], pr[S];
    double2 w[S];
    const double2 *row[S];
#pragma unroll
    for (int q = 0; q < S; ++q) {
        // a sample past the end repeats the last one; its sum is dropped
        const long long i = i0 + q < N ? i0 + q : N - 1;
        pp[q] = Pphi[i];
        pt[q] = Pth[i];
        pr[q] = Pr[i];
        row[q] = teuk + i * K;
        w[q] = make_double2(0.0, 0.0);
    }
    for (int j0 = lane; j0 < K; j0 += kFlush * G) {
        double2 u[S];
#pragma unroll
        for (int q = 0; q < S; ++q) u[q] = make_double2(0.0, 0.0);
        for (int j = j0, end = min(K, j0 + kFlush * G); j < end; j += G) {
            double2 a[S];
#pragma unroll
            for (int q = 0; q < S; ++q) a[q] = __ldcs(row[q] + j);
            const int mi = m[j];
            const double mj = (double)mi, kj = (double)k[j], nj = (double)n[j];
            // Y b + (-1)^l Y' conj(b) = (xx b.x + xy b.y) + i (yx b.x + yy b.y), b = A exp(-i phi)
            const double2 yp = ylms[j];
            double2 ym = make_double2(0.0, 0.0);
            if (mi > 0) {
                ym = ylms[K + j];
                if (l[j] & 1) ym = make_double2(-ym.x, -ym.y);
            }
            const double xx = yp.x + ym.x, xy = ym.y - yp.y, yx = yp.y + ym.y, yy = yp.x - ym.x;
            double ph[S], sn[S], cs[S];
            bool any = false;
#pragma unroll
            for (int q = 0; q < S; ++q) {
                ph[q] = __dadd_rn(__dadd_rn(__dmul_rn(mj, pp[q]), __dmul_rn(kj, pt[q])), __dmul_rn(nj, pr[q]));
                any |= phase_too_large(ph[q]);
                sincos_phase_core(ph[q], &sn[q], &cs[q]);
            }
            if (any) {
#pragma unroll
                for (int q = 0; q < S; ++q) {
                    if (phase_too_large(ph[q])) {
                        const double2 e = phasor_any(ph[q]);
                        cs[q] = e.x;
                        sn[q] = e.y;
                    }
                }
            }
#pragma unroll
            for (int q = 0; q < S; ++q) {
                const double bx = __fma_rn(a[q].x, cs[q], a[q].y * sn[q]);
                const double by = __fma_rn(a[q].y, cs[q], -(a[q].x * sn[q]));
                u[q].x = __dadd_rn(u[q].x, __fma_rn(xx, bx, xy * by));
                u[q].y = __dadd_rn(u[q].y, __fma_rn(yx, bx, yy * by));
            }
        }
#pragma unroll
        for (int q = 0; q < S; ++q) {
            w[q].x += u[q].x;
            w[q].y += u[q].y;
        }
    }
#pragma unroll
    for (int q = 0; q < S; ++q) {
#pragma unroll
        for (int off = G / 2; off > 0; off >>= 1) {
            w[q].x += __shfl_xor_sync(0xffffffffu, w[q].x, off);
            w[q].y += __shfl_xor_sync(0xffffffffu, w[q].y, off);
        }
        if (lane == q && i0 + q < N) out[i0 + q] = w[q];
    }
}

template <int G, int S, int MB>
void launch(const double2 *teuk, const double2 *ylms, const double *phases, const int *l, const int *m, const int *k,
            const int *n, int N, int K, double2 *out, cudaStream_t st) {
    const int per_block = 128 / G * S;
    k_direct_sum<G, S, MB><<<(int)(((long long)N + per_block - 1) / per_block), 128, 0, st>>>(
        teuk, ylms, phases, phases + N, phases + 2LL * N, l, m, k, n, N, K, out);
}

}  // namespace direct
}  // namespace few

// DirectModeSum.sum's kernel: teuk [device] (N, K) complex, ylms [device] (2K)
// complex (+m, then -m), phases [device] (3, N) = (Phi_phi, Phi_theta, Phi_r),
// l, m, k, n [device] (K,) int; out [device] (N,) complex.
extern "C" FEW_API int few_direct_sum(const void *teuk, const void *ylms, const double *phases, const int *l,
                                      const int *m, const int *k, const int *n, int N, int K, void *out,
                                      void *stream) {
    few::clear_error();
    if (N < 0 || K < 0) return few::fail(FEW_ERR_SIZE, "few_direct_sum: N=%d K=%d", N, K);
    if (N == 0) return FEW_OK;
    if (!out || (K > 0 && (!teuk || !ylms || !phases || !l || !m || !k || !n)))
        return few::fail(FEW_ERR_ARG, "few_direct_sum: null pointer");
    if (K == 0) {
        FEW_CUDA_TRY(cudaMemsetAsync(out, 0, (size_t)N * 16, static_cast<cudaStream_t>(stream)));
        return FEW_OK;
    }
    // Many modes on few samples leave the chip idle at 8 lanes per sample.  With 8 and 32
    // lanes: 200 modes, 8000 samples 21 and 14 us, 16000 28 and 24, 24000 31 and 35; 400
    // modes, 16000 samples 58 and 43, 24000 61 and 61; 37 modes, 12000 samples 6.5 and
    // 7.5.  Up to 32 modes 32 lanes gain nothing (3000 samples, 12 modes: 3.2 and 2.8;
    // 100000, 31 modes: 19 and 31).
    const bool few_samples = K > 32 && N < (K > 64 ? 20000 : 10000);
    auto *f = few_samples ? few::direct::launch<32, 1, 8> : few::direct::launch<8, 2, 7>;
    f(static_cast<const double2 *>(teuk), static_cast<const double2 *>(ylms), phases, l, m, k, n, N, K,
      static_cast<double2 *>(out), static_cast<cudaStream_t>(stream));
    FEW_LAUNCH_CHECK("k_direct_sum");
    return FEW_OK;
}
