// The unfolded correlation of one kernel row: shapes and the CTA body shared
// by corr_kernel (jerk_kernels.cu) and the merged launch (jerk_fold.cu).
#pragma once

#include "jerk_async.cuh"
#include "jerk_fft.cuh"
#include "jerk_kernels.cuh"

namespace jerk {

// Occupancy target for corr_kernel: enough CTAs per SM that 128-thread CTAs
// give 16 resident warps (registers are capped to fit); CTAs of 384 threads
// or more run one per SM (two would cap them at 64 registers and spill).
template <int N>
struct CorrOcc {
    static constexpr int T = FftPlan<N>::T;
    static constexpr int value = T >= 384 ? 1 : (T >= 256 ? 2 : (T >= 128 ? 4 : 8));
};

// Shared memory of corr_kernel<N>, in float2: the FFT buffer, the twiddle
// tables and (when that still leaves CorrOcc CTAs per SM) a staging row for
// the next rstep's prepared data.
// Lengths whose twiddle tables do not fit beside the buffer (15360: 158 KB of
// tables) read twiddles and kernel rows from global memory (L1/L2) instead of
// shared memory and registers; 960 threads leave 68 registers a thread.
template <int N>
struct CorrBig {
    static constexpr bool value =
        (size_t)(fft_buf_len<N>() + FftPlan<N>::twsize()) * 8 > 200 * 1024;
};

template <int N>
struct CorrSmem {
    static constexpr int kBase =
        (fft_buf_len<N>() + (CorrBig<N>::value ? 0 : FftPlan<N>::twsize()) + 1) & ~1;
    // the staged row is the prepared chunk's first half (see corr_body)
    static constexpr bool kStage = (size_t)(kBase + N / 2) * 8 * CorrOcc<N>::value <= 220 * 1024;
    static constexpr int value = kBase + (kStage ? N / 2 : 0);
};

// Kernel row lrow of subharmonic s (fftlen N, one of the short lengths of the
// merged launch), rsteps [b0, b1) of the batch, by the CTA's first warps that
// hold its T threads.  (corr_kernel runs the long lengths, whose rows need not
// fit in registers nor their data beside the tables, with its own loop.)
template <int N>
__device__ __forceinline__ void corr_body(const SearchDev &P, const int s, const int lrow,
                                          const int b0, const int b1)
{
    constexpr int R0 = FftPlan<N>::R0;
    constexpr int T = FftPlan<N>::T;
    constexpr int TWN = FftPlan<N>::twsize();
    static_assert(CorrSmem<N>::kStage && !CorrBig<N>::value, "a short length");
    extern __shared__ __align__(16) float2 sm2[];
    __shared__ uint64_t s_bar;
    float2 *buf = sm2;
    float2 *tws = sm2 + fft_buf_len<N>();
    float2 *dsm = sm2 + CorrSmem<N>::kBase;  // staged data row
    const int tid = threadIdx.x;
    const SubDev sd = P.subs[s];
    const float2 *D0 = P.prepped + sd.data_off;

    // The prepared chunk is the FFT of data spread to even interbins, which
    // repeats with period N/2 (X[k + N/2] = X[k]); prep_kernel stores its
    // first half only, and element m of the product reads X[m mod N/2].  In
    // the first-stage butterfly of thread tid, input r is element
    // tid + r N/R0, so inputs r and r + R0/2 read the same value.
    static_assert(R0 % 2 == 0 && (N / R0) * (R0 / 2) == N / 2, "half-row reads");
    constexpr unsigned kRowBytes = N / 2 * sizeof(float2);
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_u32(&s_bar)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (tid == 0 && b0 < b1)
        bulk_row_load(dsm, D0 + (long long)b0 * N, kRowBytes, &s_bar);

    for (int i = tid; i < TWN; i += T)
        tws[i] = P.twiddles[sd.twoff + i];

    // the kernel row, in the order this thread's first-stage butterfly reads it
    float2 kreg[R0];
    const float2 *K = P.bank + sd.kern_off + (long long)lrow * N;
#pragma unroll
    for (int r = 0; r < R0; r++)
        kreg[r] = tid < T ? K[tid + r * (N / R0)] : make_float2(0.f, 0.f);
    __syncthreads();

    const int offset = sd.halfwidth * 2;  // binoffset * ACCEL_NUMBETWEEN
    const float norm = sd.pownorm;
    for (int b = b0; b < b1; b++) {
        const int numrs = P.steps[(P.first_rstep + b) * P.nsubs + s].numrs;
        float *outp = P.planes + sd.plane_off + (long long)b * sd.plane_size +
                      (long long)lrow * sd.stride;
        // the power is formed for every output and the store predicated on
        // the good-bin range (one unsigned compare): measured faster than a
        // branch around both.  Power-of-two fftlen: 1/fftlen^2 is already in
        // the chunk.
        auto out = [&](int m, float2 y) {
            const int kk = m - offset;
            const float pw = fmaf(y.x, y.x, y.y * y.y);
            const float o = IsPow2<N>::value ? pw : pw * norm;
            if ((unsigned)kk < (unsigned)numrs)
                outp[kk] = o;
        };
        // rstep b's row is (or will shortly be) in dsm; once every thread
        // has read it, thread 0 starts the copy of rstep b + 1's row
        if (!bar_wait(&s_bar, (b - b0) & 1) && P.status)
            atomicOr(P.status, kStatusCopy);
        auto in = [&](int r) -> float2 {
            return cmulconj(dsm[tid + (r % (R0 / 2)) * (N / R0)], kreg[r]);
        };
        auto mid = [&] {
            if (tid == 0 && b + 1 < b1) {
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                bulk_row_load(dsm, D0 + (long long)(b + 1) * N, kRowBytes, &s_bar);
            }
        };
        fft_block<N, +1>(buf, tws, tid, in, out, mid);
        __syncthreads();
    }
}

}  // namespace jerk
