// Jerk-search kernels for sm_100a (FP32 SIMT; the method is spectral, not a
// dense contraction, so there is no tensor-core path).
//
// Per batch of rsteps (one rstep = corr_uselen interbinned fundamental
// bins), three steps run on one stream; rows of fftlen 512 to 4096 are correlated
// by jerk_fold.cu (half-length transforms of folded rows), and large volumes
// summed by jerk_harm.cu (rows copied through shared memory):
//
//  1. prep_kernel      one CTA per (rstep, subharmonic): gathers fftlen/2
//                      spectral bins, block-median normalises them exactly as
//                      the reference does, spreads them to interbins, takes
//                      the forward FFT, and writes the rinds lookup table.
//                      (reference: src/accel_utils.c:1107-1210, done there on
//                      the host; src/accel_utils_cu.c:464-588)
//  2. corr_kernel<N>   one CTA per response-kernel row (w, z) of every
//                      subharmonic with fftlen N; the kernel row stays in
//                      registers while the CTA walks all rsteps of the batch:
//                      multiply by conj(kernel), inverse FFT in shared memory,
//                      |.|^2 / fftlen^2 of the numrs good bins straight to the
//                      ffdot volume.  (reference: src/accel_utils.c:1245-1285;
//                      src/accel_kernels.cu:930-988 + cuFFT)
//  3. harmsum_kernel   one thread per fundamental (w, z, r): the stage-0
//                      threshold, then the subharmonic adds in the reference's
//                      order with a threshold after each stage; hits go to a
//                      compact list through atomics.
//                      (reference: src/accel_utils.c:1356-1377, 1507-1555;
//                      src/accel_kernels.cu:781-862)
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>

#include "jerk_async.cuh"
#include "jerk_corr.cuh"
#include "jerk_fft.cuh"
#include "jerk_kernels.cuh"

namespace jerk {

// ---------------------------------------------------------------------------
// Exact double-precision index arithmetic (no FMA contraction), as the
// reference's host code computes it (src/accel_utils.c:54-97).

__device__ __forceinline__ double calc_required_r_d(double hf, double rfull)
{
    return __dmul_rn(rint(__dmul_rn(__dmul_rn(2.0, rfull), hf)), 0.5);
}

__device__ __forceinline__ int index_from_r_d(double r, double lor)
{
    return __double2int_rz(__dadd_rn(__dmul_rn(__dsub_rn(r, lor), 2.0), 1e-14));
}

// ---------------------------------------------------------------------------
// 1. Data preparation.

constexpr double kLn2 = 0.69314718055994530942;  // log(2.0), correctly rounded

// -locpow local power levels (src/corr_routines.c:309-366): the double
// top-hat of weight ((M/2)/NUMLOCPOWAVG, integer division) * 2/M at offsets
// DELTAAVGBINS+1 .. NUMLOCPOWAVG/2+DELTAAVGBINS either side -- the reference
// applies it by FFT correlation, restated as the direct sum -- with the first
// and last kern_half_width bins taking the nearest interior value.
constexpr int kLocAvg = 20;   // NUMLOCPOWAVG (include/presto.h:100)
constexpr int kLocDelta = 5;  // DELTAAVGBINS (include/presto.h:104)

__device__ __forceinline__ float local_power(const float *pw, int M, int i)
{
    constexpr int khw = kLocAvg / 2 + kLocDelta;
    const double w = (double)((M / 2) / kLocAvg) * 2.0 / (double)M;
    const int c = i < khw ? khw : (i >= M - khw ? M - 1 - khw : i);
    double s = 0.0;
#pragma unroll
    for (int d = kLocDelta + 1; d <= khw; d++)
        s = __dadd_rn(s, __dadd_rn((double)pw[c + d], (double)pw[c - d]));
    return __double2float_rn(__dmul_rn(w, s));
}

// Whether prep_impl<N> keeps the FFT twiddles in shared memory beside its
// buffer, data chunk and powers (every length up to 7680), or reads them
// from global memory (10240, whose tables alone take 100 KB).
template <int N>
struct PrepTwInSmem {
    static constexpr int M = N / 2;
    static constexpr bool value =
        (size_t)(fft_buf_len<N>() + FftPlan<N>::twsize() + M) * 8 + (size_t)M * 4 <= 200 * 1024;
};

// The k-th smallest (0-based) of M non-negative floats, by the whole block
// (at least kSelThreads threads): a radix select on their bit patterns, which
// order as the values do, 11 + 10 + 10 bits.  Each pass counts the digits of
// the values that still match in a shared histogram, and the thread whose
// bins hold rank k names the digit.  The result is the element a full sort
// would put at position k.  What bounds it is the chain of barriers, so few
// passes: it replaced a bitonic sort of the padded chunk (55 dependent
// barriers at 1024 values): a prep launch of 64 CTAs went from 31.2 to 14.7 us
// (CUDA events), one of 1024 CTAs from 68.4 to 34.3 us.
constexpr int kSelBins = 2048, kSelThreads = 256;
constexpr int kSelInts = kSelBins + 16;  // histogram, warp totals, result

__device__ __forceinline__ float select_rank(const float *keys, int M, unsigned k, unsigned *hist)
{
    unsigned *wtot = hist + kSelBins;       // 8 warp totals
    unsigned *found = hist + kSelBins + 8;  // digit, rank inside its bin
    const int tid = threadIdx.x, nt = blockDim.x;
    unsigned prefix = 0;  // bits chosen so far, at their place
    int shift = 20;
#pragma unroll
    for (int pass = 0; pass < 3; pass++) {
        const int bins = pass == 0 ? kSelBins : kSelBins / 2;
        const unsigned keep = pass == 0 ? 0u : ~0u << (shift + 10);
        for (int i = tid; i < bins; i += nt)
            hist[i] = 0;
        __syncthreads();
        for (int i = tid; i < M; i += nt) {
            const unsigned u = __float_as_uint(keys[i]);
            if ((u & keep) == prefix)
                atomicAdd(&hist[(u >> shift) & (bins - 1)], 1u);
        }
        __syncthreads();
        const int per = bins / kSelThreads;
        unsigned sum = 0, incl = 0;
        if (tid < kSelThreads) {
            for (int i = 0; i < per; i++)
                sum += hist[tid * per + i];
            incl = sum;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const unsigned o = __shfl_up_sync(0xffffffffu, incl, d);
                if ((tid & 31) >= d)
                    incl += o;
            }
            if ((tid & 31) == 31)
                wtot[tid >> 5] = incl;
        }
        __syncthreads();
        if (tid < kSelThreads) {
            unsigned before = incl - sum;
            for (int w = 0; w < (tid >> 5); w++)
                before += wtot[w];
            if (k >= before && k < before + sum) {
                int i = tid * per;
                while (k >= before + hist[i])
                    before += hist[i++];
                found[0] = (unsigned)i;
                found[1] = k - before;
            }
        }
        __syncthreads();
        prefix |= found[0] << shift;
        k = found[1];
        shift -= 10;
    }
    return __uint_as_float(prefix);
}

// Shared float2 of prep_impl's FFT buffer, which also holds the select's
// histogram before the transform starts.
template <int N>
__host__ __device__ constexpr int prep_buf_len()
{
    return fft_buf_len<N>() * 2 > kSelInts ? fft_buf_len<N>() : kSelInts / 2;
}

// The chunk of (rstep b, subharmonic s): gather its M bins into data (the
// powers into keys), normalise.  hist: kSelInts words of shared memory that
// nothing else uses until the next barrier after this.
__device__ __forceinline__ void prep_chunk(const SearchDev &P, const SubDev &sd, const StepDev &st,
                                           int M, float2 *data, float *keys, unsigned *hist)
{
    const int tid = threadIdx.x, nt = blockDim.x;
    // get_fourier_amplitudes: M bins from lobin, zero outside the file
    const long long lobin = st.rlo - sd.halfwidth;
    for (int i = tid; i < M; i += nt) {
        const long long bi = lobin - P.lobin + i;
        float2 v = make_float2(0.f, 0.f);
        if (bi >= 0 && bi < P.numbins)
            v = P.spec[bi];
        data[i] = v;
        keys[i] = __fadd_rn(__fmul_rn(v.x, v.x), __fmul_rn(v.y, v.y));
    }
    __syncthreads();

    if (!(P.nph > 0.0f) && P.norm_type == 1) {
        // -locpow: a float norm per bin (src/accel_utils.c:1186-1203)
        for (int i = tid; i < M; i += nt) {
            const float nrm = invsqrtf_ref(local_power(keys, M, i));
            float2 v = data[i];
            v.x = __fmul_rn(v.x, nrm);
            v.y = __fmul_rn(v.y, nrm);
            data[i] = v;
        }
    } else {
        double norm;
        if (P.nph > 0.0f) {
            norm = __ddiv_rn(1.0, __dsqrt_rn((double)P.nph));
        } else {
            // median(): the order statistic of rank (M-1)/2 (src/median.c)
            const double med = (double)select_rank(keys, M, (M - 1) / 2, hist);
            norm = __ddiv_rn(1.0, __dsqrt_rn(__ddiv_rn(med, kLn2)));
        }
        for (int i = tid; i < M; i += nt) {
            float2 v = data[i];
            v.x = __double2float_rn(__dmul_rn((double)v.x, norm));
            v.y = __double2float_rn(__dmul_rn((double)v.y, norm));
            data[i] = v;
        }
    }
    __syncthreads();
}

// rinds: fundamental r -> subharmonic r index (src/accel_utils.c:1114-1123)
__device__ __forceinline__ void prep_rinds(const SearchDev &P, const SubDev &sd, const StepDev &st,
                                           int b, int s)
{
    if (sd.numharm <= 1)
        return;
    uint16_t *rinds = P.rinds + ((long long)b * P.nsubs + s) * P.corr_uselen;
    const double rlo = (double)st.rlo;
    for (int ii = threadIdx.x; ii < P.corr_uselen; ii += blockDim.x) {
        const double rr = __dadd_rn(st.fullrlo, __dmul_rn((double)ii, 0.5));
        const double subr = calc_required_r_d(sd.harm_fract, rr);
        rinds[ii] = (uint16_t)index_from_r_d(subr, rlo);
    }
}

template <int N>
__device__ void prep_impl(const SearchDev &P, int b, int s, float *smem)
{
    constexpr int M = N / 2;  // numdata = fftlen / ACCEL_NUMBETWEEN
    static_assert(M >= 2 * (kLocAvg / 2 + kLocDelta), "chunk too short for -locpow");
    constexpr int R0 = FftPlan<N>::R0;
    const SubDev sd = P.subs[s];
    const StepDev st = P.steps[(P.first_rstep + b) * P.nsubs + s];
    constexpr int TWN = FftPlan<N>::twsize();
    float2 *buf = reinterpret_cast<float2 *>(smem);
    // buffer, twiddles, data chunk, powers; at the longest fftlen the
    // twiddles stay in global memory (read through L1) to leave room
    constexpr bool kTwS = PrepTwInSmem<N>::value;
    float2 *tws = buf + prep_buf_len<N>();
    float2 *data = tws + (kTwS ? TWN : 0);
    float *keys = reinterpret_cast<float *>(data + M);
    const float2 *tw = kTwS ? tws : P.twiddles + sd.twoff;
    const int tid = threadIdx.x, nt = blockDim.x;

    if constexpr (kTwS) {
        for (int i = tid; i < TWN; i += nt)
            tws[i] = P.twiddles[sd.twoff + i];
    }
    prep_chunk(P, sd, st, M, data, keys, reinterpret_cast<unsigned *>(buf));

    // spread_no_pad (data at even interbins) + forward FFT (sign -1).  For a
    // power-of-two fftlen the chunk is scaled by 1/fftlen here, exactly (a
    // power of two), so the correlation's |y|^2 already carries the
    // reference's 1/fftlen^2 and needs no multiply; other lengths keep it.
    // The transform of the spread chunk repeats with period N/2; only the
    // first half is stored (the correlation reads it twice).
    float2 *outp = P.prepped + sd.data_off + (long long)b * N;
    auto in = [&](int r) -> float2 {
        const int m = tid + r * (N / R0);
        return (m & 1) ? make_float2(0.f, 0.f) : data[m >> 1];
    };
    auto out = [&](int m, float2 y) {
        if constexpr (IsPow2<N>::value) {
            constexpr float inv = 1.0f / (float)N;
            y.x = __fmul_rn(y.x, inv);
            y.y = __fmul_rn(y.y, inv);
        }
        if (m < N / 2)
            outp[m] = y;
    };
    fft_block<N, -1>(buf, tw, tid, in, out);
    prep_rinds(P, sd, st, b, s);
}

// Forward transform of one window of the normalised chunk (FoldClass).
template <int L>
__device__ __forceinline__ void prep_window(float2 *buf, const float2 *tw, const float2 *data,
                                            float2 *outp)
{
    const int tid = threadIdx.x;
    auto in = [&](int r) -> float2 { return data[tid + r * (L / FftPlan<L>::R0)]; };
    auto out = [&](int m, float2 y) { outp[m] = y; };
    fft_block<L, -1>(buf, tw, tid, in, out);
    __syncthreads();  // buf is the next window's too
}

// Shared float2 of prep_folded's FFT buffer for an M-bin chunk.
__host__ __device__ inline int prep_folded_buf(int M)
{
    return fft_buf_len_rt(M) * 2 > kSelInts ? fft_buf_len_rt(M) : kSelInts / 2;
}

// A folded subharmonic (jerk_fold.cu): the same chunk, then the transform of
// each of its windows.  The spread to interbins drops out (the folded rows
// hold both output parities), so a window of L bins takes an L-point
// transform.
__device__ void prep_folded(const SearchDev &P, const SubDev &sd, int b, int s, float *smem)
{
    const StepDev st = P.steps[(P.first_rstep + b) * P.nsubs + s];
    const int M = sd.fftlen / 2;
    float2 *buf = reinterpret_cast<float2 *>(smem);
    float2 *data = buf + prep_folded_buf(M);
    float *keys = reinterpret_cast<float *>(data + M);
    prep_chunk(P, sd, st, M, data, keys, reinterpret_cast<unsigned *>(buf));
    for (int c = sd.cls0; c < sd.cls0 + sd.ncls; c++) {
        const FoldClass fc = P.classes[c];
        float2 *outp = P.prepped + fc.data_off + (long long)b * fc.len;
        const float2 *tw = P.twiddles + fc.twoff;
        switch (fc.len) {
#define JERK_WIN(LL) case LL: prep_window<LL>(buf, tw, data + fc.wstart, outp); break;
        JERK_WIN(256) JERK_WIN(384) JERK_WIN(512) JERK_WIN(640) JERK_WIN(768)
        JERK_WIN(1024) JERK_WIN(1280) JERK_WIN(1536) JERK_WIN(1792) JERK_WIN(2048)
#undef JERK_WIN
        default: break;
        }
    }
    prep_rinds(P, sd, st, b, s);
}

// LONG: the lengths whose FFT plans need more than 256 threads too.
template <bool LONG>
__device__ __forceinline__ void prep_dispatch(const SearchDev &P, int b, int s)
{
    extern __shared__ float smem[];
    if (P.subs[s].ncls > 0) {
        prep_folded(P, P.subs[s], b, s, smem);
        return;
    }
    switch (P.subs[s].fftlen) {
#define JERK_PREP_CASE(NN)                   \
    case NN:                                 \
        prep_impl<NN>(P, b, s, smem);        \
        break;
        JERK_PREP_CASE(128)
        JERK_PREP_CASE(192)
        JERK_PREP_CASE(256)
        JERK_PREP_CASE(384)
        JERK_PREP_CASE(512)
        JERK_PREP_CASE(768)
        JERK_PREP_CASE(1024)
        JERK_PREP_CASE(1280)
        JERK_PREP_CASE(2048)
        JERK_PREP_CASE(4096)
    default:
        if constexpr (LONG) {
            switch (P.subs[s].fftlen) {
                JERK_PREP_CASE(5120)
                JERK_PREP_CASE(7680)
                JERK_PREP_CASE(10240)
                JERK_PREP_CASE(15360)
#undef JERK_PREP_CASE
            default:
                break;
            }
        }
        break;
    }
}

// Threads of a prep CTA: 256 serve every length up to 4096 (and leave the
// compiler 128 registers); the longer ones take their FFT plan's count.
constexpr int kPrepLong = 4096;

template <bool LONG>
__global__ void __launch_bounds__(LONG ? 1024 : 256, LONG ? 1 : 2)
    prep_kernel(const __grid_constant__ SearchDev P)
{
    wait_before();
    let_follow();
    prep_dispatch<LONG>(P, blockIdx.x, blockIdx.y);
}

// plan i of the wave: index of the plan that owns flat CTA x
__device__ __forceinline__ int group_plan(const GroupLaunch &M, int x)
{
    int i = 0;
    while (i + 1 < M.n && x >= M.cta0[i + 1])
        i++;
    return i;
}

template <bool LONG>
__global__ void __launch_bounds__(LONG ? 1024 : 256, LONG ? 1 : 2)
    prep_group_kernel(const __grid_constant__ GroupLaunch M)
{
    wait_before();
    let_follow();
    const int i = group_plan(M, blockIdx.x);
    const int local = blockIdx.x - M.cta0[i];
    const int nsubs = M.P[i].nsubs;
    prep_dispatch<LONG>(M.P[i], local / nsubs, local % nsubs);
}

// ---------------------------------------------------------------------------
// 2. Correlation: one CTA per kernel row, all rsteps of the batch.

// A wait that must run out: the correlation's bounded wait (bar_wait) on an
// mbarrier whose phase 0 nothing completes (no copy is involved, so nothing
// is left in flight).  It gives up after its poll limit and reports as a copy
// that never completed would: the correlation's or the harmonic sum's, by
// `bits`.  Launched by plans whose wait probe is on (jerk_debug_wait_probe),
// one thread.
__global__ void wait_probe_kernel(unsigned int *status, unsigned bits)
{
    __shared__ uint64_t s_probe;
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_u32(&s_probe)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    if (!bar_wait(&s_probe, 0) && status)
        atomicOr(status, bits);
}

cudaError_t launch_wait_probe(unsigned int *status, bool sum, cudaStream_t st)
{
    wait_probe_kernel<<<1, 1, 0, st>>>(status, sum ? kStatusSumCopy : kStatusCopy);
    return cudaGetLastError();
}

// A plan's own launch: one CTA per kernel row (blockIdx.x) of the group,
// rsteps of chunk blockIdx.y of gridDim.y.
template <int N>
__global__ void __launch_bounds__(FftPlan<N>::T, CorrOcc<N>::value)
    corr_kernel(const __grid_constant__ SearchDev P, const __grid_constant__ RowGroup G)
{
    constexpr int R0 = FftPlan<N>::R0;
    constexpr int T = FftPlan<N>::T;
    constexpr int TWN = FftPlan<N>::twsize();
    constexpr bool kStage = CorrSmem<N>::kStage;
    constexpr bool kBig = CorrBig<N>::value;
    extern __shared__ __align__(16) float2 sm2[];
    __shared__ uint64_t s_bar;
    float2 *buf = sm2;
    float2 *tws = sm2 + fft_buf_len<N>();
    float2 *dsm = sm2 + CorrSmem<N>::kBase;  // staged data row (kStage)
    const int tid = threadIdx.x;
    wait_before();
    const int row = blockIdx.x;
    int gi = 0;
    while (gi + 1 < G.n && row >= G.rowstart[gi + 1])
        gi++;
    const int s = G.sub[gi];
    const int lrow = row - G.rowstart[gi];
    const SubDev sd = P.subs[s];
    const float2 *D0 = P.prepped + sd.data_off;
    // this CTA's rsteps: all of the batch, or a share of them when a small
    // group's rows alone would leave SMs idle (gridDim.y > 1)
    const int bchunk = (P.nb + (int)gridDim.y - 1) / (int)gridDim.y;
    const int b0 = min(P.nb, (int)blockIdx.y * bchunk), b1 = min(P.nb, b0 + bchunk);

    // The prepared chunk is the FFT of data spread to even interbins, which
    // repeats with period N/2 (X[k + N/2] = X[k]); prep_kernel stores its
    // first half only, and element m of the product reads X[m mod N/2].  In
    // the first-stage butterfly of thread tid, input r is element
    // tid + r N/R0, so inputs r and r + R0/2 read the same value.
    static_assert(R0 % 2 == 0 && (N / R0) * (R0 / 2) == N / 2, "half-row reads");
    constexpr unsigned kRowBytes = N / 2 * sizeof(float2);
    if constexpr (kStage) {
        if (tid == 0) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_u32(&s_bar)) : "memory");
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        __syncthreads();
        if (tid == 0 && b0 < b1)
            bulk_row_load(dsm, D0 + (long long)b0 * N, kRowBytes, &s_bar);
    }

    const float2 *tw = kBig ? P.twiddles + sd.twoff : tws;
    if constexpr (!kBig) {
        for (int i = tid; i < TWN; i += T)
            tws[i] = P.twiddles[sd.twoff + i];
    }


    // the kernel row, in the order this thread's first-stage butterfly reads it
    // (kBig: read from global memory at every rstep instead)
    float2 kreg[R0];
    const float2 *K = P.bank + sd.kern_off + (long long)lrow * N;
    if constexpr (!kBig) {
#pragma unroll
        for (int r = 0; r < R0; r++)
            kreg[r] = K[tid + r * (N / R0)];
    }
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
        if constexpr (kStage) {
            // rstep b's row is (or will shortly be) in dsm; once every thread
            // has read it, thread 0 starts the copy of rstep b + 1's row
            if (!bar_wait(&s_bar, (b - b0) & 1) && P.status)
                atomicOr(P.status, kStatusCopy);
            auto in = [&](int r) -> float2 {
                // kBig: the kernel row is read from global memory here too
                return cmulconj(dsm[tid + (r % (R0 / 2)) * (N / R0)],
                                kBig ? K[tid + r * (N / R0)] : kreg[r]);
            };
            auto mid = [&] {
                if (tid == 0 && b + 1 < b1) {
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    bulk_row_load(dsm, D0 + (long long)(b + 1) * N, kRowBytes, &s_bar);
                }
            };
            fft_block<N, +1>(buf, tw, tid, in, out, mid);
        } else {
            const float2 *D = D0 + (long long)b * N;
            auto in = [&](int r) -> float2 {
                const int m = tid + r * (N / R0);
                return cmulconj(D[tid + (r % (R0 / 2)) * (N / R0)], kBig ? K[m] : kreg[r]);
            };
            fft_block<N, +1>(buf, tw, tid, in, out);
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// 3. Harmonic summing + threshold + compaction.

constexpr int kHarmThreads = 128;

// Append one hit.  Hits are rare (a few per rstep at the usual sigma
// cutoffs), so a plain per-thread atomic costs less than a warp vote on every
// comparison; the host sorts the keys, so their order here does not matter.
__device__ __forceinline__ void record_hit(const SearchDev &P, unsigned long long key, float v)
{
    const unsigned int idx = atomicAdd(P.hit_count, 1u);
    if ((long long)idx < P.max_hits) {
        P.hit_keys[idx] = key;
        P.hit_pows[idx] = v;
    }
}

// Shared memory (dynamic): zrow[s][jj] = zinds_s[jj] * stride_s, the row
// offset inside subharmonic s's volume for fundamental z row jj; rows are
// padded to a multiple of 8 entries (zero offsets past numz0) so a thread's
// 4 or 8 rows load as int4s.
__host__ __device__ __forceinline__ int zrow_pitch(int numz0) { return (numz0 + 7) & ~7; }

size_t harmsum_smem_bytes(int nsubs, int numz0)
{
    return sizeof(int) * (size_t)nsubs * zrow_pitch(numz0);
}

// Thread = one fundamental r (kk) of one w row (ii) of one rstep (b); it
// walks all z rows ZU at a time.  Used where the TMA path's boxes (below)
// do not fit in shared memory.  Per point the float adds run in the
// reference's order: stage 1 adds 1/2, stage 2 adds 1/4 then 3/4, ...
// (src/accel_utils.c:1356-1377 applied stage by stage); after each stage the
// value is compared with that stage's cutoff.  Offsets are 32-bit (the
// batch's volumes hold fewer than 2^32 floats; checked on the host).
template <int S, int ZU>
struct HarmOcc {
    // S <= 5, 4 rows per step: 7 CTAs of 128 threads (72 registers) measured
    // 6 % faster than 6 CTAs (80 registers); 8 CTAs spill
    static constexpr int value = ZU <= 4 ? (S <= 5 ? 7 : 4) : (S <= 5 ? 4 : 2);
};

// L2 prefetch, by the copy engine, of the boxes (HarmTma) that fundamental
// rows [j0, j0 + kPrefetchRows) of this CTA will gather: one tensor prefetch
// per subharmonic, no shared memory, nothing to wait for.
constexpr int kPrefetchRows = 16;

template <int NS>
__device__ __forceinline__ void prefetch_tile(const SearchDev &P, const HarmTma &T, int j0,
                                              const int *rstart, const int *wind, int b)
{
    if (j0 >= P.numz0)
        return;
    for (int s = 0; s < NS; s++) {
        const int zs = s == 0 ? j0 : P.zinds[P.subs[s].zinds_off + j0];
        asm volatile("cp.async.bulk.prefetch.tensor.4d.L2.global.tile [%0, {%1, %2, %3, %4}];"
                     :: "l"(reinterpret_cast<uint64_t>(&T.map[s])), "r"(rstart[s]), "r"(zs),
                        "r"(wind[s]), "r"(b)
                     : "memory");
    }
}

// Rare path of harmsum_kernel: the main loop only collects, per step, which
// (stage, row) pairs crossed their cutoff (bit stage * zu + u of hm); this
// redoes those rows' sums -- the same adds in the same order, so the same
// values -- and records each crossing with the value it had at its stage.
// Offsets are rebuilt here (out of line), so the main loop keeps nothing
// extra live for it: measured 11 % faster than testing and recording inside
// the loop.
template <int S>
__device__ __noinline__ void harmsum_rare_hits(const SearchDev &P, const int *hsm, int pitch,
                                               const unsigned int *s_base, int b, int ii, int kk,
                                               int jj0, unsigned int hm, int zu)
{
    constexpr int NS = 1 << (S - 1);
    const long long rstep = P.first_rstep + b;
    for (int u = 0; u < zu; u++) {
        unsigned int bits = 0;
        for (int st = 0; st < S; st++)
            bits |= ((hm >> (st * zu + u)) & 1u) << st;
        if (!bits)
            continue;
        const int jj = jj0 + u;
        float w = P.planes[s_base[0] + kk + hsm[jj]];
        int s = 1;
        for (int st = 0; st < S; st++) {
            if (st > 0) {
                for (int h = 0; h < (1 << (st - 1)); h++, s++) {
                    unsigned int ri = P.rinds[((long long)b * NS + s) * P.corr_uselen + kk];
                    if (ri >= (unsigned int)P.steps[rstep * NS + s].numrs)
                        ri = 0;  // as the main loop does (and flags)
                    w = __fadd_rn(w, P.planes[s_base[s] + ri + hsm[s * pitch + jj]]);
                }
            }
            if (bits & (1u << st))
                record_hit(P,
                           ((((unsigned long long)rstep * S + st) * P.numw0 + ii) * P.numz0 + jj) *
                                   P.corr_uselen + kk,
                           w);
        }
    }
}

// One CTA: r block bx of fundamental w row ii of rstep b.  T (the tensor maps)
// is read only with PF.
template <int S, int ZU, bool PF>
__device__ __forceinline__ void harmsum_body(const SearchDev &P, const HarmTma *T, const int bx,
                                             const int ii, const int b)
{
    constexpr int kHarmZ = ZU;
    static_assert(ZU == 4 || ZU == 8, "whole int4s of z offsets");
    // the crossing mask hm holds one bit per (stage, row): with more than 32
    // the shifts would be undefined and the compiler may drop whole stages
    static_assert(S * ZU <= 32, "hit mask wider than 32 bits");
    constexpr int NS = 1 << (S - 1);
    extern __shared__ int hsm[];
    __shared__ unsigned int s_base[NS];
    __shared__ int s_numrs[NS];
    const int numz0 = P.numz0;
    const int pitch = zrow_pitch(numz0);
    const int tid = threadIdx.x;
    const int kk = bx * kHarmThreads + tid;
    const bool valid = kk < P.corr_uselen;
    const long long rstep = P.first_rstep + b;

    __shared__ int s_pwind[NS], s_prstart[NS];  // prefetch box corners (PF)
    if (tid < NS) {
        const SubDev sd = P.subs[tid];
        const int wind = tid == 0 ? ii : P.wind[sd.wind_off + ii];
        s_base[tid] = (unsigned int)(sd.plane_off + (long long)b * sd.plane_size +
                                     (long long)wind * sd.numz * sd.stride);
        s_numrs[tid] = P.steps[rstep * NS + tid].numrs;
        if constexpr (PF) {
            const int k0 = bx * kHarmThreads;
            s_pwind[tid] = wind;
            s_prstart[tid] = tid == 0 ? k0
                                      : (int)(P.rinds[((long long)b * NS + tid) * P.corr_uselen + k0] &
                                              ~3u);
        }
    }
    for (int i = tid; i < NS * pitch; i += kHarmThreads) {
        const int s = i / pitch, jj = i - s * pitch;
        const SubDev &sd = P.subs[s];
        int zi = 0;
        if (jj < numz0)
            zi = s == 0 ? jj : P.zinds[sd.zinds_off + jj];
        hsm[i] = zi * sd.stride;
    }
    __syncthreads();

    // per-thread offsets: volume row base + this thread's r index
    unsigned int off[NS];
    off[0] = s_base[0] + (valid ? kk : 0);
#pragma unroll
    for (int s = 1; s < NS; s++) {
        unsigned int ri = valid ? P.rinds[((long long)b * NS + s) * P.corr_uselen + kk] : 0u;
        if (ri >= (unsigned int)s_numrs[s]) {
            // cannot happen for tables built as the reference builds them;
            // record it and read a cell that exists
            atomicOr(P.status, kStatusRind);
            ri = 0;
        }
        off[s] = s_base[s] + ri;
    }
    float cut[S];
#pragma unroll
    for (int st = 0; st < S; st++)
        cut[st] = P.powcut[st];

    const float *planes = P.planes;
    // subharmonics [0, NA) belong to stages 0 .. S-2, [NA, NS) to the last
    constexpr int NA = NS > 1 ? NS / 2 : 1;
    if constexpr (PF) {
        if (tid == 0) {
            prefetch_tile<NS>(P, *T, 0, s_prstart, s_pwind, b);
            prefetch_tile<NS>(P, *T, kPrefetchRows, s_prstart, s_pwind, b);
        }
    }
    for (int jj0 = 0; jj0 < numz0; jj0 += kHarmZ) {
        const bool full = jj0 + kHarmZ <= numz0;
        if constexpr (PF) {
            // one tile ahead of the rows being gathered
            if (tid == 0 && jj0 > 0 && jj0 % kPrefetchRows == 0)
                prefetch_tile<NS>(P, *T, jj0 + kPrefetchRows, s_prstart, s_pwind, b);
        }
        float v[kHarmZ];
        unsigned int hm = 0;  // bit stage * ZU + u: row u crossed that stage's cutoff
        // phase 1: every gather of stages 0 .. S-2 for the four rows in flight
        // at once, then the adds in the reference's order
        {
            float x[NA][kHarmZ];
#pragma unroll
            for (int s = 0; s < NA; s++) {
#pragma unroll
                for (int q = 0; q < kHarmZ / 4; q++) {
                    const int4 z = *reinterpret_cast<const int4 *>(hsm + s * pitch + jj0 + 4 * q);
                    x[s][4 * q + 0] = planes[off[s] + z.x];
                    x[s][4 * q + 1] = planes[off[s] + z.y];
                    x[s][4 * q + 2] = planes[off[s] + z.z];
                    x[s][4 * q + 3] = planes[off[s] + z.w];
                }
            }
#pragma unroll
            for (int u = 0; u < kHarmZ; u++)
                v[u] = x[0][u];
            int s = 1;
#pragma unroll
            for (int stage = 0; stage < (S > 1 ? S - 1 : 1); stage++) {
                if (stage > 0) {
#pragma unroll
                    for (int h = 0; h < (1 << (stage - 1)); h++, s++) {
#pragma unroll
                        for (int u = 0; u < kHarmZ; u++)
                            v[u] = __fadd_rn(v[u], x[s][u]);
                    }
                }
#pragma unroll
                for (int u = 0; u < kHarmZ; u++)
                    hm |= v[u] > cut[stage] ? 1u << (stage * kHarmZ + u) : 0u;
            }
        }
        // phase 2: the last stage's subharmonics
        if constexpr (S > 1) {
            float x[NS - NA][kHarmZ];
#pragma unroll
            for (int s = NA; s < NS; s++) {
#pragma unroll
                for (int q = 0; q < kHarmZ / 4; q++) {
                    const int4 z = *reinterpret_cast<const int4 *>(hsm + s * pitch + jj0 + 4 * q);
                    x[s - NA][4 * q + 0] = planes[off[s] + z.x];
                    x[s - NA][4 * q + 1] = planes[off[s] + z.y];
                    x[s - NA][4 * q + 2] = planes[off[s] + z.z];
                    x[s - NA][4 * q + 3] = planes[off[s] + z.w];
                }
            }
#pragma unroll
            for (int s = NA; s < NS; s++) {
#pragma unroll
                for (int u = 0; u < kHarmZ; u++)
                    v[u] = __fadd_rn(v[u], x[s - NA][u]);
            }
            constexpr int stage = S - 1;
#pragma unroll
            for (int u = 0; u < kHarmZ; u++)
                hm |= v[u] > cut[stage] ? 1u << (stage * kHarmZ + u) : 0u;
        }
        if (!valid)
            hm = 0;
        if (!full) {
            const unsigned int rows = (1u << (numz0 - jj0)) - 1u;
            unsigned int m = 0;
#pragma unroll
            for (int st = 0; st < S; st++)
                m |= rows << (st * kHarmZ);
            hm &= m;
        }
        if (hm)
            harmsum_rare_hits<S>(P, hsm, pitch, s_base, b, ii, kk, jj0, hm, kHarmZ);
    }
}

template <int S, int ZU, bool PF>
__global__ void __launch_bounds__(kHarmThreads, HarmOcc<S, ZU>::value)
    harmsum_kernel(const __grid_constant__ SearchDev P, const __grid_constant__ HarmTma T)
{
    wait_before();
    harmsum_body<S, ZU, PF>(P, &T, blockIdx.x, blockIdx.y, blockIdx.z);
}

// The gather form over a wave of plans with S stages each (no prefetch).
template <int S>
__global__ void __launch_bounds__(kHarmThreads, HarmOcc<S, 4>::value)
    harmsum_group_kernel(const __grid_constant__ GroupLaunch M)
{
    wait_before();
    const int i = group_plan(M, blockIdx.x);
    const int local = blockIdx.x - M.cta0[i];
    const int nx = M.nx[i], nw = M.P[i].numw0;
    harmsum_body<S, 4, false>(M.P[i], nullptr, local % nx, (local / nx) % nw, local / (nx * nw));
}

// ---------------------------------------------------------------------------
// 3b. Harmonic summing fed by TMA (harm_mode 3 and 4; the default forms are the
// gathers above and the ring of row copies in jerk_harm.cu).
//
// Same thread mapping, same float adds in the same order and the same hit
// keys as harmsum_kernel, so the results are bitwise the same; the
// difference is where the operands come from.  The CTA walks the fundamental
// z rows in tiles of ZT.  For each tile, one thread issues one tensor copy per
// subharmonic (cp.async.bulk.tensor.4d): the box of that subharmonic's
// volume that the tile's 128 fundamental r x ZT fundamental z can touch --
// rows zinds_s[z0] .. + Z[s], cells from the tile's first r index (rounded
// down to 4, the 16-byte rule of the x coordinate) .. + W[s] -- into shared
// memory, completing on an mbarrier.  The threads then gather from shared
// memory, so the global-memory latency that bounds harmsum_kernel is paid by
// the copy engine, many tiles in flight per SM.

template <int S, int ZT>
struct HarmTmaOcc {
    static constexpr int value = S <= 5 ? (ZT <= 8 ? 5 : 3) : (ZT <= 8 ? 3 : 2);
};

template <int S, int ZT>
__global__ void __launch_bounds__(kHarmThreads, HarmTmaOcc<S, ZT>::value)
    harmsum_tma_kernel(const SearchDev P, const __grid_constant__ HarmTma T)
{
    constexpr int NS = 1 << (S - 1);
    constexpr int NA = NS > 1 ? NS / 2 : 1;
    constexpr int ZU = 4;  // z rows per compute step
    static_assert(ZT % ZU == 0, "tile of whole steps");
    extern __shared__ __align__(128) float tsm[];
    // tensor-copy destinations 128-byte aligned whatever the static shared
    // variables before the dynamic block (128 bytes of slack are allocated)
    float *box = tsm + ((128u - (smem_u32(tsm) & 127u)) & 127u) / 4u;
    int *zoff = reinterpret_cast<int *>(box + T.box_floats);  // [NS][pitch]
    __shared__ uint64_t s_bar;
    __shared__ int s_wind[NS], s_rstart[NS], s_numrs[NS];
    const int numz0 = P.numz0;
    const int pitch = zrow_pitch(numz0);
    const int b = blockIdx.z;
    const int ii = blockIdx.y;
    const int tid = threadIdx.x;
    const int k0 = blockIdx.x * kHarmThreads;
    const int kk = k0 + tid;
    const bool valid = kk < P.corr_uselen;
    const long long rstep = P.first_rstep + b;

    if (tid < NS) {
        const SubDev sd = P.subs[tid];
        s_wind[tid] = tid == 0 ? ii : P.wind[sd.wind_off + ii];
        s_rstart[tid] = tid == 0 ? k0
                                 : (int)(P.rinds[((long long)b * NS + tid) * P.corr_uselen + k0] & ~3u);
        s_numrs[tid] = P.steps[rstep * NS + tid].numrs;
    }
    // zoff[s][jj]: offset in the shared buffer of subharmonic s's row for
    // fundamental row jj, within the box of jj's tile
    for (int i = tid; i < NS * pitch; i += kHarmThreads) {
        const int s = i / pitch, jj = i - s * pitch;
        int o = T.boxoff[s];
        if (jj < numz0) {
            const int j0 = jj - jj % ZT;
            const int zi = s == 0 ? jj : P.zinds[P.subs[s].zinds_off + jj];
            const int z0 = s == 0 ? j0 : P.zinds[P.subs[s].zinds_off + j0];
            int dz = zi - z0;
            if (dz < 0 || dz >= T.Z[s]) {  // cannot happen for tables built as the reference builds them
                atomicOr(P.status, kStatusRind);
                dz = 0;
            }
            o += dz * T.W[s];
        }
        zoff[i] = o;
    }
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_u32(&s_bar)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (smem_u32(box) & 127u) {  // unreachable by construction; never issue a misaligned copy
        if (tid == 0)
            atomicOr(P.status, kStatusSumCopy);
        return;
    }

    // this thread's cell in every box
    int col[NS];
    col[0] = tid;
#pragma unroll
    for (int s = 1; s < NS; s++) {
        int c = 0;
        if (valid) {
            const unsigned int ri = P.rinds[((long long)b * NS + s) * P.corr_uselen + kk];
            c = (int)ri - s_rstart[s];
            if (ri >= (unsigned int)s_numrs[s] || c < 0 || c >= T.W[s]) {
                atomicOr(P.status, kStatusRind);
                c = 0;
            }
        }
        col[s] = c;
    }
    float cut[S];
#pragma unroll
    for (int st = 0; st < S; st++)
        cut[st] = P.powcut[st];

    const int ntiles = (numz0 + ZT - 1) / ZT;
    for (int t = 0; t < ntiles; t++) {
        const int z0 = t * ZT;
        if (tid == 0) {
            // the previous tile's reads (generic proxy) are ordered before
            // this tile's writes by the copy engine (async proxy)
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;"
                         :: "r"(smem_u32(&s_bar)), "r"(T.box_bytes) : "memory");
            for (int s = 0; s < NS; s++) {
                const int zs = s == 0 ? z0 : P.zinds[P.subs[s].zinds_off + z0];
                asm volatile(
                    "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
                    " [%0], [%1, {%2, %3, %4, %5}], [%6];"
                    :: "r"(smem_u32(box + T.boxoff[s])), "l"(reinterpret_cast<uint64_t>(&T.map[s])),
                       "r"(s_rstart[s]), "r"(zs), "r"(s_wind[s]), "r"(b), "r"(smem_u32(&s_bar))
                    : "memory");
            }
        }
        const bool ok = bar_wait(&s_bar, t & 1);
        if (__syncthreads_or(!ok)) {
            if (tid == 0) {
                atomicOr(P.status, kStatusSumCopy);
                bar_wait(&s_bar, t & 1);  // once more, bounded, for the copies in flight
            }
            return;
        }
        const int nrows = min(ZT, numz0 - z0);
        for (int u0 = 0; u0 < nrows; u0 += ZU) {
            const int jj0 = z0 + u0;
            const bool full = u0 + ZU <= nrows;
            float v[ZU];
            {
                float x[NA][ZU];
#pragma unroll
                for (int s = 0; s < NA; s++) {
                    const int4 z = *reinterpret_cast<const int4 *>(zoff + s * pitch + jj0);
                    x[s][0] = box[z.x + col[s]];
                    x[s][1] = box[z.y + col[s]];
                    x[s][2] = box[z.z + col[s]];
                    x[s][3] = box[z.w + col[s]];
                }
#pragma unroll
                for (int u = 0; u < ZU; u++)
                    v[u] = x[0][u];
                int s = 1;
#pragma unroll
                for (int stage = 0; stage < (S > 1 ? S - 1 : 1); stage++) {
                    if (stage > 0) {
#pragma unroll
                        for (int h = 0; h < (1 << (stage - 1)); h++, s++) {
#pragma unroll
                            for (int u = 0; u < ZU; u++)
                                v[u] = __fadd_rn(v[u], x[s][u]);
                        }
                    }
#pragma unroll
                    for (int u = 0; u < ZU; u++) {
                        if (valid && (full || u0 + u < nrows) && v[u] > cut[stage])
                            record_hit(P,
                                       ((((unsigned long long)rstep * S + stage) * P.numw0 + ii) *
                                            numz0 + (jj0 + u)) * P.corr_uselen + kk,
                                       v[u]);
                    }
                }
            }
            if constexpr (S > 1) {
                float x[NS - NA][ZU];
#pragma unroll
                for (int s = NA; s < NS; s++) {
                    const int4 z = *reinterpret_cast<const int4 *>(zoff + s * pitch + jj0);
                    x[s - NA][0] = box[z.x + col[s]];
                    x[s - NA][1] = box[z.y + col[s]];
                    x[s - NA][2] = box[z.z + col[s]];
                    x[s - NA][3] = box[z.w + col[s]];
                }
#pragma unroll
                for (int s = NA; s < NS; s++) {
#pragma unroll
                    for (int u = 0; u < ZU; u++)
                        v[u] = __fadd_rn(v[u], x[s - NA][u]);
                }
                constexpr int stage = S - 1;
#pragma unroll
                for (int u = 0; u < ZU; u++) {
                    if (valid && (full || u0 + u < nrows) && v[u] > cut[stage])
                        record_hit(P,
                                   ((((unsigned long long)rstep * S + stage) * P.numw0 + ii) *
                                        numz0 + (jj0 + u)) * P.corr_uselen + kk,
                                   v[u]);
                }
            }
        }
        __syncthreads();  // every read of this tile's boxes is done
    }
}

// ---------------------------------------------------------------------------
// Launchers (host side of this translation unit).

template <int N>
static size_t prep_bytes_n()
{
    constexpr int M = N / 2;
    constexpr int TW = PrepTwInSmem<N>::value ? FftPlan<N>::twsize() : 0;
    return sizeof(float2) * (size_t)(prep_buf_len<N>() + TW + M) + sizeof(float) * (size_t)M;
}

// Shared memory of a prep CTA for one subharmonic's length.
size_t prep_smem_bytes(int fftlen, bool folded)
{
    if (folded) {
        const int M = fftlen / 2;
        return sizeof(float2) * (size_t)(prep_folded_buf(M) + M) + sizeof(float) * (size_t)M;
    }
    switch (fftlen) {
#define JERK_PB(NN) case NN: return prep_bytes_n<NN>();
    JERK_PB(128) JERK_PB(192) JERK_PB(256) JERK_PB(384) JERK_PB(512) JERK_PB(768)
    JERK_PB(1024) JERK_PB(1280) JERK_PB(2048) JERK_PB(4096) JERK_PB(5120) JERK_PB(7680) JERK_PB(10240) JERK_PB(15360)
#undef JERK_PB
    default: return 0;
    }
}

// twiddle tables of every supported fftlen's plan (host)
int fft_twiddle_size(int N)
{
    switch (N) {
#define JERK_TS(NN) case NN: return FftPlan<NN>::twsize();
    JERK_TS(128) JERK_TS(192) JERK_TS(256) JERK_TS(384) JERK_TS(512) JERK_TS(768)
    JERK_TS(640) JERK_TS(1536) JERK_TS(1792)
    JERK_TS(1024) JERK_TS(1280) JERK_TS(2048) JERK_TS(4096) JERK_TS(5120) JERK_TS(7680) JERK_TS(10240) JERK_TS(15360)
#undef JERK_TS
    default: return -1;
    }
}

void fft_twiddle_table(int N, float2 *out)
{
    switch (N) {
#define JERK_TT(NN) case NN: fft_stage_twiddles<NN>(out); break;
    JERK_TT(128) JERK_TT(192) JERK_TT(256) JERK_TT(384) JERK_TT(512) JERK_TT(768)
    JERK_TT(640) JERK_TT(1536) JERK_TT(1792)
    JERK_TT(1024) JERK_TT(1280) JERK_TT(2048) JERK_TT(4096) JERK_TT(5120) JERK_TT(7680) JERK_TT(10240) JERK_TT(15360)
#undef JERK_TT
    default: break;
    }
}

static int prep_threads(int maxfft)
{
    int t = 256;
#define JERK_PT(NN)                                  \
    if (NN <= maxfft && FftPlan<NN>::T > t)          \
        t = FftPlan<NN>::T;
    JERK_PT(4096) JERK_PT(5120) JERK_PT(7680) JERK_PT(10240) JERK_PT(15360)
#undef JERK_PT
    return (t + 31) / 32 * 32;
}

// Function attributes are set when a plan is made (and by the plan-free entry
// point), not at every launch.
cudaError_t prep_attrs(int maxfft)
{
    cudaError_t e = cudaSuccess;
    if (maxfft > kPrepLong) {
        e = smem_attrs(prep_kernel<true>, false);
        return e == cudaSuccess ? smem_attrs(prep_group_kernel<true>, false) : e;
    }
    e = smem_attrs(prep_kernel<false>, false);
    return e == cudaSuccess ? smem_attrs(prep_group_kernel<false>, false) : e;
}

// maxfft, smem: the longest fftlen of the launch and the largest
// prep_smem_bytes over its subharmonics
cudaError_t launch_prep(const SearchDev &P, int maxfft, size_t smem, cudaStream_t st)
{
    const dim3 grid(P.nb, P.nsubs);
    if (maxfft > kPrepLong)
        return launch_follow(prep_kernel<true>, grid, prep_threads(maxfft), smem, st, P);
    return launch_follow(prep_kernel<false>, grid, 256, smem, st, P);
}

template <int N>
static cudaError_t launch_corr_n(const SearchDev &P, const RowGroup &G, int rows, cudaStream_t st)
{
    const size_t smem = sizeof(float2) * CorrSmem<N>::value;
    // a group with fewer rows than two waves of CTAs also splits its rsteps
    const int wave = sm_count() * CorrOcc<N>::value;
    const int split = rows >= 2 * wave ? 1 : std::max(1, std::min(P.nb, (2 * wave + rows - 1) / rows));
    return launch_follow(corr_kernel<N>, dim3(rows, split), FftPlan<N>::T, smem, st, P, G);
}

cudaError_t corr_attrs(int fftlen)
{
    switch (fftlen) {
#define JERK_CA(NN) case NN: return smem_attrs(corr_kernel<NN>, true);
    JERK_CA(128) JERK_CA(192) JERK_CA(256) JERK_CA(384) JERK_CA(512) JERK_CA(768) JERK_CA(1024)
    JERK_CA(1280) JERK_CA(2048) JERK_CA(4096) JERK_CA(5120) JERK_CA(7680) JERK_CA(10240) JERK_CA(15360)
#undef JERK_CA
    default: return cudaErrorInvalidValue;
    }
}

bool fftlen_supported(int n)
{
    switch (n) {
    case 128: case 192: case 256: case 384: case 512: case 768: case 1024: case 1280:
    case 2048: case 4096: case 5120: case 7680: case 10240: case 15360:
        return true;
    default:
        return false;
    }
}

cudaError_t launch_corr(const SearchDev &P, int fftlen, const RowGroup &G, int rows,
                        cudaStream_t st)
{
    switch (fftlen) {
    case 128: return launch_corr_n<128>(P, G, rows, st);
    case 192: return launch_corr_n<192>(P, G, rows, st);
    case 256: return launch_corr_n<256>(P, G, rows, st);
    case 384: return launch_corr_n<384>(P, G, rows, st);
    case 512: return launch_corr_n<512>(P, G, rows, st);
    case 768: return launch_corr_n<768>(P, G, rows, st);
    case 1024: return launch_corr_n<1024>(P, G, rows, st);
    case 1280: return launch_corr_n<1280>(P, G, rows, st);
    case 2048: return launch_corr_n<2048>(P, G, rows, st);
    case 4096: return launch_corr_n<4096>(P, G, rows, st);
    case 5120: return launch_corr_n<5120>(P, G, rows, st);
    case 7680: return launch_corr_n<7680>(P, G, rows, st);
    case 10240: return launch_corr_n<10240>(P, G, rows, st);
    case 15360: return launch_corr_n<15360>(P, G, rows, st);
    default: return cudaErrorInvalidValue;
    }
}

template <int S, bool PF>
static cudaError_t launch_harmsum_s(const SearchDev &P, const HarmTma &T, cudaStream_t st)
{
    const size_t smem = harmsum_smem_bytes(P.nsubs, P.numz0);
    const dim3 grid((P.corr_uselen + kHarmThreads - 1) / kHarmThreads, P.numw0, P.nb);
    return launch_follow(harmsum_kernel<S, 4, PF>, grid, kHarmThreads, smem, st, P, T);
}

template <bool PF>
static cudaError_t launch_harmsum_p(const SearchDev &P, const HarmTma &T, cudaStream_t st)
{
    switch (P.nstages) {
    case 1: return launch_harmsum_s<1, PF>(P, T, st);
    case 2: return launch_harmsum_s<2, PF>(P, T, st);
    case 3: return launch_harmsum_s<3, PF>(P, T, st);
    case 4: return launch_harmsum_s<4, PF>(P, T, st);
    case 5: return launch_harmsum_s<5, PF>(P, T, st);
    case 6: return launch_harmsum_s<6, PF>(P, T, st);
    default: return cudaErrorInvalidValue;
    }
}

// The gather kernel; with prefetch, T holds tensor maps whose boxes were
// sized for tiles of kPrefetchRows rows.
cudaError_t launch_harmsum(const SearchDev &P, const HarmTma &T, bool prefetch, cudaStream_t st)
{
    return prefetch ? launch_harmsum_p<true>(P, T, st) : launch_harmsum_p<false>(P, T, st);
}

// ---------------------------------------------------------------------------
// Waves: one launch per kernel kind over the current batches of several
// plans.  The caller fills M.n and M.P; the launchers fill the CTA ranges.

cudaError_t launch_prep_group(GroupLaunch M, int maxfft, size_t smem, cudaStream_t st)
{
    if (M.n < 1 || M.n > kMaxGroupPlans)
        return cudaErrorInvalidValue;
    int x = 0;
    for (int i = 0; i < M.n; i++) {
        M.cta0[i] = x;
        x += M.P[i].nb * M.P[i].nsubs;
    }
    M.cta0[M.n] = x;
    if (maxfft > kPrepLong)
        return launch_follow(prep_group_kernel<true>, (unsigned)x, prep_threads(maxfft), smem, st,
                             M);
    return launch_follow(prep_group_kernel<false>, (unsigned)x, 256, smem, st, M);
}

int harmsum_wave_ctas(int nstages)
{
    return sm_count() * (nstages <= 5 ? HarmOcc<5, 4>::value : HarmOcc<6, 4>::value);
}

template <int S>
static cudaError_t launch_harmsum_group_s(GroupLaunch &M, cudaStream_t st)
{
    size_t smem = 0;
    long long x = 0;
    for (int i = 0; i < M.n; i++) {
        const SearchDev &P = M.P[i];
        smem = std::max(smem, harmsum_smem_bytes(P.nsubs, P.numz0));
        M.cta0[i] = (int)x;
        M.nx[i] = (P.corr_uselen + kHarmThreads - 1) / kHarmThreads;
        x += (long long)M.nx[i] * P.numw0 * P.nb;
    }
    if (x >= (1ll << 31))
        return cudaErrorInvalidValue;
    M.cta0[M.n] = (int)x;
    return launch_follow(harmsum_group_kernel<S>, (unsigned)x, kHarmThreads, smem, st, M);
}

// Every plan of M must have nstages stages.
cudaError_t launch_harmsum_group(GroupLaunch M, int nstages, cudaStream_t st)
{
    if (M.n < 1 || M.n > kMaxGroupPlans)
        return cudaErrorInvalidValue;
    switch (nstages) {
    case 1: return launch_harmsum_group_s<1>(M, st);
    case 2: return launch_harmsum_group_s<2>(M, st);
    case 3: return launch_harmsum_group_s<3>(M, st);
    case 4: return launch_harmsum_group_s<4>(M, st);
    case 5: return launch_harmsum_group_s<5>(M, st);
    case 6: return launch_harmsum_group_s<6>(M, st);
    default: return cudaErrorInvalidValue;
    }
}

size_t harmsum_tma_smem_bytes(const HarmTma &T, int nsubs, int numz0)
{
    return 128 + sizeof(float) * (size_t)T.box_floats + harmsum_smem_bytes(nsubs, numz0);
}

template <int S, int ZT>
static cudaError_t launch_harmsum_tma_s(const SearchDev &P, const HarmTma &T, cudaStream_t st)
{
    const size_t smem = harmsum_tma_smem_bytes(T, P.nsubs, P.numz0);
    const dim3 grid((P.corr_uselen + kHarmThreads - 1) / kHarmThreads, P.numw0, P.nb);
    harmsum_tma_kernel<S, ZT><<<grid, kHarmThreads, smem, st>>>(P, T);
    return cudaGetLastError();
}

template <int ZT>
static cudaError_t launch_harmsum_tma_z(const SearchDev &P, const HarmTma &T, cudaStream_t st)
{
    switch (P.nstages) {
    case 1: return launch_harmsum_tma_s<1, ZT>(P, T, st);
    case 2: return launch_harmsum_tma_s<2, ZT>(P, T, st);
    case 3: return launch_harmsum_tma_s<3, ZT>(P, T, st);
    case 4: return launch_harmsum_tma_s<4, ZT>(P, T, st);
    case 5: return launch_harmsum_tma_s<5, ZT>(P, T, st);
    case 6: return launch_harmsum_tma_s<6, ZT>(P, T, st);
    default: return cudaErrorInvalidValue;
    }
}

template <int S>
static cudaError_t harmsum_attrs_s(int harm_mode)
{
    // (the gather forms keep the default carveout: their gathers live in L1)
    cudaError_t e = harm_mode >= 4   ? smem_attrs(harmsum_tma_kernel<S, 16>, true)
                    : harm_mode == 3 ? smem_attrs(harmsum_tma_kernel<S, 8>, true)
                    : harm_mode == 2 ? smem_attrs(harmsum_kernel<S, 4, true>, false)
                                     : smem_attrs(harmsum_kernel<S, 4, false>, false);
    return e == cudaSuccess ? smem_attrs(harmsum_group_kernel<S>, false) : e;
}

cudaError_t harmsum_attrs(int nstages, int harm_mode)
{
    switch (nstages) {
    case 1: return harmsum_attrs_s<1>(harm_mode);
    case 2: return harmsum_attrs_s<2>(harm_mode);
    case 3: return harmsum_attrs_s<3>(harm_mode);
    case 4: return harmsum_attrs_s<4>(harm_mode);
    case 5: return harmsum_attrs_s<5>(harm_mode);
    case 6: return harmsum_attrs_s<6>(harm_mode);
    default: return cudaErrorInvalidValue;
    }
}

// zt: fundamental z rows per tile (8 or 16), as the boxes in T were sized
cudaError_t launch_harmsum_tma(const SearchDev &P, const HarmTma &T, int zt, cudaStream_t st)
{
    return zt == 8 ? launch_harmsum_tma_z<8>(P, T, st) : launch_harmsum_tma_z<16>(P, T, st);
}

}  // namespace jerk

// ---------------------------------------------------------------------------
// Allocation-free entry point.
//
// Some callers cannot allocate device memory at the moment they need a search
// step: a process whose device memory is handed out up front by a pool it
// does not own, a real-time pipeline that forbids allocation after start-up,
// or code running where cudaMalloc would stall or fail.  For them
// jerk_volume_static computes one subharmonic's ffdot volume for one rstep
// (the prep and correlation kernels above) with all of its working memory --
// the subharmonic and rstep descriptors, the FFT twiddles, the prepared
// spectrum chunk and the rinds table -- in one fixed device array,
// g_static_scratch, compiled into this library.  The caller passes only its
// inputs (spectrum, kernel rows) and its output (the volume).
//
// The array is JERK_STATIC_SCRATCH_BYTES (192 KiB) on every GPU that loads
// the library, held until the process exits; it bounds fftlen to 7680 and
// corr_uselen to 16384.  Every call shares it and it keeps the last call's
// contents (each call rewrites all of it that it reads, so nothing needs
// clearing); calls that overlap on the GPU -- two streams, or two host
// threads -- race on it and must be serialised by the caller.  Host code
// cannot use the array's name as a device address, so the first call on each
// device looks the address up with cudaGetSymbolAddress (with that device
// current); make that first call before any stream capture.  After that a
// call only launches kernels on its stream: the descriptors travel as kernel
// parameters and the FFT twiddles are computed on the device, so nothing is
// copied from host memory.

#define JERK_STATIC_SCRATCH_BYTES (192 * 1024)
static __device__ __align__(256) unsigned char g_static_scratch[JERK_STATIC_SCRATCH_BYTES];

#include <cstdio>
#include <mutex>

#include "jerk.h"

namespace jerk {
namespace {

constexpr int kStaticMaxFft = 7680;
constexpr int kStaticMaxUselen = 16384;
// scratch layout (byte offsets)
constexpr size_t kOffSub = 0;
constexpr size_t kOffStep = 256;
constexpr size_t kOffTw = 512;
constexpr size_t kOffData = kOffTw + 81920;                    // twiddles <= 10240 float2
constexpr size_t kOffRinds = kOffData + 8 * (size_t)kStaticMaxFft;
static_assert(kOffRinds + 2 * (size_t)kStaticMaxUselen <= JERK_STATIC_SCRATCH_BYTES,
              "static scratch layout");

std::mutex g_static_mu;
unsigned char *g_static_addr[64];

int static_fail(int code, const char *msg)
{
    char buf[256];
    snprintf(buf, sizeof buf, "jerk_volume_static: %s", msg);
    return set_error(code, buf);
}

// Radices of one FFT plan, passed by value to the set-up kernel.
struct StaticRadices {
    int n;
    int r[kMaxStages];
};

template <int N>
StaticRadices static_radices()
{
    StaticRadices R{};
    R.n = FftPlan<N>::nstages;
    for (int i = 0; i < R.n; i++)
        R.r[i] = FftPlan<N>::radices[i];
    return R;
}

StaticRadices static_radices_of(int N)
{
    switch (N) {
#define JERK_SR(NN) case NN: return static_radices<NN>();
    JERK_SR(128) JERK_SR(192) JERK_SR(256) JERK_SR(384) JERK_SR(512) JERK_SR(768)
    JERK_SR(1024) JERK_SR(1280) JERK_SR(2048) JERK_SR(4096) JERK_SR(5120) JERK_SR(7680)
#undef JERK_SR
    default: return StaticRadices{};
    }
}

}  // namespace

// Writes the call's descriptors and the plan's per-stage twiddle tables (the
// layout fft_stage_twiddles writes on the host: stage s >= 1 holds
// W_{Ns R}^(r k) at [r Ns + k]) into the static array.  Twiddles are taken in
// double, as on the host, and rounded to float.
__global__ void static_setup_kernel(SubDev sd, StepDev sp, StaticRadices R, int tws,
                                    SubDev *dsub, StepDev *dstep, float2 *dtw)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) {
        *dsub = sd;
        *dstep = sp;
    }
    if (i >= tws)
        return;
    int off = 0, ns = R.r[0];
    for (int s = 1; s < R.n; s++) {
        const int size = ns * R.r[s];
        if (i < off + size) {
            const int idx = i - off, r = idx / ns, k = idx % ns;
            const double a = -2.0 * 3.14159265358979323846264338327950288 * (double)(r * k) /
                             (double)size;
            double sa, ca;
            sincos(a, &sa, &ca);
            dtw[i] = make_float2((float)ca, (float)sa);
            return;
        }
        off += size;
        ns *= R.r[s];
    }
}

}  // namespace jerk

extern "C" int jerk_volume_static(const void *spectrum, long long numbins, long long lobin,
                                  const jerk_subharm *sub, const void *kernels, double fullrlo,
                                  int corr_uselen, float nph, float *volume, int *numrs_out,
                                  long long *rlo_out, void *stream)
{
    using namespace jerk;
    if (!spectrum || !sub || !kernels || !volume || numbins < 1)
        return static_fail(JERK_EINVAL, "null argument");
    const int N = sub->fftlen;
    const int tws = fft_twiddle_size(N);
    if (N > kStaticMaxFft || !fftlen_supported(N) || tws < 0 || (size_t)tws * sizeof(float2) > kOffData - kOffTw)
        return static_fail(JERK_EINVAL, "fftlen beyond the static scratch (at most 7680, and supported)");
    if (corr_uselen <= 0 || corr_uselen % 2 || corr_uselen > kStaticMaxUselen)
        return static_fail(JERK_EINVAL, "corr_uselen beyond the static scratch (even, at most 16384)");
    if (sub->numharm < 1 || sub->harmnum < 1 || sub->numz < 1 || sub->numw < 1)
        return static_fail(JERK_EINVAL, "bad subharmonic");

    // rstep geometry, as jerk_plan_create computes it (src/accel_utils.c:1107-1141)
    const double hf = (double)sub->harmnum / (double)sub->numharm;
    const int rstep = corr_uselen / 2;
    const double lastr = fullrlo + rstep - 0.5;
    const double drlo = rint(2.0 * fullrlo * hf) * 0.5, drhi = rint(2.0 * lastr * hf) * 0.5;
    int numrs = (int)((ceil(drhi) - floor(drlo)) * 2 + 1e-14) + 1;
    if (sub->numharm == 1 && sub->harmnum == 1)
        numrs = corr_uselen;
    else if (numrs % 2)
        numrs = (numrs / 2 + 1) * 2;
    if (numrs + 2 * sub->halfwidth > N)
        return static_fail(JERK_EINVAL, "fftlen too short for the good bins");

    cudaStream_t st = (cudaStream_t)stream;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess)
        return static_fail(JERK_ECUDA, "cudaGetDevice failed");
    if (dev < 0 || dev >= 64)
        return static_fail(JERK_EUNSUPPORTED, "device ordinal above 63");
    unsigned char *base = nullptr;
    {
        std::lock_guard<std::mutex> lock(g_static_mu);
        if (!g_static_addr[dev]) {
            void *addr = nullptr;
            const cudaError_t e = cudaGetSymbolAddress(&addr, g_static_scratch);
            if (e != cudaSuccess || !addr) {
                char msg[160];
                snprintf(msg, sizeof msg, "cudaGetSymbolAddress: %s", cudaGetErrorString(e));
                return static_fail(JERK_ECUDA, msg);
            }
            g_static_addr[dev] = (unsigned char *)addr;
        }
        base = g_static_addr[dev];
    }

    SubDev sd{};
    sd.numharm = sub->numharm;
    sd.harmnum = sub->harmnum;
    sd.harm_fract = hf;
    sd.numz = sub->numz;
    sd.numw = sub->numw;
    sd.fftlen = N;
    sd.halfwidth = sub->halfwidth;
    sd.stride = numrs;
    sd.pownorm = (float)(1.0 / (double)(N * N));
    sd.twoff = 0;
    sd.kern_off = 0;
    sd.plane_off = 0;
    sd.plane_size = (long long)sub->numw * sub->numz * numrs;
    sd.data_off = 0;
    StepDev sp{};
    sp.rlo = (long long)floor(drlo);
    sp.fullrlo = fullrlo;
    sp.numrs = numrs;

    // descriptors and twiddles into the array, by a kernel on the call's
    // stream: no copy from host memory
    static_setup_kernel<<<(tws + 255) / 256 > 0 ? (tws + 255) / 256 : 1, 256, 0, st>>>(
        sd, sp, static_radices_of(N), tws, (SubDev *)(base + kOffSub),
        (StepDev *)(base + kOffStep), (float2 *)(base + kOffTw));
    cudaError_t e = cudaGetLastError();

    SearchDev P{};
    P.spec = (const float2 *)spectrum;
    P.numbins = numbins;
    P.lobin = lobin;
    P.nsubs = 1;
    P.nstages = 1;
    P.corr_uselen = corr_uselen;
    P.numz0 = sub->numz;
    P.numw0 = sub->numw;
    P.norm_type = 0;
    P.nph = nph;
    P.subs = (const SubDev *)(base + kOffSub);
    P.steps = (const StepDev *)(base + kOffStep);
    P.bank = (const float2 *)kernels;
    P.twiddles = (const float2 *)(base + kOffTw);
    P.prepped = (float2 *)(base + kOffData);
    P.planes = volume;
    P.rinds = (uint16_t *)(base + kOffRinds);
    P.first_rstep = 0;
    P.nb = 1;
    if (e == cudaSuccess)
        e = prep_attrs(N);
    if (e == cudaSuccess)
        e = corr_attrs(N);
    if (e == cudaSuccess)
        e = launch_prep(P, N, prep_smem_bytes(N, false), st);
    if (e == cudaSuccess) {
        RowGroup G{};
        G.n = 1;
        G.sub[0] = 0;
        G.rowstart[0] = 0;
        G.rowstart[1] = sub->numw * sub->numz;
        e = launch_corr(P, N, G, G.rowstart[1], st);
    }
    if (e != cudaSuccess)
        return static_fail(JERK_ECUDA, cudaGetErrorString(e));
    if (numrs_out)
        *numrs_out = numrs;
    if (rlo_out)
        *rlo_out = sp.rlo;
    return JERK_OK;
}
