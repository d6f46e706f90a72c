// The spectrum of a time series on the GPU, as the reference prepares a
// ".dat" input before its search (src/accel_utils.c:1696-1753): a forward
// real FFT in PRESTO's packing (realfft, src/fastffts.c:163-235, isign -1)
// followed by red-noise removal (deredden, src/accel_utils.c:1557-1633).
//
// Real FFT of n = 2M samples.  The samples are read as M complex values
// z[m] = x[2m] + i x[2m+1]; their M-point FFT Z is taken in four steps with
// M = R1 * R2 (R1, R2 block-FFT sizes from 128 to 10240: powers of two and
// products with 3 and 5), each step one block-wide FFT per CTA from
// jerk_fft.cuh:
//   1. columns: for each m2 < R2, the R1-point FFT over m1 of z[m2 + R2 m1],
//      times exp(-2 pi i m2 k1 / M), stored as row k1 of an R1 x R2 scratch;
//   2. rows: for each k1 < R1, the R2-point FFT of that row, stored to
//      Z[k1 + R1 k2] in the output (a CTA of either takes up to four
//      neighbouring columns or rows, so that the strided side moves whole
//      32-byte sectors);
//   3. in place on the output: X[k] = (Z[k] + conj Z[M-k]) / 2
//      - (i/2) exp(-2 pi i k / n) (Z[k] - conj Z[M-k]), one thread per
//      pair (k, M-k) in double, and X[0] = (DC, Nyquist) packed as the
//      reference packs them.
// Every kernel is launched early and waits for the one before in its first
// instruction: of a 786432-sample series' 37 us the six launches' gaps took 7.
// No scaling (the reference's forward transform is unnormalised).  The
// FFTs run in FP32 like the reference's, so values agree with the
// reference's to FP32 rounding, not bitwise.
//
// Red-noise removal is bit-exact with the reference.  Its blocks depend only
// on where the walk stops: block 0 is bins [1, 7); each later block starts
// where the previous one ended and is (int)(6 ln(start)) bins long (at most
// 200); a block exists while it ends below numamps.  The host walks this
// sequence once with the C library's log, as the reference does, and keeps it
// as runs of blocks of equal length (about 130 runs cover 2^31 bins), passed
// to the kernels by value.  One warp per block takes the median power (the
// value of rank (n-1)/2, which the reference's quickselect returns) over
// ln 2 (a selection by ballots); one warp per segment between block
// midpoints then scales its bins by
// invsqrtf of the linearly interpolated level, in the reference's float and
// double steps.

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <mutex>
#include <vector>

#include "jerk.h"
#include "jerk_async.cuh"
#include "jerk_fft.cuh"
#include "jerk_kernels.cuh"

namespace jerk {
namespace {

// R1, R2: the block-FFT sizes from 128 to 10240 (powers of two and the mixed
// sizes with factors 3 and 5 that jerk_fft.cuh plans)
constexpr int kRfSizes[] = {128, 192, 256, 384, 512, 768, 1024, 1280, 2048,
                            4096, 5120, 7680, 8192, 10240};

// ---------------------------------------------------------------------------
// real FFT kernels

// The radices of one FFT plan, and where its tables go.
struct RfTable {
    int n, size;
    int r[8];
    float2 *tw;
};

// The per-stage twiddle tables of both block FFTs in one launch (the layout
// fft_stage_twiddles writes on the host: stage s >= 1 of radix R after ns
// points holds W_{ns R}^(r k) at [r ns + k]), computed in double.
__global__ void rf_twiddle_kernel(RfTable A, RfTable B)
{
    wait_before();
    let_follow();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    const RfTable &t = i < A.size ? A : B;
    if (i >= A.size)
        i -= A.size;
    if (i >= t.size)
        return;
    int off = 0, ns = t.r[0];
    for (int s = 1; s < t.n; s++) {
        const int size = ns * t.r[s];
        if (i < off + size) {
            const int r = (i - off) / ns, k = (i - off) % ns;
            double sn, cs;
            sincospi(-2.0 * (double)(r * k) / (double)size, &sn, &cs);
            t.tw[i] = make_float2((float)cs, (float)sn);
            return;
        }
        off += size;
        ns *= t.r[s];
    }
}

// Columns (rows) of a CTA: four where their threads fit in one CTA, whose
// 8-byte accesses then make whole sectors on the strided side.  The buffers
// lie 4 banks of 8 bytes apart, so that a half warp (four columns of four
// neighbouring threads) touches every bank once.  At 2^25 samples one column
// per CTA took 230 us and one row 161 (a quarter of each sector used).
template <int R>
struct RfShape {
    static constexpr int T = FftPlan<R>::T;
    static constexpr int C = T <= 256 ? 4 : T <= 512 ? 2 : 1;
    static constexpr int Pitch = (fft_buf_len<R>() + 15) / 16 * 16 + 4;  // float2
    static constexpr int Smem = C * Pitch * 8;
};

// Step 1: a CTA transforms columns m2 of z (stride R2) and stores row k1 of
// the scratch at a[k1 * R2 + m2], times exp(-2 pi i m2 k1 / M).  The twiddle
// is the double product of two per-column tables, exp(-2 pi i m2 lo / M) and
// exp(-2 pi i m2 64 hi / M) for k1 = 64 hi + lo (exponents reduced mod M
// exactly), rounded once to float.
constexpr int kTwLo = 64;
template <int R1>
__global__ void __launch_bounds__(RfShape<R1>::T * RfShape<R1>::C)
    rf_column_kernel(const float2 *z, int R2, const float2 *tw,
                     float2 *a)
{
    wait_before();
    let_follow();
    using H = RfShape<R1>;
    constexpr int T = H::T, C = H::C;
    constexpr int NHI = (R1 + kTwLo - 1) / kTwLo;
    extern __shared__ float2 rf_buf[];
    __shared__ double2 t_lo[kTwLo][C], t_hi[NHI][C];
    const int c = threadIdx.x % C, tid = threadIdx.x / C;
    const int m2 = blockIdx.x * C + c;
    const long long M = (long long)R1 * R2;
    for (int i = tid; i < kTwLo + NHI; i += T) {
        const long long e = i < kTwLo ? ((long long)m2 * i) % M
                                      : ((long long)m2 * kTwLo * (i - kTwLo)) % M;
        double sn, cs;
        sincospi(-2.0 * (double)e / (double)M, &sn, &cs);
        if (i < kTwLo)
            t_lo[i][c] = make_double2(cs, sn);
        else
            t_hi[i - kTwLo][c] = make_double2(cs, sn);
    }
    // fft_block's first barrier orders these writes before the reads in out()
    auto in = [&](int r) -> float2 { return z[m2 + (size_t)R2 * (size_t)(tid + r * T)]; };
    auto out = [&](int k1, float2 y) {
        const double2 u = t_hi[k1 / kTwLo][c], v = t_lo[k1 % kTwLo][c];
        const float2 w = make_float2((float)(u.x * v.x - u.y * v.y), (float)(u.x * v.y + u.y * v.x));
        a[(size_t)k1 * R2 + m2] = cmul(y, w);
    };
    fft_block<R1, -1>(rf_buf + c * H::Pitch, tw, tid, in, out);
}

// Step 2: a CTA transforms rows k1 of the scratch and stores Z[k1 + R1 k2].
template <int R2>
__global__ void __launch_bounds__(RfShape<R2>::T * RfShape<R2>::C)
    rf_row_kernel(const float2 *a, int R1, const float2 *tw,
                  float2 *zout)
{
    wait_before();
    let_follow();
    using H = RfShape<R2>;
    constexpr int T = H::T, C = H::C;
    extern __shared__ float2 rf_buf[];
    const int c = threadIdx.x % C, tid = threadIdx.x / C;
    const int k1 = blockIdx.x * C + c;
    const float2 *row = a + (size_t)k1 * R2;
    auto in = [&](int r) -> float2 { return row[tid + r * T]; };
    auto out = [&](int k2, float2 y) { zout[k1 + (size_t)R1 * k2] = y; };
    fft_block<R2, -1>(rf_buf + c * H::Pitch, tw, tid, in, out);
}

// Step 3, in place: thread k (0 <= k <= M/2) turns Z[k], Z[M-k] into X[k],
// X[M-k].  With h = (Z[k] + conj Z[M-k]) / 2, d = Z[k] - conj Z[M-k] and
// g = W d, W = exp(-i pi k / M):
//   X[k]   = (h.x + g.y / 2,  h.y - g.x / 2)
//   X[M-k] = (h.x - g.y / 2, -h.y - g.x / 2)
__global__ void rf_post_kernel(float2 *x, long long M)
{
    wait_before();
    let_follow();
    const long long half = M / 2;
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k <= half;
         k += (long long)gridDim.x * blockDim.x) {
        if (k == 0) {
            const float2 z0 = x[0];
            x[0] = make_float2(z0.x + z0.y, z0.x - z0.y);
            continue;
        }
        const float2 a = x[k], b = x[M - k];
        const double hx = 0.5 * ((double)a.x + (double)b.x);
        const double hy = 0.5 * ((double)a.y - (double)b.y);
        const double dx = (double)a.x - (double)b.x;
        const double dy = (double)a.y + (double)b.y;
        double s, c;
        sincospi(-(double)k / (double)M, &s, &c);
        const double gx = c * dx - s * dy, gy = c * dy + s * dx;
        x[k] = make_float2((float)(hx + 0.5 * gy), (float)(hy - 0.5 * gx));
        if (k != M - k)
            x[M - k] = make_float2((float)(hx - 0.5 * gy), (float)(-hy - 0.5 * gx));
    }
}

template <int R1>
cudaError_t rf_launch_columns(const float2 *z, int R2, const float2 *tw, float2 *a, cudaStream_t st)
{
    using H = RfShape<R1>;
    cudaError_t e = cudaFuncSetAttribute(rf_column_kernel<R1>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, H::Smem);
    if (e != cudaSuccess)
        return e;
    return launch_follow(rf_column_kernel<R1>, R2 / H::C, H::T * H::C, H::Smem, st, z, R2, tw, a);
}

template <int R2>
cudaError_t rf_launch_rows(const float2 *a, int R1, const float2 *tw, float2 *zout, cudaStream_t st)
{
    using H = RfShape<R2>;
    cudaError_t e = cudaFuncSetAttribute(rf_row_kernel<R2>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, H::Smem);
    if (e != cudaSuccess)
        return e;
    return launch_follow(rf_row_kernel<R2>, R1 / H::C, H::T * H::C, H::Smem, st, a, R1, tw, zout);
}

// Runtime dispatch over kRfSizes.
template <template <int> class F, class... A>
cudaError_t rf_dispatch(int R, A... args)
{
    switch (R) {
    case 128: return F<128>::run(args...);
    case 192: return F<192>::run(args...);
    case 256: return F<256>::run(args...);
    case 384: return F<384>::run(args...);
    case 512: return F<512>::run(args...);
    case 768: return F<768>::run(args...);
    case 1024: return F<1024>::run(args...);
    case 1280: return F<1280>::run(args...);
    case 2048: return F<2048>::run(args...);
    case 4096: return F<4096>::run(args...);
    case 5120: return F<5120>::run(args...);
    case 7680: return F<7680>::run(args...);
    case 8192: return F<8192>::run(args...);
    case 10240: return F<10240>::run(args...);
    default: return cudaErrorInvalidValue;
    }
}
template <int R> struct RfRadices {
    static cudaError_t run(RfTable *t)
    {
        using P = FftPlan<R>;
        static_assert(P::nstages <= 8, "radices");
        t->n = P::nstages;
        t->size = P::twsize();
        for (int i = 0; i < P::nstages; i++)
            t->r[i] = P::radices[i];
        return cudaSuccess;
    }
};
template <int R> struct RfCol {
    static cudaError_t run(const float2 *z, int R2, const float2 *tw, float2 *a, cudaStream_t st)
    {
        return rf_launch_columns<R>(z, R2, tw, a, st);
    }
};
template <int R> struct RfRow {
    static cudaError_t run(const float2 *a, int R1, const float2 *tw, float2 *zo, cudaStream_t st)
    {
        return rf_launch_rows<R>(a, R1, tw, zo, st);
    }
};

template <int R> struct RfTwSize {
    static cudaError_t run(int *out)
    {
        *out = FftPlan<R>::twsize();
        return cudaSuccess;
    }
};

int rf_twsize(int R)
{
    int n = -1;
    return rf_dispatch<RfTwSize>(R, &n) == cudaSuccess ? n : -1;
}

size_t align256(size_t b) { return (b + 255) & ~(size_t)255; }

// M = n / 2 = R1 * R2 with R1, R2 in kRfSizes, the most balanced pair
// (R1 >= R2); false when n is odd or M has no such factorisation.
bool rf_split(long long n, int *R1, int *R2)
{
    if (n < 2 || (n & 1))
        return false;
    const long long M = n / 2;
    bool found = false;
    for (int a : kRfSizes)
        for (int b : kRfSizes)
            if (a >= b && (long long)a * b == M && (!found || a - b < *R1 - *R2)) {
                *R1 = a;
                *R2 = b;
                found = true;
            }
    return found;
}

// scratch: [M float2 | R1 twiddles | R2 twiddles], each region 256-aligned
size_t rf_scratch(int R1, int R2)
{
    return align256(sizeof(float2) * (size_t)R1 * R2) + align256(sizeof(float2) * rf_twsize(R1)) +
           align256(sizeof(float2) * rf_twsize(R2));
}

// ---------------------------------------------------------------------------
// red-noise removal

constexpr int kDrInit = 6, kDrMax = 200;  // initialbuflen, maxbuflen
constexpr int kDrRuns = 192;

// Blocks first .. first + count - 1 start at start + (b - first) * len.
struct DrRun {
    int first, start, len, count;
};
struct DrRuns {
    int n;
    DrRun r[kDrRuns];
};
static_assert(sizeof(DrRuns) <= 4000, "kernel parameter space");

// the run that holds block b
__device__ __forceinline__ int dr_run(const DrRuns &R, int b)
{
    int lo = 0, hi = R.n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (R.r[mid].first <= b)
            lo = mid;
        else
            hi = mid - 1;
    }
    return lo;
}

__device__ __forceinline__ float dr_power(float2 v)
{
    return __fadd_rn(__fmul_rn(v.x, v.x), __fmul_rn(v.y, v.y));
}

constexpr int kDrWarps = 8;

// The k-th smallest (0-based) of the first n <= 128 values held 4 per lane
// (value e = lane + 32 j as bit pattern u[j], ~0 past n; non-negative floats
// order as their bits do), by one warp: thresholds -- first where the median
// of exponential noise of this mean would lie, then steps by that density --
// until the count below one is k or k + 1, whose neighbour is the value; ties
// and other distributions end in a walk over the values from the lower bound.
// The thresholds only set the speed.  (For 2^24 bins: 71 us; sorting in
// registers, a hundred shuffles a block, 110; a quickselect by ballots 119.)
__device__ __forceinline__ int warp_count_below(const unsigned (&u)[4], unsigned t)
{
    const unsigned c = (u[0] < t) + (u[1] < t) + (u[2] < t) + (u[3] < t);
    return (int)__reduce_add_sync(0xffffffffu, c);
}

__device__ __forceinline__ unsigned warp_select(const unsigned (&u)[4], float mean, int n, int k)
{
    // counts below flo and fhi: cl <= k < ch
    float flo = 0.f, fhi = __int_as_float(0x7f800000);
    int cl = 0, ch = n;
    float p = 0.69314718f * mean;
    const float step = 2.0f * mean / (float)n;  // one rank at the median
#pragma unroll 1
    for (int round = 0; round < 7 && cl < k && ch > k + 1; round++) {
        const int c = warp_count_below(u, __float_as_uint(p));
        if (c <= k) {
            flo = p;
            cl = c;
        } else {
            fhi = p;
            ch = c;
        }
        // the next threshold aims half a rank past the one wanted
        const float d = ((float)(k - c) + 0.5f) * step;
        const float q = p + d;
        p = q > flo && q < fhi ? q : 0.5f * (flo + fhi);
    }
    if (ch == k + 1) {  // the largest value below fhi
        unsigned m = 0u;
        const unsigned t = __float_as_uint(fhi);
#pragma unroll
        for (int j = 0; j < 4; j++)
            m = max(m, u[j] < t ? u[j] : 0u);
        return __reduce_max_sync(0xffffffffu, m);
    }
    unsigned lo = __float_as_uint(flo);
    for (;;) {  // the smallest value from lo on, until its rank passes k
        unsigned m = ~0u;
#pragma unroll
        for (int j = 0; j < 4; j++)
            m = min(m, u[j] >= lo ? u[j] : ~0u);
        m = __reduce_min_sync(0xffffffffu, m);
        if (cl == k || m == ~0u || warp_count_below(u, m + 1u) > k)
            return m;
        lo = m + 1u;
        cl = -1;
    }
}

// One warp per block: level[b] = median power / ln 2, its middle bin and
// its length.  Blocks are at most 128 bins long below 2^31 bins ((int)(6 ln
// 2^31) = 128); the value of rank (n-1)/2 is the one the reference's
// quickselect returns.  (Longer blocks, which the walk never makes, would take
// the stable-rank count.)
__global__ void __launch_bounds__(32 * kDrWarps)
    dr_level_kernel(const float2 *x, const __grid_constant__ DrRuns runs, int nb,
                    double ln2, float *level, int *mid, int *len)
{
    wait_before();
    let_follow();
    __shared__ float pw[kDrWarps][kDrMax];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int b = blockIdx.x * kDrWarps + w;
    // the run of the CTA's first block, once; the others step on from it
    __shared__ int s_run;
    if (threadIdx.x == 0)
        s_run = dr_run(runs, blockIdx.x * kDrWarps);
    __syncthreads();
    if (b >= nb)
        return;  // whole warps leave; only warp-level syncs below
    int run = s_run;
    while (run + 1 < runs.n && runs.r[run + 1].first <= b)
        run++;
    const int2 blk = make_int2(runs.r[run].start + (b - runs.r[run].first) * runs.r[run].len,
                               runs.r[run].len);
    const int n = blk.y;
    const int k = (n - 1) / 2;
    if (lane == 0) {
        mid[b] = blk.x + n / 2;
        len[b] = n;
    }
    if (n <= 128) {
        unsigned u[4];
        float sum = 0.f;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int i = lane + 32 * j;
            const float p = i < n ? dr_power(x[blk.x + i]) : 0.f;
            u[j] = i < n ? __float_as_uint(p) : ~0u;
            sum += p;
        }
#pragma unroll
        for (int d = 16; d > 0; d >>= 1)
            sum += __shfl_xor_sync(0xffffffffu, sum, d);
        const float med = __uint_as_float(warp_select(u, sum / (float)n, n, k));
        if (lane == 0)
            level[b] = (float)((double)med / ln2);
        return;
    }
    float *p = pw[w];
    for (int i = lane; i < n; i += 32)
        p[i] = dr_power(x[blk.x + i]);
    __syncwarp();
    for (int i = lane; i < n; i += 32) {
        const float v = p[i];
        int pos = 0;
        for (int j = 0; j < n; j++) {
            const float u = p[j];
            pos += (u < v) | ((u == v) & (j < i));
        }
        if (pos == k)
            level[b] = (float)((double)v / ln2);
    }
}

// One warp per segment s = 0..nb: segment 0 is bins [1, mid(0)) at the
// constant level[0]; segment s is [mid(s-1), mid(s)) (mid(nb) = numamps)
// running from level[s-1] with the slope toward level[s] (the tail keeps the
// last slope, or 1 when there is one block).  mid(b) = start + len / 2.
// Bin 0 becomes (1, bin0_imag).  A segment is about a hundred bins: its loads
// go out together, and the blocks' places come from the level pass (the walk
// over the runs three times a warp, and one load at a time, took 97 us for
// 2^24 bins).
__global__ void __launch_bounds__(32 * kDrWarps)
    dr_scale_kernel(float2 *x, int nb, int numamps, const float *level,
                    const int *mid, const int *len, float bin0_imag)
{
    wait_before();
    let_follow();
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int s = blockIdx.x * kDrWarps + w;
    if (s > nb)
        return;
    const bool flat = s == 0;
    const int lo = flat ? 1 : mid[s - 1];
    const int hi = s < nb ? mid[s] : numamps;
    const float base = level[flat ? 0 : s - 1];
    float slope = 0.0f;
    if (flat) {
        if (lane == 0)
            x[0] = make_float2(1.0f, bin0_imag);
    } else {
        const int bb = s < nb ? s : nb - 1;
        slope = bb >= 1 ? (float)((double)__fsub_rn(level[bb], level[bb - 1]) /
                                  (0.5 * (double)(len[bb - 1] + len[bb])))
                        : 1.0f;
    }
    for (int i0 = lo + lane; i0 < hi; i0 += 128) {
        float2 v[4];
#pragma unroll
        for (int j = 0; j < 4; j++)
            if (i0 + 32 * j < hi)
                v[j] = x[i0 + 32 * j];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int ind = i0 + 32 * j;
            if (ind >= hi)
                break;
            const float lv = flat ? base : __fadd_rn(base, __fmul_rn(slope, (float)(ind - lo)));
            const float nrm = invsqrtf_ref(lv);
            x[ind] = make_float2(__fmul_rn(v[j].x, nrm), __fmul_rn(v[j].y, nrm));
        }
    }
}

// The block walk from bin 1, kept as runs of equal length.  Shared by every
// call; extended under the lock as longer spectra arrive.
std::mutex g_dr_mu;
std::vector<DrRun> g_dr_runs;  // complete runs plus the open last one
long long g_dr_next = 0;       // start of the first block not yet walked

int dr_len(long long binnum)
{
    const int l = (int)(kDrInit * std::log((double)binnum));
    return l > kDrMax ? kDrMax : l;
}

// Walk until the next block's start passes limit.
void dr_extend(long long limit)
{
    if (g_dr_runs.empty()) {
        g_dr_runs.push_back({0, 1, kDrInit, 1});
        g_dr_next = 1 + kDrInit;
    }
    while (g_dr_next <= limit) {
        const int len = dr_len(g_dr_next);
        DrRun &last = g_dr_runs.back();
        const int nblk = last.first + last.count;
        if (len == last.len && last.first > 0)
            last.count++;
        else
            g_dr_runs.push_back({nblk, (int)g_dr_next, len, 1});
        g_dr_next += len;
    }
}

// The runs of the blocks of a numamps-bin spectrum: block 0, then every
// block b >= 1 with start + len < numamps.  Returns the block count, or -1.
int dr_layout(int numamps, DrRuns *out)
{
    std::lock_guard<std::mutex> lock(g_dr_mu);
    dr_extend(numamps);
    int nb = 0, nr = 0;
    for (const DrRun &u : g_dr_runs) {
        int take = 0;
        if (u.first == 0) {
            take = 1;
        } else {
            // blocks j < count with start + j len + len < numamps
            const long long room = (long long)numamps - u.start - u.len;  // need j * len < room
            if (room > 0)
                take = (int)std::min<long long>(u.count, (room + u.len - 1) / u.len);
        }
        if (take == 0)
            break;
        if (nr == kDrRuns)
            return -1;
        out->r[nr++] = {u.first, u.start, u.len, take};
        nb = u.first + take;
        if (take < u.count)
            break;
    }
    out->n = nr;
    return nb;
}

// Three words a block: level, mid, len.  There are far fewer blocks than
// numamps / kDrInit (their length grows from 6 bins to 17 by bin 18 and 35 by
// bin 400), and the first 21 fit in the rounding to 256 bytes: a size for one
// word per kDrInit bins, which a caller may have allocated once, holds them.
size_t dr_scratch(int numamps)
{
    return align256(sizeof(float) * (size_t)(numamps / kDrInit + 2));
}

// ---------------------------------------------------------------------------
// birdie zapping (zapbirds from memory, src/zapping.c:29-81)

constexpr int kZapBins = 200;  // MEDIANBINS (src/zapping.c:3)
constexpr int kZapThreads = 512;
constexpr int kZapGroup = 128;

struct ZapGroup {
    double lo[kZapGroup], hi[kZapGroup];
};

// One birdie per CTA.  The median powers (rank 99 of 200) of the bins
// [lobin - 300, lobin - 100) and [hibin - 100, hibin + 100), read before any
// bin is written (bins at or past numamps read as zeros, as the reference's
// zero-padded buffer gives them), set avgamp = sqrt(0.5 (mlo + mhi) / ln 2);
// bins [floor(lobin), ceil(hibin)) become (avgamp, 0).  The birdies of a
// launch touch no bin that another writes (one launch per birdie, as the
// order of the list would have it, took 7 us each).
__global__ void __launch_bounds__(kZapThreads)
    zap_kernel(float2 *x, long long numamps, const __grid_constant__ ZapGroup g,
               double neg_log_half)
{
    wait_before();
    let_follow();
    __shared__ __align__(16) float p[2][kZapBins];
    __shared__ float med[2];
    const double lobin = g.lo[blockIdx.x], hibin = g.hi[blockIdx.x];
    const int w = threadIdx.x / 256, i = threadIdx.x % 256;
    const long long first = w == 0 ? (long long)(lobin - 3 * kZapBins / 2)
                                   : (long long)(hibin - kZapBins / 2);
    float v = 0.f;
    if (i < kZapBins) {
        const long long b = first + i;
        v = dr_power((b >= 0 && b < numamps) ? x[b] : make_float2(0.f, 0.f));
        p[w][i] = v;
    }
    __syncthreads();
    constexpr int k = (kZapBins - 1) / 2;
    if (i < kZapBins) {
        int pos = 0;
#pragma unroll 5
        for (int j = 0; j < kZapBins; j += 4) {
            const float4 u = *reinterpret_cast<const float4 *>(&p[w][j]);
            pos += (u.x < v) | ((u.x == v) & (j < i));
            pos += (u.y < v) | ((u.y == v) & (j + 1 < i));
            pos += (u.z < v) | ((u.z == v) & (j + 2 < i));
            pos += (u.w < v) | ((u.w == v) & (j + 3 < i));
        }
        if (pos == k)
            med[w] = v;
    }
    __syncthreads();
    const float avgamp =
        (float)__dsqrt_rn(__ddiv_rn(0.5 * (double)__fadd_rn(med[0], med[1]), neg_log_half));
    const long long lo = (long long)floor(lobin), hi = (long long)ceil(hibin);
    for (long long b = lo + threadIdx.x; b < hi; b += kZapThreads)
        if (b >= 0 && b < numamps)
            x[b] = make_float2(avgamp, 0.f);
}

}  // namespace
}  // namespace jerk

using namespace jerk;

extern "C" long long jerk_realfft_scratch_bytes(long long n)
{
    int R1, R2;
    if (!rf_split(n, &R1, &R2))
        return 0;
    return (long long)rf_scratch(R1, R2);
}

extern "C" int jerk_realfft(const float *timeseries, long long n, void *spectrum, void *scratch,
                            long long scratch_bytes, void *stream)
{
    int R1, R2;
    if (!rf_split(n, &R1, &R2))
        return set_error(JERK_EUNSUPPORTED,
                         "jerk_realfft: n must be 2 R1 R2 with R1, R2 in {128, 192, 256, 384, "
                         "512, 768, 1024, 1280, 2048, 4096, 5120, 7680, 8192, 10240}");
    if (!timeseries || !spectrum || !scratch)
        return set_error(JERK_EINVAL, "jerk_realfft: null pointer");
    if (((uintptr_t)timeseries | (uintptr_t)spectrum) & 7 || (uintptr_t)scratch & 255)
        return set_error(JERK_EINVAL,
                         "jerk_realfft: series and spectrum must be 8-byte aligned, scratch 256");
    if (scratch_bytes < (long long)rf_scratch(R1, R2))
        return set_error(JERK_EINVAL, "jerk_realfft: scratch smaller than jerk_realfft_scratch_bytes");
    cudaStream_t st = (cudaStream_t)stream;
    unsigned char *base = (unsigned char *)scratch;
    float2 *a = (float2 *)base;
    float2 *tw1 = (float2 *)(base + align256(sizeof(float2) * (size_t)R1 * R2));
    float2 *tw2 = (float2 *)((unsigned char *)tw1 + align256(sizeof(float2) * rf_twsize(R1)));
    float2 *out = (float2 *)spectrum;
    RfTable t1{}, t2{};
    rf_dispatch<RfRadices>(R1, &t1);
    rf_dispatch<RfRadices>(R2, &t2);
    t1.tw = tw1;
    t2.tw = tw2;
    cudaError_t e =
        launch_follow(rf_twiddle_kernel, (t1.size + t2.size + 255) / 256, 256, 0, st, t1, t2);
    if (e == cudaSuccess)
        e = rf_dispatch<RfCol>(R1, (const float2 *)timeseries, R2, (const float2 *)tw1, a, st);
    if (e == cudaSuccess)
        e = rf_dispatch<RfRow>(R2, (const float2 *)a, R1, (const float2 *)tw2, out, st);
    if (e == cudaSuccess) {
        const long long M = (long long)R1 * R2;
        const long long threads = M / 2 + 1;
        const int grid = (int)std::min<long long>((threads + 255) / 256, 148LL * 16);
        e = launch_follow(rf_post_kernel, grid, 256, 0, st, out, M);
    }
    if (e != cudaSuccess)
        return set_error(JERK_ECUDA, cudaGetErrorString(e));
    return JERK_OK;
}

extern "C" long long jerk_deredden_scratch_bytes(long long numamps)
{
    if (numamps < 8 || numamps > 0x7fffffffLL)
        return 0;
    return (long long)dr_scratch((int)numamps);
}

namespace {
int deredden_impl(void *spectrum, long long numamps, void *scratch, long long scratch_bytes,
                  void *stream, float bin0_imag)
{
    if (numamps < 8 || numamps > 0x7fffffffLL)
        return set_error(JERK_EINVAL, "jerk_deredden: numamps must be 8 .. 2^31-1");
    if (!spectrum || !scratch)
        return set_error(JERK_EINVAL, "jerk_deredden: null pointer");
    if ((uintptr_t)spectrum & 7 || (uintptr_t)scratch & 3)
        return set_error(JERK_EINVAL, "jerk_deredden: misaligned spectrum or scratch");
    if (scratch_bytes < (long long)dr_scratch((int)numamps))
        return set_error(JERK_EINVAL,
                         "jerk_deredden: scratch smaller than jerk_deredden_scratch_bytes");
    DrRuns runs;
    const int nb = dr_layout((int)numamps, &runs);
    if (nb < 1 || 3 * sizeof(float) * (size_t)nb > dr_scratch((int)numamps))
        return set_error(JERK_EUNSUPPORTED, "jerk_deredden: block layout too long");
    cudaStream_t st = (cudaStream_t)stream;
    float *level = (float *)scratch;
    int *mid = (int *)scratch + nb, *len = mid + nb;
    float2 *x = (float2 *)spectrum;
    const int threads = 32 * kDrWarps;
    cudaError_t e = launch_follow(dr_level_kernel, (nb + kDrWarps - 1) / kDrWarps, threads, 0, st, x,
                                  runs, nb, std::log(2.0), level, mid, len);
    if (e == cudaSuccess)
        e = launch_follow(dr_scale_kernel, (nb + 1 + kDrWarps - 1) / kDrWarps, threads, 0, st, x, nb,
                          (int)numamps, level, mid, len, bin0_imag);
    if (e != cudaSuccess)
        return set_error(JERK_ECUDA, cudaGetErrorString(e));
    return JERK_OK;
}
}  // namespace

// deredden sets bin 0 to (1, 0) (src/accel_utils.c:1569-1570).
extern "C" int jerk_deredden(void *spectrum, long long numamps, void *scratch,
                             long long scratch_bytes, void *stream)
{
    return deredden_impl(spectrum, numamps, scratch, scratch_bytes, stream, 0.0f);
}

extern "C" long long jerk_spectrum_scratch_bytes(long long n)
{
    const long long a = jerk_realfft_scratch_bytes(n), b = jerk_deredden_scratch_bytes(n / 2);
    return a && b ? std::max(a, b) : 0;
}

extern "C" int jerk_spectrum_from_timeseries(const float *timeseries, long long n, void *spectrum,
                                             void *scratch, long long scratch_bytes, void *stream)
{
    const int rc = jerk_realfft(timeseries, n, spectrum, scratch, scratch_bytes, stream);
    if (rc != JERK_OK)
        return rc;
    // create_accelobs then sets bin 0 of a .dat input to (1, 1) when the
    // powers are not photon-normalised (src/accel_utils.c:1829-1834)
    return deredden_impl(spectrum, n / 2, scratch, scratch_bytes, stream, 1.0f);
}

// The caller's loop around zapbirds (src/accelsearch_lib.c:393-418): birdies
// in list order, stopping at the first one at or above N/2, high edges
// clamped to N/2 - 1; birdies at or below 1.5 * 200 + 1 bins are left alone.
extern "C" int jerk_zap_birdies(void *spectrum, long long numbins, long long N,
                                const double *lobins, const double *hibins, int nbirds,
                                void *stream)
{
    if (!spectrum || numbins < 1 || N < 2 || nbirds < 0 || (nbirds && (!lobins || !hibins)))
        return set_error(JERK_EINVAL, "jerk_zap_birdies: bad argument");
    if ((uintptr_t)spectrum & 7)
        return set_error(JERK_EINVAL, "jerk_zap_birdies: misaligned spectrum");
    cudaStream_t st = (cudaStream_t)stream;
    const double top = (double)(N / 2);
    const double neg_log_half = -std::log(0.5);
    // birdies in list order; a launch takes as many as touch none of each
    // other's bins: a birdie reads within [lo - 301, lo - 99) and [hi - 101,
    // hi + 101) and writes within [lo - 1, hi + 1)
    ZapGroup g;
    cudaError_t e = cudaSuccess;
    int n = 0;
    auto flush = [&] {
        if (n && e == cudaSuccess)
            e = launch_follow(zap_kernel, n, kZapThreads, 0, st, (float2 *)spectrum, numbins, g,
                              neg_log_half);
        n = 0;
    };
    auto clear_of = [](double alo, double ahi, double blo, double bhi) {  // a's bins, b's writes
        return std::min(alo - 302.0, ahi - 102.0) >= bhi + 1.0 ||
               std::max(alo - 99.0, ahi + 102.0) <= blo - 1.0;
    };
    for (int i = 0; i < nbirds; i++) {
        if (lobins[i] >= top)
            break;
        const double lo = lobins[i], hi = hibins[i] >= top ? top - 1 : hibins[i];
        if (!(lo - 1.5 * kZapBins > 1))
            continue;
        bool apart = n < kZapGroup;
        for (int j = 0; j < n && apart; j++)
            apart = clear_of(lo, hi, g.lo[j], g.hi[j]) && clear_of(g.lo[j], g.hi[j], lo, hi);
        if (!apart)
            flush();
        g.lo[n] = lo;
        g.hi[n++] = hi;
    }
    flush();
    if (e != cudaSuccess)
        return set_error(JERK_ECUDA, cudaGetErrorString(e));
    return JERK_OK;
}
