// Correlation on folded kernel rows (sm_100a, FP32 SIMT).
//
// The prepared chunk of one (rstep, subharmonic) is fftlen/2 = M normalised
// bins spread to even half bins; a kernel row is the fftlen-point transform
// of the row's response k[t], t in half bins.  Only the good outputs are
// kept, and the two output parities separate:
//   y[2m]     = sum_j conj k[2j]     d[m + j]
//   y[2m + 1] = sum_j conj k[2j - 1] d[m + j]
// two correlations of the M bins d.  A row whose response lies within
// [-2h, 2h) half bins reads, for its nr/2 good outputs of each parity, no
// more than nr/2 + 2h bins, so a circular transform of L >= nr/2 + 2h bins
// around the good ones gives exactly those outputs, whatever fftlen the
// search geometry names.  FFT lengths come in coarse steps (1280, then 2048)
// and most rows are narrower than the widest one, so at zmax 200, wmax 300,
// 16 harmonics the rows need 0.85 of the points that M-point transforms take
// (at 300, 600, 32 harmonics 0.77): the correlation of 64 rsteps went from
// 7.44 to 6.53 ms a batch; at 300, 600, 2 harmonics, 16 rsteps, from 3.68
// (4096-point transforms of unfolded rows) to 2.98.
//
// A plan therefore takes, for a row of support h, the shortest L of kFoldLens
// that holds it.  In a generated bank h is the halfwidth of the row's response,
// which is checked while the rows are folded; of other rows, or where that
// check fails, h is measured from the row itself (fold_support_kernel).  The row
// is written as A = conj(FFT_L k[2j]) / L and B = conj(FFT_L k[2j-1]) / L
// (fold_rows_kernel; both in double, each value rounded once).  L = M needs
// no support: there A and B are sums of the row's own values, the same
// circular correlation the row defines.  The 1/L in the row makes |y|^2 the
// power, with no multiply left in the loop.
//
// The rows of one L form one launch: corr_fold_kernel<L>.  The half-length
// plan is [8, 16, R2], L = 128 R2, on T = L/8 threads a row, and a CTA takes
// as many rows (of one class, so that they share the staged chunk transform)
// as make whole warps.  Stage 0 runs the two transforms in the two lanes of
// packed FP32 instructions: every butterfly of the even transform has its
// twin in the odd one at the same position with the same twiddle and data
// value, so each instruction does both.  Thread j does butterfly j of both
// from the same 8 data values, and applies stage 1's input twiddles.  Stage 1
// (radix 16, T/2 butterflies per transform): one transform per thread in
// scalar FP32, the first half of a row's threads the even one and the second
// half the odd one, so every warp works (a scalar instruction holds the FP32
// pipe for one cycle, a packed one for two: the pipe time is the same either
// way).  Stage 2 (radix R2, 128 butterflies, Ns = 128): up to R2 = 8 packed,
// butterfly j of both, and the lane pair of powers (outputs 2m, 2m + 1) is
// one 8-byte store; above that the packed values would not fit in registers,
// so neighbouring threads take the even and the odd transform of a butterfly
// in scalar FP32 and their 4-byte stores are consecutive.
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
// Plan-time: row support and folded rows, in double.

// Threads for N-point rows: one radix-4 butterfly each.  The transforms are
// latency bound (at fftlen 4096 the buffers leave one CTA an SM), so as many
// threads as there are butterflies: making a plan of 23,000 such rows spent
// 18 ms here with 256 threads a CTA.
constexpr int kFoldThreads = 1024;
static int fold_threads(int N) { return std::max(128, std::min(N / 4 / 32 * 32, kFoldThreads)); }

// Element i of a transform buffer in shared memory: a word of 16 bytes is left
// out after every eight, or a stage's stores, four elements apart between
// neighbouring threads, would meet in a quarter of the banks (29371 rows of 2048
// points transformed back: 1.90 -> 1.58 ms, with shifts for the division by ns).
__host__ __device__ constexpr int dpad(int i) { return i + (i >> 3); }

__device__ __forceinline__ double2 dmulw(double2 a, double2 w, bool inv)
{
    const double wy = inv ? -w.y : w.y;
    return make_double2(a.x * w.x - a.y * wy, a.x * wy + a.y * w.x);
}

// One Stockham stage of radix R from x to y in shared memory, ns (the product
// of the radices before it) a power of two.  roots[m] = exp(-2 pi i m / n);
// inv: the conjugate transform.
template <int R>
__device__ __forceinline__ void dstage(const double2 *x, double2 *y, int n, int ns,
                                       const double2 *__restrict__ roots, bool inv)
{
    const int nb = n / R, step = nb / ns;
    for (int j = threadIdx.x; j < nb; j += blockDim.x) {
        const int k = j & (ns - 1);
        double2 v[R];
        // the powers of one root: a read of each, from L2, costs more than the
        // products, whose error is far below the rows' rounding (plans of 23042
        // rows of 4096 points 7.7 -> 6.8 ms, of 31,000 rows to 2048 12.5 -> 11.1)
        const double2 w1 = roots[k * step];
        double2 wr = w1;
#pragma unroll
        for (int r = 0; r < R; r++) {
            v[r] = x[dpad(j + r * nb)];
            if (r > 0) {
                v[r] = dmulw(v[r], wr, inv);
                wr = dmulw(wr, w1, false);
            }
        }
        const int o = (j - k) * R + k;
        if constexpr (R == 4) {
            const double2 a = make_double2(v[0].x + v[2].x, v[0].y + v[2].y);
            const double2 b = make_double2(v[0].x - v[2].x, v[0].y - v[2].y);
            const double2 c = make_double2(v[1].x + v[3].x, v[1].y + v[3].y);
            double2 d = make_double2(v[1].y - v[3].y, v[3].x - v[1].x);  // -i (v1 - v3)
            if (inv)
                d = make_double2(-d.x, -d.y);
            y[dpad(o)] = make_double2(a.x + c.x, a.y + c.y);
            y[dpad(o + ns)] = make_double2(b.x + d.x, b.y + d.y);
            y[dpad(o + 2 * ns)] = make_double2(a.x - c.x, a.y - c.y);
            y[dpad(o + 3 * ns)] = make_double2(b.x - d.x, b.y - d.y);
        } else {
#pragma unroll
            for (int q = 0; q < R; q++) {
                double2 s = v[0];
#pragma unroll
                for (int r = 1; r < R; r++) {
                    const double2 t = dmulw(v[r], roots[((q * r) % R) * nb], inv);
                    s.x += t.x;
                    s.y += t.y;
                }
                y[dpad(o + q * ns)] = s;
            }
        }
    }
    __syncthreads();
}

// n-point transform (n a power of two times 1, 3, 5 or 7, whose stage comes
// last) of x, ping-pong with y, both laid out by dpad; the whole block calls it
// after a barrier.  Returns where the result is.
__device__ double2 *dfft(double2 *x, double2 *y, int n, const double2 *__restrict__ roots, bool inv)
{
    int ns = 1;
    while (ns < n) {
        const int rem = n / ns;
        const int R = rem % 4 == 0 ? 4 : rem % 2 == 0 ? 2 : rem % 3 == 0 ? 3 : rem % 5 == 0 ? 5 : 7;
        switch (R) {
        case 2: dstage<2>(x, y, n, ns, roots, inv); break;
        case 3: dstage<3>(x, y, n, ns, roots, inv); break;
        case 4: dstage<4>(x, y, n, ns, roots, inv); break;
        case 5: dstage<5>(x, y, n, ns, roots, inv); break;
        default: dstage<7>(x, y, n, ns, roots, inv); break;
        }
        double2 *t = x;
        x = y;
        y = t;
        ns *= R;
    }
    return x;
}

// roots[m] = exp(-2 pi i m / n)
__global__ void fold_roots_kernel(double2 *roots, int n)
{
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= n)
        return;
    double s, c;
    sincospi(-2.0 * (double)m / (double)n, &s, &c);
    roots[m] = make_double2(c, s);
}

// The response k[t] (times N) of a bank row: the inverse transform of the row.
__device__ double2 *row_response(const float2 *K, int N, double2 *x, double2 *y,
                                 const double2 *__restrict__ rootsN)
{
    for (int i = threadIdx.x; i < N; i += blockDim.x) {
        const float2 v = K[i];
        x[dpad(i)] = make_double2((double)v.x, (double)v.y);
    }
    __syncthreads();
    return dfft(x, y, N, rootsN, true);
}

// A row's support: the smallest h whose taps outside [-2h, 2h) carry no more
// than (2e-7)^2 of the row's energy -- the rounding of the row's own FP32
// values puts about (1e-7)^2 there -- or N/4, the whole circle.  (A response
// cut at its half width ends on values near 1e-2 of its peak, far above.)
constexpr double kSupportTol2 = 4e-14;

__global__ void __launch_bounds__(kFoldThreads)
    fold_support_kernel(const float2 *__restrict__ bank, const long long *__restrict__ src, int N,
                        const double2 *__restrict__ rootsN, int *__restrict__ half)
{
    extern __shared__ double2 dsm2[];
    __shared__ double part[32];
    __shared__ int first[32];
    const double2 *k = row_response(bank + src[blockIdx.x], N, dsm2, dsm2 + dpad(N), rootsN);
    // shell h = 1 .. N/4: the four taps that [-2h, 2h) adds to [-2h+2, 2h-2).
    // Lane l of warp 0 holds shells [l per + 1, (l + 1) per]: sums, then the
    // energy outside each shell from the top down.
    const int shells = N / 4, per = shells / 32;  // N a multiple of 128
    if (threadIdx.x >= 32)
        return;
    const int lane = threadIdx.x;
    auto shell = [&](int h) {
        double e = 0.0;
        const int t[4] = {2 * h - 2, 2 * h - 1, N - 2 * h, N - 2 * h + 1};
        for (int i = 0; i < 4; i++) {
            const double2 v = k[dpad(t[i])];
            e += v.x * v.x + v.y * v.y;
        }
        return e;
    };
    double sum = 0.0;
    for (int i = 1; i <= per; i++)
        sum += shell(lane * per + i);
    part[lane] = sum;
    __syncwarp();
    double total = 0.0, outside = 0.0;
    for (int l = 31; l >= 0; l--) {
        total += part[l];
        if (l > lane)
            outside += part[l];
    }
    // smallest h of this lane whose outside energy is within the bound
    int best = N / 4 + 1;
    for (int i = per; i >= 1; i--) {
        if (!(outside <= kSupportTol2 * total))
            break;
        best = lane * per + i;
        outside += shell(best);
    }
    first[lane] = best;
    __syncwarp();
    if (lane == 0) {
        int h = N / 4;
        for (int l = 31; l >= 0 && first[l] <= N / 4; l--)
            h = first[l];
        half[blockIdx.x] = h;
    }
}

// Whether h is the support of the response k (that fold_support_kernel would
// find); the answer is the whole block's, which calls it after a barrier.
__device__ bool support_is(const double2 *k, int N, int h)
{
    double total = 0.0, out = 0.0, in = 0.0;  // outside [-2h, 2h); outside [-2h+2, 2h-2)
    for (int i = threadIdx.x; i < N; i += blockDim.x) {
        const double2 v = k[dpad(i)];
        const double e = v.x * v.x + v.y * v.y;
        const int t = i < N / 2 ? i : i - N;
        total += e;
        if (t < -2 * h || t >= 2 * h)
            out += e;
        if (t < 2 - 2 * h || t >= 2 * h - 2)
            in += e;
    }
    __shared__ double part[3][32];
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
        total += __shfl_xor_sync(0xffffffffu, total, d);
        out += __shfl_xor_sync(0xffffffffu, out, d);
        in += __shfl_xor_sync(0xffffffffu, in, d);
    }
    if ((threadIdx.x & 31) == 0) {
        part[0][threadIdx.x >> 5] = total;
        part[1][threadIdx.x >> 5] = out;
        part[2][threadIdx.x >> 5] = in;
    }
    __syncthreads();
    total = out = in = 0.0;
    for (int w = 0; w < (int)blockDim.x / 32; w++) {
        total += part[0][w];
        out += part[1][w];
        in += part[2][w];
    }
    const double tol = kSupportTol2 * total;
    return out <= tol && (h == 1 || in > tol);
}

// One folded row per CTA: src[i] the bank row, (N, h) its length and support
// (h < 0: fold the row's own values, L = N/2), off = -1 for a padding row of
// zeros.  A row whose support is not the one expected of it sets *differs, and
// the CTAs that come after leave at once.
__global__ void __launch_bounds__(kFoldThreads)
    fold_rows_kernel(const float2 *__restrict__ bank, const FoldSrc *__restrict__ src, int L,
                     const double2 *__restrict__ roots, const int *__restrict__ roots_at,
                     float2 *__restrict__ out, int *differs)
{
    extern __shared__ double2 dsm2[];
    const FoldSrc f = src[blockIdx.x];
    float2 *o = out + (long long)blockIdx.x * 2 * L;
    const int N = f.N;
    if (f.off < 0) {
        for (int i = threadIdx.x; i < 2 * L; i += blockDim.x)
            o[i] = make_float2(0.f, 0.f);
        return;
    }
    if (__syncthreads_or(differs && *(volatile int *)differs))
        return;
    const float2 *K = bank + f.off;
    double2 *k = nullptr;
    if (f.h >= 0 || f.expect > 0)
        k = row_response(K, N, dsm2, dsm2 + dpad(N), roots + roots_at[N / 128]);
    if (f.expect > 0 && !support_is(k, N, f.expect)) {
        if (threadIdx.x == 0)
            *differs = 1;
        return;
    }
    if (f.h < 0) {
        // A = conj K[k] + conj K[k + L], B = (conj K[k] - conj K[k + L]) e^{+2 pi i k/N}, over N
        const double sc = 1.0 / (double)N;
        for (int k = threadIdx.x; k < L; k += blockDim.x) {
            const float2 k0 = K[k], k1 = K[k + L];
            const double ar = (double)k0.x + (double)k1.x, ai = -(double)k0.y - (double)k1.y;
            const double dr = (double)k0.x - (double)k1.x, di = -(double)k0.y + (double)k1.y;
            double sn, cs;
            sincospi((double)k / (double)L, &sn, &cs);
            o[k] = make_float2((float)(sc * ar), (float)(sc * ai));
            o[k + L] = make_float2((float)(sc * (dr * cs - di * sn)), (float)(sc * (dr * sn + di * cs)));
        }
        return;
    }
    double2 *w = k == dsm2 ? dsm2 + dpad(N) : dsm2;
    // taps of the two parities at j mod L, one after the other (2 L <= N, L a
    // multiple of 128)
    double2 *w2 = w + dpad(L);
    for (int i = threadIdx.x; i < 2 * L; i += blockDim.x)
        w[dpad(i)] = make_double2(0.0, 0.0);
    __syncthreads();
    for (int i = threadIdx.x; i < 4 * f.h; i += blockDim.x) {
        const int t = i - 2 * f.h;  // [-2h, 2h)
        const double2 v = k[dpad(t < 0 ? t + N : t)];
        const int j = t & 1 ? (t + 1) / 2 : t / 2;
        (t & 1 ? w2 : w)[dpad(j < 0 ? j + L : j)] = v;
    }
    __syncthreads();
    const double2 *rl = roots + roots_at[L / 128];
    const double sc = 1.0 / ((double)L * (double)N);
    double2 *a = dfft(w, k, L, rl, false);
    for (int i = threadIdx.x; i < L; i += blockDim.x)
        o[i] = make_float2((float)(sc * a[dpad(i)].x), (float)(-sc * a[dpad(i)].y));
    __syncthreads();
    a = dfft(w2, k + dpad(L), L, rl, false);
    for (int i = threadIdx.x; i < L; i += blockDim.x)
        o[L + i] = make_float2((float)(sc * a[dpad(i)].x), (float)(-sc * a[dpad(i)].y));
}

cudaError_t fold_plan_attrs()
{
    cudaError_t e = smem_attrs(fold_support_kernel, true);
    return e == cudaSuccess ? smem_attrs(fold_rows_kernel, true) : e;
}

cudaError_t launch_fold_roots(double2 *roots, int n, cudaStream_t st)
{
    fold_roots_kernel<<<(n + 255) / 256, 256, 0, st>>>(roots, n);
    return cudaGetLastError();
}

cudaError_t launch_fold_support(const float2 *bank, const long long *src, int nrows, int N,
                                const double2 *rootsN, int *half, cudaStream_t st)
{
    fold_support_kernel<<<nrows, fold_threads(N), 2 * dpad(N) * sizeof(double2), st>>>(bank, src, N, rootsN,
                                                                             half);
    return cudaGetLastError();
}

// maxN: the longest bank row among src; differs: null where no row is checked
cudaError_t launch_fold_rows(const float2 *bank, const FoldSrc *src, int nrows, int L, int maxN,
                             const double2 *roots, const int *roots_at, float2 *out, int *differs,
                             cudaStream_t st)
{
    fold_rows_kernel<<<nrows, fold_threads(maxN), 2 * dpad(maxN) * sizeof(double2), st>>>(
        bank, src, L, roots, roots_at, out, differs);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// The correlation.

// Rows per CTA and CTAs per SM of each half length: rows so that the row
// threads (L/8 each) fill whole warps, CTAs for up to 20 warps an SM within
// 228 KB of shared memory and the registers (about 95) the loop needs.
// Measured at zmax 200, wmax 300 (ns per row and rstep, 64 rsteps a launch):
// 1024 3.41, 768 2.74 (two rows, 3 CTAs: 2.78), 640 2.46 (one row, 6 CTAs:
// 2.67), 512 1.76, 384 1.55.  There is no 896: its 112 threads make whole
// warps only in pairs (7 warps; 3.88 ns, more than the 1024 points it saves),
// and with idle lanes it takes 3.38.
template <int L>
struct FoldShape;
template <> struct FoldShape<256> { static constexpr int Rows = 4, Occ = 5; };
template <> struct FoldShape<384> { static constexpr int Rows = 2, Occ = 6; };
template <> struct FoldShape<512> { static constexpr int Rows = 2, Occ = 5; };
template <> struct FoldShape<640> { static constexpr int Rows = 2, Occ = 4; };
template <> struct FoldShape<768> { static constexpr int Rows = 1, Occ = 6; };
template <> struct FoldShape<1024> { static constexpr int Rows = 1, Occ = 5; };
template <> struct FoldShape<1280> { static constexpr int Rows = 1, Occ = 4; };
template <> struct FoldShape<1536> { static constexpr int Rows = 1, Occ = 3; };
template <> struct FoldShape<1792> { static constexpr int Rows = 1, Occ = 2; };
template <> struct FoldShape<2048> { static constexpr int Rows = 1, Occ = 2; };

constexpr int kFoldTw1 = 8 * 16;  // stage 1's roots W_128^(r k) at [r 8 + k] (every length)

// RowsT: rows per CTA, if other than the length's own launch takes (the
// merged launch's CTAs have 128 threads).
template <int L, int RowsT = FoldShape<L>::Rows>
struct Fold : FoldShape<L> {
    static constexpr int Rows = RowsT;
    static constexpr int R2 = L / 128;
    static constexpr int T = L / 8;  // threads of a row, stage-0 butterflies
    static constexpr int Threads = (T * Rows + 31) / 32 * 32;
    static constexpr bool Whole = Threads == T * Rows;  // no idle threads
    static constexpr int Step2 = Whole ? T : Threads;  // threads of a row in stage 2
    static constexpr bool Pairs = R2 > 8;          // stage 2 by lane pairs
    static constexpr int Plane = fft_buf_len<L>();  // float2 per transform buffer
    // the odd output buffer of the lane-pair form starts 16 banks off the
    // even one, so that the pair's reads never meet
    static constexpr int OddShift = Pairs ? 8 : 0;
    static constexpr int RowBuf = 4 * Plane + OddShift;
    // shared memory: four buffers per row, stage 0's table, the data row
    static constexpr int Smem = (Rows * RowBuf + kFoldTw1 + L) * 8;
    static_assert(L == 128 * R2 && T % 16 == 0 && (Whole || Rows == 1), "[8, 16, R2]");
    static_assert((Rows * RowBuf + kFoldTw1) % 2 == 0, "16-byte aligned data row");
    static_assert((Smem + 1200) * FoldShape<L>::Occ <= 228 * 1024, "shared memory of the SM");
};

int fold_twiddle_size(int L) { return kFoldTw1 + L; }

// Host: the two tables of a half length, forward sign, in double rounded to
// float: stage 1's, then stage 2's W_L^(r k) at [r 128 + k].
void fold_twiddle_table(int L, float2 *out)
{
    const double tau = 2.0 * 3.14159265358979323846264338327950288;
    for (int r = 0; r < 16; r++)
        for (int k = 0; k < 8; k++) {
            const double a = -tau * (double)(r * k) / 128.0;
            out[r * 8 + k] = make_float2((float)cos(a), (float)sin(a));
        }
    for (int r = 0; r < L / 128; r++)
        for (int k = 0; k < 128; k++) {
            const double a = -tau * (double)(r * k) / (double)L;
            out[kFoldTw1 + r * 128 + k] = make_float2((float)cos(a), (float)sin(a));
        }
}

// v (c + i s) with (c, s) the conjugate of a forward table root w: the
// inverse transform's twiddle
__device__ __forceinline__ Cp pmul_conj(const Cp &v, float2 w) { return pmul(v, w.x, -w.y); }

// One CTA: rows [row0, row0 + Rows) of the launch's folded rows, rsteps
// [b0, b1).  Shared memory holds, per row, four padded float2 planes (stage 0
// writes even / odd, stage 1 reads them and writes the other two, stage 2
// reads those; conflict-free for all three stages), so a rstep needs two
// barriers; then stage 0's table and the staged data row, which a bulk copy
// refills for the next rstep as soon as stage 0 has read it.  Stage 2's roots
// are read through L1, shared by the CTAs of an SM.
template <int L, int RowsT = FoldShape<L>::Rows>
__device__ __forceinline__ void fold_cta(const SearchDev &P, const FoldRows &R, const int row0,
                                         const int b0, const int b1)
{
    using F = Fold<L, RowsT>;
    constexpr int T = F::T, R2 = F::R2, NB1 = T / 2, Rows = F::Rows;
    extern __shared__ __align__(16) float2 smf[];
    __shared__ uint64_t s_bar;
    float2 *tws = smf + Rows * F::RowBuf;
    float2 *dsm = tws + kFoldTw1;
    const int rr = Rows == 1 ? 0 : (int)threadIdx.x / T;
    const int tid = Rows == 1 ? (int)threadIdx.x : (int)threadIdx.x - rr * T;
    float2 *bufE = smf + rr * F::RowBuf, *bufO = bufE + F::Plane;
    float2 *outE = bufO + F::Plane, *outO = outE + F::Plane + F::OddShift;

    // the rows of a CTA share one class (padding rows, class -1, follow the
    // class's last row; a CTA of the merged launch may hold only such)
    const int cls = R.map[row0].x;
    if (cls < 0)
        return;
    const FoldClass fc = P.classes[cls];
    const int2 rm = R.map[row0 + rr];
    const float2 *D0 = P.prepped + fc.data_off;
    constexpr unsigned kRowBytes = L * sizeof(float2);
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_u32(&s_bar)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (threadIdx.x == 0 && b0 < b1)
        bulk_row_load(dsm, D0 + (long long)b0 * L, kRowBytes, &s_bar);
    for (int i = threadIdx.x; i < kFoldTw1; i += F::Threads)
        tws[i] = R.tw[i];
    const float2 *tw2 = R.tw + kFoldTw1;
    // the lane pairs (re A, re B), (im A, im B) of this thread's folded values
    float2 kr[8], ki[8];
    {
        const float2 *Fr = R.rows + (long long)(row0 + rr) * 2 * L;
#pragma unroll
        for (int r = 0; r < 8; r++) {
            const int i = F::Whole || tid < T ? tid + T * r : 0;
            const float2 a = Fr[i], bb = Fr[L + i];
            kr[r] = make_float2(a.x, bb.x);
            ki[r] = make_float2(a.y, bb.y);
        }
    }
    const int out0 = fc.out0;
    float *out = P.planes + fc.plane_off + (long long)rm.y * fc.stride;
    const long long plane_size = fc.plane_size;
    const StepDev *steps = P.steps + P.first_rstep * P.nsubs + fc.sub;
    const bool live = rm.x >= 0;
    __syncthreads();

    for (int b = b0; b < b1; b++) {
        const int numrs = live ? steps[(long long)b * P.nsubs].numrs : 0;
        float *outp = out + (long long)b * plane_size;
        if (!bar_wait(&s_bar, (b - b0) & 1) && P.status)
            atomicOr(P.status, kStatusCopy);
        // stage 0: radix 8 of both transforms from the same data values
        if (F::Whole || tid < T) {
            Cp v[8];
#pragma unroll
            for (int r = 0; r < 8; r++) {
                const float2 d = dsm[tid + T * r];
                // d A and d B: (dr ar - di ai, dr ai + di ar) per lane
                v[r].re = fma2(bc(d.x), kr[r], mul2(bc(-d.y), ki[r]));
                v[r].im = fma2(bc(d.x), ki[r], mul2(bc(d.y), kr[r]));
            }
            pdft8(v);
            // stage 1's input twiddles, applied here: element 8 t + r of
            // this stage is input t / (T/16) of stage-1 butterfly
            // (8 t + r) mod (T/2), whose twiddle is W_128^((t / (T/16)) r)
            const float2 *w1 = tws + (tid / (T / 16)) * 8;
#pragma unroll
            for (int r = 1; r < 8; r++)
                v[r] = pmul_conj(v[r], w1[r]);
            const int pd = pad(tid * 8);
#pragma unroll
            for (int r = 0; r < 8; r++) {
                bufE[pad_add(pd, r)] = make_float2(v[r].re.x, v[r].im.x);
                bufO[pad_add(pd, r)] = make_float2(v[r].re.y, v[r].im.y);
            }
        }
        __syncthreads();
        // every thread has read the staged row: start the next rstep's copy
        if (threadIdx.x == 0 && b + 1 < b1) {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            bulk_row_load(dsm, D0 + (long long)(b + 1) * L, kRowBytes, &s_bar);
        }
        // stage 1: radix 16 (Ns = 8), one transform per thread (scalar); its
        // input twiddles were applied by stage 0
        if (F::Whole || tid < T) {
            const bool odd = tid >= NB1;
            const int j = odd ? tid - NB1 : tid;
            const float2 *src = odd ? bufO : bufE;
            float2 *dst = odd ? outO : outE;
            float2 x[16];
            const int pj = pad(j);
            if constexpr (NB1 % 16 == 0) {
#pragma unroll
                for (int r = 0; r < 16; r++)
                    x[r] = src[pad_add(pj, r * NB1)];
            } else {  // NB1 = 8 mod 16: odd r start half a pad group on
                const int pj8 = pad(j + 8);
#pragma unroll
                for (int r = 0; r < 16; r++)
                    x[r] = r & 1 ? src[pad_add(pj8, r * NB1 - 8)] : src[pad_add(pj, r * NB1)];
            }
            Dft<16, +1>::run(x);
            const int pq = pad((j >> 3) * 128 + (j & 7));
#pragma unroll
            for (int r = 0; r < 16; r++)
                dst[pad_add(pq, r * 8)] = x[r];
        }
        __syncthreads();
        // stage 2: radix R2 (Ns = 128)
        if constexpr (!F::Pairs) {
            // butterflies j = tid, tid + T, ... < 128 of both transforms
#pragma unroll
            for (int jb = 0; jb < 128; jb += F::Step2) {
                const int j = jb + tid;
                if (128 % F::Step2 == 0 || j < 128) {
                    Cp v[R2];
                    const int pj = pad(j);
#pragma unroll
                    for (int r = 0; r < R2; r++) {
                        const float2 e = outE[pad_add(pj, r * 128)], o = outO[pad_add(pj, r * 128)];
                        v[r].re = make_float2(e.x, o.x);
                        v[r].im = make_float2(e.y, o.y);
                    }
#pragma unroll
                    for (int r = 1; r < R2; r++)
                        v[r] = pmul_conj(v[r], __ldg(tw2 + r * 128 + j));
                    pdft<R2>(v);
                    // window outputs 2 m and 2 m + 1, m = j + 128 r: the lane
                    // pair of powers is one 8-byte store (numrs is even)
#pragma unroll
                    for (int r = 0; r < R2; r++) {
                        const int kk = 2 * (j + 128 * r - out0);
                        const float2 pw = fma2(v[r].re, v[r].re, mul2(v[r].im, v[r].im));
                        if ((unsigned)kk < (unsigned)numrs)
                            *reinterpret_cast<float2 *>(outp + kk) = pw;
                    }
                }
            }
        } else {
            // item q: butterfly q / 2 of the even (q even) or odd transform
#pragma unroll
            for (int qb = 0; qb < 256; qb += F::Step2) {
                const int q = qb + tid, j = q >> 1;
                if (256 % F::Step2 == 0 || q < 256) {
                    const float2 *src = q & 1 ? outO : outE;
                    float2 x[R2];
                    const int pj = pad(j);
#pragma unroll
                    for (int r = 0; r < R2; r++)
                        x[r] = src[pad_add(pj, r * 128)];
#pragma unroll
                    for (int r = 1; r < R2; r++) {
                        const float2 w = __ldg(tw2 + r * 128 + j);
                        x[r] = cmul(x[r], make_float2(w.x, -w.y));
                    }
                    Dft<R2, +1>::run(x);
#pragma unroll
                    for (int r = 0; r < R2; r++) {
                        const int kk = 2 * (j + 128 * r - out0) + (q & 1);
                        const float pw = fmaf(x[r].x, x[r].x, x[r].y * x[r].y);
                        if ((unsigned)kk < (unsigned)numrs)
                            outp[kk] = pw;
                    }
                }
            }
        }
        // no barrier: the next rstep's stage 0 writes bufE / bufO, last read
        // in stage 1 before the barrier above, and its stage 1 writes outE /
        // outO only after the barrier that follows its stage 0
    }
}

// A plan's own launch: CTA x takes rsteps of chunk x mod ny for row group
// x / ny (the chunks of a group run side by side, so its rows come from HBM
// once).  A batch's correlation launches read the same prepared rows and write
// rows of their own, so each may start on the SMs that the last CTAs of the
// one before leave idle: six trials of 2^21 samples in waves of 96 rsteps,
// zmax 50, wmax 150, 8 harmonics, 124 ms one after the other, 101 ms so.
template <int L>
__global__ void __launch_bounds__(Fold<L>::Threads, Fold<L>::Occ)
    corr_fold_kernel(const __grid_constant__ SearchDev P, const __grid_constant__ FoldRows R,
                     const int ny, const bool first)
{
    if (first)  // of its batch: the rows come from the kernel before
        wait_before();
    let_follow();
    int b0, b1;
    rstep_chunk(P.nb, ny, blockIdx.x % ny, &b0, &b1);
    fold_cta<L>(P, R, (blockIdx.x / ny) * Fold<L>::Rows, b0, b1);
    wait_before();
}

// The merged launch: every row set of up to NP plans that would leave SMs idle
// in a launch of its own -- half lengths to 1024 and the short unfolded
// lengths -- in CTAs of 128 threads.  Small searches are bound by launches of
// a fraction of a wave: at zmax 20, wmax 60, 8 harmonics seven launches took
// 73 us per batch of 8 rsteps one after the other, the merged one takes 28
// (CUDA events); at zmax 100, 16 harmonics, 32 rsteps 176 against 108.
constexpr int kMultiThreads = 128, kMultiOcc = 5;

template <int L>
struct Multi {
    static constexpr int Rows = kMultiThreads / (L / 8);
    using F = Fold<L, Rows>;
    static_assert(F::Threads <= kMultiThreads, "merged CTA");
};

template <int NP>
__global__ void __launch_bounds__(kMultiThreads, kMultiOcc)
    corr_multi_kernel(const __grid_constant__ MultiLaunch<NP> M, const bool first)
{
    if (first)
        wait_before();
    let_follow();
    int j = 0;
    while (j + 1 < M.n && (int)blockIdx.x >= M.seg[j + 1].cta0)
        j++;
    const MultiSeg S = M.seg[j];
    const SearchDev &P = M.P[NP == 1 ? 0 : S.plan];
    const int local = blockIdx.x - S.cta0, g = local / S.ny;
    const FoldRows R = P.rowsets[S.set];
    int b0, b1;
    rstep_chunk(P.nb, S.ny, local % S.ny, &b0, &b1);
    // Warps past the row's own leave at once: the barriers of the row's body
    // count the threads that have not left, and one that waited for the kernel
    // before would hold its CTA's first barrier until that kernel had ended.
    switch (R.len) {
#define JERK_MF(LL)                                                       \
    case LL:                                                              \
        if (threadIdx.x >= Multi<LL>::F::Threads)                         \
            return;                                                       \
        fold_cta<LL, Multi<LL>::Rows>(P, R, g * Multi<LL>::Rows, b0, b1); \
        break;
    JERK_MF(256) JERK_MF(384) JERK_MF(512) JERK_MF(640) JERK_MF(768) JERK_MF(1024)
#undef JERK_MF
#define JERK_MC(NN)                                        \
    case -NN: {                                            \
        if (threadIdx.x >= (FftPlan<NN>::T + 31) / 32 * 32) \
            return;                                        \
        const int2 rm = R.map[g];                          \
        corr_body<NN>(P, rm.x, rm.y, b0, b1);              \
        break;                                             \
    }
    JERK_MC(128) JERK_MC(192) JERK_MC(256) JERK_MC(384)
#undef JERK_MC
    default: break;
    }
    wait_before();
}

// rstep chunks per row group: at least eight waves of CTAs, so that the last,
// partly filled one costs little, as long as a chunk keeps eight rsteps for
// the rows it loads; and two waves whatever the chunk, so that few rows still
// fill the GPU.
static int fold_split(long long groups, int wave, int nb)
{
    const long long tail = std::min<long long>((8LL * wave + groups - 1) / groups, nb / 8);
    const long long fill = std::min<long long>((2LL * wave + groups - 1) / groups, nb);
    return (int)std::max<long long>(1, std::max(tail, fill));
}

template <int L>
struct FoldOps {
    using F = Fold<L>;
    static cudaError_t attrs() { return smem_attrs(corr_fold_kernel<L>, true); }
    static cudaError_t launch(const SearchDev &P, const FoldRows &R, bool first, cudaStream_t st)
    {
        const int groups = R.n / F::Rows;
        const int split = fold_split(groups, sm_count() * F::Occ, P.nb);
        return launch_follow(corr_fold_kernel<L>, (unsigned)(groups * split), F::Threads, F::Smem,
                             st, P, R, split, first);
    }
};

#define JERK_FOLD_DISPATCH(L, call)                                                       \
    switch (L) {                                                                          \
    case 256: return FoldOps<256>::call;                                                  \
    case 384: return FoldOps<384>::call;                                                  \
    case 512: return FoldOps<512>::call;                                                  \
    case 640: return FoldOps<640>::call;                                                  \
    case 768: return FoldOps<768>::call;                                                  \
    case 1024: return FoldOps<1024>::call;                                                \
    case 1280: return FoldOps<1280>::call;                                                \
    case 1536: return FoldOps<1536>::call;                                                \
    case 1792: return FoldOps<1792>::call;                                                \
    case 2048: return FoldOps<2048>::call;                                                \
    default: return cudaErrorInvalidValue;                                                \
    }

cudaError_t fold_attrs(int L) { JERK_FOLD_DISPATCH(L, attrs()) }

cudaError_t launch_corr_fold(int L, const SearchDev &P, const FoldRows &R, bool first,
                             cudaStream_t st)
{
    JERK_FOLD_DISPATCH(L, launch(P, R, first, st))
}

// Row groups and shared memory of one row set in the merged launch; groups 0
// where it does not run there.
static void multi_shape(const FoldRows &R, int *groups, int *smem)
{
    *groups = *smem = 0;
    switch (R.len) {
#define JERK_MS(LL)                                                                \
    case LL:                                                                       \
        *groups = (R.n + Multi<LL>::Rows - 1) / Multi<LL>::Rows;                   \
        *smem = Multi<LL>::F::Smem;                                                \
        break;
    JERK_MS(256) JERK_MS(384) JERK_MS(512) JERK_MS(640) JERK_MS(768) JERK_MS(1024)
#undef JERK_MS
#define JERK_MS(NN)                                                                \
    case -NN:                                                                      \
        *groups = R.n;                                                             \
        *smem = (int)sizeof(float2) * CorrSmem<NN>::value;                         \
        break;
    JERK_MS(128) JERK_MS(192) JERK_MS(256) JERK_MS(384)
#undef JERK_MS
    default: break;
    }
}

bool multi_takes(const FoldRows &R)
{
    int groups, smem;
    multi_shape(R, &groups, &smem);
    return groups > 0;
}

cudaError_t multi_attrs()
{
    cudaError_t e = smem_attrs(corr_multi_kernel<1>, true);
    return e == cudaSuccess ? smem_attrs(corr_multi_kernel<kMaxGroupPlans>, true) : e;
}

template <int NP>
static cudaError_t launch_multi_n(const SearchDev *P, int np, const int (*sets)[2],
                                  const FoldRows *const *rows, int nsets, bool first,
                                  cudaStream_t st)
{
    MultiLaunch<NP> M;
    M.n = nsets;
    for (int i = 0; i < np; i++)
        M.P[i] = P[i];
    // rsteps per CTA: as many as leave four waves of CTAs over all row sets,
    // and two at least (a CTA's set-up costs more than one rstep).  Measured
    // with 1 / 2 / 4 / 6 waves, us per launch: zmax 100, 16 harmonics, 32
    // rsteps 163 / 120 / 108 / 109; zmax 50, wmax 150, 8 harmonics, 32 rsteps
    // 157 / 145 / 142 / 138; zmax 20, wmax 60, 8 rsteps 28.2 at two rsteps a
    // CTA, 33.1 at one.
    const long long wave = (long long)sm_count() * kMultiOcc;
    long long total = 0;
    int smem = 0;
    int groups[NP * kMaxRowSets];
    for (int j = 0; j < nsets; j++) {
        int sm;
        multi_shape(rows[j][0], &groups[j], &sm);
        smem = std::max(smem, sm);
        total += (long long)groups[j] * P[sets[j][0]].nb;
    }
    const int chunk = (int)std::max<long long>(2, total / (4 * wave));
    long long x = 0;
    for (int j = 0; j < nsets; j++) {
        M.seg[j].cta0 = (int)x;
        M.seg[j].plan = (short)sets[j][0];
        M.seg[j].set = (short)sets[j][1];
        M.seg[j].ny = (P[sets[j][0]].nb + chunk - 1) / chunk;
        x += (long long)groups[j] * M.seg[j].ny;
    }
    if (x <= 0 || x >= (1ll << 31))
        return cudaErrorInvalidValue;
    return launch_follow(corr_multi_kernel<NP>, (unsigned)x, kMultiThreads, smem, st, M,
                         first);
}

// Row sets sets[j] = (plan, row set), rows[j] their host copies; P the np
// plans' arguments.
cudaError_t launch_corr_multi(const SearchDev *P, int np, const int (*sets)[2],
                              const FoldRows *const *rows, int nsets, bool first,
                              cudaStream_t st)
{
    if (np < 1 || np > kMaxGroupPlans || nsets < 1 || nsets > np * kMaxRowSets)
        return cudaErrorInvalidValue;
    return np == 1 ? launch_multi_n<1>(P, np, sets, rows, nsets, first, st)
                   : launch_multi_n<kMaxGroupPlans>(P, np, sets, rows, nsets, first, st);
}

// kernel rows a CTA takes, and CTAs of one full wave
int fold_cta_rows(int L)
{
    switch (L) {
#define JERK_FR(LL) case LL: return Fold<LL>::Rows;
    JERK_FR(256) JERK_FR(384) JERK_FR(512) JERK_FR(640) JERK_FR(768)
    JERK_FR(1024) JERK_FR(1280) JERK_FR(1536) JERK_FR(1792) JERK_FR(2048)
#undef JERK_FR
    default: return 1;
    }
}

int fold_wave_ctas(int L)
{
    switch (L) {
#define JERK_FO(LL) case LL: return sm_count() * Fold<LL>::Occ;
    JERK_FO(256) JERK_FO(384) JERK_FO(512) JERK_FO(640) JERK_FO(768)
    JERK_FO(1024) JERK_FO(1280) JERK_FO(1536) JERK_FO(1792) JERK_FO(2048)
#undef JERK_FO
    default: return sm_count();
    }
}

}  // namespace jerk
