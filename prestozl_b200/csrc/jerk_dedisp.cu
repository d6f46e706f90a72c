// Subband dedispersion on the GPU: the two steps prepsubband_cu runs on
// every block of subband data before the DM trials go to the search
// (src/prepsubband_cu.c:1140-1165):
//
//   jerk_downsample_subbands  DownsampDataArray (src/prepsubband_kernels.cu:
//                             23-46; the CPU form src/prepsubband.c:984-1001):
//                             ds[t][s] = (sum over k < bs of in[t bs + k][s]) / bs
//   jerk_dedisp_subbands      getDedisp (src/prepsubband_kernels.cu:48-74; the
//                             CPU form float_dedisp, src/dispersion.c:208-231):
//                             out[dm][t] = sum over s of x[t + off[dm][s]][s],
//                             x = last ++ cur, the previous and the current
//                             block of worklen samples of nsub subbands
//
// Both sum in the reference's order (k, then s ascending) in FP32, so the
// results are bit-exact with the reference's.
//
// The reference's getDedisp runs one thread per (dm, t) and makes nsub
// global loads each nsub floats apart.  Here one CTA takes a tile of T
// samples for a group of G consecutive DMs: for every subband s it stages
// the window of x that the group's DMs read -- T + (largest - smallest
// offset of s in the group) samples -- into shared memory once, transposed
// to [s][t] so that a warp's reads are consecutive words, and every staged
// value serves all G DMs.  Windows of four subbands come in as one 16-byte
// load per sample when nsub is a multiple of 4 and neighbouring subbands'
// windows overlap.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstdint>
#include <cstdio>
#include <vector>

#include "jerk.h"
#include "jerk_async.cuh"
#include "jerk_kernels.cuh"

using jerk::set_error;

namespace {

constexpr int kDdThreads = 256;
constexpr int kDsThreads = 256;
constexpr size_t kSmemPreferred = 100 * 1024;  // two CTAs per SM
constexpr size_t kSmemTwo = 112 * 1024;        // what two CTAs per SM leave each
constexpr size_t kSmemMax = 227 * 1024;

// V: subbands per window load (4: one 16-byte load per sample; 1: one);
// KT: outputs per thread per pass, T / KT apart.
template <int V, int KT>
__global__ void __launch_bounds__(kDdThreads)
dedisp_kernel(const float *__restrict__ cur, const float *__restrict__ last,
              float *__restrict__ out, const int *__restrict__ offsets,
              const int *__restrict__ glo, const int *__restrict__ gbase,
              const int *__restrict__ grel, const int *__restrict__ glen, int worklen, int nsub,
              int ps, int numdms, int G, int T)
{
    extern __shared__ float sm[];
    const int g = blockIdx.y;
    const int t0 = blockIdx.x * T;
    const int d0 = g * G;
    const int gd = min(G, numdms - d0);
    const int *lo_g = glo + (size_t)g * nsub;
    const int *base_g = gbase + (size_t)g * (nsub + 1);
    const int *rel_g = grel + (size_t)g * nsub;
    const int *len_g = glen + (size_t)g * ((nsub + 31) / 32);
    const int total = base_g[nsub];
    float *win = sm;                             // [s][T + span_s], rows at base[s]
    int *pos = (int *)(sm + ((total + 3) & ~3));  // [d][s]: row base + offset - lowest offset
    int *lo = pos + G * ps;           // [s]: the group's lowest offset
    int *base = lo + nsub;            // [s + 1]
    for (int i = threadIdx.x; i < nsub; i += kDdThreads)
        lo[i] = lo_g[i];
    for (int i = threadIdx.x; i <= nsub; i += kDdThreads)
        base[i] = base_g[i];
    __syncthreads();
    for (int i = threadIdx.x; i < gd * nsub; i += kDdThreads) {
        const int d = i / nsub, s = i - d * nsub;
        pos[d * ps + s] = base[s] + offsets[(size_t)(d0 + d) * nsub + s] - lo[s];
    }
    // x[tau] = last[tau] for tau < worklen, cur[tau - worklen] after
    const long long tau_end = 2LL * worklen;
    // (the window stores share the array with lo and base, so the loops
    // below keep what they need of those in registers)
    if (V == 4) {
        // Neighbouring threads take neighbouring quads of subbands of one
        // sample (a whole sector; 16 lines a warp's load instead of 32), and
        // four pairs of quads go out together.  65536 samples x 64 subbands,
        // 512 DMs: 466 us with one load at a time, 425 with four, 414 with
        // the pairs.  The rows' bases put a warp's stores on distinct banks
        // (dd_tables).  What bounds the kernel now is one shared-memory load
        // per addition: the load pipe is at 85 %.
        constexpr int QB = 4;
        const int nq = nsub / 4, par = threadIdx.x & 1;
        for (int q0 = 0; q0 < nq; q0 += 2 * QB) {
            const int len = __ldg(len_g + q0 / 8);
            int plo[QB], rel[QB][4], sw[QB][4], sb[QB][4];
#pragma unroll
            for (int h = 0; h < QB; h++) {
                const int q = q0 + 2 * h + par;
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const int s = 4 * min(q, nq - 1) + j;
                    sb[h][j] = base[s];
                    sw[h][j] = q < nq ? base[s + 1] - sb[h][j] : 0;
                    rel[h][j] = __ldg(rel_g + s);
                }
                plo[h] = lo[4 * min(q, nq - 1)] + rel[h][0];
            }
            for (int i = threadIdx.x >> 1; i < len; i += kDdThreads / 2) {
                float4 v[QB];
#pragma unroll
                for (int h = 0; h < QB; h++) {
                    const int q = q0 + 2 * h + par;
                    v[h] = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (q < nq) {
                        const long long tau = (long long)t0 + plo[h] + i;
                        if (tau < tau_end) {
                            const float *src = tau < worklen ? last + tau * nsub
                                                             : cur + (tau - worklen) * nsub;
                            v[h] = __ldg((const float4 *)(src + 4 * q));
                        }
                    }
                }
#pragma unroll
                for (int h = 0; h < QB; h++) {
                    const float vv[4] = {v[h].x, v[h].y, v[h].z, v[h].w};
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        const int p = rel[h][j] + i;
                        if (p >= 0 && p < sw[h][j])
                            win[sb[h][j] + p] = vv[j];
                    }
                }
            }
        }
    } else {
        // Eight neighbouring threads take eight neighbouring subbands of one
        // sample, four such groups' loads together: a warp along the samples of
        // one subband took a sector for every word (65536 samples x 51
        // subbands, 300 DMs: 436 us, 312 now, with positions by fours).
        constexpr int SB = 4;
        const int c = threadIdx.x & 7;
        for (int s0 = 0; s0 < nsub; s0 += 8 * SB) {
            const int len = __ldg(len_g + s0 / 32);
            int plo[SB], rel[SB], sw[SB], sb[SB];
#pragma unroll
            for (int h = 0; h < SB; h++) {
                const int s = s0 + 8 * h + c, r = min(s, nsub - 1);
                sb[h] = base[r];
                sw[h] = s < nsub ? base[r + 1] - sb[h] : 0;
                rel[h] = __ldg(rel_g + r);
                plo[h] = lo[r] + rel[h];
            }
            for (int i = threadIdx.x >> 3; i < len; i += kDdThreads / 8) {
                float v[SB];
#pragma unroll
                for (int h = 0; h < SB; h++) {
                    const int p = rel[h] + i;
                    v[h] = 0.f;
                    if (p >= 0 && p < sw[h]) {
                        const long long tau = (long long)t0 + plo[h] + i;
                        const int s = s0 + 8 * h + c;
                        if (tau < tau_end)
                            v[h] = tau < worklen ? __ldg(last + tau * nsub + s)
                                                 : __ldg(cur + (tau - worklen) * nsub + s);
                    }
                }
#pragma unroll
                for (int h = 0; h < SB; h++) {
                    const int p = rel[h] + i;
                    if (p >= 0 && p < sw[h])
                        win[sb[h] + p] = v[h];
                }
            }
        }
    }
    __syncthreads();
    // float_dedisp starts each sum at -approx_mean = -0.0f and adds the
    // subbands in ascending order
    const int TQ = T / KT;
    for (int it = threadIdx.x; it < gd * TQ; it += kDdThreads) {
        const int d = it / TQ, tq = it - d * TQ;
        const int *pd = pos + d * ps;
        float v[KT];
#pragma unroll
        for (int k = 0; k < KT; k++)
            v[k] = -0.0f;
        int s = 0;
        const int s4 = V == 4 ? nsub : ps % 4 == 0 ? nsub & ~3 : 0;
        for (; s < s4; s += 4) {  // rows of pos start on 16 bytes
            const int4 p4 = *(const int4 *)(pd + s);
            const int pp[4] = {p4.x, p4.y, p4.z, p4.w};
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const float *w = win + pp[j] + tq;
#pragma unroll
                for (int k = 0; k < KT; k++)
                    v[k] += w[k * TQ];
            }
        }
        for (; s < nsub; s++) {
            const float *w = win + pd[s] + tq;
#pragma unroll
            for (int k = 0; k < KT; k++)
                v[k] += w[k * TQ];
        }
        float *o = out + (size_t)(d0 + d) * worklen + t0;
#pragma unroll
        for (int k = 0; k < KT; k++) {
            const int t = tq + k * TQ;
            if (t0 + t < worklen)
                o[t] = v[k];
        }
    }
}

// F: float, or float4 for four subbands of a sample at a time (nv: subbands
// in units of F).  A thread's sample and subband advance by the grid's stride,
// divided once: with a 64-bit division per output the arithmetic, not memory,
// took its share (65536 samples x 64 subbands from four times as many:
// 10 us less, against 12.5 us that its bytes take).
template <class F>
__global__ void __launch_bounds__(kDsThreads)
downsample_kernel(F *__restrict__ out, const F *__restrict__ in, long long n, int bs, int nv)
{
    const long long step = gridDim.x * (long long)kDsThreads;
    const long long step_t = step / nv;
    const int step_s = (int)(step - step_t * nv);
    long long i = blockIdx.x * (long long)kDsThreads + threadIdx.x;
    long long t = i / nv;
    int s = (int)(i - t * nv);
    for (; i < n; i += step) {
        const F *p = in + t * bs * nv + s;
        float v[sizeof(F) / sizeof(float)] = {};
        for (int k = 0; k < bs; k++) {
            const F x = __ldg(p + (long long)k * nv);
#pragma unroll
            for (int j = 0; j < (int)(sizeof(F) / sizeof(float)); j++)
                v[j] += ((const float *)&x)[j];
        }
        F o;
#pragma unroll
        for (int j = 0; j < (int)(sizeof(F) / sizeof(float)); j++)
            ((float *)&o)[j] = v[j] / (float)bs;
        out[i] = o;
        t += step_t;
        s += step_s;
        if (s >= nv) {
            s -= nv;
            t++;
        }
    }
}

int dd_cuda(cudaError_t e, const char *what)
{
    static thread_local char buf[256];
    snprintf(buf, sizeof buf, "%s: %s", what, cudaGetErrorString(e));
    return set_error(JERK_ECUDA, buf);
}

}  // namespace

struct jerk_dedisperser {
    int worklen = 0, nsub = 0, numdms = 0, G = 1, T = 32, ngroups = 0;
    size_t smem = 0;
    int ps = 0;         // words per row of positions
    bool quads = true;  // staged by 16-byte loads where the blocks allow it
    int *d_offsets = nullptr;  // [numdms][nsub], then the other tables
    const int *d_glo = nullptr, *d_gbase = nullptr, *d_grel = nullptr, *d_glen = nullptr;
    std::vector<int> h_offsets;
};

namespace {

// Per group of G DMs and subband s: the lowest offset and the window rows'
// bases; returns the largest shared-memory footprint over the groups.
// (apart: equal samples of neighbouring quads of subbands lie 16 banks apart,
// and where the subbands are staged singly those of eight neighbours 4, for
// the staging's stores; a few words more per row.
// staged: the words of all groups' rows together.)
size_t dd_tables(const int *off, int numdms, int nsub, int G, int T, std::vector<int> *lo,
                 std::vector<int> *base, bool apart = false, double *staged = nullptr)
{
    if (staged)
        *staged = 0.0;
    const int ngroups = (numdms + G - 1) / G;
    if (lo) {
        lo->assign((size_t)ngroups * nsub, 0);
        base->assign((size_t)ngroups * (nsub + 1), 0);
    }
    size_t worst = 0;
    std::vector<int> low(nsub), high(nsub);
    for (int g = 0; g < ngroups; g++) {
        // (along the rows of the offsets, which the compiler vectorises)
        const int *o = off + (size_t)g * G * nsub;
        std::copy(o, o + nsub, low.begin());
        std::copy(o, o + nsub, high.begin());
        for (int d = g * G + 1; d < std::min(numdms, (g + 1) * G); d++) {
            o += nsub;
            for (int s = 0; s < nsub; s++) {
                low[s] = std::min(low[s], o[s]);
                high[s] = std::max(high[s], o[s]);
            }
        }
        long long total = 0;
        for (int s = 0; s < nsub; s++) {
            const int mn = low[s], mx = high[s];
            if (apart) {
                const long long want = (nsub % 4 ? 4 * (s % 8) : 16 * (s / 4 & 1)) + mn;
                total += (((want - total) % 32) + 32) % 32;
            }
            if (lo) {
                (*lo)[(size_t)g * nsub + s] = mn;
                (*base)[(size_t)g * (nsub + 1) + s] = (int)total;
            }
            total += T + (mx - mn);
        }
        if (lo)
            (*base)[(size_t)g * (nsub + 1) + nsub] = (int)total;
        if (staged)
            *staged += (double)total;
        const size_t bytes = sizeof(float) * (size_t)((total + 3) & ~3LL) +
                             sizeof(int) * ((size_t)G * nsub + 2 * nsub + 1);
        worst = std::max(worst, bytes);
    }
    return worst;
}

// How the windows are staged.  rel[s]: where the loop over a window's samples
// starts, relative to the row's own first sample; len: that loop's length, per
// 32 subbands.  Returns whether four subbands come by one 16-byte load: those
// read from the first row's start to the last row's end, and no more than four
// times the rows' words are read (64 subbands of 1200-1600 MHz, 128 DMs from
// 500, 3.7 times: 160 us, one by one 163; 350-450 MHz from 100, 6.5 times: 318
// and 272).  Neighbours -- a pair of quads, eight single subbands -- share a
// start while that does not lengthen the loop by more than half.
bool dd_staging(const std::vector<int> &lo, const std::vector<int> &base, int ngroups, int nsub,
                std::vector<int> *rel, std::vector<int> *len)
{
    const auto spans = [&](int g, int s0, int n, int *first) {  // of subbands s0 .. s0 + n
        int end = INT_MIN;
        *first = INT_MAX;
        for (int s = s0; s < std::min(s0 + n, nsub); s++) {
            const int l = lo[(size_t)g * nsub + s];
            const int *b = &base[(size_t)g * (nsub + 1) + s];
            *first = std::min(*first, l);
            end = std::max(end, l + b[1] - b[0]);
        }
        return end - *first;
    };
    const int chunks = (nsub + 31) / 32;
    long long quad = 0, rows = 0;
    for (int g = 0; g < ngroups; g++) {
        rows += base[(size_t)g * (nsub + 1) + nsub];
        int first;
        for (int s = 0; s < nsub; s += 4)
            quad += 4LL * spans(g, s, 4, &first);
    }
    const bool quads = nsub % 4 == 0 && quad <= 4 * rows;
    const int unit = quads ? 4 : 1;
    rel->assign((size_t)ngroups * nsub, 0);
    len->assign((size_t)ngroups * chunks, 0);
    for (int g = 0; g < ngroups; g++)
        for (int s0 = 0; s0 < nsub; s0 += 8) {
            int &n = (*len)[(size_t)g * chunks + s0 / 32];
            int first, own = 0;
            for (int s = s0; s < std::min(s0 + 8, nsub); s += unit)
                own = std::max(own, spans(g, s, unit, &first));
            const int all = spans(g, s0, 8, &first);
            const bool near = all <= own + own / 2;
            n = std::max(n, near ? all : own);
            for (int s = s0; s < std::min(s0 + 8, nsub); s++) {
                int start = first;
                if (!near)
                    spans(g, s - s % unit, unit, &start);
                (*rel)[(size_t)g * nsub + s] = start - lo[(size_t)g * nsub + s];
            }
        }
    return quads;
}

// The tiling a dedisperser launches: of the tiles (512, 256, 128 samples) and
// DM groups (64 .. 1) whose shared memory leaves two CTAs per SM, the least
// estimated time.  A staged word costs about 14 times an output's addition of
// one subband (fitted to 65536 samples x 64 subbands, 512 DMs of wide spread:
// groups of 16 and 32 662 and 497 us), and a tile of 128, half as many outputs
// per thread, half again as much per addition (699 us at groups of 32); one
// CTA alone on an SM takes about 0.6 of a pair's time, and 0.7 where a few SMs
// hold a pair (8192 samples x 32 subbands, 300 DMs: 160 CTAs of (64, 256) 37 us,
// 320 of (32, 256) 35).  jerk_dedisp_plan's
// widest tile first loses where only a small group fits it: 96 subbands, 300
// DMs, 20000 samples 703 us at (2, 256), 176 at (32, 128).
void launch_tiling(const int *off, int worklen, int numdms, int nsub, int sms, int *group,
                   int *tile)
{
    double best = 0.0;
    for (int gsz : {64, 32, 16, 8, 4, 2, 1}) {
        const long long ngroups = (numdms + gsz - 1) / gsz;
        if (ngroups > 65535)
            continue;
        double spans = 0.0;  // the windows' words beyond their tile
        const size_t bytes = dd_tables(off, numdms, nsub, gsz, 0, nullptr, nullptr, false, &spans);
        for (int t : {512, 256, 128}) {
            if (bytes + sizeof(float) * (size_t)((nsub * (long long)t + 3) & ~3LL) > kSmemTwo)
                continue;
            const double staged = spans + (double)ngroups * nsub * t;
            const double adds = (double)numdms * t * nsub * (t >= 256 ? 1.0 : 1.5);
            const double ctas = (double)ngroups * ((worklen + t - 1) / t);
            const double cost = (14.0 * staged + adds) / (double)ngroups *
                                std::max(ctas / (2.0 * sms), ctas <= sms ? 0.6 : 0.7);
            if (best == 0.0 || cost < best) {
                best = cost;
                *group = gsz;
                *tile = t;
            }
        }
    }
}

// The offsets table on the host: copied from device memory (as getDedisp
// receives it) when it lives there.
int host_offsets(const int *offsets, long long n, std::vector<int> &buf, const int **out)
{
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, offsets) != cudaSuccess) {
        cudaGetLastError();
        *out = offsets;
        return JERK_OK;
    }
    if (a.type != cudaMemoryTypeDevice && a.type != cudaMemoryTypeManaged) {
        *out = offsets;
        return JERK_OK;
    }
    buf.resize((size_t)n);
    const cudaError_t e = cudaMemcpy(buf.data(), offsets, sizeof(int) * n, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess)
        return dd_cuda(e, "dedisperser offsets");
    *out = buf.data();
    return JERK_OK;
}

}  // namespace

// Host only: checks the sizes and a host offsets table and gives a tiling that
// fits -- the widest tile (256, 128), then the largest DM group, whose
// shared memory fits two CTAs per SM; else tiles of 64 or 32 samples with up
// to 227 KB.
extern "C" int jerk_dedisp_plan(int worklen, int nsub, int numdms, const int *offsets,
                                int *group_dms, int *tile_samples, long long *smem_bytes)
{
    if (!offsets)
        return set_error(JERK_EINVAL, "jerk_dedisp_plan: null pointer");
    if (worklen < 1 || nsub < 1 || numdms < 1)
        return set_error(JERK_EINVAL, "jerk_dedisp_plan: worklen, nsub, numdms must be > 0");
    if ((long long)worklen * nsub * 2 >= (1LL << 40) || (long long)numdms * nsub > INT_MAX)
        return set_error(JERK_EINVAL, "jerk_dedisp_plan: sizes too large");
    for (long long i = 0; i < (long long)numdms * nsub; i++)
        if (offsets[i] < 0 || offsets[i] > worklen)
            return set_error(JERK_EINVAL, "jerk_dedisp_plan: every offset must lie in [0, worklen]");
    int G = 0, T = 0;
    size_t smem = 0;
    for (int t : {256, 128, 64, 32}) {
        const size_t cap = t >= 128 ? kSmemPreferred : kSmemMax;
        for (int gsz : {32, 16, 8, 4, 2, 1}) {
            const size_t b = dd_tables(offsets, numdms, nsub, gsz, t, nullptr, nullptr);
            if (b <= cap) {
                G = gsz;
                T = t;
                smem = b;
                break;
            }
        }
        if (G)
            break;
    }
    if (!G)
        return set_error(JERK_EUNSUPPORTED,
                         "jerk_dedisp_plan: a subband window does not fit in shared memory");
    if ((numdms + G - 1) / G > 65535)
        return set_error(JERK_EUNSUPPORTED, "jerk_dedisp_plan: too many DM groups");
    if (group_dms)
        *group_dms = G;
    if (tile_samples)
        *tile_samples = T;
    if (smem_bytes)
        *smem_bytes = (long long)smem;
    return JERK_OK;
}

extern "C" int jerk_dedisperser_create(jerk_dedisperser **out, int worklen, int nsub, int numdms,
                                       const int *offsets_in)
{
    if (!out || !offsets_in)
        return set_error(JERK_EINVAL, "jerk_dedisperser_create: null pointer");
    *out = nullptr;
    if (worklen < 1 || nsub < 1 || numdms < 1 || (long long)numdms * nsub > INT_MAX)
        return set_error(JERK_EINVAL, "jerk_dedisperser_create: bad sizes");
    std::vector<int> hbuf;
    const int *offsets = nullptr;
    int rc = host_offsets(offsets_in, (long long)numdms * nsub, hbuf, &offsets);
    if (rc != JERK_OK)
        return rc;
    int G = 0, T = 0;
    if ((rc = jerk_dedisp_plan(worklen, nsub, numdms, offsets, &G, &T, nullptr)) != JERK_OK)
        return rc;
    launch_tiling(offsets, worklen, numdms, nsub, jerk::sm_count(), &G, &T);
    jerk_dedisperser *d = new jerk_dedisperser;
    d->worklen = worklen;
    d->nsub = nsub;
    d->numdms = numdms;
    d->G = G;
    d->T = T;
    d->ngroups = (numdms + G - 1) / G;
    std::vector<int> lo, base;
    d->smem = dd_tables(offsets, numdms, nsub, G, T, &lo, &base, true);
    if (d->smem > (T >= 128 ? kSmemTwo : kSmemMax))
        d->smem = dd_tables(offsets, numdms, nsub, G, T, &lo, &base);
    std::vector<int> rel, len;
    d->quads = dd_staging(lo, base, d->ngroups, nsub, &rel, &len);
    // rows of positions on 16 bytes, where that still fits
    const size_t pad = sizeof(int) * (size_t)G * ((4 - nsub % 4) % 4);
    d->ps = nsub;
    if (d->smem + pad <= (T >= 128 ? kSmemTwo : kSmemMax)) {
        d->ps = (nsub + 3) & ~3;
        d->smem += pad;
    }
    d->h_offsets.assign(offsets, offsets + (size_t)numdms * nsub);
    // every table in one array: one allocation and one copy
    std::vector<int> all(d->h_offsets);
    size_t at[4];
    int i = 0;
    for (const std::vector<int> *t : {&lo, &base, &rel, &len}) {
        at[i++] = all.size();
        all.insert(all.end(), t->begin(), t->end());
    }
    cudaError_t e = cudaMalloc(&d->d_offsets, sizeof(int) * all.size());
    if (e == cudaSuccess)
        e = cudaMemcpy(d->d_offsets, all.data(), sizeof(int) * all.size(), cudaMemcpyHostToDevice);
    d->d_glo = d->d_offsets + at[0];
    d->d_gbase = d->d_offsets + at[1];
    d->d_grel = d->d_offsets + at[2];
    d->d_glen = d->d_offsets + at[3];
    for (auto k : {dedisp_kernel<4, 8>, dedisp_kernel<4, 4>, dedisp_kernel<1, 8>,
                   dedisp_kernel<1, 4>})
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)kSmemMax);
    if (e != cudaSuccess) {
        jerk_dedisperser_destroy(d);
        return dd_cuda(e, "jerk_dedisperser_create");
    }
    *out = d;
    return JERK_OK;
}

extern "C" void jerk_dedisperser_destroy(jerk_dedisperser *d)
{
    if (!d)
        return;
    cudaFree(d->d_offsets);
    delete d;
}

extern "C" int jerk_dedisperser_shape(const jerk_dedisperser *d, int *group_dms, int *tile_samples)
{
    if (!d)
        return set_error(JERK_EINVAL, "jerk_dedisperser_shape: null pointer");
    if (group_dms)
        *group_dms = d->G;
    if (tile_samples)
        *tile_samples = d->T;
    return JERK_OK;
}

extern "C" int jerk_dedisperser_matches(const jerk_dedisperser *d, int worklen, int nsub,
                                        int numdms, const int *offsets_in)
{
    if (!d || !offsets_in || d->worklen != worklen || d->nsub != nsub || d->numdms != numdms)
        return 0;
    std::vector<int> hbuf;
    const int *offsets = nullptr;
    if (host_offsets(offsets_in, (long long)numdms * nsub, hbuf, &offsets) != JERK_OK)
        return 0;
    return std::equal(d->h_offsets.begin(), d->h_offsets.end(), offsets) ? 1 : 0;
}

extern "C" int jerk_dedisp_subbands(jerk_dedisperser *d, const float *cur, const float *last,
                                    float *out, void *stream)
{
    if (!d || !cur || !last || !out)
        return set_error(JERK_EINVAL, "jerk_dedisp_subbands: null pointer");
    cudaStream_t st = (cudaStream_t)stream;
    const dim3 grid((d->worklen + d->T - 1) / d->T, d->ngroups);
    const bool quads = d->quads && d->nsub % 4 == 0 && ((uintptr_t)cur % 16) == 0 && ((uintptr_t)last % 16) == 0;
    // 8 outputs per thread on 256-sample tiles (a warp per DM row), else 4
    auto kern = quads ? (d->T >= 256 ? dedisp_kernel<4, 8> : dedisp_kernel<4, 4>)
                      : (d->T >= 256 ? dedisp_kernel<1, 8> : dedisp_kernel<1, 4>);
    kern<<<grid, kDdThreads, d->smem, st>>>(cur, last, out, d->d_offsets, d->d_glo, d->d_gbase,
                                            d->d_grel, d->d_glen, d->worklen, d->nsub, d->ps,
                                            d->numdms, d->G, d->T);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? JERK_OK : dd_cuda(e, "jerk_dedisp_subbands");
}

extern "C" int jerk_downsample_subbands(float *out, const float *in, int worklen, int bs, int nsub,
                                        void *stream)
{
    if (!out || !in)
        return set_error(JERK_EINVAL, "jerk_downsample_subbands: null pointer");
    if (worklen < 1 || bs < 1 || nsub < 1)
        return set_error(JERK_EINVAL, "jerk_downsample_subbands: worklen, bs, nsub must be > 0");
    const bool quads = nsub % 4 == 0 && ((uintptr_t)in % 16) == 0 && ((uintptr_t)out % 16) == 0;
    const int nv = quads ? nsub / 4 : nsub;
    const long long n = (long long)worklen * nv;
    const long long blocks = std::min<long long>((n + kDsThreads - 1) / kDsThreads, 8LL * jerk::sm_count());
    cudaStream_t st = (cudaStream_t)stream;
    if (quads)
        downsample_kernel<<<(int)blocks, kDsThreads, 0, st>>>((float4 *)out, (const float4 *)in, n,
                                                              bs, nv);
    else
        downsample_kernel<<<(int)blocks, kDsThreads, 0, st>>>(out, in, n, bs, nv);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? JERK_OK : dd_cuda(e, "jerk_downsample_subbands");
}
