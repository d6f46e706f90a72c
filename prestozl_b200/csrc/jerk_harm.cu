// Harmonic sum + threshold, fed by a ring of bulk row copies (sm_100a, FP32).
//
// Same sums as harmsum_kernel (jerk_kernels.cu): per fundamental cell (w, z, r)
// the subharmonic powers are added in the reference's order (1/1, 1/2, 1/4,
// 3/4, ...; src/accel_utils.c:1356-1377) and compared with the stage's cutoff
// after each stage, so the hits are bitwise the same.  What differs is how
// the powers arrive.  The gather form waits on HBM latency: all of its loads
// go to L1 lines that mostly miss, and it reached 0.56 of the HBM bandwidth
// with 26 warps of gathers an SM in flight.
//
// Here a CTA walks the fundamental z rows of r tiles of one (w, rstep).
// Subharmonic s's row index steps by 0 or 1 per row, so the row it needs
// changes only now and then (harm_fract of the steps), and one producer warp
// -- lane s for subharmonic s -- copies the tile's piece of each new row into
// the next slot of a ring (cp.async.bulk on the slot's mbarrier), several rows
// ahead of the sums and on into the CTA's next item.  The consumers keep the
// current value of every subharmonic in registers (their r index is fixed per
// tile) and reload only those whose row changed: 8.5 shared-memory loads per
// cell at 16 harmonics instead of 16 gathers.
//
// Measured (CUDA events, us per launch, gathers -> ring): zmax 200, wmax 300,
// 16 harmonics, 64 rsteps 2853 -> 2040 (5.1 TB/s, 0.78 of the measured copy
// bandwidth); 300, 600, 2 harmonics, 16 rsteps 1066 -> 800; 50, 150, 8
// harmonics, 32 rsteps 166 -> 139; 100, 0, 16 harmonics, 32 rsteps 70 -> 59;
// 200, 300, 4 harmonics, 32 rsteps 497 -> 485.  What is left is the consumers'
// instructions (about 50 per cell; the reload's branches are cheaper than
// predicated loads, 2469 us).
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstdint>

#include "jerk_async.cuh"
#include "jerk_kernels.cuh"

namespace jerk {

namespace {

// Fraction of subharmonic s: 1/1, then stage t holds s in [2^(t-1), 2^t) with
// the odd harmonics over 2^t.
constexpr int sub_den(int s)
{
    int n = 1;
    while (n <= s)
        n *= 2;
    return s == 0 ? 1 : n;
}
constexpr int sub_num(int s) { return s == 0 ? 1 : 2 * (s - sub_den(s) / 2) + 1; }

// Shapes.  A bulk copy costs its SM about 55 ns plus its bytes (2 harmonics,
// zmax 300, wmax 600: pieces of 1, 2, 4 and 8 KB took 2352, 1270, 986 and
// 645 us a launch), so a tile spans as much of a row as the registers allow:
// the values and indexes of Q cells per thread.  A row also costs every warp
// its waits and branches, so few subharmonics want few warps with many cells
// (8 harmonics: 31 warps of 2 cells 139 us, 15 of 4 172; 2 harmonics: 8 warps
// of 8 cells, three CTAs an SM, 800 us, 31 of 2 1559).
template <int S>
struct RingShape {  // 16 harmonics: Q = 3, or 2 where that leaves fewer threads idle
    static constexpr int Warps = 15, Q = 3, Occ = 1;
};
template <> struct RingShape<1> { static constexpr int Warps = 8, Q = 8, Occ = 3; };
template <> struct RingShape<2> { static constexpr int Warps = 8, Q = 8, Occ = 3; };
template <> struct RingShape<3> { static constexpr int Warps = 15, Q = 4, Occ = 2; };
template <> struct RingShape<4> { static constexpr int Warps = 31, Q = 2, Occ = 1; };

template <int S, int CellsPerThread>
struct Ring {
    static constexpr int NS = 1 << (S - 1);
    static constexpr int Cols = CellsPerThread;
    static constexpr int Threads = 32 * RingShape<S>::Warps;  // consumers
    static constexpr int All = Threads + 32;
    static constexpr int C = Cols * Threads;  // r cells per tile
    static constexpr int Occ = RingShape<S>::Occ;
    // whether the launch may come before the last correlation CTAs have ended:
    // it saves the gap (zmax 200, wmax 300, 4 harmonics, 96 rsteps 5110 ->
    // 4930 us a pass; zmax 100, 16 harmonics 14.33 -> 14.13 ms), but small
    // CTAs that come in one by one lose more (1 harmonic 2935 -> 3240 us; zmax
    // 300, wmax 600, 2 harmonics 12.34 -> 12.80 ms)
    static constexpr bool Early = Occ < 3;
    // cells of subharmonic s that C fundamental cells can touch: the index
    // grows by at most floor((C - 1) hf) + 1, the piece starts on a multiple
    // of kPlaneAlign cells and ends on one (whole 32-byte sectors)
    static constexpr int width(int s)
    {
        return s == 0 ? C
                      : ((C - 1) * sub_num(s) / sub_den(s) + 2 + 2 * (kPlaneAlign - 1)) /
                            kPlaneAlign * kPlaneAlign;
    }
    static constexpr int off(int s)
    {
        int o = 0;
        for (int i = 0; i < s; i++)
            o += width(i);
        return o;
    }
    static constexpr int Slot = (off(NS) + 31) / 32 * 32;  // floats
    static constexpr int Fit = (226 * 1024 / Occ - 8 * 1024) / (Slot * 4);
    static constexpr int D = Fit < 12 ? Fit : 12;  // slots
    static constexpr int Smem = D * Slot * 4;
    static_assert((Smem + 8192) * Occ <= 228 * 1024 && D >= 3 && C % kPlaneAlign == 0, "ring");
};

// Hits of a CTA, kept in shared memory and appended to the plan's list when
// the CTA is done: hits cluster around a signal (up to every row of a CTA),
// and a global atomic per hit would put its round trip into every such row.
// (The host sorts the keys, so their order here does not matter.)
constexpr int kCtaHits = 512;
struct HitBox {
    unsigned long long key[kCtaHits];
    float pow[kCtaHits];
    unsigned n, base;
};

__device__ __forceinline__ void store_hit(const SearchDev &P, unsigned idx, unsigned long long key,
                                          float v)
{
    if ((long long)idx < P.max_hits) {
        P.hit_keys[idx] = key;
        P.hit_pows[idx] = v;
    }
}

__device__ __noinline__ void ring_hit(const SearchDev &P, HitBox *box, unsigned long long key,
                                      float v)
{
    const unsigned i = atomicAdd(&box->n, 1u);
    if (i < kCtaHits) {
        box->key[i] = key;
        box->pow[i] = v;
    } else {
        store_hit(P, atomicAdd(P.hit_count, 1u), key, v);
    }
}

__device__ __forceinline__ void bar_init(uint64_t *bar, unsigned count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(smem_u32(bar)), "r"(count)
                 : "memory");
}

template <int IMM>
__device__ __forceinline__ float ring_load(unsigned addr)
{
    float v;
    asm volatile("ld.shared.f32 %0, [%1+%2];" : "=f"(v) : "r"(addr), "n"(IMM));
    return v;
}

// x[s][c] of the subharmonics whose row is new in the slot `so` bytes into the
// ring (bits of mask).
template <class R, int s>
struct RingLoads {
    __device__ __forceinline__ static void run(float (&x)[R::NS][R::Cols],
                                               const unsigned (&at)[R::NS][R::Cols], unsigned mask,
                                               unsigned so)
    {
        if constexpr (s == 0) {  // cell c Threads on from this thread's first
            first<0>(x, at[0][0] + so);
        } else if (mask & 1u << s) {
#pragma unroll
            for (int c = 0; c < R::Cols; c++)
                x[s][c] = ring_load<R::off(s) * 4>(at[s][c] + so);
        }
        if constexpr (s + 1 < R::NS)
            RingLoads<R, s + 1>::run(x, at, mask, so);
    }
    template <int c>
    __device__ __forceinline__ static void first(float (&x)[R::NS][R::Cols], unsigned at0)
    {
        x[0][c] = ring_load<c * R::Threads * 4>(at0);
        if constexpr (c + 1 < R::Cols)
            first<c + 1>(x, at0);
    }
};

// One fundamental row: sum, test.
template <int S, class R>
struct RingRow {
    __device__ __forceinline__ static bool sums(const float (&x)[R::NS][R::Cols],
                                                const float (&cut)[S], int c)
    {
        float v = x[0][c];
        bool hit = v > cut[0];
        int s = 1;
#pragma unroll
        for (int st = 1; st < S; st++) {
#pragma unroll
            for (int h = 0; h < (1 << (st - 1)); h++, s++)
                v = __fadd_rn(v, x[s][c]);
            hit |= v > cut[st];
        }
        return hit;
    }
    // The rare path: the same adds again, from the registers, recording each
    // crossing (a first form that read the volumes again took tens of
    // microseconds a call and, in the few CTAs around a pulsar, set the
    // launch's time).
    __device__ __forceinline__ static void record(const SearchDev &P, HitBox *box,
                                                  const float (&x)[R::NS][R::Cols],
                                                  const float (&cut)[S], int c, int b, int ii,
                                                  int jj, int kk, int klast)
    {
        if (kk > klast)  // the tile's threads past its last cell
            return;
        const long long rstep = P.first_rstep + b;
        float v = x[0][c];
        int s = 1;
#pragma unroll
        for (int st = 0; st < S; st++) {
            if (st > 0) {
#pragma unroll
                for (int h = 0; h < (1 << (st - 1)); h++, s++)
                    v = __fadd_rn(v, x[s][c]);
            }
            if (v > cut[st])
                ring_hit(P, box, ((((unsigned long long)rstep * S + st) * P.numw0 + ii) * P.numz0 + jj) *
                                    P.corr_uselen + kk, v);
        }
    }
};

// A plan's work in items: one r tile (of `cells` cells), `nz` fundamental z
// rows of one w row, one rstep.  Item order (rstep, z chunk, w, tile): the
// items in flight at a time lie close together in the volumes (a walk that
// gave each CTA a distant range of its own ran at half the bandwidth), and
// neighbouring w rows read most subharmonic rows together.
struct RingPlan {
    int ntiles, cells, nz, nzc, items;
};

struct RingItem {
    int b, tile, ii, z, zend;
    __device__ __forceinline__ RingItem(const RingPlan &W, const SearchDev &P, int item)
    {
        tile = item % W.ntiles;
        item /= W.ntiles;
        ii = item % P.numw0;
        item /= P.numw0;
        const int zc = item % W.nzc;
        b = item / W.nzc;
        z = zc * W.nz;
        zend = min(z + W.nz, P.numz0);
    }
};

// First cell of subharmonic s's piece of its rows (of the tile from k0 on).
__device__ __forceinline__ int ring_first(const SearchDev &P, int ns, int s, int b, int k0)
{
    const int lo = s == 0 ? k0 : P.rinds[((long long)b * ns + s) * P.corr_uselen + k0];
    const int numrs = P.steps[(P.first_rstep + b) * ns + s].numrs;
    return min(lo, numrs - 1) & ~(kPlaneAlign - 1);
}

// This thread's indexes in every piece of the tile's rows, and the tile's
// first and last cells.
template <class R>
__device__ __forceinline__ void ring_tile(const SearchDev &P, const RingPlan &W, int b, int tile,
                                          unsigned base, unsigned (&at)[R::NS][R::Cols])
{
    const int tid = threadIdx.x;
    const int k0 = tile * W.cells, klast = min(k0 + W.cells, P.corr_uselen) - 1;
#pragma unroll
    for (int s = 1; s < R::NS; s++) {
        const int numrs = P.steps[(P.first_rstep + b) * R::NS + s].numrs;
        const uint16_t *rinds = P.rinds + ((long long)b * R::NS + s) * P.corr_uselen;
        const unsigned a = ring_first(P, R::NS, s, b, k0);
#pragma unroll
        for (int q = 0; q < R::Cols; q++) {
            unsigned ri = rinds[min(k0 + tid + q * R::Threads, klast)];
            if (ri >= (unsigned)numrs) {
                // cannot happen for tables built as the reference builds
                // them; record it and read a cell that exists
                atomicOr(P.status, kStatusRind);
                ri = a;
            }
            at[s][q] = base + 4u * min((unsigned)R::width(s) - 1u, ri - a);
        }
    }
}

// One CTA: items first, first + stride, ... of plan P.
template <int S, class R>
__device__ __forceinline__ void ring_body(const SearchDev &P, const RingPlan &W, const int first,
                                          const int stride)
{
    constexpr int NS = R::NS;
    extern __shared__ __align__(128) float ring[];
    __shared__ uint64_t full[R::D], empty[R::D];
    __shared__ unsigned s_mask[R::D];
    __shared__ int s_dead;
    __shared__ HitBox s_hits;
    const int tid = threadIdx.x;
    if (tid < R::D) {
        bar_init(&full[tid], 1);
        bar_init(&empty[tid], R::Threads / 32);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (tid == 0) {
        s_dead = 0;
        s_hits.n = 0;
    }
    __syncthreads();
    if (tid >= R::Threads) {
        // producer warp: lane s copies subharmonic s's rows
        const int s = tid - R::Threads;
        const bool have = s < NS;
        const SubDev &sd = P.subs[have ? s : 0];
        const uint16_t *zinds = P.zinds + sd.zinds_off;
        const int *wind = P.wind + sd.wind_off;
        const long long wrow = (long long)sd.numz * sd.stride;
        const int rowlen = sd.stride;
        unsigned dst = smem_u32(ring);
        int most = R::C;
#pragma unroll
        for (int i = 0; i < NS; i++)
            if (i == s) {
                dst += 4u * R::off(i);
                most = R::width(i);
            }
        const float *piece = nullptr;
        unsigned bytes = 0;
        int slot = 0, have_b = -1, have_tile = -1;
        unsigned phase = 1;  // a fresh barrier's "previous" phase is complete
        for (int item = first; item < W.items; item += stride) {
            RingItem I(W, P, item);
            if (have && (I.b != have_b || I.tile != have_tile)) {
                have_b = I.b;
                have_tile = I.tile;
                const int k0 = I.tile * W.cells, klast = min(k0 + W.cells, P.corr_uselen) - 1;
                const int numrs = P.steps[(P.first_rstep + I.b) * NS + s].numrs;
                const int a = ring_first(P, NS, s, I.b, k0);
                int last = s == 0 ? klast
                                  : P.rinds[((long long)I.b * NS + s) * P.corr_uselen + klast];
                last = min(last, numrs - 1);
                int n = (last - a) / kPlaneAlign * kPlaneAlign + kPlaneAlign;
                if (n > most || n < kPlaneAlign) {  // cannot happen, as above
                    atomicOr(P.status, kStatusRind);
                    n = kPlaneAlign;
                }
                bytes = 4u * n;
                piece = P.planes + sd.plane_off + (long long)I.b * sd.plane_size + a;
            }
            const float *row0 = have ? piece + (s == 0 ? I.ii : wind[I.ii]) * wrow : nullptr;
            int prev = -1;
            int znext = !have ? -1 : s == 0 ? I.z : zinds[I.z];
          for (; I.z < I.zend; I.z++) {
            const int zi = znext;
            if (have && I.z + 1 < I.zend)
                znext = s == 0 ? I.z + 1 : zinds[I.z + 1];
            const bool fresh = have && zi != prev;
            prev = zi;
            const float *src = row0 + (long long)zi * rowlen;
            const unsigned mask = __ballot_sync(0xffffffffu, fresh);
            const unsigned total = __reduce_add_sync(0xffffffffu, fresh ? bytes : 0u);
            if (!__all_sync(0xffffffffu, bar_wait(&empty[slot], phase) && !*(volatile int *)&s_dead)) {
                if (s == 0)
                    atomicOr(P.status, kStatusSumCopy);
                *(volatile int *)&s_dead = 1;
                // the copies in flight land before the CTA ends (bounded)
                for (int d = 0; d < R::D; d++)
                    bar_wait(&full[d], phase ^ (d < slot ? 1u : 0u));
                return;
            }
            if (s == 0) {
                s_mask[slot] = mask;
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;"
                             :: "r"(smem_u32(&full[slot])), "r"(total) : "memory");
            }
            __syncwarp();
            if (fresh)
                asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes "
                             "[%0], [%1], %2, [%3];"
                             :: "r"(dst + (unsigned)(slot * R::Slot * 4)), "l"(src), "r"(bytes),
                                "r"(smem_u32(&full[slot])) : "memory");
            if (++slot == R::D) {
                slot = 0;
                phase ^= 1u;
            }
          }
        }
        return;
    }

    float x[NS][R::Cols];
    unsigned at[NS][R::Cols];
    float cut[S];
    const unsigned base = smem_u32(ring);
    at[0][0] = base + 4u * tid;  // (a tile starts on a multiple of kPlaneAlign)
#pragma unroll
    for (int st = 0; st < S; st++)
        cut[st] = P.powcut[st];
#pragma unroll
    for (int s = 0; s < NS; s++) {
#pragma unroll
        for (int q = 0; q < R::Cols; q++)
            x[s][q] = 0.f;
    }
    int slot = 0, have_b = -1, have_tile = -1;
    unsigned phase = 0;
    bool ok = true;
#pragma unroll 1
    for (int item = first; item < W.items && ok; item += stride) {
        RingItem I(W, P, item);
        if (I.b != have_b || I.tile != have_tile) {
            have_b = I.b;
            have_tile = I.tile;
            ring_tile<R>(P, W, I.b, I.tile, base, at);
        }
#pragma unroll 1
        for (; I.z < I.zend; I.z++) {
            if (!bar_wait(&full[slot], phase)) {
                *(volatile int *)&s_dead = 1;
                atomicOr(P.status, kStatusSumCopy);
                ok = false;
                break;
            }
            RingLoads<R, 0>::run(x, at, *(volatile unsigned *)&s_mask[slot],
                                 (unsigned)slot * (R::Slot * 4u));
            // every lane has read the slot: one arrival per warp frees it
            __syncwarp();
            if ((tid & 31) == 0)
                asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];"
                             :: "r"(smem_u32(&empty[slot])) : "memory");
            if (++slot == R::D) {
                slot = 0;
                phase ^= 1u;
            }
            bool hit = false;
#pragma unroll
            for (int c = 0; c < R::Cols; c++)
                hit |= RingRow<S, R>::sums(x, cut, c);
            if (hit) {
                const int k0 = I.tile * W.cells, klast = min(k0 + W.cells, P.corr_uselen) - 1;
#pragma unroll
                for (int c = 0; c < R::Cols; c++)
                    RingRow<S, R>::record(P, &s_hits, x, cut, c, I.b, I.ii, I.z,
                                          k0 + tid + c * R::Threads, klast);
            }
        }
    }
    // the CTA's hits to the plan's list (the producers have left or will)
    asm volatile("bar.sync 1, %0;" :: "n"(R::Threads) : "memory");
    const unsigned n = min(s_hits.n, (unsigned)kCtaHits);
    if (n == 0)
        return;
    if (tid == 0)
        s_hits.base = atomicAdd(P.hit_count, n);
    asm volatile("bar.sync 1, %0;" :: "n"(R::Threads) : "memory");
    for (unsigned i = tid; i < n; i += R::Threads)
        store_hit(P, s_hits.base + i, s_hits.key[i], s_hits.pow[i]);
}

template <int S, int Q>
__global__ void __launch_bounds__(Ring<S, Q>::All, Ring<S, Q>::Occ)
    harmsum_ring_kernel(const __grid_constant__ SearchDev P, const __grid_constant__ RingPlan W)
{
    wait_before();
    ring_body<S, Ring<S, Q>>(P, W, blockIdx.x, gridDim.x);
}

// A wave of plans with S stages each.
struct RingGroup {
    GroupLaunch M;
    RingPlan W[kMaxGroupPlans];
};

template <int S, int Q>
__global__ void __launch_bounds__(Ring<S, Q>::All, Ring<S, Q>::Occ)
    harmsum_ring_group_kernel(const __grid_constant__ RingGroup G)
{
    wait_before();
    int i = 0;
    while (i + 1 < G.M.n && (int)blockIdx.x >= G.M.cta0[i + 1])
        i++;
    ring_body<S, Ring<S, Q>>(G.M.P[i], G.W[i], blockIdx.x - G.M.cta0[i],
                             G.M.cta0[i + 1] - G.M.cta0[i]);
}

// r tiles of at most `most` cells, evenly sized; z rows per item for `ctas`
// CTAs: the fewest rows a CTA ends up with, where an item costs about two
// rows more than it has (its first row brings every subharmonic's).
RingPlan ring_plan(const SearchDev &P, int most, int ctas)
{
    RingPlan W;
    const int uselen = P.corr_uselen;
    W.ntiles = (uselen + most - 1) / most;
    W.cells = ((uselen + W.ntiles - 1) / W.ntiles + kPlaneAlign - 1) / kPlaneAlign * kPlaneAlign;
    W.ntiles = (uselen + W.cells - 1) / W.cells;
    const long long lines = (long long)P.nb * W.ntiles * P.numw0;
    long long best = LLONG_MAX;
    W.nz = P.numz0;
    for (int n = 1; n <= P.numz0; n++) {
        const int nz = (P.numz0 + n - 1) / n;
        if (nz < 4 && n > 1)
            break;
        const long long items = lines * ((P.numz0 + nz - 1) / nz);
        const long long cost = (items + ctas - 1) / ctas * (nz + 2);
        if (cost < best && items < (1 << 30)) {
            best = cost;
            W.nz = nz;
        }
    }
    W.nzc = (P.numz0 + W.nz - 1) / W.nz;
    W.items = (int)(lines * W.nzc);
    return W;
}

template <int S>
struct RingOps {
    static constexpr int QMax = RingShape<S>::Q;
    static cudaError_t attrs()
    {
        cudaError_t e = smem_attrs(harmsum_ring_kernel<S, QMax>, true);
        if constexpr (S == 5) {
            if (e == cudaSuccess)
                e = smem_attrs(harmsum_ring_kernel<S, 2>, true);
        }
        return e == cudaSuccess ? smem_attrs(harmsum_ring_group_kernel<S, QMax>, true) : e;
    }
    template <int Q>
    static cudaError_t launch_q(const SearchDev &P, const RingPlan &W, cudaStream_t st)
    {
        using R = Ring<S, Q>;
        const int x = std::min(W.items, sm_count() * R::Occ);
        if (R::Early)
            return launch_follow(harmsum_ring_kernel<S, Q>, (unsigned)x, R::All, R::Smem, st, P, W);
        harmsum_ring_kernel<S, Q><<<x, R::All, R::Smem, st>>>(P, W);
        return cudaGetLastError();
    }
    static cudaError_t launch(const SearchDev &P, cudaStream_t st)
    {
        const int wave = sm_count() * Ring<S, QMax>::Occ;
        const RingPlan w = ring_plan(P, Ring<S, QMax>::C, wave);
        if constexpr (S == 5) {
            // the fewer idle threads; on a tie the wider tile
            const RingPlan w2 = ring_plan(P, Ring<S, 2>::C, wave);
            if (2 * w2.ntiles < QMax * w.ntiles)
                return launch_q<2>(P, w2, st);
        }
        return launch_q<QMax>(P, w, st);
    }
    static cudaError_t launch_group(const GroupLaunch &M, cudaStream_t st)
    {
        using R = Ring<S, QMax>;
        RingGroup G;
        G.M = M;
        // CTAs in proportion to the plans' tile rows, what is left over to
        // whichever has the most rows per CTA
        const int wave = sm_count() * R::Occ;
        double work[kMaxGroupPlans], all = 0.0;
        int share[kMaxGroupPlans], dealt = 0;
        for (int i = 0; i < M.n; i++) {
            const SearchDev &P = M.P[i];
            work[i] = (double)P.nb * P.numw0 * P.numz0 * ((P.corr_uselen + R::C - 1) / R::C);
            all += work[i];
        }
        for (int i = 0; i < M.n; i++)
            dealt += share[i] = std::max(1, (int)(work[i] / all * wave));
        for (; dealt < wave; dealt++) {
            int most = 0;
            for (int i = 1; i < M.n; i++)
                if (work[i] * share[most] > work[most] * share[i])
                    most = i;
            share[most]++;
        }
        int x = 0;
        for (int i = 0; i < M.n; i++) {
            G.W[i] = ring_plan(M.P[i], R::C, share[i]);
            G.M.cta0[i] = x;
            x += std::min(G.W[i].items, share[i]);
        }
        G.M.cta0[M.n] = x;
        if (R::Early)
            return launch_follow(harmsum_ring_group_kernel<S, QMax>, (unsigned)x, R::All, R::Smem,
                                 st, G);
        harmsum_ring_group_kernel<S, QMax><<<x, R::All, R::Smem, st>>>(G);
        return cudaGetLastError();
    }
};

}  // namespace

#define JERK_RING_DISPATCH(S, call)              \
    switch (S) {                                 \
    case 1: return RingOps<1>::call;             \
    case 2: return RingOps<2>::call;             \
    case 3: return RingOps<3>::call;             \
    case 4: return RingOps<4>::call;             \
    case 5: return RingOps<5>::call;             \
    default: return cudaErrorInvalidValue;       \
    }

cudaError_t harm_ring_attrs(int nstages) { JERK_RING_DISPATCH(nstages, attrs()) }

// Whether the ring is the faster form for a batch whose volumes take `bytes`:
// below about 48 MB a launch is latency, and the gathers' chain is the shorter
// (25 MB: 17.8 us against 19.4; 8 MB: 13.5 against 14.9; 134 MB: 69.9 against
// 58.9).
bool harm_ring_wins(double bytes) { return bytes >= 48e6; }

cudaError_t launch_harm_ring(const SearchDev &P, cudaStream_t st)
{
    JERK_RING_DISPATCH(P.nstages, launch(P, st))
}

// Every plan of M must have nstages stages.
cudaError_t launch_harm_ring_group(const GroupLaunch &M, int nstages, cudaStream_t st)
{
    if (M.n < 1 || M.n > kMaxGroupPlans)
        return cudaErrorInvalidValue;
    JERK_RING_DISPATCH(nstages, launch_group(M, st))
}

}  // namespace jerk
