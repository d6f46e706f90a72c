// Host side of libjerk: search geometry, the device plan, the batch loop,
// candidate assembly, and the C ABI of include/jerk.h.
//
// The plan owns every device buffer of one search configuration (kernel bank,
// twiddles, lookup tables, per-batch volumes, hit buffer) so that a search
// allocates nothing per rstep (the reference allocates and frees per call,
// src/accel_utils_cu.c:451-455, 591-611).
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <functional>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <string>
#include <thread>
#include <vector>

#include "jerk.h"
#include "jerk_async.cuh"
#include "jerk_kernels.cuh"

namespace jerk {
size_t prep_smem_bytes(int fftlen, bool folded);
cudaError_t prep_attrs(int maxfft);
cudaError_t launch_prep(const SearchDev &P, int maxfft, size_t smem, cudaStream_t st);
cudaError_t corr_attrs(int fftlen);
cudaError_t launch_corr(const SearchDev &P, int fftlen, const RowGroup &G, int rows,
                        cudaStream_t st);
cudaError_t harmsum_attrs(int nstages, int harm_mode);
cudaError_t launch_harmsum(const SearchDev &P, const HarmTma &T, bool prefetch, cudaStream_t st);
cudaError_t harm_ring_attrs(int nstages);
cudaError_t launch_harm_ring(const SearchDev &P, cudaStream_t st);
bool harm_ring_wins(double bytes);
cudaError_t launch_harm_ring_group(const GroupLaunch &M, int nstages, cudaStream_t st);
cudaError_t launch_harmsum_tma(const SearchDev &P, const HarmTma &T, int zt, cudaStream_t st);
size_t harmsum_tma_smem_bytes(const HarmTma &T, int nsubs, int numz0);
bool fftlen_supported(int n);
cudaError_t launch_prep_group(GroupLaunch M, int maxfft, size_t smem, cudaStream_t st);
cudaError_t launch_harmsum_group(GroupLaunch M, int nstages, cudaStream_t st);
cudaError_t launch_wait_probe(unsigned int *status, bool sum, cudaStream_t st);
cudaError_t fold_plan_attrs();
cudaError_t launch_fold_roots(double2 *roots, int n, cudaStream_t st);
cudaError_t launch_fold_support(const float2 *bank, const long long *src, int nrows, int N,
                                const double2 *rootsN, int *half, cudaStream_t st);
cudaError_t launch_fold_rows(const float2 *bank, const FoldSrc *src, int nrows, int L, int maxN,
                             const double2 *roots, const int *roots_at, float2 *out, int *differs,
                             cudaStream_t st);
int fold_twiddle_size(int L);
void fold_twiddle_table(int L, float2 *out);
cudaError_t fold_attrs(int L);
cudaError_t launch_corr_fold(int L, const SearchDev &P, const FoldRows &R, bool first,
                             cudaStream_t st);
bool multi_takes(const FoldRows &R);
cudaError_t multi_attrs();
cudaError_t launch_corr_multi(const SearchDev *P, int np, const int (*sets)[2],
                              const FoldRows *const *rows, int nsets, bool first,
                              cudaStream_t st);
int fold_cta_rows(int L);
int fold_wave_ctas(int L);
int harmsum_wave_ctas(int nstages);
int fft_twiddle_size(int N);
void fft_twiddle_table(int N, float2 *out);
cudaError_t launch_bank_response(const BankRow *rows, int nrows, int max_pts, float2 *bank,
                                 cudaStream_t st);
cudaError_t launch_bank_fft_any(int N, const BankRow *rows, int first, int count, const float2 *tw,
                                int twoff, float2 *bank, cudaStream_t st);
}  // namespace jerk

using namespace jerk;

// ---------------------------------------------------------------------------
// errors

static thread_local std::string g_err;

static int fail(int code, const std::string &msg)
{
    // an error that has been reported (an allocation that did not fit) is not
    // the next launch's
    if (code == JERK_ECUDA)
        cudaGetLastError();
    g_err = msg;
    return code;
}

static int cuda_fail(cudaError_t e, const char *what)
{
    return fail(JERK_ECUDA, std::string(what) + ": " + cudaGetErrorString(e));
}

#define JERK_CUDA(call)                                  \
    do {                                                 \
        cudaError_t e_ = (call);                         \
        if (e_ != cudaSuccess)                           \
            return cuda_fail(e_, #call);                 \
    } while (0)

extern "C" const char *jerk_last_error(void) { return g_err.c_str(); }

// Error reporting for the entry points compiled in other files.
int jerk::set_error(int code, const char *msg) { return fail(code, msg); }
extern "C" void jerk_free(void *p) { free(p); }

// ---------------------------------------------------------------------------
// Reference index arithmetic (src/accel_utils.c:36-97), host side.

static constexpr double kDR = 0.5;
static constexpr int kRDR = 2;
static constexpr int kDZ = 2;
static constexpr double kRDZ = 0.5;
static constexpr int kDW = 20;
static constexpr double kRDW = 0.05;
static constexpr double kDblCorrect = 1e-14;
static constexpr double kClosestR = 15.0;

static inline int nearest_int(double x) { return (int)(x < 0 ? x - 0.5 : x + 0.5); }
static inline double calc_required_r(double hf, double rfull) { return rint(kRDR * rfull * hf) * kDR; }
static inline int calc_required_z(double hf, double zfull) { return nearest_int(kRDZ * zfull * hf) * kDZ; }
static inline int calc_required_w(double hf, double wfull) { return nearest_int(kRDW * wfull * hf) * kDW; }
static inline int index_from_z(double z, double loz) { return (int)((z - loz) * kRDZ + kDblCorrect); }
static inline int index_from_w(double w, double low) { return (int)((w - low) * kRDW + kDblCorrect); }

// src/responses.c:27-84 (LOWACC)
static int z_resp_halfwidth(double z) { return (int)(0.5 * 1.1 * fabs(z)) + 16; }
static int w_resp_halfwidth(double z, double w)
{
    if (fabs(w) < 1.0e-7)
        return z_resp_halfwidth(z);
    const double r0 = 0.5 * (w / 6.0 - z), r1 = 0.5 * (w / 6.0 + z);
    double maxdev = fabs(r0) > fabs(r1) ? fabs(r0) : fabs(r1);
    const double u_ext = 0.5 - z / w;
    if (u_ext > 0.0 && u_ext < 1.0) {
        const double z0 = z - w / 2.0;
        const double r_ext = 0.5 * w * u_ext * u_ext + z0 * u_ext + r0;
        maxdev = fabs(r_ext) > maxdev ? fabs(r_ext) : maxdev;
    }
    return (int)(1.1 * maxdev) + 16;
}

int jerk::w_resp_halfwidth_lowacc(double z, double w) { return w_resp_halfwidth(z, w); }

static long long next2_to_n(long long x)
{
    long long n = 1;
    while (n < x)
        n <<= 1;
    return n;
}

// src/corr_prep.c:3-35
static int next_good_fftlen(int N)
{
    static const int lens[17] = {128, 192, 256, 384, 512, 768, 1024, 1280, 2048,
                                 4096, 5120, 7680, 10240, 12288, 15360, 16384, 25600};
    int ii = 0;
    if (N <= lens[0])
        return lens[0];
    if (N > lens[16])
        return (int)next2_to_n(N);
    while (N > lens[ii])
        ii++;
    return lens[ii];
}

static int fftlen_from_kernwidth(int kw)
{
    if (kw < 6) return 128;
    if (kw < 52) return 256;
    if (kw < 67) return 512;
    if (kw < 378) return 1024;
    if (kw < 664) return 2048;
    if (kw < 1672) return 4096;
    if (kw < 3015) return 10240;
    if (kw < 3554) return 15360;
    if (kw < 6000) return 25600;
    return (int)next2_to_n(kw * 5);
}

// ---------------------------------------------------------------------------
// Statistics: candidate_sigma / power_for_sigma (src/characteristics.c:400-705)
// for the integer numsum the search uses, written from the published
// formulas the reference's code evaluates.

// ln Gamma(a, z), the upper incomplete gamma function, for large z by its
// asymptotic series (Abramowitz & Stegun 6.5.32):
//   Gamma(a, z) ~ z^(a-1) e^(-z) sum_k (a-1)(a-2)...(a-k) / z^k,
// summed until a term drops below 1e-15.
static double log_upper_gamma_large_z(double a, double z)
{
    double sum = 1.0, term = 1.0;
    for (int k = 1; fabs(term) > 1e-15; k++) {
        term *= (a - k) / z;
        sum += term;
    }
    return (a - 1.0) * log(z) - z + log(sum);
}

// ln Gamma(z) by Stirling's series (Abramowitz & Stegun 6.1.41), to the
// z^-7 term: (z - 1/2) ln z - z + ln(2 pi)/2 + 1/(12 z) - 1/(360 z^3)
// + 1/(1260 z^5) - 1/(1680 z^7).
static double log_gamma_stirling(double z)
{
    const double half_log_2pi = 0.91893853320467274178;
    const double u = 1.0 / (z * z);
    const double series =
        (((-1.0 / 1680.0) * u + 1.0 / 1260.0) * u - 1.0 / 360.0) * u + 1.0 / 12.0;
    return (z - 0.5) * log(z) - z + half_log_2pi + series / z;
}

// Q(a, x) for integer a: exp(-x) sum_{n<a} x^n / n!
static double q_gamma_int(int a, double x)
{
    if (x <= 0.0)
        return 1.0;
    double t = exp(-x), sum = t;
    for (int n = 1; n < a; n++) {
        t = t * x / n;
        sum += t;
    }
    return sum;
}

static double chi2_logp(double chi2, double dof)
{
    if (chi2 <= 0.0)
        return -INFINITY;
    if (chi2 / dof > 15.0 || (dof > 150 && chi2 / dof > 6.0))
        return log_upper_gamma_large_z(0.5 * dof, 0.5 * chi2) -
               log_gamma_stirling(0.5 * dof);
    return log(q_gamma_int((int)(0.5 * dof + 0.5), 0.5 * chi2));
}

// The rational approximation of the upper normal quantile, Abramowitz &
// Stegun 26.2.23, on log p for p <= 1/2 (|error| < 4.5e-4)
static double normal_quantile_rational(double logp)
{
    const double t = sqrt(-2.0 * logp);
    const double num = 2.515517 + t * (0.802853 + t * 0.010328);
    const double den = 1.0 + t * (1.432788 + t * (0.189269 + t * 0.001308));
    return t - num / den;
}

// x with 1 - Phi(x) = q for 0 < q < 1/2, full double precision: Newton steps
// from the rational approximation (three square its error, up to x = 35, away
// below the last bit; the fourth settles rounding).  A search has thousands
// of hits, and a bisection with 55 erfc calls each took 2 us a hit.
static double upper_normal_quantile(double logq, double q)
{
    double x = normal_quantile_rational(logq);
    for (int it = 0; it < 4; it++) {
        const double dens = exp(-0.5 * x * x) / sqrt(2.0 * M_PI);
        x += (0.5 * erfc(x / M_SQRT2) - q) / dens;
    }
    return x;
}

static double equivalent_gaussian_sigma(double logp)
{
    if (logp < -600.0)
        return std::max(0.0, normal_quantile_rational(logp));
    const double q = exp(logp);
    /* p = 1 - q < 0 has no normal quantile: the reference's cdfnor2 gives
       NaN there; at q >= 1/2 the quantile is not positive, which is 0 */
    if (q > 1.0)
        return NAN;
    if (!(q < 0.5))
        return 0.0;
    const double x = upper_normal_quantile(logp, q);
    return x < 0.0 ? 0.0 : x;
}

extern "C" double jerk_candidate_sigma(double power, int numsum, double numtrials)
{
    if (power <= 0.0)
        return 0.0;
    double logp = chi2_logp(2.0 * power, 2.0 * numsum);
    logp += log(numtrials);
    return equivalent_gaussian_sigma(logp);
}

extern "C" double jerk_power_for_sigma(double sigma, int numsum, double numtrials)
{
    const double q = 0.5 * erfc(sigma / M_SQRT2) / numtrials;
    const double logq = log(q);
    double lo = 0.0, hi = 1.0;
    while (log(q_gamma_int(numsum, hi)) > logq)
        hi *= 2.0;
    for (int it = 0; it < 200; it++) {
        const double mid = 0.5 * (lo + hi);
        if (log(q_gamma_int(numsum, mid)) > logq)
            lo = mid;
        else
            hi = mid;
        if (hi - lo <= 1e-15 * hi)
            break;
    }
    return 0.5 * (lo + hi);
}

// ---------------------------------------------------------------------------
// Geometry (the sizing part of create_accelobs, src/accel_utils.c:1795-2004)

extern "C" int jerk_obs_from_params(long long numbins, long long N, double dt, int zmax, int wmax,
                                    int wmax_given, int numharm, float sigma, double flo,
                                    double fhi, jerk_obs *obs, int *fftlen_out,
                                    int *maxkernlen_out)
{
    if (!obs || numbins < 2 || dt <= 0.0)
        return fail(JERK_EINVAL, "jerk_obs_from_params: bad arguments");
    if (numharm != 1 && numharm != 2 && numharm != 4 && numharm != 8 && numharm != 16 &&
        numharm != 32)
        return fail(JERK_EINVAL, "numharm must be a power of two <= 32");
    memset(obs, 0, sizeof(*obs));
    if (zmax % kDZ)
        zmax = (zmax / kDZ + 1) * kDZ;
    const double T = dt * (double)N;
    obs->numbins = numbins;
    obs->lobin = 0;
    int stages = 0;
    while ((1 << stages) < numharm)
        stages++;
    obs->numharmstages = stages + 1;
    obs->numz = (zmax / kDZ) * 2 + 1;
    double whi = 0.0;
    int numw = 0;
    if (wmax_given) {
        if (wmax % kDW)
            wmax = (wmax / kDW + 1) * kDW;
        whi = wmax;
        numw = (wmax / kDW) * 2 + 1;
        if (wmax == 0)
            numw = 0;
    } else {
        wmax = 0;
    }
    obs->numw = numw;
    obs->zlo = -zmax;
    obs->wlo = -whi;
    obs->rlo = floor(flo * T);
    if (obs->rlo < obs->lobin)
        obs->rlo = obs->lobin;
    if (obs->rlo > numbins - 1)
        return fail(JERK_EINVAL, "flo is above the highest frequency");
    obs->highestbin = numbins - 1;
    obs->highestbin = (long long)ceil(fhi * T);
    if (obs->highestbin > numbins - 1)
        obs->highestbin = numbins - 1;
    const double rhi = (double)obs->highestbin;
    if (obs->highestbin < obs->rlo)
        return fail(JERK_EINVAL, "fhi is below flo");
    const double dz = kDZ, dw = wmax_given ? kDW : 0.0;
    for (int ii = 0; ii < obs->numharmstages; ii++) {
        const int h = 1 << ii;
        if (obs->numz == 1 && obs->numw == 0)
            obs->numindep[ii] = (long long)((rhi - obs->rlo) / h);
        else if (obs->numz > 1 && obs->numw == 0)
            obs->numindep[ii] = (long long)((rhi - obs->rlo) * (obs->numz + 1) * (dz / 6.95) / h);
        else
            obs->numindep[ii] = (long long)((rhi - obs->rlo) * (obs->numz + 1) * (dz / 6.95) *
                                            (obs->numw + 1) * (dw / 44.2) / h);
        obs->powcut[ii] = (float)jerk_power_for_sigma(sigma, h, (double)obs->numindep[ii]);
    }
    const int maxkernlen = 2 * 2 * w_resp_halfwidth(zmax, whi);
    int fftlen = fftlen_from_kernwidth(maxkernlen);
    if (fftlen < 2048)
        fftlen = 2048;
    int uselen = fftlen - maxkernlen;
    if (uselen % kRDR)
        uselen = uselen / kRDR * kRDR;
    obs->corr_uselen = uselen;
    if (fftlen_out)
        *fftlen_out = fftlen;
    if (maxkernlen_out)
        *maxkernlen_out = maxkernlen;
    return JERK_OK;
}

extern "C" int jerk_subharm_count(int numharmstages)
{
    return numharmstages < 1 ? 0 : (1 << (numharmstages - 1));
}

// Bank order (src/accel_utils.c:236-282): (1/1), (1/2), (1/4), (3/4), (1/8), ...
static void index_to_harm(int index, int *numharm, int *harmnum)
{
    if (index == 0) {
        *numharm = 1;
        *harmnum = 1;
        return;
    }
    int stage = 1;
    while (index >= (1 << stage))
        stage++;
    // stage s holds subharmonics 2^(s-1) .. 2^s - 1, harm = 2*(index - 2^(s-1)) + 1
    *numharm = 1 << stage;
    *harmnum = 2 * (index - (1 << (stage - 1))) + 1;
}

extern "C" int jerk_subharm_sizes(const jerk_obs *obs, int fftlen, int index, jerk_subharm *out)
{
    if (!obs || !out || index < 0 || index >= jerk_subharm_count(obs->numharmstages))
        return fail(JERK_EINVAL, "jerk_subharm_sizes: bad index");
    int nh, hn;
    index_to_harm(index, &nh, &hn);
    const double hf = (double)hn / (double)nh;
    const int zmax = (int)-obs->zlo, wmax = (int)-obs->wlo;
    memset(out, 0, sizeof(*out));
    out->numharm = nh;
    out->harmnum = hn;
    out->zmax = calc_required_z(hf, zmax);
    out->wmax = calc_required_w(hf, wmax);
    out->numz = (out->zmax / kDZ) * 2 + 1;
    out->numw = (out->wmax / kDW) * 2 + 1;
    if (nh == 1 && hn == 1) {
        out->fftlen = fftlen;
    } else {
        const int bins_needed = (int)ceil(obs->corr_uselen * hf) + 2;
        const int end_effects = 2 * 2 * w_resp_halfwidth(calc_required_z(hf, zmax),
                                                         calc_required_w(hf, wmax));
        out->fftlen = next_good_fftlen(bins_needed + end_effects);
    }
    out->halfwidth = w_resp_halfwidth((double)-out->zmax, (double)-out->wmax);
    out->kernels = nullptr;
    return JERK_OK;
}

// ---------------------------------------------------------------------------
// Candidate list: insert_new_accelcand (src/accel_utils.c:382-480).
//
// The reference walks a linked list from its head to the first node with
// r >= rr (or to the last node).  The list is not always sorted -- when the
// walk ends at the last node and only the node before it is overwritten, a
// larger r lands before a smaller one -- so the walk cannot be replaced by a
// binary search.  CandList keeps the list in blocks with each block's max r:
// "first node with r >= rr" skips whole blocks whose max is below rr, which
// gives the walk's exact answer in O(sqrt n) instead of O(n).

namespace {

class CandList {
  public:
    struct Pos {
        size_t b, o;
    };

    bool empty() const { return n_ == 0; }

    // the reference walk's stopping node
    Pos walk(double rr) const
    {
        for (size_t b = 0; b < blocks_.size(); b++) {
            if (blocks_[b].maxr >= rr) {
                const auto &v = blocks_[b].v;
                for (size_t o = 0; o < v.size(); o++)
                    if (!(v[o].r < rr))
                        return {b, o};
            }
        }
        return last();
    }
    Pos last() const { return {blocks_.size() - 1, blocks_.back().v.size() - 1}; }
    bool is_last(Pos p) const { return p.b == blocks_.size() - 1 && p.o == blocks_[p.b].v.size() - 1; }
    bool has_prev(Pos p) const { return p.o > 0 || p.b > 0; }
    Pos prev(Pos p) const { return p.o > 0 ? Pos{p.b, p.o - 1} : Pos{p.b - 1, blocks_[p.b - 1].v.size() - 1}; }
    const jerk_cand &at(Pos p) const { return blocks_[p.b].v[p.o]; }

    void push_back(const jerk_cand &c)
    {
        if (blocks_.empty() || blocks_.back().v.size() >= 2 * kBlock)
            blocks_.push_back(Block{});
        Block &B = blocks_.back();
        B.v.push_back(c);
        B.maxr = B.v.size() == 1 ? c.r : std::max(B.maxr, c.r);
        n_++;
    }
    void replace(Pos p, const jerk_cand &c)
    {
        Block &B = blocks_[p.b];
        B.v[p.o] = c;
        remax(B);
    }
    void insert_before(Pos p, const jerk_cand &c)
    {
        Block &B = blocks_[p.b];
        B.v.insert(B.v.begin() + p.o, c);
        B.maxr = std::max(B.maxr, c.r);
        n_++;
        if (B.v.size() > 2 * kBlock)
            split(p.b);
    }
    void erase(Pos p)
    {
        Block &B = blocks_[p.b];
        B.v.erase(B.v.begin() + p.o);
        n_--;
        if (B.v.empty())
            blocks_.erase(blocks_.begin() + p.b);
        else
            remax(B);
    }
    void export_to(std::vector<jerk_cand> &out) const
    {
        out.clear();
        out.reserve(n_);
        for (const auto &B : blocks_)
            out.insert(out.end(), B.v.begin(), B.v.end());
    }

  private:
    static constexpr size_t kBlock = 256;
    struct Block {
        std::vector<jerk_cand> v;
        double maxr = -INFINITY;
    };
    static void remax(Block &B)
    {
        double m = -INFINITY;
        for (const auto &c : B.v)
            m = std::max(m, c.r);
        B.maxr = m;
    }
    void split(size_t b)
    {
        Block nb;
        Block &B = blocks_[b];
        nb.v.assign(B.v.begin() + kBlock, B.v.end());
        B.v.resize(kBlock);
        remax(B);
        remax(nb);
        blocks_.insert(blocks_.begin() + b + 1, std::move(nb));
    }
    std::vector<Block> blocks_;
    size_t n_ = 0;
};

bool insert_cand(CandList &L, const jerk_cand &v)
{
    if (L.empty()) {
        L.push_back(v);
        return true;
    }
    const CandList::Pos tmp = L.walk(v.r);
    const bool have_prev = L.has_prev(tmp);
    const double next_diff = fabs(v.r - L.at(tmp).r);
    const double prev_diff = have_prev ? fabs(v.r - L.at(L.prev(tmp)).r) : kClosestR + 1.0;
    bool added = false;
    if (prev_diff < kClosestR) {
        const CandList::Pos prev = L.prev(tmp);
        if (L.at(prev).sigma < v.sigma) {
            L.replace(prev, v);
            added = true;
        }
        if (next_diff < kClosestR && L.at(tmp).sigma < v.sigma) {
            if (added)
                L.erase(tmp);
            else {
                L.replace(tmp, v);
                added = true;
            }
        }
    } else if (next_diff < kClosestR) {
        if (L.at(tmp).sigma < v.sigma) {
            L.replace(tmp, v);
            added = true;
        }
    } else {
        added = true;
        if (L.is_last(tmp) && L.at(tmp).r < v.r - kClosestR)
            L.push_back(v);
        else
            L.insert_before(tmp, v);
    }
    return added;
}

long long export_list(const CandList &CL, jerk_cand **out)
{
    std::vector<jerk_cand> L;
    CL.export_to(L);
    if (!out)
        return (long long)L.size();
    *out = (jerk_cand *)malloc(sizeof(jerk_cand) * (L.size() ? L.size() : 1));
    if (!*out)
        return -1;
    if (!L.empty())
        memcpy(*out, L.data(), sizeof(jerk_cand) * L.size());
    return (long long)L.size();
}

}  // namespace

extern "C" long long jerk_insert_hits(const jerk_cand *hits, long long nhits, jerk_cand **cands)
{
    CandList L;
    for (long long i = 0; i < nhits; i++)
        insert_cand(L, hits[i]);
    return export_list(L, cands);
}

// ---------------------------------------------------------------------------
// the per-stage twiddle tables of fftlen N's FFT plan (jerk_fft.cuh)

static void append_twiddles(int N, std::vector<float2> &tw)
{
    const size_t at = tw.size();
    tw.resize(at + fft_twiddle_size(N));
    fft_twiddle_table(N, tw.data() + at);
}

// ---------------------------------------------------------------------------
// Kernel bank (create_subharminfos / init_kernel, src/accel_utils.c:151-282)

extern "C" long long jerk_bank_elements(const jerk_subharm *subs, int nsubs)
{
    long long n = 0;
    for (int s = 0; s < nsubs; s++)
        n += (long long)subs[s].numw * subs[s].numz * subs[s].fftlen;
    return n;
}

extern "C" int jerk_device_alloc(long long bytes, void **out)
{
    if (!out || bytes <= 0)
        return fail(JERK_EINVAL, "jerk_device_alloc: bad argument");
    JERK_CUDA(cudaMalloc(out, (size_t)bytes));
    return JERK_OK;
}

extern "C" void jerk_device_free(void *p) { cudaFree(p); }

extern "C" int jerk_copy_to_host(void *dst, const void *src, long long bytes)
{
    JERK_CUDA(cudaMemcpy(dst, src, (size_t)bytes, cudaMemcpyDeviceToHost));
    return JERK_OK;
}

extern "C" int jerk_bank_generate(const jerk_subharm *subs, int nsubs, void *device_bank,
                                  void *stream)
{
    if (!subs || nsubs <= 0 || !device_bank)
        return fail(JERK_EINVAL, "jerk_bank_generate: bad argument");
    cudaStream_t st = (cudaStream_t)stream;
    // rows grouped by fftlen so each FFT launch covers a contiguous range
    std::map<int, std::vector<BankRow>> byN;
    long long off = 0;
    int max_pts = 1;
    for (int s = 0; s < nsubs; s++) {
        const jerk_subharm &sh = subs[s];
        if (!fftlen_supported(sh.fftlen))
            return fail(JERK_EUNSUPPORTED, "unsupported fftlen " + std::to_string(sh.fftlen));
        for (int ii = 0; ii < sh.numw; ii++)
            for (int jj = 0; jj < sh.numz; jj++) {
                BankRow r{};
                r.z = -sh.zmax + jj * kDZ;
                r.w = -sh.wmax + ii * kDW;
                r.fftlen = sh.fftlen;
                const int hw = w_resp_halfwidth((double)r.z, (double)r.w);
                r.numkern = 2 * 2 * hw;
                r.num_pts = 0;
                if (fabs((double)r.w) >= 1e-4) {
                    r.num_pts = (int)next2_to_n(6 * hw + 200 + r.numkern / 2);
                    max_pts = std::max(max_pts, r.num_pts);
                }
                if (r.numkern > sh.fftlen)
                    return fail(JERK_EINVAL, "response wider than its fftlen");
                r.off = off + ((long long)ii * sh.numz + jj) * sh.fftlen;
                byN[sh.fftlen].push_back(r);
            }
        off += (long long)sh.numw * sh.numz * sh.fftlen;
    }
    if ((size_t)max_pts * sizeof(float) > 200 * 1024)
        return fail(JERK_EUNSUPPORTED, "response series too long for shared memory");
    std::vector<BankRow> rows;
    std::vector<std::pair<int, std::pair<int, int>>> groups;  // N, (first, count)
    std::vector<float2> tw;
    std::map<int, int> twoff;
    for (auto &kv : byN) {
        groups.push_back({kv.first, {(int)rows.size(), (int)kv.second.size()}});
        rows.insert(rows.end(), kv.second.begin(), kv.second.end());
        twoff[kv.first] = (int)tw.size();
        append_twiddles(kv.first, tw);
    }
    BankRow *d_rows = nullptr;
    float2 *d_tw = nullptr;
    int rc = JERK_OK;
    cudaError_t e = cudaMalloc(&d_rows, sizeof(BankRow) * rows.size());
    if (e == cudaSuccess)
        e = cudaMalloc(&d_tw, sizeof(float2) * tw.size());
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(d_rows, rows.data(), sizeof(BankRow) * rows.size(),
                            cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(d_tw, tw.data(), sizeof(float2) * tw.size(), cudaMemcpyHostToDevice,
                            st);
    if (e == cudaSuccess)
        e = launch_bank_response(d_rows, (int)rows.size(), max_pts, (float2 *)device_bank, st);
    for (size_t g = 0; g < groups.size() && e == cudaSuccess; g++)
        e = launch_bank_fft_any(groups[g].first, d_rows, groups[g].second.first,
                                groups[g].second.second, d_tw, twoff[groups[g].first],
                                (float2 *)device_bank, st);
    if (e == cudaSuccess)
        e = cudaStreamSynchronize(st);
    if (e != cudaSuccess)
        rc = cuda_fail(e, "jerk_bank_generate");
    cudaFree(d_rows);
    cudaFree(d_tw);
    return rc;
}

// ---------------------------------------------------------------------------
// Half lengths of the folded correlation (jerk_fold.cu)

// The window of half length L of a subharmonic whose chunk holds M = fftlen/2
// bins with the good outputs from bin H (the halfwidth) on, nr/2 of each
// parity: its first bin (the good bins in the middle, inside the chunk), and
// the widest support it holds.  L = M holds any row.
static int fold_window(int M, int H, int nr, int L, int *hmax)
{
    const int w = std::max(0, std::min(H - (L - nr / 2) / 2, M - L));
    *hmax = L >= M ? 1 << 30 : std::min(H - w, L - nr / 2 - (H - w));
    return w;
}

// The shortest half length (index into kFoldLens) for a row of support h.
static int fold_choose(int fftlen, int H, int nr, int h)
{
    const int M = fftlen / 2;
    int hmax = 0;
    for (int i = 0; i < kNumFoldLens; i++) {
        fold_window(M, H, nr, kFoldLens[i], &hmax);
        if (kFoldLens[i] >= M || h <= hmax)
            return i;
    }
    return kNumFoldLens - 1;
}

// Bytes of the folded rows of one subharmonic whose rows are the generated
// bank's (jerk_bank_generate), each as wide as its response.
long long jerk::fold_bytes(const jerk_subharm &s, int maxnumrs)
{
    if (!folded_fftlen(s.fftlen))
        return 0;
    std::map<int, long long> rows;
    for (int ii = 0; ii < s.numw; ii++)
        for (int jj = 0; jj < s.numz; jj++)
            rows[kFoldLens[fold_choose(s.fftlen, s.halfwidth, maxnumrs,
                                       w_resp_halfwidth(-s.zmax + jj * kDZ, -s.wmax + ii * kDW))]]++;
    long long b = 0;
    for (auto &kv : rows) {
        const long long per = fold_cta_rows(kv.first);
        b += (kv.second + per - 1) / per * per * 2 * kv.first * (long long)sizeof(float2);
    }
    return b;
}

// ---------------------------------------------------------------------------
// The plan

// per kernel class: launches, device time (CUDA events on the plan's stream,
// only while profiling is on), and algorithmic bytes / flops of the launches
struct KernelClass {
    std::string name;
    long long launches = 0;
    double ms = 0.0, bytes = 0.0, flops = 0.0;
};

constexpr int kHarmRing = 5;  // the default harmonic sum

struct PendingTiming {
    int cls;
    cudaEvent_t start, stop;
};

struct jerk_plan {
    int device = 0;
    cudaStream_t stream = nullptr;   // prep + correlation (and the caller's work)
    bool own_stream = false;
    jerk_obs obs{};
    int nsubs = 0, maxfft = 0, batch = 8;
    size_t prep_smem = 0;
    // harmonic-sum kernel (jerk_config.harm_mode, 0 resolved to kHarmRing):
    // 1 gather, 2 gather + TMA L2 prefetch, 3 / 4 TMA tiles of harm_tile
    // (8 / 16) rows, kHarmRing the ring of row copies (jerk_harm.cu); tma
    // holds the tensor maps of modes 2-4
    int harm_mode = kHarmRing;
    int harm_tile = 16;
    std::unique_ptr<HarmTma> tma;
    // graph mode: a whole pass captured once per (first, count) and replayed;
    // the spectrum is always staged into d_spec so one graph fits any input
    bool use_graph = false;
    cudaGraphExec_t graph_exec = nullptr;
    long long graph_first = -1, graph_count = -1;
    long long graph_replays = 0;
    int zlo0 = 0, wlo0 = 0;
    long long nrsteps = 0;
    std::vector<jerk_subharm> subs;
    std::vector<SubDev> hsubs;
    std::vector<StepDev> hsteps;  // [nrsteps][nsubs]
    std::map<int, std::vector<int>> groups;  // fftlen -> subs, the long unfolded lengths
    std::vector<FoldRows> rowsets;  // folded half lengths, then short unfolded lengths
    std::vector<char> own_launch;   // per row set: launched by itself (own_launch_wins)
    FoldRows *d_rowsets = nullptr;
    std::vector<FoldClass> fold_classes;
    std::vector<std::vector<double>> class_rows;  // [half length index][class] live rows
    // device
    float2 *d_bank = nullptr;
    bool own_bank = false;
    float2 *d_tw = nullptr;
    float2 *d_fold = nullptr;   // every half length's folded rows
    int2 *d_foldmap = nullptr;  // and their maps
    long long fold_f2 = 0;
    FoldClass *d_classes = nullptr;
    SubDev *d_subs = nullptr;
    StepDev *d_steps = nullptr;
    uint16_t *d_zinds = nullptr;
    int *d_wind = nullptr;
    // prepared rows and row indices of a batch, and of the next, which is
    // prepared while this one is correlated (null: not allocated, in turn)
    float2 *d_prepped[2] = {};
    float *d_planes = nullptr;
    uint16_t *d_rinds[2] = {};
    float2 *d_spec = nullptr;
    long long spec_cap = 0;
    unsigned long long *d_hit_keys = nullptr;
    float *d_hit_pows = nullptr;
    unsigned int *d_hit_count = nullptr;
    unsigned int *d_status = nullptr;
    int wait_probe = 0;                // jerk_debug_wait_probe
    long long max_hits = 0;
    long long plane_floats = 0, prepped_f2 = 0;
    // a search pass being enqueued batch by batch
    struct Pass {
        SearchDev a{};
        long long first = 0, count = 0, next = 0, nbatch = 0, ndone = 0;
        bool all_enqueued = false;
        int buf = 0;            // the buffers of the batch at next
        bool prepared = false;  // its rows are prepared there
        bool capturing = false;  // being recorded into a graph: no host-side event queries
        int error = 0;  // first enqueue failure (the pass is then abandoned)
    } pass;
    static constexpr int kRing = 16;
    cudaEvent_t ev_batch[kRing] = {};  // harmonic sum of batch n done (n % kRing)
    // asynchronous search in flight (jerk_search_async / jerk_search_collect)
    bool in_flight = false;
    const float2 *inflight_spec = nullptr;
    long long inflight_first = 0, inflight_count = 0;
    unsigned int *h_counts = nullptr;  // pinned: hit count, status
    cudaEvent_t ev_done = nullptr;
    // instrumentation
    bool profiling = false;
    std::vector<KernelClass> classes;
    std::map<std::string, int> class_index;
    std::vector<PendingTiming> pending;
    std::vector<cudaEvent_t> event_pool;
    long long h2d_bytes = 0, d2h_bytes = 0;
};

static int kclass(jerk_plan *p, const std::string &name)
{
    auto it = p->class_index.find(name);
    if (it != p->class_index.end())
        return it->second;
    KernelClass k;
    k.name = name;
    p->classes.push_back(k);
    p->class_index[name] = (int)p->classes.size() - 1;
    return (int)p->classes.size() - 1;
}

static cudaEvent_t take_event(jerk_plan *p)
{
    if (!p->event_pool.empty()) {
        cudaEvent_t e = p->event_pool.back();
        p->event_pool.pop_back();
        return e;
    }
    cudaEvent_t e = nullptr;
    cudaEventCreate(&e);
    return e;
}

// Bracket one launch: returns a token to pass to launch_end.
static int launch_begin(jerk_plan *p, int cls, double bytes, double flops)
{
    KernelClass &k = p->classes[cls];
    k.launches++;
    k.bytes += bytes;
    k.flops += flops;
    if (!p->profiling)
        return -1;
    PendingTiming t{cls, take_event(p), take_event(p)};
    cudaEventRecord(t.start, p->stream);
    p->pending.push_back(t);
    return (int)p->pending.size() - 1;
}

static void launch_end(jerk_plan *p, int token)
{
    if (token >= 0)
        cudaEventRecord(p->pending[token].stop, p->stream);
}

// after a stream synchronisation: fold the recorded intervals into the classes
static void collect_timings(jerk_plan *p)
{
    for (auto &t : p->pending) {
        float ms = 0.f;
        if (cudaEventElapsedTime(&ms, t.start, t.stop) == cudaSuccess)
            p->classes[t.cls].ms += ms;
        p->event_pool.push_back(t.start);
        p->event_pool.push_back(t.stop);
    }
    p->pending.clear();
}

extern "C" int jerk_plan_set_profiling(jerk_plan *p, int on)
{
    if (!p)
        return fail(JERK_EINVAL, "null plan");
    p->profiling = on != 0;
    return JERK_OK;
}

extern "C" void jerk_plan_reset_stats(jerk_plan *p)
{
    if (!p)
        return;
    for (auto &k : p->classes) {
        k.launches = 0;
        k.ms = k.bytes = k.flops = 0.0;
    }
    p->h2d_bytes = p->d2h_bytes = 0;
}

extern "C" int jerk_plan_kernel_stats(const jerk_plan *p, int max, jerk_kernel_stat *out)
{
    if (!p)
        return 0;
    int n = 0;
    for (const auto &k : p->classes) {
        if (n < max && out) {
            memset(&out[n], 0, sizeof(out[n]));
            strncpy(out[n].name, k.name.c_str(), sizeof(out[n].name) - 1);
            out[n].launches = k.launches;
            out[n].ms = k.ms;
            out[n].bytes = k.bytes;
            out[n].flops = k.flops;
        }
        n++;
    }
    return n;
}

extern "C" void jerk_plan_transfer_stats(const jerk_plan *p, long long *h2d, long long *d2h)
{
    if (h2d)
        *h2d = p ? p->h2d_bytes : 0;
    if (d2h)
        *d2h = p ? p->d2h_bytes : 0;
}

static void drop_graph(jerk_plan *p)
{
    if (p->graph_exec)
        cudaGraphExecDestroy(p->graph_exec);
    p->graph_exec = nullptr;
    p->graph_first = p->graph_count = -1;
}

static void plan_free_device(jerk_plan *p)
{
    if (p->own_bank)
        cudaFree(p->d_bank);
    cudaFree(p->d_tw);
    cudaFree(p->d_fold);
    cudaFree(p->d_foldmap);
    cudaFree(p->d_classes);
    cudaFree(p->d_rowsets);
    cudaFree(p->d_subs);
    cudaFree(p->d_steps);
    cudaFree(p->d_zinds);
    cudaFree(p->d_wind);
    for (int i = 0; i < 2; i++) {
        cudaFree(p->d_prepped[i]);
        cudaFree(p->d_rinds[i]);
    }
    cudaFree(p->d_planes);
    cudaFree(p->d_spec);
    cudaFree(p->d_hit_keys);
    cudaFree(p->d_hit_pows);
    cudaFree(p->d_hit_count);
    cudaFree(p->d_status);
}

extern "C" void jerk_plan_destroy(jerk_plan *p)
{
    if (!p)
        return;
    int cur = 0;
    cudaGetDevice(&cur);
    cudaSetDevice(p->device);
    if (p->stream)
        cudaStreamSynchronize(p->stream);
    drop_graph(p);
    plan_free_device(p);
    for (auto &t : p->pending) {
        cudaEventDestroy(t.start);
        cudaEventDestroy(t.stop);
    }
    for (auto e : p->event_pool)
        cudaEventDestroy(e);
    if (p->ev_done)
        cudaEventDestroy(p->ev_done);
    for (int i = 0; i < jerk_plan::kRing; i++)
        if (p->ev_batch[i])
            cudaEventDestroy(p->ev_batch[i]);
    if (p->h_counts)
        cudaFreeHost(p->h_counts);
    if (p->own_stream && p->stream)
        cudaStreamDestroy(p->stream);
    cudaSetDevice(cur);
    delete p;
}

// Device memory for a plan that holds its own already (a larger hit buffer, a
// staged spectrum).  Where there is none left, the buffers that let a batch be
// prepared ahead make room: the plan works without them, and a batch prepared
// there is prepared again in its turn.
template <class T>
static cudaError_t plan_malloc(jerk_plan *p, T **ptr, size_t bytes)
{
    *ptr = nullptr;
    cudaError_t e = cudaMalloc(ptr, bytes);
    if (e != cudaErrorMemoryAllocation || !p->d_rinds[1])
        return e;
    cudaGetLastError();
    e = cudaStreamSynchronize(p->stream);
    if (e != cudaSuccess)
        return e;
    drop_graph(p);  // a captured pass holds them
    for (void *b : {(void *)p->d_prepped[1], (void *)p->d_rinds[1]})
        cudaFree(b);
    p->d_prepped[1] = nullptr;
    p->d_rinds[1] = nullptr;
    p->pass.prepared = false;
    p->pass.buf = 0;
    return cudaMalloc(ptr, bytes);
}

static int alloc_hits(jerk_plan *p, long long cap)
{
    drop_graph(p);  // the captured pass holds the old hit buffers
    cudaFree(p->d_hit_keys);
    cudaFree(p->d_hit_pows);
    p->d_hit_keys = nullptr;
    p->d_hit_pows = nullptr;
    p->max_hits = 0;  // a pass without them stores nothing
    JERK_CUDA(plan_malloc(p, &p->d_hit_keys, sizeof(unsigned long long) * cap));
    JERK_CUDA(plan_malloc(p, &p->d_hit_pows, sizeof(float) * cap));
    p->max_hits = cap;
    return JERK_OK;
}

static long long count_rsteps(const jerk_obs &o)
{
    const int rstep = (int)(o.corr_uselen * kDR);
    long long n = 0;
    double startr = o.rlo;
    while (startr + rstep < (double)o.highestbin) {
        n++;
        startr += rstep;
    }
    return n;
}

extern "C" long long jerk_num_rsteps(const jerk_plan *p) { return p ? p->nrsteps : 0; }

// cuTensorMapEncodeTiled from the driver, without linking libcuda.
static PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder()
{
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (PFN_cuTensorMapEncodeTiled_v12000)f;
    });
    return fn;
}

// The harmonic sum's TMA boxes and tensor maps (HarmTma in jerk_kernels.cuh).
// A tile covers kThreads fundamental r (one CTA) x harm_tile fundamental z.
// Subharmonic index steps are 0 or 1 per fundamental step (harm_fract <= 1),
// so over n steps an index grows by at most floor(n * harm_fract) + 1: the box
// spans that + 1 cells / rows, plus 3 cells for rounding its first r index
// down to a multiple of 4.  For the tile kernel (in_smem) the boxes must fit
// next to the z tables in shared memory; if they do not, or the driver has no
// tensor-map encoder, tma stays null and the plan uses the gather kernel.
static int build_harm_tma(jerk_plan *p, bool in_smem)
{
    constexpr int kThreads = 128;  // harmonic-sum CTA width (kHarmThreads)
    auto T = std::make_unique<HarmTma>();
    memset(T.get(), 0, sizeof(HarmTma));
    const int zt = p->harm_tile;
    int off = 0;
    long long bytes = 0;
    for (int s = 0; s < p->nsubs; s++) {
        const SubDev &d = p->hsubs[s];
        const double hf = d.harm_fract;
        const int W = s == 0 ? kThreads : ((int)floor((kThreads - 1) * hf) + 5 + 3) & ~3;
        const int Z = s == 0 ? zt : (int)floor((zt - 1) * hf) + 2;
        if (W > 256 || Z > 256)
            return JERK_OK;
        T->W[s] = W;
        T->Z[s] = Z;
        T->boxoff[s] = off;
        off += (W * Z + 31) & ~31;  // 128-byte aligned boxes
        bytes += 4LL * W * Z;
    }
    T->box_floats = off;
    T->box_bytes = (int)bytes;
    const size_t smem = harmsum_tma_smem_bytes(*T, p->nsubs, p->subs[0].numz);
    if (in_smem && smem + 1024 > 200 * 1024)
        return JERK_OK;  // boxes too large: gather kernel
    PFN_cuTensorMapEncodeTiled_v12000 enc = tensor_map_encoder();
    if (!enc)
        return JERK_OK;  // no driver entry point: gather kernel
    for (int s = 0; s < p->nsubs; s++) {
        const SubDev &d = p->hsubs[s];
        const cuuint64_t dims[4] = {(cuuint64_t)d.stride, (cuuint64_t)d.numz, (cuuint64_t)d.numw,
                                    (cuuint64_t)p->batch};
        const cuuint64_t strides[3] = {4ull * d.stride, 4ull * d.stride * d.numz,
                                       4ull * (cuuint64_t)d.plane_size};
        const cuuint32_t box[4] = {(cuuint32_t)T->W[s], (cuuint32_t)T->Z[s], 1, 1};
        const cuuint32_t estr[4] = {1, 1, 1, 1};
        const CUresult r = enc(&T->map[s], CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4,
                               (void *)(p->d_planes + d.plane_off), dims, strides, box, estr,
                               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                               CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS)
            return fail(JERK_ECUDA, "cuTensorMapEncodeTiled failed for a volume tensor map");
    }
    p->tma = std::move(T);
    return JERK_OK;
}

// Whether a row set is launched by itself rather than merged with others: its
// CTAs make two waves; or, for the half lengths whose rows leave a warp of the
// merged launch's four idle (768, 640, 384), four waves over the rsteps --
// the launches overlap, so that a last partial wave is no loss.  Measured (ms
// per pass; merged against own): 6 trials of 2^21 samples, zmax 50, wmax 150,
// 8 harmonics 103.4 / 100.3; 2^22 samples, zmax 100, 16 harmonics 13.75 /
// 13.70, and 14.32 with its 359 rows of 1024 by themselves as well; against it
// 2^21 samples, zmax 100, wmax 100, 4 harmonics, batches of 8, 18.2 / 19.0.
static bool own_launch_wins(int L, long long n, int batch)
{
    const long long groups = n / fold_cta_rows(L), wave = fold_wave_ctas(L);
    const bool idle = L == 768 || L == 640 || L == 384;
    return groups >= 2 * wave || (idle && groups * batch >= 4 * wave);
}

// Scratch of folding a bank on the device, freed on every path (cudaFree waits
// for the kernels reading it), and the tables in it.
struct FoldScratch {
    char *mem = nullptr;
    double2 *roots = nullptr;     // exp(-2 pi i m / n) of every length n taken
    int *roots_at = nullptr;      // [n / 128]: where they start
    long long *src = nullptr;     // the rows' places in the bank
    FoldSrc *fsrc = nullptr;
    int *half = nullptr;          // their supports
    int *differs = nullptr;       // set where a support is not the expected one
    ~FoldScratch() { cudaFree(mem); }
};

// The plan's row sets for supports `half` (of subharmonic s from first_row[s]
// on): the rows of every folded length in the shortest half length that holds
// them, laid out by class (their prepared windows from *data_off on) and written
// class after class, longest half length first; then the maps of the short
// lengths that do not fold (fftlen 128 to 384).  check: the supports are what
// generated rows have; *same says whether the bank's do.
static int fold_rows(jerk_plan *p, const std::vector<int> &maxnumrs, const std::vector<int> &half,
                     const std::vector<long long> &first_row, const FoldScratch &sc, bool check,
                     long long *data_off, bool *same)
{
    cudaStream_t st = p->stream;
    // classes: a subharmonic's rows of one half length
    struct Built {
        std::vector<FoldSrc> src;
        std::vector<int2> map;
        int maxN = 0;
    };
    std::vector<Built> built(kNumFoldLens);
    p->class_rows.assign(kNumFoldLens, {});
    for (int s = 0; s < p->nsubs; s++) {
        const jerk_subharm &sh = p->subs[s];
        if (!folded_fftlen(sh.fftlen))
            continue;
        SubDev &d = p->hsubs[s];
        const int M = sh.fftlen / 2, rows = sh.numw * sh.numz;
        const int *h = half.data() + first_row[s];
        std::vector<std::vector<int>> of(kNumFoldLens);
        for (int r = 0; r < rows; r++)
            of[fold_choose(sh.fftlen, sh.halfwidth, maxnumrs[s], h[r])].push_back(r);
        d.cls0 = (int)p->fold_classes.size();
        for (int i = 0; i < kNumFoldLens; i++) {
            if (of[i].empty())
                continue;
            FoldClass c{};
            int hmax = 0;
            c.sub = s;
            c.len = kFoldLens[i];
            c.wstart = fold_window(M, sh.halfwidth, maxnumrs[s], c.len, &hmax);
            c.out0 = sh.halfwidth - c.wstart;
            c.stride = d.stride;
            c.plane_off = d.plane_off;
            c.plane_size = d.plane_size;
            c.data_off = *data_off;
            *data_off += (long long)c.len * p->batch;
            const int ci = (int)p->fold_classes.size();
            Built &B = built[i];
            B.maxN = std::max(B.maxN, sh.fftlen);
            for (int r : of[i]) {
                // (rows of the whole length fold whatever their support: a
                // sixteenth of them is checked)
                const bool whole = c.len == M;
                B.src.push_back({d.kern_off + (long long)r * sh.fftlen, sh.fftlen,
                                 whole ? -1 : h[r], check && !(whole && r % 16) ? h[r] : 0});
                B.map.push_back(make_int2(ci, r));
            }
            while (B.src.size() % fold_cta_rows(c.len)) {
                B.src.push_back({-1, sh.fftlen, -1, 0});
                B.map.push_back(make_int2(-1, 0));
            }
            p->fold_classes.push_back(c);
            p->class_rows[i].resize(p->fold_classes.size(), 0.0);
            p->class_rows[i][ci] = (double)of[i].size();
        }
        d.ncls = (int)p->fold_classes.size() - d.cls0;
    }

    std::map<int, std::vector<int2>> shorts;  // unfolded fftlen -> map
    for (int s = 0; s < p->nsubs; s++) {
        const jerk_subharm &sh = p->subs[s];
        if (!folded_fftlen(sh.fftlen) && sh.fftlen < 512)
            for (int r = 0; r < sh.numw * sh.numz; r++)
                shorts[sh.fftlen].push_back(make_int2(s, r));
    }
    long long total = 0, f2 = 0;
    for (int i = 0; i < kNumFoldLens; i++) {
        total += (long long)built[i].src.size();
        f2 += (long long)built[i].src.size() * 2 * kFoldLens[i];
    }
    for (auto &kv : shorts)
        total += (long long)kv.second.size();
    p->fold_f2 = f2;
    if (f2)
        JERK_CUDA(cudaMalloc(&p->d_fold, sizeof(float2) * f2));
    if (total)
        JERK_CUDA(cudaMalloc(&p->d_foldmap, sizeof(int2) * total));
    if (check)
        JERK_CUDA(cudaMemsetAsync(sc.differs, 0, sizeof(int), st));
    long long row = 0, at = 0;
    for (int i = kNumFoldLens - 1; i >= 0; i--) {
        const Built &B = built[i];
        const long long n = (long long)B.src.size();
        if (!n)
            continue;
        const int L = kFoldLens[i];
        JERK_CUDA(cudaMemcpyAsync(sc.fsrc + row, B.src.data(), sizeof(FoldSrc) * n,
                                  cudaMemcpyHostToDevice, st));
        JERK_CUDA(cudaMemcpyAsync(p->d_foldmap + row, B.map.data(), sizeof(int2) * n,
                                  cudaMemcpyHostToDevice, st));
        JERK_CUDA(launch_fold_rows(p->d_bank, sc.fsrc + row, (int)n, L, B.maxN, sc.roots,
                                   sc.roots_at, p->d_fold + at, check ? sc.differs : nullptr, st));
        FoldRows R{};
        R.len = L;
        R.n = (int)n;
        R.rows = p->d_fold + at;
        R.map = p->d_foldmap + row;
        p->rowsets.push_back(R);
        p->own_launch.push_back(!multi_takes(R) || own_launch_wins(L, n, p->batch));
        row += n;
        at += n * 2 * L;
    }
    for (auto kv = shorts.rbegin(); kv != shorts.rend(); ++kv) {
        const long long n = (long long)kv->second.size();
        JERK_CUDA(cudaMemcpyAsync(p->d_foldmap + row, kv->second.data(), sizeof(int2) * n,
                                  cudaMemcpyHostToDevice, st));
        FoldRows R{};
        R.len = -kv->first;
        R.n = (int)n;
        R.map = p->d_foldmap + row;
        p->rowsets.push_back(R);
        p->own_launch.push_back(0);
        row += n;
    }
    if (p->rowsets.size() > (size_t)kMaxRowSets)
        return fail(JERK_EUNSUPPORTED, "too many row sets");
    int differs = 0;
    if (check) {
        JERK_CUDA(cudaMemcpyAsync(&differs, sc.differs, sizeof(int), cudaMemcpyDeviceToHost, st));
        JERK_CUDA(cudaStreamSynchronize(st));
    }
    *same = !differs;
    // the host tables above are pageable: copied before these calls returned
    return JERK_OK;
}

// Folds the bank's rows into the plan's row sets.  Generated rows are as wide as
// their responses, which the folding checks; measuring every row first
// transforms each back twice (a plan on a shared bank, zmax 300, wmax 600, 2
// harmonics: 10.8 ms with that, 7.7 without; 200, 300, 16: 12.9 and 12.5).
static int fold_bank(jerk_plan *p, const std::vector<int> &maxnumrs, long long *data_off)
{
    std::map<int, std::vector<int>> subs_of;  // fftlen -> subharmonics
    for (int s = 0; s < p->nsubs; s++)
        if (folded_fftlen(p->subs[s].fftlen))
            subs_of[p->subs[s].fftlen].push_back(s);
    cudaStream_t st = p->stream;
    JERK_CUDA(fold_plan_attrs());

    // root tables of every length the folding may take
    int roots_at[4096 / 128 + 1];
    int nroots = 0, maxN = 0;
    std::fill(std::begin(roots_at), std::end(roots_at), -1);
    std::vector<int> lens(std::begin(kFoldLens), std::end(kFoldLens));
    for (auto &kv : subs_of) {
        lens.push_back(kv.first);
        maxN = std::max(maxN, kv.first);
    }
    for (int n : lens)
        if (n <= maxN && roots_at[n / 128] < 0) {
            roots_at[n / 128] = nroots;
            nroots += n;
        }

    long long nrows = 0;
    bool generated = !p->own_bank;  // as the rows' (z, w) would be by the sizes
    std::vector<long long> first_row(p->nsubs, 0);
    for (auto &kv : subs_of)
        for (int s : kv.second) {
            const jerk_subharm &sh = p->subs[s];
            first_row[s] = nrows;
            nrows += (long long)sh.numw * sh.numz;
            generated = generated && sh.numz == sh.zmax / kDZ * 2 + 1 &&
                        sh.numw == sh.wmax / kDW * 2 + 1;
        }
    if (nrows > INT_MAX)
        return fail(JERK_EUNSUPPORTED, "too many kernel rows");
    // (the padding adds at most three rows a class)
    FoldScratch sc;
    const size_t pad_rows = 4 * (size_t)kNumFoldLens * p->nsubs;
    const size_t b_roots = sizeof(double2) * nroots, b_at = 256,
                 b_src = sizeof(long long) * (size_t)nrows,
                 b_fsrc = sizeof(FoldSrc) * ((size_t)nrows + pad_rows),
                 b_half = sizeof(int) * (size_t)nrows;
    static_assert(sizeof(roots_at) <= 256, "roots_at");
    JERK_CUDA(cudaMalloc(&sc.mem, b_roots + b_at + b_src + b_fsrc + b_half + 16));
    sc.roots = (double2 *)sc.mem;
    sc.roots_at = (int *)(sc.mem + b_roots);
    sc.src = (long long *)(sc.mem + b_roots + b_at);
    sc.fsrc = (FoldSrc *)(sc.mem + b_roots + b_at + b_src);
    sc.half = (int *)(sc.mem + b_roots + b_at + b_src + b_fsrc);
    sc.differs = sc.half + nrows;
    for (int n : lens)
        if (n <= maxN && roots_at[n / 128] >= 0)
            JERK_CUDA(launch_fold_roots(sc.roots + roots_at[n / 128], n, st));
    JERK_CUDA(cudaMemcpyAsync(sc.roots_at, roots_at, sizeof(roots_at), cudaMemcpyHostToDevice, st));

    std::vector<int> half(nrows);
    bool same = false;
    if (generated) {
        for (auto &kv : subs_of)
            for (int s : kv.second) {
                const jerk_subharm &sh = p->subs[s];
                for (int ii = 0; ii < sh.numw; ii++)
                    for (int jj = 0; jj < sh.numz; jj++)
                        half[first_row[s] + (long long)ii * sh.numz + jj] =
                            w_resp_halfwidth(-sh.zmax + jj * kDZ, -sh.wmax + ii * kDW);
            }
        const long long at = *data_off;
        const int rc = fold_rows(p, maxnumrs, half, first_row, sc, true, data_off, &same);
        if (rc != JERK_OK || same)
            return rc;
        *data_off = at;
        cudaFree(p->d_fold);
        cudaFree(p->d_foldmap);
        p->d_fold = nullptr;
        p->d_foldmap = nullptr;
        p->fold_classes.clear();
        p->rowsets.clear();
        p->own_launch.clear();
        for (SubDev &d : p->hsubs)
            d.cls0 = d.ncls = 0;
    }
    std::vector<long long> src(nrows);
    for (auto &kv : subs_of)
        for (int s : kv.second)
            for (long long r = 0; r < (long long)p->subs[s].numw * p->subs[s].numz; r++)
                src[first_row[s] + r] = p->hsubs[s].kern_off + r * kv.first;
    JERK_CUDA(cudaMemcpyAsync(sc.src, src.data(), b_src, cudaMemcpyHostToDevice, st));
    for (auto &kv : subs_of) {
        const long long at = first_row[kv.second.front()];
        long long n = 0;
        for (int s : kv.second)
            n += (long long)p->subs[s].numw * p->subs[s].numz;
        JERK_CUDA(launch_fold_support(p->d_bank, sc.src + at, (int)n, kv.first,
                                      sc.roots + roots_at[kv.first / 128], sc.half + at, st));
    }
    JERK_CUDA(cudaMemcpyAsync(half.data(), sc.half, b_half, cudaMemcpyDeviceToHost, st));
    JERK_CUDA(cudaStreamSynchronize(st));
    return fold_rows(p, maxnumrs, half, first_row, sc, false, data_off, &same);
}

static int plane_stride(int numrs) { return (numrs + kPlaneAlign - 1) / kPlaneAlign * kPlaneAlign; }

extern "C" int jerk_plan_create(jerk_plan **out, const jerk_obs *obs, const jerk_subharm *subs,
                                int nsubs, const jerk_config *cfg)
{
    if (!out || !obs || !subs)
        return fail(JERK_EINVAL, "jerk_plan_create: null argument");
    *out = nullptr;
    if (obs->numharmstages < 1 || obs->numharmstages > kMaxStages ||
        nsubs != jerk_subharm_count(obs->numharmstages))
        return fail(JERK_EINVAL, "jerk_plan_create: nsubs does not match numharmstages");
    if (obs->norm_type != 0 && obs->norm_type != 1 && !(obs->nph > 0.0f))
        return fail(JERK_EINVAL, "norm_type must be 0 (block median) or 1 (local power)");
    if (obs->corr_uselen <= 0 || obs->corr_uselen % 2 || obs->corr_uselen > 65535)
        return fail(JERK_EINVAL, "bad corr_uselen");
    for (int s = 0; s < nsubs; s++)  // before any device work
        if (!fftlen_supported(subs[s].fftlen))
            return fail(JERK_EUNSUPPORTED, "unsupported fftlen " + std::to_string(subs[s].fftlen) +
                                               " (at most 15360 here)");

    jerk_plan *p = new jerk_plan();
    cudaGetDevice(&p->device);
    p->obs = *obs;
    p->nsubs = nsubs;
    p->subs.assign(subs, subs + nsubs);
    p->batch = (cfg && cfg->batch_rsteps > 0) ? cfg->batch_rsteps : 8;
    const int hm = cfg ? cfg->harm_mode : 0;
    if (hm < 0 || hm > 4) {
        delete p;
        return fail(JERK_EINVAL, "jerk_plan_create: harm_mode must be 0 .. 4");
    }
    // the ring up to 16 harmonics; at 32 its registers would hold one cell a
    // thread, and the gathers stay
    p->harm_mode = hm != 0 ? hm : obs->numharmstages <= 5 ? kHarmRing : 1;
    p->harm_tile = p->harm_mode == 3 ? 8 : 16;
    p->use_graph = cfg && cfg->use_graph;
    const long long want_hits = (cfg && cfg->max_hits > 0) ? cfg->max_hits : (1LL << 22);
    if (cfg && cfg->stream) {
        p->stream = (cudaStream_t)cfg->stream;
    } else {
        cudaError_t e = cudaStreamCreateWithFlags(&p->stream, cudaStreamNonBlocking);
        if (e != cudaSuccess) {
            delete p;
            return cuda_fail(e, "cudaStreamCreate");
        }
        p->own_stream = true;
    }
    auto bail = [&](int code) {
        jerk_plan_destroy(p);
        return code;
    };

    const jerk_subharm &f = subs[0];
    if (f.numharm != 1 || f.harmnum != 1 || f.numz != obs->numz)
        return bail(fail(JERK_EINVAL, "subharmonic 0 must be the fundamental (1/1)"));
    p->zlo0 = calc_required_z(1.0, obs->zlo);
    p->wlo0 = calc_required_w(1.0, obs->wlo);
    p->nrsteps = count_rsteps(*obs);

    // steps: rlo / numrs of every (rstep, subharmonic)
    p->hsteps.resize((size_t)p->nrsteps * nsubs);
    std::vector<int> maxnumrs(nsubs, 0);
    const int rstep = (int)(obs->corr_uselen * kDR);
    for (long long k = 0; k < p->nrsteps; k++) {
        const double startr = obs->rlo + (double)k * rstep;
        const double lastr = startr + rstep - kDR;
        for (int s = 0; s < nsubs; s++) {
            const double hf = (double)subs[s].harmnum / (double)subs[s].numharm;
            const double drlo = calc_required_r(hf, startr), drhi = calc_required_r(hf, lastr);
            StepDev &st = p->hsteps[(size_t)k * nsubs + s];
            st.rlo = (long long)floor(drlo);
            st.fullrlo = startr;
            int numrs = (int)((ceil(drhi) - floor(drlo)) * kRDR + kDblCorrect) + 1;
            if (s == 0)
                numrs = obs->corr_uselen;
            else if (numrs % kRDR)
                numrs = (numrs / kRDR + 1) * kRDR;
            st.numrs = numrs;
            st.pad = 0;
            maxnumrs[s] = std::max(maxnumrs[s], numrs);
        }
    }

    // The harmonic sum addresses one batch's volumes with 32-bit offsets, so
    // the rsteps per batch (a speed knob only) are capped to what fits: at
    // zmax 600, wmax 1200 one rstep's volumes already hold 1.6 G floats.
    {
        long long per_rstep = 0;
        for (int s = 0; s < nsubs; s++)
            per_rstep += (long long)subs[s].numw * subs[s].numz * plane_stride(maxnumrs[s]);
        const long long cap = per_rstep > 0 ? ((1LL << 32) - 1) / per_rstep : p->batch;
        if (cap < 1)
            return bail(fail(JERK_EUNSUPPORTED, "ffdot volumes of one rstep exceed 2^32 floats"));
        p->batch = (int)std::min<long long>(p->batch, cap);
    }

    // subharmonic layout
    p->hsubs.resize(nsubs);
    long long kern_off = 0, plane_off = 0, data_off = 0;
    int zinds_off = 0, wind_off = 0;
    std::vector<uint16_t> zinds;
    std::vector<int> wind;
    std::map<int, int> twoff;
    int twtotal = 0;
    for (int s = 0; s < nsubs; s++) {
        const jerk_subharm &sh = subs[s];
        if (!fftlen_supported(sh.fftlen))
            return bail(fail(JERK_EUNSUPPORTED, "unsupported fftlen " + std::to_string(sh.fftlen)));
        if (maxnumrs[s] + 2 * sh.halfwidth > sh.fftlen)
            return bail(fail(JERK_EINVAL, "fftlen too short for the good bins"));
        SubDev &d = p->hsubs[s];
        d.numharm = sh.numharm;
        d.harmnum = sh.harmnum;
        d.harm_fract = (double)sh.harmnum / (double)sh.numharm;
        d.numz = sh.numz;
        d.numw = sh.numw;
        d.fftlen = sh.fftlen;
        d.halfwidth = sh.halfwidth;
        d.stride = plane_stride(maxnumrs[s]);
        d.zlo = calc_required_z(d.harm_fract, obs->zlo);
        d.wlo = calc_required_w(d.harm_fract, obs->wlo);
        d.pownorm = (float)(1.0 / (double)(sh.fftlen * sh.fftlen));
        const bool folded = folded_fftlen(sh.fftlen);
        if (!folded && !twoff.count(sh.fftlen)) {
            twoff[sh.fftlen] = twtotal;
            twtotal += fft_twiddle_size(sh.fftlen);
        }
        d.twoff = folded ? 0 : twoff[sh.fftlen];
        d.cls0 = d.ncls = 0;  // set with the folded rows below
        d.kern_off = kern_off;
        kern_off += (long long)sh.numw * sh.numz * sh.fftlen;
        d.plane_size = (long long)sh.numw * sh.numz * d.stride;
        d.plane_off = plane_off;
        plane_off += d.plane_size * p->batch;
        d.data_off = data_off;
        if (!folded)
            data_off += (long long)sh.fftlen * p->batch;
        d.zinds_off = zinds_off;
        d.wind_off = wind_off;
        // zinds (src/accel_utils.c:1124-1130) and wind (src/accel_utils.c:1362-1364)
        for (int ii = 0; ii < obs->numz; ii++) {
            const double zz = obs->zlo + ii * kDZ;
            const int subz = calc_required_z(d.harm_fract, zz);
            const int zi = index_from_z(subz, d.zlo);
            if (s > 0 && (zi < 0 || zi >= sh.numz))
                return bail(fail(JERK_EINVAL, "zinds out of range"));
            zinds.push_back((uint16_t)zi);
        }
        for (int ii = 0; ii < subs[0].numw; ii++) {
            const int ww = p->wlo0 + ii * kDW;
            const int subw = calc_required_w(d.harm_fract, ww);
            const int wi = index_from_w(subw, d.wlo);
            if (s > 0 && (wi < 0 || wi >= sh.numw))
                return bail(fail(JERK_EINVAL, "wind out of range"));
            wind.push_back(wi);
        }
        zinds_off += obs->numz;
        wind_off += subs[0].numw;
        p->maxfft = std::max(p->maxfft, sh.fftlen);
        p->prep_smem = std::max(p->prep_smem, prep_smem_bytes(sh.fftlen, folded));
        if (!folded && sh.fftlen > 512)
            p->groups[sh.fftlen].push_back(s);
    }
    p->plane_floats = plane_off;
    if (plane_off >= (1LL << 32))
        return bail(fail(JERK_EINVAL, "ffdot volumes of one batch exceed 2^32 floats: lower batch_rsteps"));

#define JERK_CUDA_B(call)                                \
    do {                                                 \
        cudaError_t e_ = (call);                         \
        if (e_ != cudaSuccess)                           \
            return bail(cuda_fail(e_, #call));           \
    } while (0)

    // kernel bank
    if (cfg && cfg->device_bank) {
        p->d_bank = (float2 *)cfg->device_bank;
        p->own_bank = false;
    } else {
        JERK_CUDA_B(cudaMalloc(&p->d_bank, sizeof(float2) * kern_off));
        p->own_bank = true;
        for (int s = 0; s < nsubs; s++) {
            if (!subs[s].kernels)
                return bail(fail(JERK_EINVAL, "subharmonic without kernels and no device bank"));
            const size_t n = (size_t)subs[s].numw * subs[s].numz * subs[s].fftlen;
            JERK_CUDA_B(cudaMemcpyAsync(p->d_bank + p->hsubs[s].kern_off, subs[s].kernels,
                                        sizeof(float2) * n, cudaMemcpyHostToDevice, p->stream));
        }
    }
    // folded rows (the bank must be complete when the plan is made;
    // jerk_bank_generate returns once it is)
    {
        const int rc = fold_bank(p, maxnumrs, &data_off);
        if (rc != JERK_OK)
            return bail(rc);
    }
    p->prepped_f2 = data_off;

    // twiddles: exp(-2 pi i m / N), double on the host
    std::vector<float2> tw;
    {
        std::vector<std::pair<int, int>> byoff;
        for (auto &kv : twoff)
            byoff.push_back({kv.second, kv.first});
        std::sort(byoff.begin(), byoff.end());
        for (auto &o : byoff)
            append_twiddles(o.second, tw);
    }
    std::map<int, int> fold_tw;
    for (const FoldRows &R : p->rowsets) {
        if (R.len < 0)
            continue;
        const int at = (int)tw.size();
        for (FoldClass &c : p->fold_classes)
            if (c.len == R.len)
                c.twoff = at;
        append_twiddles(R.len, tw);
        tw.resize(tw.size() + (tw.size() & 1));  // 16-byte aligned tables
        fold_tw[R.len] = (int)tw.size();
        tw.resize(tw.size() + fold_twiddle_size(R.len));
        fold_twiddle_table(R.len, tw.data() + fold_tw[R.len]);
    }
    JERK_CUDA_B(cudaMalloc(&p->d_tw, sizeof(float2) * (tw.size() + 1)));
    JERK_CUDA_B(cudaMemcpyAsync(p->d_tw, tw.data(), sizeof(float2) * tw.size(),
                                cudaMemcpyHostToDevice, p->stream));
    for (FoldRows &R : p->rowsets)
        if (R.len > 0)
            R.tw = p->d_tw + fold_tw[R.len];
    if (!p->rowsets.empty()) {
        JERK_CUDA_B(cudaMalloc(&p->d_rowsets, sizeof(FoldRows) * p->rowsets.size()));
        JERK_CUDA_B(cudaMemcpyAsync(p->d_rowsets, p->rowsets.data(),
                                    sizeof(FoldRows) * p->rowsets.size(), cudaMemcpyHostToDevice,
                                    p->stream));
    }
    if (!p->fold_classes.empty()) {
        JERK_CUDA_B(cudaMalloc(&p->d_classes, sizeof(FoldClass) * p->fold_classes.size()));
        JERK_CUDA_B(cudaMemcpyAsync(p->d_classes, p->fold_classes.data(),
                                    sizeof(FoldClass) * p->fold_classes.size(), cudaMemcpyHostToDevice,
                                    p->stream));
    }
    JERK_CUDA_B(cudaMalloc(&p->d_subs, sizeof(SubDev) * nsubs));
    JERK_CUDA_B(cudaMemcpyAsync(p->d_subs, p->hsubs.data(), sizeof(SubDev) * nsubs,
                                cudaMemcpyHostToDevice, p->stream));
    if (p->nrsteps > 0) {
        JERK_CUDA_B(cudaMalloc(&p->d_steps, sizeof(StepDev) * p->hsteps.size()));
        JERK_CUDA_B(cudaMemcpyAsync(p->d_steps, p->hsteps.data(),
                                    sizeof(StepDev) * p->hsteps.size(), cudaMemcpyHostToDevice,
                                    p->stream));
    }
    JERK_CUDA_B(cudaMalloc(&p->d_zinds, sizeof(uint16_t) * zinds.size()));
    JERK_CUDA_B(cudaMemcpyAsync(p->d_zinds, zinds.data(), sizeof(uint16_t) * zinds.size(),
                                cudaMemcpyHostToDevice, p->stream));
    JERK_CUDA_B(cudaMalloc(&p->d_wind, sizeof(int) * wind.size()));
    JERK_CUDA_B(cudaMemcpyAsync(p->d_wind, wind.data(), sizeof(int) * wind.size(),
                                cudaMemcpyHostToDevice, p->stream));
    const size_t rinds_bytes = sizeof(uint16_t) * (size_t)p->batch * nsubs * obs->corr_uselen;
    JERK_CUDA_B(cudaMalloc(&p->d_prepped[0], sizeof(float2) * p->prepped_f2));
    JERK_CUDA_B(cudaMalloc(&p->d_rinds[0], rinds_bytes));
    // one volume buffer: every launch of a pass runs on the plan's
    // stream, so batch k + 1's correlation starts after batch k's harmonic
    // sum has read the volumes (running the two side by side on two streams
    // measured slower than back to back: their CTAs then share SMs)
    JERK_CUDA_B(cudaMalloc(&p->d_planes, sizeof(float) * p->plane_floats));
    if (p->harm_mode >= 2 && p->harm_mode <= 4) {
        const int rc = build_harm_tma(p, p->harm_mode >= 3);
        if (rc != JERK_OK)
            return bail(rc);
        if (!p->tma)
            p->harm_mode = 1;  // no tensor maps here: the plain gather kernel
    }
    JERK_CUDA_B(prep_attrs(p->maxfft));
    JERK_CUDA_B(harmsum_attrs(obs->numharmstages, p->harm_mode == kHarmRing ? 1 : p->harm_mode));
    if (p->harm_mode == kHarmRing)
        JERK_CUDA_B(harm_ring_attrs(obs->numharmstages));
    for (auto &kv : p->groups)
        JERK_CUDA_B(corr_attrs(kv.first));
    for (const FoldRows &R : p->rowsets)
        if (R.len > 0)
            JERK_CUDA_B(fold_attrs(R.len));
    JERK_CUDA_B(multi_attrs());
    JERK_CUDA_B(cudaEventCreateWithFlags(&p->ev_done, cudaEventDisableTiming));
    for (int i = 0; i < jerk_plan::kRing; i++)
        JERK_CUDA_B(cudaEventCreateWithFlags(&p->ev_batch[i], cudaEventDisableTiming));
    JERK_CUDA_B(cudaHostAlloc(&p->h_counts, 2 * sizeof(unsigned int), cudaHostAllocDefault));
    JERK_CUDA_B(cudaMalloc(&p->d_hit_count, sizeof(unsigned int)));
    JERK_CUDA_B(cudaMalloc(&p->d_status, sizeof(unsigned int)));
    JERK_CUDA_B(cudaMemsetAsync(p->d_status, 0, sizeof(unsigned int), p->stream));
    {
        int rc = alloc_hits(p, want_hits);
        if (rc != JERK_OK)
            return bail(rc);
    }
    // the next batch's buffers come last and may be missing; what is allocated
    // later (plan_malloc) may take their place
    if (cudaMalloc(&p->d_prepped[1], sizeof(float2) * p->prepped_f2) != cudaSuccess ||
        cudaMalloc(&p->d_rinds[1], rinds_bytes) != cudaSuccess) {
        cudaGetLastError();
        cudaFree(p->d_prepped[1]);
        p->d_prepped[1] = nullptr;
        p->d_rinds[1] = nullptr;
    }
    JERK_CUDA_B(cudaStreamSynchronize(p->stream));
#undef JERK_CUDA_B
    *out = p;
    return JERK_OK;
}

static int copy_spectrum(jerk_plan *p, float2 *dst, const void *spectrum, int on_device)
{
    JERK_CUDA(cudaMemcpyAsync(dst, spectrum, sizeof(float2) * p->obs.numbins,
                              on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice,
                              p->stream));
    if (!on_device)
        p->h2d_bytes += (long long)sizeof(float2) * p->obs.numbins;
    return JERK_OK;
}

static int stage_spectrum(jerk_plan *p, const void *spectrum, int on_device, const float2 **spec)
{
    if (on_device && !p->use_graph) {
        *spec = (const float2 *)spectrum;
        return JERK_OK;
    }
    if (p->spec_cap < p->obs.numbins) {
        cudaFree(p->d_spec);
        p->d_spec = nullptr;
        JERK_CUDA(plan_malloc(p, &p->d_spec, sizeof(float2) * p->obs.numbins));
        p->spec_cap = p->obs.numbins;
    }
    *spec = p->d_spec;
    return copy_spectrum(p, p->d_spec, spectrum, on_device);
}

static SearchDev make_args(const jerk_plan *p, const float2 *spec)
{
    SearchDev a{};
    a.spec = spec;
    a.numbins = p->obs.numbins;
    a.lobin = p->obs.lobin;
    a.nsubs = p->nsubs;
    a.nstages = p->obs.numharmstages;
    a.corr_uselen = p->obs.corr_uselen;
    a.numz0 = p->subs[0].numz;
    a.numw0 = p->subs[0].numw;
    a.norm_type = p->obs.norm_type;
    a.nph = p->obs.nph;
    for (int i = 0; i < kMaxStages; i++)
        a.powcut[i] = i < p->obs.numharmstages ? p->obs.powcut[i] : INFINITY;
    a.subs = p->d_subs;
    a.steps = p->d_steps;
    a.bank = p->d_bank;
    a.twiddles = p->d_tw;
    a.classes = p->d_classes;
    a.rowsets = p->d_rowsets;
    a.zinds = p->d_zinds;
    a.wind = p->d_wind;
    a.prepped = p->d_prepped[0];
    a.planes = p->d_planes;
    a.rinds = p->d_rinds[0];
    a.hit_keys = p->d_hit_keys;
    a.hit_pows = p->d_hit_pows;
    a.hit_count = p->d_hit_count;
    a.max_hits = p->max_hits;
    a.status = p->d_status;
    return a;
}

// prep + correlation for one batch (volumes only)
static inline double fft_flops(int n)
{
    return 5.0 * n * log2((double)n);
}

// algorithmic traffic and operations of one row set over a batch: each row
// read once, each prepared window once, every good power written once; the
// product and the transforms
static void rowset_work(const jerk_plan *p, const SearchDev &a, const FoldRows &R, double *bytes,
                        double *flops)
{
    auto add = [&](double rows, int sub, double row_f2, double fl) {
        double numrs = 0;
        for (int b = 0; b < a.nb; b++)
            numrs += p->hsteps[(size_t)(a.first_rstep + b) * p->nsubs + sub].numrs;
        *bytes += rows * row_f2 * 8.0 + a.nb * row_f2 * 4.0 + rows * numrs * 4.0;
        *flops += rows * (a.nb * fl + numrs * 3.0);
    };
    if (R.len < 0) {
        for (int s = 0; s < p->nsubs; s++)
            if (p->subs[s].fftlen == -R.len)
                add((double)p->subs[s].numw * p->subs[s].numz, s, -R.len,
                    fft_flops(-R.len) + 6.0 * -R.len);
        return;
    }
    int li = 0;
    while (kFoldLens[li] != R.len)
        li++;
    const std::vector<double> &rows = p->class_rows[li];
    for (size_t c = 0; c < rows.size(); c++)
        if (rows[c] > 0.0)
            add(rows[c], p->fold_classes[c].sub, 2.0 * R.len,
                2 * (fft_flops(R.len) + 6.0 * R.len));
}

// The rows of the subharmonics subs (one fftlen), numbered consecutively.
static RowGroup row_group(const jerk_plan *p, const std::vector<int> &subs)
{
    RowGroup G{};
    G.n = (int)subs.size();
    int rows = 0;
    for (int i = 0; i < G.n; i++) {
        const int s = subs[i];
        G.sub[i] = s;
        G.rowstart[i] = rows;
        rows += p->subs[s].numw * p->subs[s].numz;
    }
    G.rowstart[G.n] = rows;
    return G;
}

// Batch arguments: rsteps from k on (to the pass's end at most), in buffers buf.
static void batch_args(const jerk_plan *p, long long k, int buf, SearchDev &a)
{
    const jerk_plan::Pass &ps = p->pass;
    a.first_rstep = k;
    a.nb = (int)std::min<long long>(p->batch, ps.first + ps.count - k);
    a.planes = p->d_planes;
    a.prepped = p->d_prepped[buf];
    a.rinds = p->d_rinds[buf];
}

// The batch at the pass's next rstep, and whether the one after it is to be
// prepared beside it (into *ahead).
static bool next_batch(jerk_plan *p, SearchDev *ahead)
{
    jerk_plan::Pass &ps = p->pass;
    batch_args(p, ps.next, ps.buf, ps.a);
    const long long after = ps.next + ps.a.nb;
    if (!p->d_rinds[1] || after >= ps.first + ps.count)
        return false;
    *ahead = ps.a;
    batch_args(p, after, ps.buf ^ 1, *ahead);
    return true;
}

static void batch_enqueued(jerk_plan *p, bool ahead)
{
    jerk_plan::Pass &ps = p->pass;
    ps.next += ps.a.nb;
    ps.nbatch++;
    ps.prepared = ahead;
    if (ahead)
        ps.buf ^= 1;
}

static void prep_work(const jerk_plan *p, const SearchDev &a, double *bytes, double *flops)
{
    for (int s = 0; s < p->nsubs; s++) {
        const int N = p->subs[s].fftlen;
        *bytes += (double)a.nb * (N / 2 * 8.0 + N / 2 * 8.0);
        *flops += (double)a.nb * fft_flops(N);
    }
}

static int run_prep(jerk_plan *p, const SearchDev &a)
{
    double bytes = 0, flops = 0;
    prep_work(p, a, &bytes, &flops);
    const int tok = launch_begin(p, kclass(p, "prep"), bytes, flops);
    cudaError_t e = launch_prep(a, p->maxfft, p->prep_smem, p->stream);
    launch_end(p, tok);
    return e == cudaSuccess ? JERK_OK : cuda_fail(e, "prep_kernel");
}

// A batch's volumes (prepared: its rows are there already).  ahead, if not
// null: the next batch's arguments, whose preparation runs beside this one's
// correlation.  Preparation is a chain of latencies on a few CTAs: 16 us of a
// 62-us batch at zmax 20, wmax 60, 8 harmonics; a pass takes 4.71 ms with it
// in turn, 4.30 beside (zmax 100, 16 harmonics, 2^22 samples 14.07 and 13.68,
// zmax 50, wmax 150 36.2 and 35.5).  Order: it waits for the last harmonic
// sum, which reads the buffers it writes; the correlation starts once its CTAs
// have, needing only what came before it.
static int run_volumes(jerk_plan *p, const SearchDev &a, bool prepared, const SearchDev *ahead)
{
    if (!prepared) {
        const int rc = run_prep(p, a);
        if (rc != JERK_OK)
            return rc;
    }
    if (ahead) {
        const int rc = run_prep(p, *ahead);
        if (rc != JERK_OK)
            return rc;
    }
    cudaError_t e = cudaSuccess;
    // The next launch needs the kernel before (as in enqueue_wave): after the
    // next batch's preparation the rows are older than it, and whatever waited
    // for it lets the others go.
    bool first = !ahead;
    for (auto &kv : p->groups) {
        const RowGroup G = row_group(p, kv.second);
        // algorithmic traffic: each kernel row read once per batch, each
        // prepared chunk read once, every good power written once
        const int N = kv.first;
        double bytes = 0, flops = 0;
        for (int i = 0; i < G.n; i++) {
            const int s = G.sub[i];
            const double nrow = (double)p->subs[s].numw * p->subs[s].numz;
            double numrs = 0;
            for (int b = 0; b < a.nb; b++)
                numrs += p->hsteps[(size_t)(a.first_rstep + b) * p->nsubs + s].numrs;
            bytes += nrow * N * 8.0 + a.nb * N / 2 * 8.0 + nrow * numrs * 4.0;
            flops += nrow * a.nb * (fft_flops(N) + 6.0 * N) + nrow * numrs * 3.0;
        }
        const int tok = launch_begin(p, kclass(p, "corr_" + std::to_string(N)), bytes, flops);
        e = launch_corr(a, N, G, G.rowstart[G.n], p->stream);  // (waits)
        launch_end(p, tok);
        first = false;
        if (e != cudaSuccess)
            return cuda_fail(e, "corr_kernel");
    }
    int sets[kMaxRowSets][2], nsets = 0;
    const FoldRows *rows[kMaxRowSets];
    double mbytes = 0, mflops = 0;
    for (size_t i = 0; i < p->rowsets.size(); i++) {
        const FoldRows &R = p->rowsets[i];
        if (!p->own_launch[i]) {
            if (p->profiling)
                rowset_work(p, a, R, &mbytes, &mflops);
            sets[nsets][0] = 0;
            sets[nsets][1] = (int)i;
            rows[nsets++] = &R;
            continue;
        }
        double bytes = 0, flops = 0;
        if (p->profiling)
            rowset_work(p, a, R, &bytes, &flops);
        const int tok = launch_begin(p, kclass(p, "corr_fold_" + std::to_string(R.len)), bytes,
                                     flops);
        e = launch_corr_fold(R.len, a, R, first, p->stream);
        first = false;
        launch_end(p, tok);
        if (e != cudaSuccess)
            return cuda_fail(e, "corr_fold_kernel");
    }
    if (nsets) {
        const int tok = launch_begin(p, kclass(p, "corr_multi"), mbytes, mflops);
        e = launch_corr_multi(&a, 1, sets, rows, nsets, first, p->stream);
        launch_end(p, tok);
        if (e != cudaSuccess)
            return cuda_fail(e, "corr_multi_kernel");
    }
    return JERK_OK;
}

// A search pass is enqueued batch by batch, so a host thread driving several
// plans can keep each a few batches ahead of the device instead of filling
// the launch queue with one whole spectrum.

static int pass_begin(jerk_plan *p, const float2 *spec, long long first, long long count)
{
    jerk_plan::Pass &ps = p->pass;
    ps = jerk_plan::Pass();
    ps.a = make_args(p, spec);
    ps.first = first;
    ps.count = count;
    ps.next = first;
    JERK_CUDA(cudaMemsetAsync(p->d_hit_count, 0, sizeof(unsigned int), p->stream));
    // a pass that reported a failed wait or index leaves no trace in the next
    JERK_CUDA(cudaMemsetAsync(p->d_status, 0, sizeof(unsigned int), p->stream));
    if (p->wait_probe)
        JERK_CUDA(launch_wait_probe(p->d_status, p->wait_probe == 2, p->stream));
    return JERK_OK;
}

// Batches whose harmonic sums have finished (non-blocking).
static long long pass_done_batches(jerk_plan *p)
{
    jerk_plan::Pass &ps = p->pass;
    while (ps.ndone < ps.nbatch && cudaEventQuery(p->ev_batch[ps.ndone % jerk_plan::kRing]) ==
                                       cudaSuccess)
        ps.ndone++;
    return ps.ndone;
}

// Whether a batch takes the ring of row copies: the default form, on volumes
// large enough for it.
static bool use_ring(const jerk_plan *p, const SearchDev &a)
{
    return p->harm_mode == kHarmRing &&
           harm_ring_wins(4.0 * (double)p->plane_floats / p->batch * a.nb);
}

// The plan's own harmonic-sum launch for batch arguments a.
static cudaError_t launch_harmsum_of(const jerk_plan *p, const SearchDev &a, cudaStream_t st)
{
    static const HarmTma no_maps{};
    if (p->harm_mode == kHarmRing)
        return use_ring(p, a) ? launch_harm_ring(a, st) : launch_harmsum(a, no_maps, false, st);
    return p->harm_mode >= 3 ? launch_harmsum_tma(a, *p->tma, p->harm_tile, st)
           : p->harm_mode == 2 ? launch_harmsum(a, *p->tma, true, st)
                               : launch_harmsum(a, no_maps, false, st);
}

// algorithmic traffic of one batch's harmonic sum: every volume read once
static void harmsum_work(const jerk_plan *p, const SearchDev &a, double *bytes, double *flops)
{
    double b = 0;
    const double npts = (double)a.nb * p->subs[0].numw * p->subs[0].numz * p->obs.corr_uselen;
    for (int s = 0; s < p->nsubs; s++) {
        double numrs = 0;
        for (int k = 0; k < a.nb; k++)
            numrs += p->hsteps[(size_t)(a.first_rstep + k) * p->nsubs + s].numrs;
        b += (double)p->subs[s].numw * p->subs[s].numz * numrs * 4.0;
    }
    *bytes += b;
    *flops += npts * p->nsubs;
}

static int pass_enqueue_one(jerk_plan *p)
{
    jerk_plan::Pass &ps = p->pass;
    SearchDev &a = ps.a;
    SearchDev after;
    const bool ahead = next_batch(p, &after);
    int rc = run_volumes(p, a, ps.prepared, ahead ? &after : nullptr);
    if (rc != JERK_OK)
        return rc;
    double bytes = 0, flops = 0;
    harmsum_work(p, a, &bytes, &flops);
    const int tok = launch_begin(p, kclass(p, "harmsum"), bytes, flops);
    cudaError_t e = launch_harmsum_of(p, a, p->stream);
    launch_end(p, tok);
    if (e != cudaSuccess)
        return cuda_fail(e, "harmsum_kernel");
    if (!ps.capturing)
        JERK_CUDA(cudaEventRecord(p->ev_batch[ps.nbatch % jerk_plan::kRing], p->stream));
    batch_enqueued(p, ahead);
    return JERK_OK;
}

static int pass_finish_enqueue(jerk_plan *p)
{
    jerk_plan::Pass &ps = p->pass;
    JERK_CUDA(cudaMemcpyAsync(p->h_counts, p->d_hit_count, sizeof(unsigned int),
                              cudaMemcpyDeviceToHost, p->stream));
    JERK_CUDA(cudaMemcpyAsync(p->h_counts + 1, p->d_status, sizeof(unsigned int),
                              cudaMemcpyDeviceToHost, p->stream));
    // (inside a capture an event record is only a dependency marker; graph
    // mode records ev_done after each launch of the graph instead)
    if (!ps.capturing)
        JERK_CUDA(cudaEventRecord(p->ev_done, p->stream));
    ps.all_enqueued = true;
    return JERK_OK;
}

// Enqueue batches until `ahead` of them are queued or running beyond those
// finished (ahead <= 0: all of them).  Returns 1 while batches remain to be
// enqueued, 0 once the pass is fully enqueued, < 0 on error.
static int pass_advance(jerk_plan *p, int ahead)
{
    jerk_plan::Pass &ps = p->pass;
    if (ps.error)
        return ps.error;
    if (ps.all_enqueued)
        return 0;
    const int limit = ahead <= 0 ? 1 << 30 : std::min(ahead, jerk_plan::kRing - 2);
    while (ps.next < ps.first + ps.count) {
        if (!ps.capturing && ps.nbatch - pass_done_batches(p) >= limit)
            return 1;
        int rc = pass_enqueue_one(p);
        if (rc != JERK_OK)
            return ps.error = rc;
    }
    int rc = pass_finish_enqueue(p);
    if (rc != JERK_OK)
        ps.error = rc;
    return rc == JERK_OK ? 0 : rc;
}

// Enqueue one whole search pass (no host synchronisation beyond the
// bookkeeping of pass_advance).
static int enqueue_search_pass(jerk_plan *p, const float2 *spec, long long first, long long count)
{
    int rc = pass_begin(p, spec, first, count);
    if (rc != JERK_OK)
        return rc;
    rc = pass_advance(p, 0);
    return rc < 0 ? rc : JERK_OK;
}

// Wait for an enqueued pass and read its hit count.
static int finish_search_pass(jerk_plan *p, unsigned int *nhits_out)
{
    JERK_CUDA(cudaEventSynchronize(p->ev_done));
    collect_timings(p);
    p->d2h_bytes += 2 * sizeof(unsigned int);
    const unsigned status = p->h_counts[1];  // kStatus* (jerk_async.cuh)
    if (status & kStatusCopy)
        return fail(JERK_ECUDA, "correlation: a data-row copy into shared memory timed out");
    if (status & kStatusSumCopy)
        return fail(JERK_ECUDA, "harmonic sum: a row copy into shared memory timed out");
    if (status)
        return fail(JERK_EINVAL, "harmonic sum: a subharmonic r index left its row");
    *nhits_out = p->h_counts[0];
    return JERK_OK;
}

static int run_search_pass(jerk_plan *p, const float2 *spec, long long first, long long count,
                           unsigned int *nhits_out)
{
    int rc = enqueue_search_pass(p, spec, first, count);
    if (rc != JERK_OK)
        return rc;
    return finish_search_pass(p, nhits_out);
}

static int check_range(const jerk_plan *p, long long first_rstep, long long num_rsteps,
                       long long *count)
{
    if (first_rstep < 0 || first_rstep > p->nrsteps)
        return fail(JERK_EINVAL, "jerk_search: first_rstep out of range");
    *count = p->nrsteps - first_rstep;
    if (num_rsteps > 0 && num_rsteps < *count)
        *count = num_rsteps;
    return JERK_OK;
}

// Graph mode: the first pass over (first, count) is captured from the plan's
// stream into a CUDA graph (every batch's prep, correlation and harmonic-sum
// launches, the hit-count read-back and the completion event) and replayed
// for every later spectrum; the spectrum is staged into d_spec beforehand, so
// the graph's pointers never change.  A hit-buffer reallocation drops it.
static int launch_graph_pass(jerk_plan *p, const float2 *spec, long long first, long long count)
{
    jerk_plan::Pass &ps = p->pass;
    if (!p->graph_exec || p->graph_first != first || p->graph_count != count) {
        drop_graph(p);
        JERK_CUDA(cudaStreamBeginCapture(p->stream, cudaStreamCaptureModeThreadLocal));
        int rc = pass_begin(p, spec, first, count);
        ps.capturing = true;
        if (rc == JERK_OK)
            rc = pass_advance(p, 0);
        cudaGraph_t g = nullptr;
        const cudaError_t ec = cudaStreamEndCapture(p->stream, &g);
        ps.capturing = false;
        if (rc < 0 || ec != cudaSuccess) {
            if (g)
                cudaGraphDestroy(g);
            ps.error = rc < 0 ? rc : JERK_ECUDA;
            return rc < 0 ? rc : cuda_fail(ec, "cudaStreamEndCapture");
        }
        const cudaError_t ei = cudaGraphInstantiate(&p->graph_exec, g, 0);
        cudaGraphDestroy(g);
        if (ei != cudaSuccess) {
            p->graph_exec = nullptr;
            return cuda_fail(ei, "cudaGraphInstantiate");
        }
        p->graph_first = first;
        p->graph_count = count;
    }
    // the host bookkeeping of a fully enqueued pass
    ps = jerk_plan::Pass();
    ps.a = make_args(p, spec);
    ps.first = first;
    ps.count = count;
    ps.next = first + count;
    ps.all_enqueued = true;
    JERK_CUDA(cudaGraphLaunch(p->graph_exec, p->stream));
    JERK_CUDA(cudaEventRecord(p->ev_done, p->stream));
    p->graph_replays++;
    return JERK_OK;
}

extern "C" int jerk_search_async(jerk_plan *p, const void *spectrum, int spectrum_on_device,
                                 long long first_rstep, long long num_rsteps)
{
    if (!p || !spectrum)
        return fail(JERK_EINVAL, "jerk_search_async: null argument");
    if (p->in_flight)
        return fail(JERK_EINVAL, "jerk_search_async: a search is already in flight on this plan");
    long long count = 0;
    int rc = check_range(p, first_rstep, num_rsteps, &count);
    if (rc != JERK_OK)
        return rc;
    int cur = 0;
    cudaGetDevice(&cur);
    if (cur != p->device)
        JERK_CUDA(cudaSetDevice(p->device));
    const float2 *spec = nullptr;
    rc = stage_spectrum(p, spectrum, spectrum_on_device, &spec);
    if (rc != JERK_OK)
        return rc;
    if (p->use_graph && !p->profiling) {
        rc = launch_graph_pass(p, spec, first_rstep, count);
    } else {
        rc = pass_begin(p, spec, first_rstep, count);
        if (rc == JERK_OK)
            rc = pass_advance(p, 4);
    }
    if (rc < 0)
        return rc;
    p->in_flight = true;
    p->inflight_spec = spec;
    p->inflight_first = first_rstep;
    p->inflight_count = count;
    return JERK_OK;
}

extern "C" int jerk_search_advance(jerk_plan *p, int ahead)
{
    if (!p || !p->in_flight)
        return 0;
    return pass_advance(p, ahead);
}

extern "C" int jerk_search_ready(jerk_plan *p)
{
    if (!p || !p->in_flight)
        return 1;
    if (p->pass.error)
        return p->pass.error;
    if (!p->pass.all_enqueued)
        return 0;
    const cudaError_t e = cudaEventQuery(p->ev_done);
    if (e == cudaSuccess)
        return 1;
    if (e == cudaErrorNotReady)
        return 0;
    return cuda_fail(e, "jerk_search_ready");
}

// ---------------------------------------------------------------------------
// Waves: the current batches of several plans' passes in merged launches, each
// covering every plan of the wave (up to kMaxGroupPlans): one preparation (and
// one of the next batches), one correlation and one harmonic sum per stage count
// and form, so spectra of uneven length and geometry share launches and small
// ones fill the GPU together; what fills it by itself (a plan's row sets, long
// unfolded lengths, large volumes) keeps launches of its own.  Every plan's sums
// run as in its own launches, so its results are bitwise the same.

extern "C" int jerk_search_begin(jerk_plan *p, const void *spectrum, int spectrum_on_device,
                                 long long first_rstep, long long num_rsteps)
{
    if (!p || !spectrum)
        return fail(JERK_EINVAL, "jerk_search_begin: null argument");
    if (p->in_flight)
        return fail(JERK_EINVAL, "jerk_search_begin: a search is already in flight on this plan");
    long long count = 0;
    int rc = check_range(p, first_rstep, num_rsteps, &count);
    if (rc != JERK_OK)
        return rc;
    int cur = 0;
    cudaGetDevice(&cur);
    if (cur != p->device)
        JERK_CUDA(cudaSetDevice(p->device));
    const float2 *spec = nullptr;
    rc = stage_spectrum(p, spectrum, spectrum_on_device, &spec);
    if (rc == JERK_OK)
        rc = pass_begin(p, spec, first_rstep, count);
    if (rc != JERK_OK)
        return rc;
    p->in_flight = true;
    p->inflight_spec = spec;
    p->inflight_first = first_rstep;
    p->inflight_count = count;
    return JERK_OK;
}

// One wave over W (same stream): every plan's next batch.
static int enqueue_wave(const std::vector<jerk_plan *> &W)
{
    jerk_plan *p0 = W[0];
    cudaStream_t st = p0->stream;
    const int n = (int)W.size();
    int maxfft = 0;
    size_t prep_smem = 0;
    // rows to prepare before this wave's correlation, and beside it
    GroupLaunch M{}, now{}, next{};
    bool ahead[kMaxGroupPlans];
    double work[2][2] = {};  // bytes, operations of either
    for (int i = 0; i < n; i++) {
        jerk_plan *p = W[i];
        ahead[i] = next_batch(p, &next.P[next.n]);
        M.P[M.n++] = p->pass.a;
        if (!p->pass.prepared) {
            prep_work(p, p->pass.a, &work[0][0], &work[0][1]);
            now.P[now.n++] = p->pass.a;
        }
        if (ahead[i]) {
            prep_work(p, next.P[next.n], &work[1][0], &work[1][1]);
            next.n++;
        }
        maxfft = std::max(maxfft, p->maxfft);
        prep_smem = std::max(prep_smem, p->prep_smem);
    }
    auto fail_all = [&](cudaError_t e, const char *what) {
        const int rc = cuda_fail(e, what);
        for (jerk_plan *p : W)
            p->pass.error = rc;
        return rc;
    };
    cudaError_t e = cudaSuccess;
    int tok = 0;
    for (const GroupLaunch *G : {&now, &next}) {
        if (!G->n)
            continue;
        tok = launch_begin(p0, kclass(p0, "wave_prep"), work[G == &next][0],
                           work[G == &next][1]);
        e = launch_prep_group(*G, maxfft, prep_smem, st);
        launch_end(p0, tok);
        if (e != cudaSuccess)
            return fail_all(e, "prep_group_kernel");
    }

    // correlation: the row sets that fill the GPU twice over by themselves
    // (and the long unfolded lengths) in their plan's own launches, all the
    // others of every plan in one
    int sets[kMaxGroupPlans * kMaxRowSets][2], nsets = 0;
    const FoldRows *rows[kMaxGroupPlans * kMaxRowSets];
    double mbytes = 0, mflops = 0;
    bool first = !next.n;  // the next launch needs the one before
    for (int i = 0; i < n; i++) {
        jerk_plan *p = W[i];
        const SearchDev &a = p->pass.a;
        for (auto &kv : p->groups) {
            const RowGroup G = row_group(p, kv.second);
            tok = launch_begin(p0, kclass(p0, "wave_corr_" + std::to_string(kv.first)), 0.0, 0.0);
            e = launch_corr(a, kv.first, G, G.rowstart[G.n], st);
            launch_end(p0, tok);
            first = false;
            if (e != cudaSuccess)
                return fail_all(e, "corr_kernel");
        }
        for (size_t k = 0; k < p->rowsets.size(); k++) {
            const FoldRows &R = p->rowsets[k];
            double bytes = 0, flops = 0;
            if (p0->profiling)
                rowset_work(p, a, R, &bytes, &flops);
            if (!p->own_launch[k]) {
                sets[nsets][0] = i;
                sets[nsets][1] = (int)k;
                rows[nsets++] = &R;
                mbytes += bytes;
                mflops += flops;
                continue;
            }
            tok = launch_begin(p0, kclass(p0, "wave_corr_fold_" + std::to_string(R.len)), bytes,
                               flops);
            e = launch_corr_fold(R.len, a, R, first, st);
            first = false;
            launch_end(p0, tok);
            if (e != cudaSuccess)
                return fail_all(e, "corr_fold_kernel");
        }
    }
    if (nsets) {
        tok = launch_begin(p0, kclass(p0, "wave_corr_multi"), mbytes, mflops);
        e = launch_corr_multi(M.P, n, sets, rows, nsets, first, st);
        launch_end(p0, tok);
        if (e != cudaSuccess)
            return fail_all(e, "corr_multi_kernel");
    }

    // harmonic sums: the ring and the gather form merged per stage count;
    // plans that fill the GPU twice over, or are tuned to another form, launch
    // their own
    std::map<std::pair<int, bool>, std::vector<int>> byS;  // (stages, ring)
    for (int i = 0; i < n; i++) {
        jerk_plan *p = W[i];
        const SearchDev &a = p->pass.a;
        // The gather form merges what does not fill two waves.  The ring splits
        // its rows over the resident CTAs, alone or merged: merged, small plans
        // share one start and end (three of 0.5 GB volumes, 66.6 -> 64.7 ms a
        // search); beside a large plan they get one CTA or two, whose rounding is
        // then the whole launch's time (two plans of 2.6 GB and two of 0.1 GB:
        // 399 ms of sums, 202 so), so a large one is launched by itself.
        const bool ring = use_ring(p, a);
        const long long ctas = (long long)((a.corr_uselen + 127) / 128) * a.numw0 * a.nb;
        if (ring ? 4.0 * (double)p->plane_floats / p->batch * a.nb < 1e9
                 : (p->harm_mode <= 1 || p->harm_mode == kHarmRing) &&
                       ctas < 2 * harmsum_wave_ctas(a.nstages)) {
            byS[{p->obs.numharmstages, ring}].push_back(i);
            continue;
        }
        double bytes = 0, flops = 0;
        harmsum_work(p, p->pass.a, &bytes, &flops);
        tok = launch_begin(p0, kclass(p0, "wave_harmsum"), bytes, flops);
        e = launch_harmsum_of(p, p->pass.a, st);
        launch_end(p0, tok);
        if (e != cudaSuccess)
            return fail_all(e, "harmsum_kernel");
    }
    for (auto &kv : byS) {
        GroupLaunch H{};
        H.n = (int)kv.second.size();
        double bytes = 0, flops = 0;
        for (int j = 0; j < H.n; j++) {
            jerk_plan *p = W[kv.second[j]];
            H.P[j] = p->pass.a;
            harmsum_work(p, p->pass.a, &bytes, &flops);
        }
        tok = launch_begin(p0, kclass(p0, "wave_harmsum"), bytes, flops);
        e = kv.first.second ? launch_harm_ring_group(H, kv.first.first, st)
                            : launch_harmsum_group(H, kv.first.first, st);
        launch_end(p0, tok);
        if (e != cudaSuccess)
            return fail_all(e, "harmsum_group_kernel");
    }

    for (int i = 0; i < n; i++) {
        jerk_plan *p = W[i];
        jerk_plan::Pass &ps = p->pass;
        JERK_CUDA(cudaEventRecord(p->ev_batch[ps.nbatch % jerk_plan::kRing], st));
        batch_enqueued(p, ahead[i]);
        if (ps.next >= ps.first + ps.count) {
            const int rc = pass_finish_enqueue(p);
            if (rc != JERK_OK)
                return ps.error = rc;
        }
    }
    return JERK_OK;
}

extern "C" int jerk_group_advance(jerk_plan *const *plans, int nplans, int ahead)
{
    if (!plans || nplans < 0)
        return fail(JERK_EINVAL, "jerk_group_advance: bad argument");
    jerk_plan *first = nullptr;
    for (int i = 0; i < nplans; i++) {
        jerk_plan *p = plans[i];
        if (!p)
            return fail(JERK_EINVAL, "jerk_group_advance: null plan");
        if (!p->in_flight || p->pass.all_enqueued || p->pass.error)
            continue;
        if (!first)
            first = p;
        else if (p->stream != first->stream || p->device != first->device)
            return fail(JERK_EINVAL, "jerk_group_advance: plans on different streams or devices");
    }
    if (!first)
        return 0;
    int cur = 0;
    cudaGetDevice(&cur);
    if (cur != first->device)
        JERK_CUDA(cudaSetDevice(first->device));
    const int limit = ahead <= 0 ? 1 << 30 : std::min(ahead, jerk_plan::kRing - 2);
    for (;;) {
        std::vector<jerk_plan *> sel;
        bool left = false;
        for (int i = 0; i < nplans; i++) {
            jerk_plan *p = plans[i];
            jerk_plan::Pass &ps = p->pass;
            if (!p->in_flight || ps.all_enqueued || ps.error)
                continue;
            left = true;
            if (ps.nbatch - pass_done_batches(p) < limit)
                sel.push_back(p);
        }
        if (sel.empty())
            return left ? 1 : 0;
        for (size_t i = 0; i < sel.size(); i += kMaxGroupPlans) {
            std::vector<jerk_plan *> W(sel.begin() + i,
                                       sel.begin() + std::min(sel.size(), i + kMaxGroupPlans));
            const int rc = enqueue_wave(W);
            if (rc != JERK_OK)
                return rc;
        }
    }
}

extern "C" int jerk_search_group(jerk_plan *const *plans, const void *const *spectra,
                                 const int *spectrum_on_device, int nplans, jerk_cand **cands,
                                 long long *ncands)
{
    if (!plans || !spectra || !spectrum_on_device || !cands || !ncands || nplans < 1)
        return fail(JERK_EINVAL, "jerk_search_group: bad argument");
    for (int i = 0; i < nplans; i++) {
        cands[i] = nullptr;
        ncands[i] = 0;
    }
    int rc = JERK_OK, began = 0;
    for (; began < nplans && rc == JERK_OK; began++)
        rc = jerk_search_begin(plans[began], spectra[began], spectrum_on_device[began], 0, 0);
    if (rc != JERK_OK)
        began--;  // the failed one holds no pass
    if (rc == JERK_OK)
        rc = jerk_group_advance(plans, nplans, 0);
    // every begun pass is collected (ends its in-flight state), even after a
    // failure; the first error is returned
    for (int i = 0; i < began; i++) {
        const int r = jerk_search_collect(plans[i], &cands[i], &ncands[i], nullptr);
        if (rc == JERK_OK)
            rc = r;
    }
    return rc;
}

// What decoding a hit key needs: the fundamental's geometry and, per rstep,
// the fundamental's first r (hsteps[rs][0].rlo).
struct HitGeom {
    int S = 1;
    long long numrs0 = 0, numz0 = 0, numw0 = 0;
    int zlo0 = 0, wlo0 = 0;
    const long long *numindep = nullptr;
    std::function<long long(long long)> rlo_of;
};

// order[i]: the index of the i-th key in ascending order.  Keys are distinct;
// many are sorted by 11-bit digits of the bits they use.
static void sort_keys(const unsigned long long *keys, uint32_t n, std::vector<uint32_t> &order)
{
    order.resize(n);
    for (uint32_t i = 0; i < n; i++)
        order[i] = i;
    if (n < 4096) {
        std::sort(order.begin(), order.end(),
                  [&](uint32_t x, uint32_t y) { return keys[x] < keys[y]; });
        return;
    }
    unsigned long long used = 0;
    for (uint32_t i = 0; i < n; i++)
        used |= keys[i];
    constexpr int kBits = 11, kBins = 1 << kBits;
    std::vector<uint32_t> other(n), start(kBins + 1);
    for (int shift = 0; shift < 64 && used >> shift; shift += kBits) {
        std::fill(start.begin(), start.end(), 0u);
        for (uint32_t i = 0; i < n; i++)
            start[(keys[i] >> shift & (kBins - 1)) + 1]++;
        for (int d = 0; d < kBins; d++)
            start[d + 1] += start[d];
        for (uint32_t i = 0; i < n; i++)
            other[start[keys[order[i]] >> shift & (kBins - 1)]++] = order[i];
        order.swap(other);
    }
}

// Hits in key order -- the reference's insertion order (rstep, stage, w, z,
// r; src/accel_utils_cu.c:857-929) -- decoded into candidates with their
// sigma and inserted with the reference's rule.  order receives the sorted
// permutation of the input.
static void hits_to_list(const HitGeom &g, const unsigned long long *keys, const float *pows,
                         uint32_t nh, std::vector<uint32_t> &order, CandList &L)
{
    sort_keys(keys, nh, order);
    // decode + sigma per hit (independent, so spread over host threads when
    // there are many), then the insertions in key order (sequential: each
    // depends on the list the earlier ones left)
    std::vector<jerk_cand> cv(nh);
    auto decode = [&](uint32_t lo, uint32_t hi) {
        for (uint32_t i = lo; i < hi; i++) {
            unsigned long long key = keys[order[i]];
            const int kk = (int)(key % g.numrs0);
            key /= g.numrs0;
            const int jj = (int)(key % g.numz0);
            key /= g.numz0;
            const int ii = (int)(key % g.numw0);
            key /= g.numw0;
            const int stage = (int)(key % g.S);
            const long long rs = (long long)(key / g.S);
            const int nhm = 1 << stage;
            jerk_cand &c = cv[i];
            c.power = pows[order[i]];
            c.sigma = (float)jerk_candidate_sigma(c.power, nhm, (double)g.numindep[stage]);
            c.numharm = nhm;
            c.r = ((double)g.rlo_of(rs) + kk * kDR) / (double)nhm;
            c.z = (g.zlo0 + jj * (double)kDZ) / (double)nhm;
            c.w = (g.wlo0 + ii * (double)kDW) / (double)nhm;
        }
    };
    // about 0.4 us a hit, some 20 us to start a thread
    const uint32_t nthr = std::max(
        1u, std::min({16u, std::thread::hardware_concurrency(), nh / 1024u}));
    if (nthr == 1) {
        decode(0, nh);
    } else {
        std::vector<std::thread> pool;
        const uint32_t per = (nh + nthr - 1) / nthr;
        for (uint32_t t = 0; t < nthr; t++) {
            const uint32_t lo = t * per, hi = std::min(nh, lo + per);
            if (lo < hi)
                pool.emplace_back(decode, lo, hi);
        }
        for (auto &th : pool)
            th.join();
    }
    for (uint32_t i = 0; i < nh; i++)
        insert_cand(L, cv[i]);
}

extern "C" int jerk_search_collect(jerk_plan *p, jerk_cand **cands, long long *ncands,
                                   jerk_hits *hits)
{
    if (!p || !p->in_flight)
        return fail(JERK_EINVAL, "jerk_search_collect: no search in flight");
    p->in_flight = false;
    unsigned int nh = 0;
    int rc = pass_advance(p, 0);  // whatever is not enqueued yet
    if (rc < 0) {
        cudaStreamSynchronize(p->stream);  // what was enqueued ends before the plan is reused
        return rc;
    }
    rc = finish_search_pass(p, &nh);
    if (rc != JERK_OK)
        return rc;
    for (int attempt = 0; (long long)nh > p->max_hits; attempt++) {
        // overflow: the counter kept counting, so one retry with the exact
        // size always suffices
        if (attempt > 2)
            return fail(JERK_OVERFLOW, "hit buffer overflow persisted");
        rc = alloc_hits(p, (long long)nh + (nh >> 3) + 1024);
        if (rc != JERK_OK)
            return rc;
        rc = run_search_pass(p, p->inflight_spec, p->inflight_first, p->inflight_count, &nh);
        if (rc != JERK_OK)
            return rc;
    }

    // hits back, in the reference's insertion order
    std::vector<unsigned long long> keys(nh);
    std::vector<float> pows(nh);
    if (nh) {
        // the pass has ended (ev_done); a synchronous copy does not wait for
        // other work queued behind it on a stream shared with other plans
        JERK_CUDA(cudaMemcpy(keys.data(), p->d_hit_keys, sizeof(unsigned long long) * nh,
                             cudaMemcpyDeviceToHost));
        JERK_CUDA(cudaMemcpy(pows.data(), p->d_hit_pows, sizeof(float) * nh,
                             cudaMemcpyDeviceToHost));
        p->d2h_bytes += (long long)nh * (sizeof(unsigned long long) + sizeof(float));
    }
    HitGeom g;
    g.S = p->obs.numharmstages;
    g.numrs0 = p->obs.corr_uselen;
    g.numz0 = p->subs[0].numz;
    g.numw0 = p->subs[0].numw;
    g.zlo0 = p->zlo0;
    g.wlo0 = p->wlo0;
    g.numindep = p->obs.numindep;
    g.rlo_of = [p](long long rs) { return p->hsteps[(size_t)rs * p->nsubs].rlo; };
    CandList L;
    std::vector<uint32_t> order;
    hits_to_list(g, keys.data(), pows.data(), nh, order, L);
    if (hits) {
        hits->count = nh;
        hits->keys = (unsigned long long *)malloc(sizeof(unsigned long long) * (nh ? nh : 1));
        hits->powers = (float *)malloc(sizeof(float) * (nh ? nh : 1));
        for (uint32_t i = 0; i < nh; i++) {
            hits->keys[i] = keys[order[i]];
            hits->powers[i] = pows[order[i]];
        }
    }
    const long long n = export_list(L, cands);
    if (n < 0)
        return fail(JERK_ENOMEM, "candidate list allocation");
    if (ncands)
        *ncands = n;
    return JERK_OK;
}

extern "C" int jerk_merge_hits(const jerk_obs *obs, const jerk_subharm *fundamental,
                               const unsigned long long *keys, const float *powers,
                               long long nhits, jerk_cand **cands, long long *ncands)
{
    if (!obs || !fundamental || !cands || nhits < 0 || (nhits && (!keys || !powers)))
        return fail(JERK_EINVAL, "jerk_merge_hits: bad argument");
    if (nhits > 0xffffffffll)
        return fail(JERK_EUNSUPPORTED, "jerk_merge_hits: more than 2^32 hits");
    if (fundamental->numharm != 1 || fundamental->harmnum != 1 || fundamental->numz != obs->numz ||
        fundamental->numw < 1 || obs->corr_uselen < 2 || obs->numharmstages < 1 ||
        obs->numharmstages > JERK_MAX_STAGES)
        return fail(JERK_EINVAL, "jerk_merge_hits: fundamental and obs do not match");
    const long long nrsteps = count_rsteps(*obs);
    const long long per_rstep = (long long)obs->numharmstages * fundamental->numw *
                                fundamental->numz * obs->corr_uselen;
    for (long long i = 0; i < nhits; i++)
        if (keys[i] / (unsigned long long)per_rstep >= (unsigned long long)nrsteps)
            return fail(JERK_EINVAL, "jerk_merge_hits: a key lies beyond the last rstep");
    HitGeom g;
    g.S = obs->numharmstages;
    g.numrs0 = obs->corr_uselen;
    g.numz0 = fundamental->numz;
    g.numw0 = fundamental->numw;
    g.zlo0 = calc_required_z(1.0, obs->zlo);
    g.wlo0 = calc_required_w(1.0, obs->wlo);
    g.numindep = obs->numindep;
    const int rstep = (int)(obs->corr_uselen * kDR);
    const double rlo = obs->rlo;
    // as the plan's step table: floor(calc_required_r(1, startr))
    g.rlo_of = [rstep, rlo](long long rs) {
        return (long long)floor(calc_required_r(1.0, rlo + (double)rs * rstep));
    };
    CandList L;
    std::vector<uint32_t> order;
    hits_to_list(g, keys, powers, (uint32_t)nhits, order, L);
    const long long n = export_list(L, cands);
    if (n < 0)
        return fail(JERK_ENOMEM, "candidate list allocation");
    if (ncands)
        *ncands = n;
    return JERK_OK;
}

extern "C" int jerk_search(jerk_plan *p, const void *spectrum, int spectrum_on_device,
                           long long first_rstep, long long num_rsteps, jerk_cand **cands,
                           long long *ncands, jerk_hits *hits)
{
    int rc = jerk_search_async(p, spectrum, spectrum_on_device, first_rstep, num_rsteps);
    if (rc != JERK_OK)
        return rc;
    return jerk_search_collect(p, cands, ncands, hits);
}

extern "C" long long jerk_plan_device_bytes(const jerk_plan *p)
{
    if (!p)
        return 0;
    return (long long)(sizeof(float) * p->plane_floats +
                       (p->d_rinds[1] ? 2 : 1) *
                           (sizeof(uint16_t) * (size_t)p->batch * p->nsubs * p->obs.corr_uselen +
                            sizeof(float2) * p->prepped_f2) +
                       (sizeof(unsigned long long) + sizeof(float)) * p->max_hits +
                       sizeof(StepDev) * p->hsteps.size() + sizeof(float2) * p->spec_cap +
                       sizeof(float2) * p->fold_f2 +
                       (p->own_bank ? sizeof(float2) * jerk_bank_elements(p->subs.data(), p->nsubs)
                                    : 0));
}

extern "C" int jerk_debug_wait_probe(jerk_plan *p, int on)
{
    if (!p)
        return fail(JERK_EINVAL, "jerk_debug_wait_probe: null plan");
    if (p->in_flight)
        return fail(JERK_EINVAL, "jerk_debug_wait_probe: a search is in flight");
    p->wait_probe = on == 2 ? 2 : on != 0;
    drop_graph(p);  // a captured pass holds the old launch arguments
    return JERK_OK;
}

extern "C" int jerk_debug_volume(jerk_plan *p, const void *spectrum, int spectrum_on_device,
                                 long long rstep, int sub, float *out, int *numrs, long long *rlo)
{
    if (!p || !spectrum || !out || sub < 0 || sub >= p->nsubs || rstep < 0 ||
        rstep >= p->nrsteps)
        return fail(JERK_EINVAL, "jerk_debug_volume: bad argument");
    const float2 *spec = nullptr;
    int rc = JERK_OK;
    // a pass in flight may read the staged spectrum: the volume's own is then
    // read in place, or copied to an array that lives until it is done
    struct Staged {
        float2 *d = nullptr;
        ~Staged() { cudaFree(d); }
    } own;
    if (p->in_flight && spectrum_on_device) {
        spec = (const float2 *)spectrum;
    } else if (p->in_flight && p->inflight_spec == p->d_spec) {
        JERK_CUDA(plan_malloc(p, &own.d, sizeof(float2) * p->obs.numbins));
        rc = copy_spectrum(p, own.d, spectrum, spectrum_on_device);
        spec = own.d;
    } else {
        rc = stage_spectrum(p, spectrum, spectrum_on_device, &spec);
    }
    if (rc != JERK_OK)
        return rc;
    SearchDev a = make_args(p, spec);
    a.first_rstep = rstep;
    a.nb = 1;
    // a pass in flight may hold its next batch's prepared rows: the volume's go
    // into the other buffers, which the batches enqueued so far have read when
    // this preparation starts
    const int buf = p->pass.prepared ? p->pass.buf ^ 1 : 0;
    a.prepped = p->d_prepped[buf];
    a.rinds = p->d_rinds[buf];
    rc = run_volumes(p, a, false, nullptr);
    if (rc != JERK_OK)
        return rc;
    JERK_CUDA(cudaStreamSynchronize(p->stream));
    collect_timings(p);
    const SubDev &d = p->hsubs[sub];
    const StepDev &st = p->hsteps[(size_t)rstep * p->nsubs + sub];
    JERK_CUDA(cudaMemcpy2DAsync(out, sizeof(float) * st.numrs, p->d_planes + d.plane_off,
                                sizeof(float) * d.stride, sizeof(float) * st.numrs,
                                (size_t)d.numw * d.numz, cudaMemcpyDeviceToHost, p->stream));
    JERK_CUDA(cudaStreamSynchronize(p->stream));
    if (numrs)
        *numrs = st.numrs;
    if (rlo)
        *rlo = st.rlo;
    return JERK_OK;
}
