// libjamma_b200: per-SNP LMM association (FP64) on B200.
//
// Uab is never materialised: the weighted dot products of [W_1..W_c, x, y] are formed on the
// fly.  Three forms of the search:
//
// Direct form (precision 0, lmm_pairs_kernel below): one warp owns one (SNP, phenotype) pair
// and streams its rotated vectors once per likelihood evaluation.
//
//   phase 1  one pass with two fixed weightings: H = 1 (Iab, for REML's logdet term)
//            and H = H0 (the null-model MLE lambda, for the score test);
//   phase 2  the shared lambda grid; every grid point's H row is tabulated once per
//            cohort (SNP independent), the x-free dot products are pre-reduced, so a
//            grid evaluation only needs the c+2 x-dependent sums; REML and MLE grid
//            log-likelihoods come from the same sums;
//   phase 3  JAX-style golden-section refinement for MLE and REML, per-SNP lambda;
//   epilogue Wald (from the final REML evaluation), LRT and score statistics.
//
// Mixed form (precision 1 and 2, lmm_search_kernel in jb_lmm_search.cuh): a pair per group of
// 4 to 32 lanes, and no likelihood evaluation streams x but those at large lambda
// (direct_fix).  The x-dependent sums come from the SNP's global Chebyshev series in log lambda
// (chunk GEMM rows), log|H^-1| and the x-free sums from per-bracket expansions; the final
// evaluation at each optimum is one more such probe.
//
// Guided form (precision 3, jb_lmm_search.cuh): the FP64 form's decisions on the same series
// where they are certain, by direct evaluations where not, and one direct pass per pair for the
// statistics.
//
// The sequence of evaluations, bracket rules and NaN behaviour follow
// src/jamma/lmm/likelihood_jax.py (148-339 likelihoods, 419-598 search, 601-798
// statistics) exactly; only the summation order of the length-n reductions differs.
#include "jb_common.cuh"
#include "jb_rotate_i8.cuh"

namespace jb {
namespace tc {
int num_sms();
}
}  // namespace jb

#include <cooperative_groups.h>

#include <cmath>
#include <type_traits>

namespace jb {
namespace lmm {

constexpr double kPhi = 0.6180339887498949;
constexpr double kPyyMin = 1e-8;
constexpr int kMaxCvt = 4;

template <int C>
struct Lay {
    static constexpr int R = C + 2;  // vector columns: W_0..W_{C-1}, X = C, Y = C+1
    static constexpr int NI = R * (R + 1) / 2;
    static constexpr int NX = C + 2;  // pairs containing X: (W_a,X) a<C, (X,X), (X,Y)
    static constexpr int NS = NI - NX;
    // GEMMA GetabIndex on 0-based columns (src/jamma/lmm/likelihood.py:25-43)
    __host__ __device__ static constexpr int idx(int a, int b) {
        return a <= b ? (2 * R - (a + 1) + 2) * a / 2 + b - a
                      : (2 * R - (b + 1) + 2) * b / 2 + a - b;
    }
};

struct Params {
    int mode;
    int64_t n;
    int phi;
    int64_t m;
    const double* evals;
    const double* W;
    int64_t ldw;
    const double* Y;
    int64_t ldy;
    const double* G;
    int64_t ldg;
    const double* logl0;
    int n_grid;
    int n_iter;
    const double* loglam;  // n_grid
    const double* logdet;  // n_grid
    const double* H;       // (n_grid + phi) x n: grid rows, then null rows
    const double* S;       // (n_grid + 1 + phi) x phi x NS shared sums
    double c_reml, c_mle, df, n_d;
    jb_lmm_out out;
    // mixed form: Chebyshev expansions of the SNP-independent terms per grid bracket
    const double* cheb;    // [n_grid][1 + phi*NS][kChebN] coefficients (NULL: direct)
    const double* cheb_mid;
    const double* cheb_half;
    const double* tgrid;   // mixed form: n_grid x kChebG Chebyshev values at the grid points
    // Weighted x-sums of every table row r (grid rows, the ones row n_grid, the null rows
    // n_grid+1+f), produced for the whole chunk by two FP64 GEMMs:
    //   CL[j*ldcl + r*(C+phi) + a] = sum_i h_r,i x_ij w_a,i  (a < C)
    //   CL[j*ldcl + r*(C+phi) + C + f] = sum_i h_r,i x_ij y_f,i
    //   CQ[j*ldcq + r] = sum_i h_r,i x_ij^2
    // In the mixed form the rows are the ones row (r = 0) and the kChebG Chebyshev
    // coefficients (r = 1 + k) of the x-dependent sums over the whole log-lambda domain
    // [log 1e-5, log 1e5] (series_xsums), so no probe streams x.
    const double* CL;
    int64_t ldcl;
    const double* CQ;
    int64_t ldcq;
    const double* lam0;  // null-model lambda per phenotype (modes 2-4)
    double gmid, ginv;   // domain centre and 1 / half-width of the global series
    // guided plain form: 2 states per pair (MLE, REML), and the searches left open
    struct SearchState* state;
    int64_t* open_list;
    unsigned long long* open_count;
};

constexpr int kChebN = 25;  // interpolation nodes (degree 24) per bracket
// Global series of the x-dependent sums: each term 1/(lambda e_i + 1) is analytic in
// t = log lambda in the strip |Im t| < pi, so over the 23-wide domain a Chebyshev series
// converges geometrically (Bernstein ellipse rho ~ 1.31): degree 95 leaves at most 7.3e-12 of
// a weight and, over a kinship's eigenvalues, ~1e-13 of the sum's scale, far below the ~1e-9
// relative error of the INT8-rotated genotypes the mixed form's sums are formed from.
constexpr int kChebG = 96;
constexpr int kCoefPerLane = kChebG / 32;  // coefficients k = lane + 32 i held by each lane
static_assert(kChebG % 32 == 0, "series length must be a multiple of the warp size");
constexpr double kDomainLo = 1e-5, kDomainHi = 1e5;

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ double jnan() { return __longlong_as_double(0x7ff8000000000000ll); }
__device__ __forceinline__ double jmax(double a, double b) {  // jnp.maximum: NaN propagates
    return (isnan(a) || isnan(b)) ? jnan() : (a > b ? a : b);
}
__device__ __forceinline__ double clamp_pyy(double v) {
    return (v >= 0.0 && v < kPyyMin) ? kPyyMin : v;
}
__device__ __forceinline__ double rlog(double v) { return v > 0 ? log(v) : 0.0; }

// ---------------------------------------------------------------- special functions
// Regularised incomplete beta I_x(a, b) by the continued fraction of DLMF 8.17.22,
// evaluated with the modified Lentz method (Numerical Recipes 2nd ed. section 6.4):
// direct when x < (a+1)/(a+b+2), else through I_x(a,b) = 1 - I_{1-x}(b,a).
__device__ double betacf(double a, double b, double x) {
    const double tiny = 1e-300, eps = 1e-16;
    const double qab = a + b, qap = a + 1.0, qam = a - 1.0;
    double c = 1.0, d = 1.0 - qab * x / qap;
    if (fabs(d) < tiny) d = tiny;
    d = 1.0 / d;
    double h = d;
    for (int k = 1; k <= 4000; ++k) {
        const double k2 = 2.0 * k;
        double aa = k * (b - k) * x / ((qam + k2) * (a + k2));
        d = 1.0 + aa * d;
        if (fabs(d) < tiny) d = tiny;
        c = 1.0 + aa / c;
        if (fabs(c) < tiny) c = tiny;
        d = 1.0 / d;
        h *= d * c;
        aa = -(a + k) * (qab + k) * x / ((a + k2) * (qap + k2));
        d = 1.0 + aa * d;
        if (fabs(d) < tiny) d = tiny;
        c = 1.0 + aa / c;
        if (fabs(c) < tiny) c = tiny;
        d = 1.0 / d;
        const double del = d * c;
        h *= del;
        if (fabs(del - 1.0) < eps) break;
    }
    return h;
}

// log Gamma(a + 1/2) - log Gamma(a) for a >= 25 from the Stirling series of both terms
// (log Gamma(z) = (z - 1/2) log z - z + log(2 pi)/2 + sum_k B_2k / (2k (2k-1) z^(2k-1)))
// expanded in 1/a: 1/2 log a - 1/(8a) + 1/(192 a^3) - 1/(640 a^5) + 17/(14336 a^7)
// - 31/(18432 a^9) + 691/(180224 a^11); the next term is below 1e-20 at a = 25.  The plain
// difference of the two log-gammas cancels ~5 digits at a = df/2 ~ 1e4.
__device__ double lgamma_ratio_half(double a) {
    const double t = 1.0 / a, t2 = t * t;
    const double s = t * (-1.0 / 8 + t2 * (1.0 / 192 + t2 * (-1.0 / 640 + t2 * (17.0 / 14336 +
                     t2 * (-31.0 / 18432 + t2 * (691.0 / 180224))))));
    return 0.5 * log(a) + s;
}

__device__ double betainc_reg(double a, double b, double x) {
    if (isnan(x)) return jnan();
    if (x <= 0.0) return 0.0;
    if (x >= 1.0) return 1.0;
    // log(1 / B(a, b)); b = 1/2 (every F test here) with large a takes the series above
    const double lb = (b == 0.5 && a >= 25.0) ? lgamma_ratio_half(a) - 0.5723649429247001
                                              : lgamma(a + b) - lgamma(a) - lgamma(b);
    const double lbt = lb + a * log(x) + b * log1p(-x);
    if (x < (a + 1.0) / (a + b + 2.0)) return exp(lbt) * betacf(a, b, x) / a;
    return 1.0 - exp(lbt) * betacf(b, a, 1.0 - x) / b;
}

// I_x(a, 1/2) for a >= kBgMinA and -log x <= kBgMaxLog by the expansion in incomplete gamma
// functions of A. R. DiDonato and A. H. Morris, ACM TOMS 18 (1992) 360-373, section 9
// ("BGRAT"), at b = 1/2, where the leading function is a complementary error function:
// with T = a - 1/4, u = -T log x,
//   I = Gamma(a + 1/2) / (Gamma(a) sqrt(T)) * sum_n p_n K_n,   K_0 = erfc(sqrt(u)),
//   K_{n+1} = ((2n + 1/2)(2n + 3/2) K_n
//              + exp(-u) sqrt(u / pi) (u + 2n + 3/2) (log x / 2)^{2n}) / (4 T^2),
// p_n the coefficients of (sinh y / y)^{-1/2} in y^2.  Eight terms leave at most a few
// rounding errors of the leading term over the whole region (checked against 40-digit
// values for a from 25 to 1e5).  The continued fraction it replaces there takes up to ~100
// steps of four dependent divisions; the figures stand at lmm_fpvalue_kernel.
constexpr double kBgMinA = 25.0, kBgMaxLog = 0.7;
constexpr int kBgTerms = 8;
struct BetaGrat {
    double t, v, scale;  // a - 1/4, 1 / (4 t^2), Gamma(a + 1/2) / (Gamma(a) sqrt(t))
};

__device__ __forceinline__ double betainc_half_large_a(const BetaGrat& g, double log_x) {
    constexpr double kP[kBgTerms] = {-1.0 / 12, 1.0 / 160, -61.0 / 120960, 1261.0 / 29030400,
                                     -79.0 / 20275200, 66643.0 / 185980354560.0,
                                     -16820653.0 / 502146957312000.0, 3.1675854343161146e-09};
    constexpr double kInvSqrtPi = 0.5641895835477563;
    const double u = -g.t * log_x, r = sqrt(u);
    const double h = r * kInvSqrtPi, l2 = 0.25 * log_x * log_x;
    double k = erfcx(r), sum = k, ln = h;  // everything over exp(-u)
#pragma unroll
    for (int n = 0; n < kBgTerms; ++n) {
        k = fma((2 * n + 0.5) * (2 * n + 1.5), k, ln * (u + (2 * n + 1.5))) * g.v;
        ln *= l2;
        sum = fma(kP[n], k, sum);
    }
    return g.scale * exp(-u) * sum;
}

// F-test p-value as jamma writes it (likelihood_jax.py:668-673,765-771).
__device__ double f_pvalue(double f, double df, const BetaGrat& g, bool large_a) {
    double z;
    if (isnan(f)) {
        z = jnan();
    } else {
        z = df / (df + (f > 1e-10 ? f : 1e-10));
        z = z < 0.0 ? 0.0 : (z > 1.0 ? 1.0 : z);
    }
    double p;
    const double lz = log(z);  // NaN or -inf outside (0, 1]: the general form decides
    if (large_a && lz < 0.0 && lz >= -kBgMaxLog)
        p = betainc_half_large_a(g, lz);
    else
        p = betainc_reg(df / 2.0, 0.5, z);
    return f <= 0.0 ? 1.0 : p;
}

// chi-square(1) survival function: P(X > s) = erfc(sqrt(s / 2)).
__device__ double chi2_1_sf(double s) {
    if (isnan(s)) return jnan();
    return erfc(sqrt(0.5 * s));
}

// ---------------------------------------------------------------- Pab
template <int C>
struct PabOut {
    double xx, xy, yy;  // level c (covariates projected out)
    double yy1;         // level c+1 (covariates and genotype projected out)
    double diag[C + 1]; // Pab[i, idx(i,i)], i = 0..c
};

// GEMMA CalcPab recursion (likelihood_jax.py:148-186); inverse of a zero pivot is 0.
template <int C>
__device__ __forceinline__ PabOut<C> pab_reduce(const double (&row0)[Lay<C>::NI]) {
    using L = Lay<C>;
    constexpr int R = L::R;
    double prev[L::NI], cur[L::NI];
    PabOut<C> o;
#pragma unroll
    for (int k = 0; k < L::NI; ++k) prev[k] = cur[k] = row0[k];
    o.diag[0] = prev[L::idx(0, 0)];
#pragma unroll
    for (int p = 1; p <= C + 1; ++p) {
        const int w = p - 1;
        const double ww = prev[L::idx(w, w)];
        const double inv = (ww != 0.0) ? 1.0 / ww : 0.0;
#pragma unroll
        for (int a = p; a < R; ++a) {
#pragma unroll
            for (int b = a; b < R; ++b) {
                const double t = __dmul_rn(__dmul_rn(prev[L::idx(a, w)], prev[L::idx(b, w)]), inv);
                cur[L::idx(a, b)] = __dsub_rn(prev[L::idx(a, b)], t);
            }
        }
        if (p <= C) o.diag[p] = cur[L::idx(p, p)];
        if (p == C) {
            o.xx = cur[L::idx(C, C)];
            o.xy = cur[L::idx(C, C + 1)];
            o.yy = cur[L::idx(C + 1, C + 1)];
        }
#pragma unroll
        for (int k = 0; k < L::NI; ++k) prev[k] = cur[k];
    }
    o.yy1 = prev[L::idx(C + 1, C + 1)];
    return o;
}

// REML log-likelihood (_reml_with_precomputed_iab, likelihood_jax.py:280-339).
template <int C>
__device__ __forceinline__ double reml_logl(const PabOut<C>& pb, const double (&log_iab)[C + 1],
                                            double logdet_h, const Params& p) {
    double ldw = 0.0;
#pragma unroll
    for (int i = 0; i <= C; ++i) {
        ldw = __dadd_rn(ldw, pb.diag[i] > 0 ? log(pb.diag[i]) : 0.0);
        ldw = __dsub_rn(ldw, log_iab[i]);
    }
    const double pyy = clamp_pyy(pb.yy1);
    double f = __dsub_rn(p.c_reml, __dmul_rn(0.5, logdet_h));
    f = __dsub_rn(f, __dmul_rn(0.5, ldw));
    return __dsub_rn(f, __dmul_rn(__dmul_rn(0.5, p.df), log(pyy)));
}

// MLE log-likelihood (mle_log_likelihood_jax, likelihood_jax.py:189-228).
template <int C>
__device__ __forceinline__ double mle_logl(const PabOut<C>& pb, double logdet_h, const Params& p) {
    const double pyy = clamp_pyy(pb.yy1);
    const double f = __dsub_rn(p.c_mle, __dmul_rn(0.5, logdet_h));
    return __dsub_rn(f, __dmul_rn(__dmul_rn(0.5, p.n_d), log(pyy)));
}

// Assemble a full row 0 from pre-reduced x-free sums and fresh x-dependent sums.
template <int C>
__device__ __forceinline__ void assemble(double (&row0)[Lay<C>::NI], const double* shared,
                                         const double (&xs)[Lay<C>::NX]) {
    using L = Lay<C>;
    int s = 0;
#pragma unroll
    for (int a = 0; a < L::R; ++a) {
#pragma unroll
        for (int b = a; b < L::R; ++b) {
            if (a == C || b == C) continue;
            row0[L::idx(a, b)] = shared[s++];
        }
    }
#pragma unroll
    for (int a = 0; a < C; ++a) row0[L::idx(a, C)] = xs[a];
    row0[L::idx(C, C)] = xs[C];
    row0[L::idx(C, C + 1)] = xs[C + 1];
}

// Full evaluation at a per-SNP lambda: H = 1/(lambda*eval + 1), all NI sums + logdet.
// Loads of UNR consecutive strided samples are issued together (memory-level parallelism).
constexpr int UNR = 4;

template <int C>
__device__ __forceinline__ void full_accumulate(double lam, double ev, double xv, double yv,
                                                const double (&w)[C > 0 ? C : 1],
                                                double (&acc)[Lay<C>::NI], double& ld) {
    using L = Lay<C>;
    const double v = __dadd_rn(__dmul_rn(lam, ev), 1.0);
    const double hi = __drcp_rn(v);  // correctly rounded, = 1.0 / v
    ld += log(fabs(v));
    double vec[L::R];
#pragma unroll
    for (int a = 0; a < C; ++a) vec[a] = w[a];
    vec[C] = xv;
    vec[C + 1] = yv;
#pragma unroll
    for (int a = 0; a < L::R; ++a) {
        const double t = hi * vec[a];
#pragma unroll
        for (int b = a; b < L::R; ++b) acc[L::idx(a, b)] = fma(t, vec[b], acc[L::idx(a, b)]);
    }
}

template <int C>
__device__ __forceinline__ void eval_full(const Params& p, const double* __restrict__ x,
                                          const double* __restrict__ y, double lam,
                                          double (&row0)[Lay<C>::NI], double& logdet) {
    using L = Lay<C>;
    double acc[L::NI];
#pragma unroll
    for (int k = 0; k < L::NI; ++k) acc[k] = 0.0;
    double ld = 0.0;
    const int lane = threadIdx.x & 31;
    int64_t i = lane;
    for (; i + 32 * (UNR - 1) < p.n; i += 32 * UNR) {
        double ev[UNR], xv[UNR], yv[UNR], w[UNR][C > 0 ? C : 1];
#pragma unroll
        for (int u = 0; u < UNR; ++u) {
            ev[u] = __ldg(p.evals + i + 32 * u);
            xv[u] = x[i + 32 * u];
            yv[u] = __ldg(y + i + 32 * u);
#pragma unroll
            for (int a = 0; a < C; ++a) w[u][a] = __ldg(p.W + a * p.ldw + i + 32 * u);
        }
#pragma unroll
        for (int u = 0; u < UNR; ++u) full_accumulate<C>(lam, ev[u], xv[u], yv[u], w[u], acc, ld);
    }
    for (; i < p.n; i += 32) {
        double w[C > 0 ? C : 1];
#pragma unroll
        for (int a = 0; a < C; ++a) w[a] = __ldg(p.W + a * p.ldw + i);
        full_accumulate<C>(lam, __ldg(p.evals + i), x[i], __ldg(y + i), w, acc, ld);
    }
#pragma unroll
    for (int k = 0; k < L::NI; ++k) row0[k] = warp_sum(acc[k]);
    logdet = warp_sum(ld);
}

template <int C, bool REML>
__device__ __forceinline__ double eval_logl(const Params& p, const double* x, const double* y,
                                            double log_lam, const double (&log_iab)[C + 1],
                                            PabOut<C>* keep) {
    double row0[Lay<C>::NI];
    double logdet;
    eval_full<C>(p, x, y, exp(log_lam), row0, logdet);
    const PabOut<C> pb = pab_reduce<C>(row0);
    if (keep) *keep = pb;
    return REML ? reml_logl<C>(pb, log_iab, logdet, p) : mle_logl<C>(pb, logdet, p);
}

// Grid bracket + golden section (_golden_section_refine, likelihood_jax.py:419-488).
template <int C, bool REML>
__device__ void golden(const Params& p, const double* x, const double* y, int best,
                       const double (&log_iab)[C + 1], double& lam_out, double& logl_out,
                       PabOut<C>& pb_out) {
    const int lo = best - 1 > 0 ? best - 1 : 0;
    const int hi = best + 1 < p.n_grid - 1 ? best + 1 : p.n_grid - 1;
    auto probe = [&](double s) { return eval_logl<C, REML>(p, x, y, s, log_iab, nullptr); };
    double a = p.loglam[lo], b = p.loglam[hi];
    double c = __dsub_rn(b, __dmul_rn(kPhi, __dsub_rn(b, a)));
    double d = __dadd_rn(a, __dmul_rn(kPhi, __dsub_rn(b, a)));
    double fc = probe(c);
    double fd = probe(d);
    for (int it = 0; it < p.n_iter; ++it) {
        const bool keep_left = fc > fd;
        const double na = keep_left ? a : c;
        const double nb = keep_left ? d : b;
        const double nc = __dsub_rn(nb, __dmul_rn(kPhi, __dsub_rn(nb, na)));
        const double nd = __dadd_rn(na, __dmul_rn(kPhi, __dsub_rn(nb, na)));
        const double nl = probe(keep_left ? nc : nd);
        const double nfc = keep_left ? nl : fd;
        const double nfd = keep_left ? fc : nl;
        a = na; b = nb; c = nc; d = nd; fc = nfc; fd = nfd;
    }
    const double log_opt = __dmul_rn(__dadd_rn(a, b), 0.5);
    lam_out = exp(log_opt);
    logl_out = eval_logl<C, REML>(p, x, y, log_opt, log_iab, &pb_out);
}

constexpr unsigned kFull = 0xffffffffu;

// jnp.argmax semantics: first maximum, NaN wins (first NaN).
struct ArgMax {
    int idx = -1;
    double v = 0.0;
    __device__ void push(int i, double x) {
        if (idx < 0) { idx = i; v = x; return; }
        if (isnan(v)) return;
        if (isnan(x) || x > v) { idx = i; v = x; }
    }
    // Merge with a partial result over other indices (any order): the lowest-index NaN
    // if there is one, else the maximum with the lowest index among ties -- the same
    // pick as pushing every index in increasing order.
    __device__ void merge(int i, double x) {
        if (i < 0) return;
        if (idx < 0) { idx = i; v = x; return; }
        const bool na = isnan(v), nb = isnan(x);
        if (na || nb) {
            if (na && nb ? i < idx : nb) { idx = i; v = x; }
            return;
        }
        if (x > v || (x == v && i < idx)) { idx = i; v = x; }
    }
    template <int GW = 32>
    __device__ void warp_reduce() {  // over groups of GW lanes
#pragma unroll
        for (int o = GW / 2; o > 0; o >>= 1) {
            const int oi = __shfl_xor_sync(0xffffffffu, idx, o);
            const double ov = __shfl_xor_sync(0xffffffffu, v, o);
            merge(oi, ov);
        }
    }
};

template <int C>
__device__ __forceinline__ void beta_se(const PabOut<C>& pb, double px_yy, double df, bool& valid,
                                        double& beta, double& tau, double& se) {
    valid = pb.xx > 0;
    const double safe_xx = valid ? pb.xx : 1.0;
    beta = valid ? pb.xy / safe_xx : jnan();
    tau = df / px_yy;
    double var = valid ? 1.0 / (tau * safe_xx) : jnan();
    var = fabs(var) < 0.001 ? fabs(var) : var;
    se = valid ? sqrt(var) : jnan();
}

// Mixed form at large lambda.  The series' error in an x-dependent sum is fixed in absolute
// terms (a small fraction of the sum's size at small lambda, where every weight
// 1/(lambda e_i + 1) is near 1), while the sums the statistics use shrink like
// 1/(lambda e): at lambda = 1e5 the projected P_xy, P_xx are ~1e-5 of their small-lambda
// size and the score and LRT p-values moved by up to 2e-4 relative against the FP64 form
// (n = 20 000, 64 phenotypes whose null lambda sat on the upper bound).  The error grows
// about linearly in lambda (4e-8 at lambda = 10), so every final evaluation at
// lambda >= kDirectLam -- the score at the null lambda, the MLE and REML optima -- reduces
// its sums directly in FP64 over the rotated genotypes instead (one pass over x).  The
// search itself stays on the series.
constexpr double kDirectLam = 20.0;
constexpr double kLogDirectLam = 2.995732273553991;  // log(kDirectLam)

// The x-dependent sums of one pair at up to three lambdas (the score's null lambda, the
// MLE and REML optima; on[q] the same in every lane) in one warp-cooperative pass over the
// rotated genotypes, each term formed as full_accumulate forms it.
template <int C>
__device__ __forceinline__ void direct_xsums3(const Params& p, const double* __restrict__ x,
                                              const double* __restrict__ y,
                                              const double (&lam)[3], const bool (&on)[3],
                                              double (&xs)[3][Lay<C>::NX]) {
    using L = Lay<C>;
    double acc[3][L::NX];
#pragma unroll
    for (int q = 0; q < 3; ++q)
#pragma unroll
        for (int k = 0; k < L::NX; ++k) acc[q][k] = 0.0;
    auto term = [&](double ev, double xv, double yv, const double (&w)[C > 0 ? C : 1]) {
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            if (!on[q]) continue;
            const double hi = __drcp_rn(__dadd_rn(__dmul_rn(lam[q], ev), 1.0));
#pragma unroll
            for (int a = 0; a < C; ++a) acc[q][a] = fma(hi * w[a], xv, acc[q][a]);
            const double t = hi * xv;
            acc[q][C] = fma(t, xv, acc[q][C]);
            acc[q][C + 1] = fma(t, yv, acc[q][C + 1]);
        }
    };
    // UNR consecutive strided samples' loads issued together (memory-level parallelism)
    int64_t i = threadIdx.x & 31;
    for (; i + 32 * (UNR - 1) < p.n; i += 32 * UNR) {
        double ev[UNR], xv[UNR], yv[UNR], w[UNR][C > 0 ? C : 1];
#pragma unroll
        for (int u = 0; u < UNR; ++u) {
            ev[u] = __ldg(p.evals + i + 32 * u);
            xv[u] = x[i + 32 * u];
            yv[u] = __ldg(y + i + 32 * u);
#pragma unroll
            for (int a = 0; a < C; ++a) w[u][a] = __ldg(p.W + a * p.ldw + i + 32 * u);
        }
#pragma unroll
        for (int u = 0; u < UNR; ++u) term(ev[u], xv[u], yv[u], w[u]);
    }
    for (; i < p.n; i += 32) {
        double w[C > 0 ? C : 1];
#pragma unroll
        for (int a = 0; a < C; ++a) w[a] = __ldg(p.W + a * p.ldw + i);
        term(__ldg(p.evals + i), x[i], __ldg(y + i), w);
    }
#pragma unroll
    for (int q = 0; q < 3; ++q)
#pragma unroll
        for (int k = 0; k < L::NX; ++k) xs[q][k] = on[q] ? warp_sum(acc[q][k]) : 0.0;
}

// Pairs with a final lambda >= kDirectLam: the whole warp takes each such pair of its
// 32 / GW groups in turn and reduces its x-dependent sums directly.  The score statistic
// is recomputed and rewritten here (the group's lane 0 overwrites the series value); the
// MLE / REML sums replace xs_m / xs_r of the owning group, which then evaluates them with
// its bracket-expanded x-free sums and log-determinant as before.
template <int C, int GW>
__device__ __forceinline__ void direct_fix(const Params& p, int64_t j, int f, bool valid_pair,
                                           bool need_score, bool need_mle, bool need_reml,
                                           double s_m, double s_r, double (&xs_m)[Lay<C>::NX],
                                           double (&xs_r)[Lay<C>::NX]) {
    using L = Lay<C>;
    const int mine = (int)(threadIdx.x & 31) / GW;
#pragma unroll 1
    for (int h = 0; h < 32 / GW; ++h) {
        const int src = h * GW;
        const int fh = __shfl_sync(kFull, f, src);
        const double sm = __shfl_sync(kFull, s_m, src), sr = __shfl_sync(kFull, s_r, src);
        const double lam0 = need_score ? p.lam0[fh] : 0.0;
        const bool on[3] = {need_score && lam0 >= kDirectLam, need_mle && sm >= kLogDirectLam,
                            need_reml && sr >= kLogDirectLam};
        if (!on[0] && !on[1] && !on[2]) continue;  // the same decision in every lane
        const long long jh = __shfl_sync(kFull, (long long)j, src);
        const bool vh = __shfl_sync(kFull, (int)valid_pair, src) != 0;
        const double lam[3] = {lam0, exp(sm), exp(sr)};
        double xs[3][L::NX];
        direct_xsums3<C>(p, p.G + jh * p.ldg, p.Y + (int64_t)fh * p.ldy, lam, on, xs);
        if (on[0]) {
            double row0[L::NI];
            assemble<C>(row0, p.S + (int64_t)(p.n_grid + 1 + fh) * p.phi * L::NS + (int64_t)fh * L::NS,
                        xs[0]);
            const PabOut<C> pb = pab_reduce<C>(row0);
            bool valid;
            double beta, tau, se;
            beta_se<C>(pb, clamp_pyy(pb.yy1), p.df, valid, beta, tau, se);
            const double fstat = p.n_d * (pb.xy * pb.xy) / (pb.yy * (valid ? pb.xx : 1.0));
            if ((int)(threadIdx.x & 31) == src && vh) {
                const int64_t o = (int64_t)fh * p.m + jh;
                if (p.out.p_score) p.out.p_score[o] = valid ? fstat : jnan();
                if (p.mode == 3) {
                    if (p.out.beta) p.out.beta[o] = beta;
                    if (p.out.se) p.out.se[o] = se;
                }
            }
        }
        if (mine == h) {
#pragma unroll
            for (int k = 0; k < L::NX; ++k) {
                if (on[1]) xs_m[k] = xs[1][k];
                if (on[2]) xs_r[k] = xs[2][k];
            }
        }
    }
}

// Statistics of the REML optimum (Wald): beta, se, the F statistic (NaN: no test;
// lmm_fpvalue_kernel turns it into the p-value), lambda and the log-likelihood.
template <int C>
__device__ __forceinline__ void write_wald(const Params& p, const PabOut<C>& pb, double logl,
                                           double lam, int64_t o, bool writer) {
    bool valid;
    double beta, tau, se;
    const double px_yy = clamp_pyy(pb.yy1);
    beta_se<C>(pb, px_yy, p.df, valid, beta, tau, se);
    const double fstat = (pb.yy - px_yy) * tau;
    if (writer) {
        if (p.out.lambda_remle) p.out.lambda_remle[o] = lam;
        if (p.out.logl_h1) p.out.logl_h1[o] = logl;
        if (p.out.beta) p.out.beta[o] = beta;
        if (p.out.se) p.out.se[o] = se;
        if (p.out.p_wald) p.out.p_wald[o] = valid ? fstat : jnan();
    }
}

// 4 warps per block; as many blocks per SM as the per-warp state allows without spills.
constexpr int kPairsThreads = 128;
template <int C>
struct PairsOccupancy {
    static constexpr int kMinBlocks = C == 1 ? 4 : (C == 2 ? 3 : 2);  // C = 1: 125 registers, no spill
};

// Plain form: one (SNP, phenotype) pair per warp, every probe a direct FP64 pass over x.
template <int C>
__global__ void __launch_bounds__(kPairsThreads, PairsOccupancy<C>::kMinBlocks)
    lmm_pairs_kernel(const Params p) {
    using L = Lay<C>;
    const int64_t wid = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / 32;
    if (wid >= p.m * p.phi) return;
    const int lane = threadIdx.x & 31;
    const int64_t j = wid / p.phi;
    const int f = (int)(wid % p.phi);
    const double* __restrict__ x = p.G + j * p.ldg;
    const double* __restrict__ y = p.Y + (int64_t)f * p.ldy;
    const bool need_reml = p.mode == 1 || p.mode == 4;
    const bool need_mle = p.mode == 2 || p.mode == 4;
    const bool need_score = p.mode == 3 || p.mode == 4;
    const int64_t o = (int64_t)f * p.m + j;
    const int64_t srow = (int64_t)p.phi * L::NS;  // stride of one S row

    // Weighted x-sums of table row r for this (SNP, phenotype), from the chunk GEMMs.
    auto row_xsums = [&](int r, double (&xs)[L::NX]) {
        const double* cl = p.CL + j * p.ldcl + (int64_t)r * (C + p.phi);
#pragma unroll
        for (int a = 0; a < C; ++a) xs[a] = cl[a];
        xs[C] = p.CQ[j * p.ldcq + r];
        xs[C + 1] = cl[C + f];
    };

    // ---------------- phase 1: H = 1 (Iab) and H = H0 (score)
    double log_iab[C + 1];
#pragma unroll
    for (int i = 0; i <= C; ++i) log_iab[i] = 0.0;
    if (need_reml) {
        double xs[L::NX], row0[L::NI];
        row_xsums(p.n_grid, xs);
        assemble<C>(row0, p.S + (int64_t)p.n_grid * srow + (int64_t)f * L::NS, xs);
        const PabOut<C> pb = pab_reduce<C>(row0);
#pragma unroll
        for (int i = 0; i <= C; ++i) log_iab[i] = pb.diag[i] > 0 ? log(pb.diag[i]) : 0.0;
    }
    if (need_score) {
        double xs[L::NX], row0[L::NI];
        row_xsums(p.n_grid + 1 + f, xs);
        assemble<C>(row0, p.S + (int64_t)(p.n_grid + 1 + f) * srow + (int64_t)f * L::NS, xs);
        const PabOut<C> pb = pab_reduce<C>(row0);
        bool valid;
        double beta, tau, se;
        beta_se<C>(pb, clamp_pyy(pb.yy1), p.df, valid, beta, tau, se);
        const double fstat = p.n_d * (pb.xy * pb.xy) / (pb.yy * (valid ? pb.xx : 1.0));
        if (lane == 0) {
            // the F statistic (NaN: no test); lmm_fpvalue_kernel turns it into the p-value
            if (p.out.p_score) p.out.p_score[o] = valid ? fstat : jnan();
            if (p.mode == 3) {
                if (p.out.beta) p.out.beta[o] = beta;
                if (p.out.se) p.out.se[o] = se;
            }
        }
    }
    if (!need_reml && !need_mle) return;

    // ---------------- phase 2: shared lambda grid
    ArgMax best_reml, best_mle;
    for (int g = 0; g < p.n_grid; ++g) {
        double xs[L::NX], row0[L::NI];
        row_xsums(g, xs);
        assemble<C>(row0, p.S + (int64_t)g * srow + (int64_t)f * L::NS, xs);
        const PabOut<C> pb = pab_reduce<C>(row0);
        const double ldh = p.logdet[g];
        if (need_reml) best_reml.push(g, reml_logl<C>(pb, log_iab, ldh, p));
        if (need_mle) best_mle.push(g, mle_logl<C>(pb, ldh, p));
    }

    // ---------------- phase 3: golden sections + statistics
    if (need_mle) {
        double lam, logl;
        PabOut<C> pb;
        golden<C, false>(p, x, y, best_mle.idx, log_iab, lam, logl, pb);
        if (lane == 0) {
            if (p.out.lambda_mle) p.out.lambda_mle[o] = lam;
            if (p.out.logl_mle) p.out.logl_mle[o] = logl;
            const double stat = jmax(2.0 * (logl - p.logl0[f]), 0.0);
            if (p.out.p_lrt) p.out.p_lrt[o] = chi2_1_sf(stat);
        }
    }
    if (need_reml) {
        double lam, logl;
        PabOut<C> pb;
        golden<C, true>(p, x, y, best_reml.idx, log_iab, lam, logl, pb);
        write_wald<C>(p, pb, logl, lam, o, lane == 0);
    }
}

}  // namespace lmm
}  // namespace jb

#include "jb_lmm_search.cuh"

namespace jb {
namespace lmm {

// ---------------------------------------------------------------- tables
// H rows: grid lambda_g = exp(loglam[g]) for g < n_grid, then the null lambda0[f];
// logdet[g] = sum_i log|lambda_g * eval_i + 1| for grid rows.
__global__ void lmm_table_kernel(int64_t n, int n_grid, int phi, const double* __restrict__ evals,
                                 const double* __restrict__ loglam, const double* __restrict__ lam0,
                                 double* __restrict__ H, double* __restrict__ logdet) {
    const int r = blockIdx.x;
    const double lam = r < n_grid ? exp(loglam[r]) : lam0[r - n_grid];
    double ld = 0.0;
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
        const double v = __dadd_rn(__dmul_rn(lam, evals[i]), 1.0);
        H[(int64_t)r * n + i] = 1.0 / v;
        ld += log(fabs(v));
    }
    if (r >= n_grid) return;
    __shared__ double red[32];
    ld = warp_sum(ld);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ld;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int k = 0; k < (int)(blockDim.x >> 5); ++k) s += red[k];
        logdet[r] = s;
    }
}

// x-free weighted sums S[row][f][s] = sum_i h_row,i * v_a,i * v_b,i over pairs without X,
// rows: grid (H), ones, null rows (H0_f).
template <int C>
__global__ void lmm_shared_kernel(int64_t n, int n_grid, int phi, const double* __restrict__ W,
                                  int64_t ldw, const double* __restrict__ Y, int64_t ldy,
                                  const double* __restrict__ H, double* __restrict__ S) {
    using L = Lay<C>;
    const int r = blockIdx.x;
    const int f = blockIdx.y;
    const double* h = r < n_grid ? H + (int64_t)r * n
                                 : (r == n_grid ? nullptr : H + (int64_t)(r - 1) * n);
    double acc[L::NS];
#pragma unroll
    for (int s = 0; s < L::NS; ++s) acc[s] = 0.0;
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
        const double hi = h ? h[i] : 1.0;
        double vec[L::R];
#pragma unroll
        for (int a = 0; a < C; ++a) vec[a] = W[a * ldw + i];
        vec[C] = 0.0;
        vec[C + 1] = Y[(int64_t)f * ldy + i];
        int s = 0;
#pragma unroll
        for (int a = 0; a < L::R; ++a) {
#pragma unroll
            for (int b = a; b < L::R; ++b) {
                if (a == C || b == C) continue;
                acc[s] = fma(hi * vec[a], vec[b], acc[s]);
                ++s;
            }
        }
    }
    __shared__ double red[L::NS][8];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int s = 0; s < L::NS; ++s) {
        const double v = warp_sum(acc[s]);
        if (lane == 0) red[s][w] = v;
    }
    __syncthreads();
    if (threadIdx.x < L::NS) {
        double t = 0.0;
        for (int k = 0; k < (int)(blockDim.x >> 5); ++k) t += red[threadIdx.x][k];
        S[((int64_t)r * phi + f) * L::NS + threadIdx.x] = t;
    }
}

// GEMM operands for the per-chunk weighted x-sums: for every table row r (grid rows, the
// ones row, the null rows) A_sq[r] = h_r and A_lin[r*(C+phi) + a] = h_r * w_a (a < C),
// A_lin[r*(C+phi) + C + f] = h_r * y_f; each row has n entries.
template <int C>
__global__ void lmm_gemm_tables_kernel(int64_t n, int n_grid, int phi, const double* __restrict__ W,
                                       int64_t ldw, const double* __restrict__ Y, int64_t ldy,
                                       const double* __restrict__ H, double* __restrict__ Alin,
                                       double* __restrict__ Asq) {
    const int r = blockIdx.x;
    const double* h = r < n_grid ? H + (int64_t)r * n
                                 : (r == n_grid ? nullptr : H + (int64_t)(r - 1) * n);
    const int64_t base = (int64_t)r * (C + phi);
    for (int64_t i = blockIdx.y * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.y * blockDim.x) {
        const double hv = h ? h[i] : 1.0;
        Asq[(int64_t)r * n + i] = hv;
#pragma unroll
        for (int a = 0; a < C; ++a) Alin[(base + a) * n + i] = hv * W[a * ldw + i];
        for (int f = 0; f < phi; ++f) Alin[(base + C + f) * n + i] = hv * Y[(int64_t)f * ldy + i];
    }
}

// ---------------------------------------------------------------- squared x-sums
// CQ[j*ldcq + r] = sum_i A[i, r] x_ij^2 (r < rows) for every SNP j of a rotated chunk X
// (column-major, ld ldx): the squared weighted sums of every table row.  One fused kernel
// reads each rotated genotype once, squares it in shared memory and forms the product with
// the row table on the FP64 tensor cores (mma.sync m8n8k4 .f64), so X^2 never goes to HBM.
//   * A is held transposed, AT[i*ldt + r] (ldt a multiple of the row tile, zero for
//     r >= rows), so a slice of kSqTK samples is one contiguous block per row tile;
//   * a CTA owns TR rows x kSqTN SNPs for one range of samples; warp w owns SNPs
//     16w..16w+15 (two 8-column MMA tiles) for all TR/8 row tiles of the CTA;
//   * shared layouts As[k][TR] (TR = 8 mod 16 doubles) and Xs[j][kSqXLD] (kSqXLD = 4 mod
//     16) make every 32-lane fragment load two conflict-free wavefronts;
//   * slices are double-buffered with cp.async; out-of-range samples and SNPs read as zero;
//   * the samples are split over kz = blockIdx.z ranges when the SNP tiles alone cannot
//     fill the GPU; partial sums go to P[(kz*m + j)*ldt + r] and sq_reduce_kernel adds
//     them in kz order, so every sum has a fixed order (bit-reproducible).
constexpr int kSqTK = 16;   // samples per slice
constexpr int kSqTN = 64;   // SNPs per CTA (4 warps x 16)
constexpr int kSqXLD = 20;  // padded sample stride of a slice's SNP
constexpr int kSqThreads = 128;
constexpr int kSqSlots = 148 * 3;  // CTAs resident at once on a B200 (3 per SM)

template <int TR>
struct SqCfg {
    static_assert(TR % 16 == 8, "row tile must be 8 mod 16 doubles (conflict-free fragments)");
    static constexpr int RT = TR / 8;              // 8-row MMA tiles
    static constexpr int A_ELEMS = kSqTK * TR;
    static constexpr int X_ELEMS = kSqTN * kSqXLD;
    static constexpr int STAGE = A_ELEMS + X_ELEMS;  // doubles (even: stages stay 16-byte aligned)
    static constexpr int SMEM = 2 * STAGE * 8;
};

// Row tile for a table of `rows` rows and the matching padded leading dimension of AT.
inline int sq_tile_rows(int64_t rows) { return rows <= 56 ? 56 : 104; }
inline int64_t sq_ldt(int64_t rows) {
    const int tr = sq_tile_rows(rows);
    return ceil_div(rows, tr) * tr;
}
// Sample-range split: at least four waves of CTAs, and among the splits up to twice that
// the one whose last wave is fullest (every CTA does the same work, so a part-filled last
// wave is idle hardware); each range at least four slices long.
inline int sq_split(int64_t n, int64_t m, int64_t rows) {
    const int64_t tiles = ceil_div(m, kSqTN) * (sq_ldt(rows) / sq_tile_rows(rows));
    const int64_t kmax = ceil_div(n, 4 * kSqTK);
    int64_t k0 = ceil_div(4 * kSqSlots, tiles);
    if (k0 > kmax) k0 = kmax;
    if (k0 < 1) k0 = 1;
    int64_t best = k0;
    double best_eff = 0.0;
    for (int64_t ks = k0; ks <= 2 * k0 && ks <= kmax; ++ks) {
        const int64_t units = tiles * ks;
        const double eff = (double)units / (double)(ceil_div(units, kSqSlots) * kSqSlots);
        if (eff > best_eff + 1e-9) {
            best_eff = eff;
            best = ks;
        }
    }
    return (int)best;
}

__device__ __forceinline__ void cp_async16(double* dst, const double* src, bool valid) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src),
                 "r"(valid ? 16 : 0)
                 : "memory");
}
__device__ __forceinline__ void cp_async8(double* dst, const double* src, bool valid) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src),
                 "r"(valid ? 8 : 0)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// D (8 x 8) += A (8 x 4) B (4 x 8) in FP64; lane l holds A[l/4][l%4], B[l%4][l/4] and
// D[l/4][2(l%4)], D[l/4][2(l%4)+1].
__device__ __forceinline__ void dmma_8x8x4(double& d0, double& d1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}

template <int TR>
__global__ void __launch_bounds__(kSqThreads, 3)
    sq_sums_kernel(const double* __restrict__ AT, int64_t ldt, const double* __restrict__ X,
                   int64_t ldx, int64_t n, int64_t m, int64_t klen, int rows,
                   double* __restrict__ out, int64_t ldo, int64_t zstride) {
    using Cfg = SqCfg<TR>;
    extern __shared__ __align__(16) double sq_smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t j0 = (int64_t)blockIdx.x * kSqTN;
    const int64_t r0 = (int64_t)blockIdx.y * TR;
    const int64_t kbeg = (int64_t)blockIdx.z * klen;
    const int64_t kend = kbeg + klen < n ? kbeg + klen : n;
    const int nsl = kend > kbeg ? (int)((kend - kbeg + kSqTK - 1) / kSqTK) : 0;

    auto issue = [&](int st, int64_t k) {
        double* As = sq_smem + st * Cfg::STAGE;
        double* Xs = As + Cfg::A_ELEMS;
        for (int e = tid; e < kSqTK * (TR / 2); e += kSqThreads) {  // A: 16-byte chunks
            const int kk = e / (TR / 2), c = e % (TR / 2);
            const bool ok = k + kk < kend;
            cp_async16(As + kk * TR + 2 * c, AT + (ok ? (k + kk) * ldt : 0) + r0 + 2 * c, ok);
        }
        for (int e = tid; e < kSqTN * kSqTK; e += kSqThreads) {  // X: one double per copy
            const int jj = e / kSqTK, kk = e % kSqTK;
            const bool ok = (k + kk < kend) && (j0 + jj < m);
            cp_async8(Xs + jj * kSqXLD + kk, X + (ok ? (j0 + jj) * ldx + k + kk : 0), ok);
        }
        cp_async_commit();
    };

    double acc[Cfg::RT][2][2];
#pragma unroll
    for (int a = 0; a < Cfg::RT; ++a)
#pragma unroll
        for (int q = 0; q < 2; ++q) acc[a][q][0] = acc[a][q][1] = 0.0;

    const int fr = lane >> 2, fk = lane & 3;  // fragment row (or column) and k of this lane
    if (nsl > 0) issue(0, kbeg);
    for (int s = 0; s < nsl; ++s) {
        if (s + 1 < nsl) {
            issue((s + 1) & 1, kbeg + (int64_t)(s + 1) * kSqTK);
            cp_async_wait<1>();
        } else {
            cp_async_wait<0>();
        }
        const double* As = sq_smem + (s & 1) * Cfg::STAGE;
        double* Xs = sq_smem + (s & 1) * Cfg::STAGE + Cfg::A_ELEMS;
        // square the X elements this thread copied (its own copies have landed)
        for (int e = tid; e < kSqTN * kSqTK; e += kSqThreads) {
            double* v = Xs + (e / kSqTK) * kSqXLD + e % kSqTK;
            *v = *v * *v;
        }
        __syncthreads();
        const double* xb = Xs + (warp * 16 + fr) * kSqXLD + fk;
        const double* ab = As + fk * TR + fr;
#pragma unroll
        for (int k0 = 0; k0 < kSqTK; k0 += 4) {
            const double b0 = xb[k0], b1 = xb[8 * kSqXLD + k0];
#pragma unroll
            for (int rt = 0; rt < Cfg::RT; ++rt) {
                const double a = ab[k0 * TR + rt * 8];
                dmma_8x8x4(acc[rt][0][0], acc[rt][0][1], a, b0);
                dmma_8x8x4(acc[rt][1][0], acc[rt][1][1], a, b1);
            }
        }
        __syncthreads();  // the next issue overwrites this stage
    }
    double* o = out + (int64_t)blockIdx.z * zstride;
#pragma unroll
    for (int nt = 0; nt < 2; ++nt) {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int64_t j = j0 + warp * 16 + nt * 8 + 2 * fk + e;
            if (j >= m) continue;
#pragma unroll
            for (int rt = 0; rt < Cfg::RT; ++rt) {
                const int64_t r = r0 + rt * 8 + fr;
                if (r < rows) o[j * ldo + r] = acc[rt][nt][e];
            }
        }
    }
}

// CQ[j*ldcq + r] = sum over kz = 0..ks-1 of P[(kz*m + j)*ldt + r], in kz order.
__global__ void sq_reduce_kernel(const double* __restrict__ P, int64_t ldt, int64_t m, int rows,
                                 int ks, double* __restrict__ CQ, int64_t ldcq) {
    const int64_t total = m * rows;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total;
         t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t j = t / rows, r = t - j * rows;
        double v = 0.0;
        for (int z = 0; z < ks; ++z) v += P[((int64_t)z * m + j) * ldt + r];
        CQ[j * ldcq + r] = v;
    }
}

// AT[i*ldt + r] = A[r*n + i] for r < rows, 0 for rows <= r < ldt.
__global__ void sq_table_kernel(const double* __restrict__ A, int64_t n, int rows, int64_t ldt,
                                double* __restrict__ AT) {
    const int64_t total = n * ldt;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total;
         t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = t / ldt, r = t - i * ldt;
        AT[t] = r < rows ? A[r * n + i] : 0.0;
    }
}

// Mixed form, global series over t = log lambda in [lo, hi]: node j of kChebG at
// t_j = mid + half * cos(pi (j + 1/2) / kChebG); hn[j * n + i] = 1 / (exp(t_j) e_i + 1).
__global__ void lmm_series_nodes_kernel(int64_t n, double mid, double half,
                                        const double* __restrict__ evals, double* __restrict__ hn) {
    const int j = blockIdx.y;
    const double lam = exp(mid + half * cos(M_PI * (j + 0.5) / kChebG));
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
        hn[(int64_t)j * n + i] = __drcp_rn(__dadd_rn(__dmul_rn(lam, evals[i]), 1.0));
}

// Two small tables in one launch.  CTAs 0..kChebG-1: the Chebyshev transform of the node
// values, column-major kChebG x kChebG: ccos[k + j * kChebG] = (2 / kChebG) cos(pi k (j + 1/2)
// / kChebG), row k = 0 halved, so coefficient k of any per-sample weight is sum_j ccos[k, j] *
// value_j.  The others: Chebyshev values of the global series at the grid points,
// tg[g * kChebG + k] = T_k(t_g), by the doubling identity.
__global__ void __launch_bounds__(kChebG) lmm_series_consts_kernel(
    double* __restrict__ ccos, int n_grid, double mid, double inv_half,
    const double* __restrict__ loglam, double* __restrict__ tg) {
    const int j = blockIdx.x, k = threadIdx.x;
    if (j < kChebG) {
        const double c = (2.0 / kChebG) * cos(M_PI * k * (j + 0.5) / kChebG);
        ccos[k + (int64_t)j * kChebG] = k == 0 ? 0.5 * c : c;
        return;
    }
    __shared__ double t[2 * kChebG];
    const int g = j - kChebG;
    if (k == 0) {
        t[0] = 1.0;
        t[1] = (loglam[g] - mid) * inv_half;
    }
    for (int a = 1; a < kChebG; a *= 2) {  // T_{a+1} .. T_{2a} from T_0 .. T_a
        __syncthreads();
        if (k >= 1 && k <= a && a + k < 2 * kChebG) t[a + k] = fma(2.0 * t[a], t[k], -t[a - k]);
    }
    __syncthreads();
    tg[(int64_t)g * kChebG + k] = t[k];
}

// GEMM operands of the mixed form: row 0 is the ones row (h = 1), row 1 + k holds the
// Chebyshev coefficient k of h_i(t) (already in Asq rows 1..kChebG from the transform
// GEMM); A_lin[r*(C+phi) + a] = Asq[r] * w_a, A_lin[r*(C+phi) + C + f] = Asq[r] * y_f.
template <int C>
__global__ void lmm_series_tables_kernel(int64_t n, int phi, const double* __restrict__ W,
                                         int64_t ldw, const double* __restrict__ Y, int64_t ldy,
                                         double* __restrict__ Alin, double* __restrict__ Asq) {
    const int r = blockIdx.x;
    const int64_t base = (int64_t)r * (C + phi);
    for (int64_t i = blockIdx.y * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.y * blockDim.x) {
        double hv = 1.0;
        if (r == 0)
            Asq[i] = 1.0;
        else
            hv = Asq[(int64_t)r * n + i];
#pragma unroll
        for (int a = 0; a < C; ++a) Alin[(base + a) * n + i] = hv * W[a * ldw + i];
        for (int f = 0; f < phi; ++f) Alin[(base + C + f) * n + i] = hv * Y[(int64_t)f * ldy + i];
    }
}

// Chebyshev node values for the mixed form: block (bracket b, node k) x phenotype f
// evaluates log|H^-1| (f == 0) and the x-free weighted sums of phenotype f exactly in
// FP64 at lambda = exp(s_k), s_k the k-th Chebyshev node of bracket b.
template <int C>
__global__ void lmm_cheb_nodes_kernel(int64_t n, int n_grid, int phi,
                                      const double* __restrict__ evals, const double* __restrict__ W,
                                      int64_t ldw, const double* __restrict__ Y, int64_t ldy,
                                      const double* __restrict__ loglam, double* __restrict__ vals,
                                      double* __restrict__ mid, double* __restrict__ half) {
    using L = Lay<C>;
    const int b = blockIdx.x / kChebN, k = blockIdx.x % kChebN, f = blockIdx.y;
    const int lo = b - 1 > 0 ? b - 1 : 0, hi = b + 1 < n_grid - 1 ? b + 1 : n_grid - 1;
    const double A = loglam[lo], B = loglam[hi];
    const double m = 0.5 * (A + B), h = 0.5 * (B - A);
    const double s = m + h * cos(M_PI * (k + 0.5) / kChebN);
    const double lam = exp(s);
    double acc[L::NS];
#pragma unroll
    for (int q = 0; q < L::NS; ++q) acc[q] = 0.0;
    double ld = 0.0;
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
        const double v = __dadd_rn(__dmul_rn(lam, evals[i]), 1.0);
        const double hv = __drcp_rn(v);
        if (f == 0) ld += log(fabs(v));
        double vec[L::R];
#pragma unroll
        for (int a = 0; a < C; ++a) vec[a] = W[a * ldw + i];
        vec[C] = 0.0;
        vec[C + 1] = Y[(int64_t)f * ldy + i];
        int q = 0;
#pragma unroll
        for (int a = 0; a < L::R; ++a) {
#pragma unroll
            for (int bb = a; bb < L::R; ++bb) {
                if (a == C || bb == C) continue;
                acc[q] = fma(hv * vec[a], vec[bb], acc[q]);
                ++q;
            }
        }
    }
    __shared__ double red[L::NS + 1][8];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int q = 0; q < L::NS; ++q) {
        const double v = warp_sum(acc[q]);
        if (lane == 0) red[q][w] = v;
    }
    {
        const double v = warp_sum(ld);
        if (lane == 0) red[L::NS][w] = v;
    }
    __syncthreads();
    const int nf = 1 + phi * L::NS;
    double* out = vals + ((int64_t)b * kChebN + k) * nf;
    if (threadIdx.x <= L::NS) {
        double t = 0.0;
        for (int q = 0; q < (int)(blockDim.x >> 5); ++q) t += red[threadIdx.x][q];
        if (threadIdx.x < L::NS)
            out[1 + f * L::NS + threadIdx.x] = t;
        else if (f == 0)
            out[0] = t;
    }
    if (threadIdx.x == 0 && k == 0 && f == 0) {
        mid[b] = m;
        half[b] = h;
    }
}

// Chebyshev coefficients c_j = (2/N) sum_k f(s_k) cos(pi j (k + 1/2) / N), c_0 halved: one CTA
// per bracket forms the N^2 cosines once, then one thread takes a coefficient at a time.
__global__ void __launch_bounds__(256) lmm_cheb_coef_kernel(int nf, const double* __restrict__ vals,
                                                            double* __restrict__ coef) {
    __shared__ double cs[kChebN * kChebN];
    const int b = blockIdx.x;
    for (int t = threadIdx.x; t < kChebN * kChebN; t += blockDim.x)
        cs[t] = cos(M_PI * (t / kChebN) * (t % kChebN + 0.5) / kChebN);
    __syncthreads();
    for (int t = blockIdx.y * blockDim.x + threadIdx.x; t < nf * kChebN; t += gridDim.y * blockDim.x) {
        const int fi = t / kChebN, j = t - fi * kChebN;
        double c = 0.0;
        for (int k = 0; k < kChebN; ++k)
            c += vals[((int64_t)b * kChebN + k) * nf + fi] * cs[j * kChebN + k];
        c *= 2.0 / kChebN;
        if (j == 0) c *= 0.5;
        coef[((int64_t)b * nf + fi) * kChebN + j] = c;
    }
}

// ---------------------------------------------------------------- null model
// One cluster of 8 CTAs per phenotype runs _golden_section_minimize (likelihood.py:395-474)
// over -mle_log_likelihood_null (349-392): 73 evaluations one after another, each a sum over
// the samples with a division and a logarithm per sample -- a latency chain on one SM.
//
// The sums are those of 256 strided partial sums (partial t over samples t, t + 256, ...)
// added up warp by warp, then over the 8 warps in order.  CTA w of the cluster forms the
// partials of warp w: its threads stage weights and logarithms of the samples, tile by tile,
// in shared memory, and its warps take one or two of the sums each and add them up in sample
// order.  The 8 warp sums cross through distributed shared memory.  Same values and order as
// one CTA of 256 threads, bit for bit.  Measured at n = 20 000, 4 phenotypes: one CTA each
// 3250 us, clusters 459 us; n = 1200, two covariate columns 228 -> 137 us.
constexpr int kNullCtas = 8, kNullThreads = 256, kNullTile = 512;
template <int C>
struct NullSmem {
    double col[C + 1][kNullTile];  // W columns, y
    double h[kNullTile], ld[kNullTile];
    double part[2][Lay<C>::NS + 1];  // this CTA's warp sums, double-buffered over evaluations
    double tot[Lay<C>::NS + 1];
};

template <int C>
__device__ double null_mle_eval(int64_t n, const double* __restrict__ W, int64_t ldw,
                                const double* __restrict__ y, const double* __restrict__ evals,
                                double lam, double c_mle, NullSmem<C>& sm, int parity) {
    using L = Lay<C>;
    constexpr int kWarps = kNullThreads / 32, kSlots = (L::NS + kWarps) / kWarps;
    constexpr int kPer = kNullTile / kNullThreads;
    cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
    const int rank = (int)cl.block_rank();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // local sample q = 32 s + lane of this CTA is sample 32 rank + lane + 256 s
    const int64_t steps = (n - 1 - 32 * rank) / 256 + 1;  // 0 or less: no sample
    const int64_t nloc = n > 32 * rank ? 32 * steps : 0;
    int ca[kSlots], cb[kSlots];  // this warp's sums: columns a <= b; log|H| is sum NS
    double acc[kSlots];
#pragma unroll
    for (int q = 0; q < kSlots; ++q) {
        acc[q] = 0.0;
        ca[q] = cb[q] = 0;
        int k = 0;
#pragma unroll
        for (int a = 0; a <= C; ++a)
#pragma unroll
            for (int b = a; b <= C; ++b, ++k)
                if (k == warp + q * kWarps) {
                    ca[q] = a;
                    cb[q] = b;
                }
    }
    double ev[kPer], col[kPer][C + 1];
    auto sample = [&](int64_t q) { return 32 * rank + (q & 31) + 256 * (q >> 5); };
    auto fetch = [&](int64_t base) {
#pragma unroll
        for (int e = 0; e < kPer; ++e) {
            const int64_t q = base + threadIdx.x + e * kNullThreads, i = sample(q);
            if (q >= nloc || i >= n) continue;
            ev[e] = __ldg(evals + i);
#pragma unroll
            for (int a = 0; a < C; ++a) col[e][a] = __ldg(W + a * ldw + i);
            col[e][C] = __ldg(y + i);
        }
    };
    fetch(0);
    for (int64_t base = 0; base < nloc; base += kNullTile) {
        __syncthreads();  // the previous tile (or evaluation) has been read
#pragma unroll
        for (int e = 0; e < kPer; ++e) {
            const int64_t q = base + threadIdx.x + e * kNullThreads;
            if (q >= nloc || sample(q) >= n) continue;
            const int t = threadIdx.x + e * kNullThreads;
            const double v = __dadd_rn(__dmul_rn(lam, ev[e]), 1.0);
            sm.h[t] = 1.0 / v;
            sm.ld[t] = log(fabs(v));
#pragma unroll
            for (int a = 0; a <= C; ++a) sm.col[a][t] = col[e][a];
        }
        __syncthreads();
        fetch(base + kNullTile);
        // this lane's samples of the tile: the last step's may lie past the end
        int len = (int)(nloc - base < kNullTile ? nloc - base : kNullTile);
        if (len > 0 && sample(base + len - 32 + lane) >= n) len -= 32;
#pragma unroll
        for (int q = 0; q < kSlots; ++q) {
            const int k = warp + q * kWarps;  // warp-uniform
            const double *pa = sm.col[ca[q]], *pb = sm.col[cb[q]];
            double t = acc[q];
            if (k < L::NS) {
#pragma unroll 8
                for (int i = lane; i < len; i += 32) t = fma(sm.h[i] * pa[i], pb[i], t);
            } else if (k == L::NS) {
#pragma unroll 8
                for (int i = lane; i < len; i += 32) t += sm.ld[i];
            }
            acc[q] = t;
        }
    }
#pragma unroll
    for (int q = 0; q < kSlots; ++q) {
        const double v = warp_sum(acc[q]);
        if (lane == 0 && warp + q * kWarps <= L::NS) sm.part[parity][warp + q * kWarps] = v;
    }
    cl.sync();  // every CTA's warp sums are there (and the other buffer's have been read)
    if (threadIdx.x <= L::NS) {
        double t = 0.0;
        for (int w = 0; w < kNullCtas; ++w)
            t += cl.map_shared_rank(sm.part[parity], w)[threadIdx.x];
        sm.tot[threadIdx.x] = t;
    }
    __syncthreads();
    double row0[L::NI], tot[L::NS];
#pragma unroll
    for (int k = 0; k < L::NS; ++k) tot[k] = sm.tot[k];
    double xs[L::NX];
#pragma unroll
    for (int k = 0; k < L::NX; ++k) xs[k] = 0.0;
    assemble<C>(row0, tot, xs);
    const PabOut<C> pb = pab_reduce<C>(row0);
    const double pyy = clamp_pyy(pb.yy);  // level n_cvt for the null model
    const double f = __dsub_rn(c_mle, __dmul_rn(0.5, sm.tot[L::NS]));
    return __dsub_rn(f, __dmul_rn(__dmul_rn(0.5, (double)n), log(pyy)));
}

template <int C>
__global__ void __cluster_dims__(kNullCtas, 1, 1) __launch_bounds__(kNullThreads)
    null_mle_kernel(int64_t n, const double* W, int64_t ldw, const double* Y, int64_t ldy,
                    const double* evals, double lo, double step, int n_grid, int n_iter,
                    double log_hi, double c_mle, double* lam0, double* logl0) {
    __shared__ NullSmem<C> sm;
    const int f = blockIdx.x / kNullCtas;
    const double* y = Y + (int64_t)f * ldy;
    int parity = 0;
    // every thread of the cluster gets the same value, so the control flow is uniform
    auto func = [&](double lam) {
        parity ^= 1;
        return -null_mle_eval<C>(n, W, ldw, y, evals, lam, c_mle, sm, parity);
    };
    int best_i = 0;
    double best_v = func(exp(lo));
    for (int i = 1; i < n_grid; ++i) {
        const double v = func(exp(__dadd_rn(lo, __dmul_rn((double)i, step))));
        if (v < best_v) {
            best_v = v;
            best_i = i;
        }
    }
    const int il = best_i - 1 > 0 ? best_i - 1 : 0;
    const int ih = best_i + 1 < n_grid - 1 ? best_i + 1 : n_grid - 1;
    double a = __dadd_rn(lo, __dmul_rn((double)il, step));
    double b = __dadd_rn(lo, __dmul_rn((double)ih, step));
    double c = __dsub_rn(b, __dmul_rn(kPhi, __dsub_rn(b, a)));
    double d = __dadd_rn(a, __dmul_rn(kPhi, __dsub_rn(b, a)));
    double fc = func(exp(c)), fd = func(exp(d));
    for (int it = 0; it < n_iter; ++it) {
        if (fc < fd) {
            b = d;
            d = c;
            fd = fc;
            c = __dsub_rn(b, __dmul_rn(kPhi, __dsub_rn(b, a)));
            fc = func(exp(c));
        } else {
            a = c;
            c = d;
            fc = fd;
            d = __dadd_rn(a, __dmul_rn(kPhi, __dsub_rn(b, a)));
            fd = func(exp(d));
        }
    }
    const double opt = exp(__dmul_rn(__dadd_rn(a, b), 0.5));
    const double v = func(opt);
    if (blockIdx.x % kNullCtas == 0 && threadIdx.x == 0) {
        lam0[f] = opt;
        logl0[f] = -v;
    }
    cooperative_groups::this_cluster().sync();  // no CTA leaves while its sums may be read
}

// ---------------------------------------------------------------- host helpers
struct WsLayout {
    int64_t loglam, logdet, H, S, cheb, cmid, chalf, tgrid, cvals, alin, asq, asqt, hn, ccos, blas,
        total;
};

inline int64_t align256(int64_t b) { return (b + 255) / 256 * 256; }

inline int ns_of(int c) { return (c + 2) * (c + 1) / 2; }

// Table rows of the chunk GEMMs: grid rows + ones row + null rows (FP64 form) or the ones
// row + kChebG series coefficients (mixed form); sized for whichever is larger.
inline int64_t table_rows(int phi, int n_grid) {
    const int64_t direct = (int64_t)n_grid + 1 + phi, series = 1 + kChebG;
    return direct > series ? direct : series;
}

inline WsLayout ws_layout(int64_t n, int c, int phi, int n_grid) {
    WsLayout w;
    int64_t off = 0;
    w.loglam = off;
    off += align256(8 * (int64_t)n_grid);
    w.logdet = off;
    off += align256(8 * (int64_t)n_grid);
    w.H = off;
    off += align256(8 * (int64_t)(n_grid + phi) * n);
    w.S = off;
    off += align256(8 * (int64_t)(n_grid + 1 + phi) * phi * ns_of(c));
    const int64_t nf = 1 + (int64_t)phi * ns_of(c);
    w.cheb = off;
    off += align256(8 * (int64_t)n_grid * nf * kChebN);
    w.cmid = off;
    off += align256(8 * (int64_t)n_grid);
    w.chalf = off;
    off += align256(8 * (int64_t)n_grid);
    w.tgrid = off;
    off += align256(8 * (int64_t)n_grid * kChebG);
    w.cvals = off;
    off += align256(8 * (int64_t)n_grid * nf * kChebN);
    const int64_t rows = table_rows(phi, n_grid);
    w.alin = off;
    off += align256(8 * rows * (c + phi) * n);
    w.asq = off;
    off += align256(8 * rows * n);
    {  // the squared-sum table transposed for sq_sums_kernel, for either form's row count
        const int64_t r1 = (int64_t)n_grid + 1 + phi, r2 = 1 + kChebG;
        const int64_t ldt = sq_ldt(r1) > sq_ldt(r2) ? sq_ldt(r1) : sq_ldt(r2);
        w.asqt = off;
        off += align256(8 * ldt * n);
    }
    w.hn = off;
    off += align256(8 * (int64_t)kChebG * n);
    w.ccos = off;
    off += align256(8 * (int64_t)kChebG * kChebG);
    w.blas = off;
    off += kCublasWorkspaceBytes;
    w.total = off;
    return w;
}

struct ChunkLayout {
    int64_t sqp, cl, cq, state, open, blas, total;
};

// Partial squared sums of sq_sums_kernel's sample ranges: the largest over the row counts a
// chunk can use (FP64 form with and without null rows, mixed form).
inline int64_t sq_partial_doubles(int64_t n, int64_t m, int phi, int n_grid) {
    const int64_t cand[3] = {(int64_t)n_grid + 1 + phi, (int64_t)n_grid + 1, 1 + (int64_t)kChebG};
    int64_t best = 0;
    for (int64_t r : cand) {
        const int ks = sq_split(n, m, r);
        const int64_t v = ks > 1 ? (int64_t)ks * m * sq_ldt(r) : 0;
        if (v > best) best = v;
    }
    return best;
}

inline ChunkLayout chunk_layout(int64_t n, int c, int phi, int n_grid, int64_t m) {
    ChunkLayout L;
    const int64_t rows = table_rows(phi, n_grid);
    int64_t off = 0;
    L.sqp = off;
    off += align256(8 * sq_partial_doubles(n, m, phi, n_grid));
    L.cl = off;
    off += align256(8 * rows * (c + phi) * m);
    L.cq = off;
    off += align256(8 * rows * m);
    L.state = off;
    off += align256(2 * (int64_t)sizeof(SearchState) * phi * m);
    L.open = off;  // counter, then the list
    off += align256(256 + 2 * (int64_t)sizeof(int64_t) * phi * m);
    L.blas = off;  // cuBLAS workspace of this chunk's DGEMMs (fixed size: same kernels alone or
    off += kCublasWorkspaceBytes;  // beside other streams' work, so results do not depend on it)
    L.total = off;
    return L;
}

// Mixed form, genotype-side linear x-sums: the chunk GEMM  CL = A_lin x~  with x~ = U^T g
// equals  (U A_lin^T)^T g, so the basis  V = U A_lin^T  (n x rows_lin, column q = basis of
// CL row q) is formed once per cohort and split into INT8 digit planes; every chunk then
// gets CL from the decoded calls on the INT8 rotation core (V has rows_lin ~ 1 % of U's n
// columns), instead of an FP64 DGEMM over the rotated chunk.
struct SeriesLayout {
    int64_t rows_lin, basis, ozaki, total;
};

inline SeriesLayout series_layout(int64_t n, int c, int phi) {
    SeriesLayout L;
    L.rows_lin = (int64_t)(1 + kChebG) * (c + phi);
    int64_t off = 0;
    L.basis = off;
    off += align256(8 * n * L.rows_lin);
    L.ozaki = off;
    off += align256(tc::ozaki_layout(L.rows_lin, n).total);
    L.total = off;
    return L;
}

// numpy.linspace(start, stop, num): start + i*step, last element = stop.
__global__ void linspace_kernel(double* out, double start, double stop, int num) {
    const int i = threadIdx.x + blockIdx.x * blockDim.x;
    if (i >= num) return;
    if (num == 1) {
        out[0] = start;
        return;
    }
    const double step = (stop - start) / (double)(num - 1);
    out[i] = (i == num - 1) ? stop : __dadd_rn(__dmul_rn((double)i, step), start);
}

// F statistics (NaN where there is no test) -> F-test p-values, in place, one thread per
// value, for up to two arrays of `count` values (Wald and score) in one launch.  Bound by
// the latency of one value's FP64 chain: the large-a expansion is ~150 dependent steps with
// one division, against up to ~100 continued-fraction steps of four divisions each.
// Measured, continued fraction -> expansion: 2 x 8192 values at df = 2e4 279 -> 3.6 us,
// 2 x 131 072 values 556 -> 6.8 us, 500 values at df = 498 37 -> 2.5 us.
__global__ void lmm_fpvalue_kernel(double* __restrict__ v0, double* __restrict__ v1,
                                   int64_t count, double df, BetaGrat g, bool large_a) {
    const int64_t total = v1 ? 2 * count : count;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (int64_t)gridDim.x * blockDim.x) {
        double* v = i < count ? v0 + i : v1 + (i - count);
        *v = f_pvalue(*v, df, g, large_a);
    }
}

// Constants of betainc_half_large_a for a = df / 2: Gamma(a + 1/2) / (Gamma(a) sqrt(a - 1/4))
// from the Stirling series of lgamma_ratio_half.
inline BetaGrat beta_grat(double df) {
    const double a = 0.5 * df, t = a - 0.25, r = 1.0 / a, r2 = r * r;
    const double s = r * (-1.0 / 8 + r2 * (1.0 / 192 + r2 * (-1.0 / 640 + r2 * (17.0 / 14336 +
                     r2 * (-31.0 / 18432 + r2 * (691.0 / 180224))))));
    return BetaGrat{t, 0.25 / (t * t), std::sqrt(a / t) * std::exp(s)};
}

// Squared x-sums of a rotated chunk: sq_sums_kernel (+ sq_reduce_kernel when the samples
// are split into ranges).  AT: the transposed table (ld sq_ldt(rows)); P: partial sums
// (sq_partial_doubles); CQ: rows x m, ld ldcq.
int32_t launch_sq_sums(const double* AT, int64_t rows, const double* X, int64_t ldx, int64_t n,
                       int64_t m, double* P, double* CQ, int64_t ldcq, cudaStream_t st) {
    const int tr = sq_tile_rows(rows);
    const int64_t ldt = sq_ldt(rows);
    const int ks = sq_split(n, m, rows);
    const int64_t klen = ceil_div(ceil_div(n, ks), kSqTK) * kSqTK;
    const int64_t gx = ceil_div(m, kSqTN);
    if (gx > 0x7fffffffll || ldt / tr > 65535) {
        set_error("squared x-sums: chunk too large");
        return JB_E_INVALID;
    }
    dim3 grid((unsigned)gx, (unsigned)(ldt / tr), (unsigned)ks);
    double* out = ks > 1 ? P : CQ;
    const int64_t ldo = ks > 1 ? ldt : ldcq;
    if (tr == 56) {
        JB_CUDA(cudaFuncSetAttribute(sq_sums_kernel<56>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     SqCfg<56>::SMEM));
        sq_sums_kernel<56><<<grid, kSqThreads, SqCfg<56>::SMEM, st>>>(
            AT, ldt, X, ldx, n, m, klen, (int)rows, out, ldo, m * ldt);
    } else {
        JB_CUDA(cudaFuncSetAttribute(sq_sums_kernel<104>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     SqCfg<104>::SMEM));
        sq_sums_kernel<104><<<grid, kSqThreads, SqCfg<104>::SMEM, st>>>(
            AT, ldt, X, ldx, n, m, klen, (int)rows, out, ldo, m * ldt);
    }
    JB_LAUNCH_CHECK("sq_sums_kernel");
    if (ks > 1) {
        const int64_t blocks = ceil_div(m * rows, 256) < 4096 ? ceil_div(m * rows, 256) : 4096;
        sq_reduce_kernel<<<(unsigned)blocks, 256, 0, st>>>(P, ldt, m, (int)rows, ks, CQ, ldcq);
        JB_LAUNCH_CHECK("sq_reduce_kernel");
    }
    return JB_OK;
}

// Lanes per pair of the series search: the most with which all pairs are resident at once (2
// CTAs per SM), where the chain of steps of one pair sets the time; beyond one wave the
// fewest, which do the least work.  Measured, every test, one covariate column, 16 / 8 / 4
// lanes: 1000 pairs 57 / 80 / 105 us, 4000 pairs 144 / 87 / 108 us, 8192 pairs 259 / 158 /
// 118 us; two columns, 16 / 8 lanes: 2000 pairs 80 / 101 us, 8192 pairs 298 / 204 us.  32
// lanes pay where 16 hold too many coefficients, for three and four columns: 1000 pairs and
// three columns 102 -> 91 us (one column, with one point at a time, 64 -> 70 us).
inline int search_lanes(int64_t pairs, int c) {
    const int64_t threads = (int64_t)2 * tc::num_sms() * kSearchThreads;
    if (c > 2 && pairs * 32 <= threads) return 32;
    if (pairs * 16 <= threads) return 16;
    return c > 1 || pairs * 8 <= threads ? 8 : 4;
}

template <int C, int LP, bool GUIDE>
void launch_search_as(const Params& p, cudaStream_t st) {
    const int64_t threads = p.m * p.phi * LP;
    auto kern = lmm_search_kernel<C, LP, GUIDE, kByMode>;
    if constexpr (C >= 2 && LP == (C > 2 ? 32 : 16)) {
        if (p.mode == 2) kern = lmm_search_kernel<C, LP, GUIDE, kMleOnly>;
        if (p.mode == 1) kern = lmm_search_kernel<C, LP, GUIDE, kRemlOnly>;
    }
    kern<<<(unsigned)ceil_div(threads, kSearchThreads), kSearchThreads, 0, st>>>(p);
}

template <int C, bool GUIDE>
void launch_search(const Params& p, cudaStream_t st) {
    const int lanes = search_lanes(p.m * p.phi, C);
    if (C > 2 && lanes == 32)
        launch_search_as<C, (C > 2 ? 32 : 16), GUIDE>(p, st);
    else if (lanes == 16)
        launch_search_as<C, 16, GUIDE>(p, st);
    else if (C == 1 && lanes == 4)
        launch_search_as<C, C == 1 ? 4 : 8, GUIDE>(p, st);
    else
        launch_search_as<C, 8, GUIDE>(p, st);
}

template <int C>
int32_t launch_pairs(const Params& p, cudaStream_t st) {
    const int64_t pairs = p.m * p.phi;
    const unsigned warps = (unsigned)ceil_div(pairs * 32, kPairsThreads);
    if (p.state) {
        if (p.mode != 3) {
            JB_CUDA(cudaMemsetAsync(p.open_count, 0, sizeof(*p.open_count), st));
            launch_search<C, true>(p, st);
            JB_LAUNCH_CHECK("lmm_search_kernel");
            const int64_t sms = tc::num_sms();
            lmm_open_kernel<C><<<(unsigned)(2 * pairs < sms ? 2 * pairs : sms), kOpenThreads, 0, st>>>(
                p, kOpenPerSm * sms);
            JB_LAUNCH_CHECK("lmm_open_kernel");
            if (2 * pairs > kOpenPerSm * sms) {
                const int64_t blocks = sms * PairsOccupancy<C>::kMinBlocks;
                lmm_close_kernel<C><<<(unsigned)(warps < blocks ? warps : blocks), kPairsThreads, 0, st>>>(
                    p, kOpenPerSm * sms);
                JB_LAUNCH_CHECK("lmm_close_kernel");
            }
        }
        lmm_finish_kernel<C><<<warps, kPairsThreads, 0, st>>>(p);
    } else if (p.cheb) {
        launch_search<C, false>(p, st);
    } else {
        lmm_pairs_kernel<C><<<warps, kPairsThreads, 0, st>>>(p);
    }
    JB_LAUNCH_CHECK("lmm search");
    // p-values of the tests this mode ran (other outputs stay untouched)
    double* v0 = (p.mode == 1 || p.mode == 4) ? p.out.p_wald : nullptr;
    double* v1 = (p.mode == 3 || p.mode == 4) ? p.out.p_score : nullptr;
    if (!v0) {
        v0 = v1;
        v1 = nullptr;
    }
    if (v0) {
        const int64_t total = v1 ? 2 * pairs : pairs;
        const int64_t blocks = ceil_div(total, 128) < 8192 ? ceil_div(total, 128) : 8192;
        lmm_fpvalue_kernel<<<(unsigned)blocks, 128, 0, st>>>(v0, v1, pairs, p.df, beta_grat(p.df),
                                                             0.5 * p.df >= kBgMinA);
        JB_LAUNCH_CHECK("lmm_fpvalue_kernel");
    }
    return JB_OK;
}

template <int C>
int32_t launch_prepare(int64_t n, int phi, int n_grid, const double* evals, const double* W,
                       int64_t ldw, const double* Y, int64_t ldy, const double* lam0,
                       double l_min, double l_max, uint8_t* ws, cudaStream_t st, bool interp,
                       bool sums_only) {
    const WsLayout L = ws_layout(n, C, phi, n_grid);
    double* loglam = reinterpret_cast<double*>(ws + L.loglam);
    double* logdet = reinterpret_cast<double*>(ws + L.logdet);
    double* H = reinterpret_cast<double*>(ws + L.H);
    double* S = reinterpret_cast<double*>(ws + L.S);
    linspace_kernel<<<(n_grid + 127) / 128, 128, 0, st>>>(loglam, std::log(l_min), std::log(l_max),
                                                        n_grid);
    JB_LAUNCH_CHECK("linspace_kernel");
    const int rows_h = n_grid + (lam0 ? phi : 0);
    lmm_table_kernel<<<rows_h, 256, 0, st>>>(n, n_grid, phi, evals, loglam, lam0, H, logdet);
    JB_LAUNCH_CHECK("lmm_table_kernel");
    const int rows_s = n_grid + 1 + (lam0 ? phi : 0);
    lmm_shared_kernel<C><<<dim3(rows_s, phi), 256, 0, st>>>(n, n_grid, phi, W, ldw, Y, ldy, H, S);
    JB_LAUNCH_CHECK("lmm_shared_kernel");
    if (sums_only) return JB_OK;  // guided plain form, score test only
    const unsigned ny = (unsigned)(ceil_div(n, 256) < 64 ? ceil_div(n, 256) : 64);
    double* Alin = reinterpret_cast<double*>(ws + L.alin);
    double* Asq = reinterpret_cast<double*>(ws + L.asq);
    if (!interp) {
        lmm_gemm_tables_kernel<C><<<dim3(rows_s, ny), 256, 0, st>>>(n, n_grid, phi, W, ldw, Y, ldy,
                                                                   H, Alin, Asq);
        JB_LAUNCH_CHECK("lmm_gemm_tables_kernel");
    } else {
        // global series tables: node values -> coefficients (one DGEMM) -> A_lin / A_sq
        const double lo = std::log(kDomainLo), hi = std::log(kDomainHi);
        double* hn = reinterpret_cast<double*>(ws + L.hn);
        double* ccos = reinterpret_cast<double*>(ws + L.ccos);
        lmm_series_nodes_kernel<<<dim3(ny, kChebG), 256, 0, st>>>(n, 0.5 * (lo + hi), 0.5 * (hi - lo),
                                                                   evals, hn);
        JB_LAUNCH_CHECK("lmm_series_nodes_kernel");
        lmm_series_consts_kernel<<<kChebG + n_grid, kChebG, 0, st>>>(
            ccos, n_grid, 0.5 * (lo + hi), 1.0 / (0.5 * (hi - lo)), loglam,
            reinterpret_cast<double*>(ws + L.tgrid));
        JB_LAUNCH_CHECK("lmm_series_consts_kernel");
        cublasHandle_t h = cublas_handle();
        if (!h) {
            set_error("cuBLAS handle creation failed");
            return JB_E_LIBRARY;
        }
        cublasStatus_t cs = bind_cublas(h, st, ws + L.blas, kCublasWorkspaceBytes);
        if (cs != CUBLAS_STATUS_SUCCESS) return cublas_status(cs, "cublasSetStream/Workspace");
        const double one = 1.0, zero = 0.0;
        // (n x K, column-major, ld n) = hn (n x K) * ccos^T: coefficient rows 1..K of Asq
        cs = cublasDgemm(h, CUBLAS_OP_N, CUBLAS_OP_T, (int)n, kChebG, kChebG, &one, hn, (int)n,
                         ccos, kChebG, &zero, Asq + n, (int)n);
        if (cs != CUBLAS_STATUS_SUCCESS) return cublas_status(cs, "cublasDgemm (series transform)");
        lmm_series_tables_kernel<C><<<dim3(1 + kChebG, ny), 256, 0, st>>>(n, phi, W, ldw, Y, ldy,
                                                                         Alin, Asq);
        JB_LAUNCH_CHECK("lmm_series_tables_kernel");
    }
    {  // the squared-sum rows transposed for sq_sums_kernel
        const int64_t rows_sq = interp ? 1 + kChebG : (int64_t)rows_s;
        const int64_t ldt = sq_ldt(rows_sq);
        const int64_t blocks = ceil_div(n * ldt, 256) < 8192 ? ceil_div(n * ldt, 256) : 8192;
        sq_table_kernel<<<(unsigned)blocks, 256, 0, st>>>(Asq, n, (int)rows_sq, ldt,
                                                          reinterpret_cast<double*>(ws + L.asqt));
        JB_LAUNCH_CHECK("sq_table_kernel");
    }
    if (interp) {
        const int nf = 1 + phi * Lay<C>::NS;
        double* vals = reinterpret_cast<double*>(ws + L.cvals);
        double* coef = reinterpret_cast<double*>(ws + L.cheb);
        lmm_cheb_nodes_kernel<C><<<dim3(n_grid * kChebN, phi), 256, 0, st>>>(
            n, n_grid, phi, evals, W, ldw, Y, ldy, loglam, vals,
            reinterpret_cast<double*>(ws + L.cmid), reinterpret_cast<double*>(ws + L.chalf));
        JB_LAUNCH_CHECK("lmm_cheb_nodes_kernel");
        lmm_cheb_coef_kernel<<<dim3(n_grid, (nf + 31) / 32), 256, 0, st>>>(nf, vals, coef);
        JB_LAUNCH_CHECK("lmm_cheb_coef_kernel");
    }
    return JB_OK;
}

}  // namespace lmm
}  // namespace jb

using namespace jb;
using namespace jb::lmm;

extern "C" {

int64_t jb_lmm_workspace_size(int64_t n, int32_t n_cvt, int32_t phi, int32_t n_grid) {
    if (n <= 0 || n_cvt < 1 || phi < 1 || n_grid < 1) return -1;
    return ws_layout(n, n_cvt, phi, n_grid).total;
}

int32_t jb_lmm_prepare(int32_t lmm_mode, int32_t precision, int64_t n, int32_t n_cvt,
                       int32_t phi, const double* evals, const double* UtW, int64_t ldw,
                       const double* Uty, int64_t ldy, const double* lam0, double l_min,
                       double l_max, int32_t n_grid, void* workspace, int64_t workspace_bytes,
                       uintptr_t stream) {
    JB_CHECK_ARG(precision == 0 || precision == 1 || precision == 3,
                 "jb_lmm_prepare: precision must be 0, 1 or 3");
    JB_CHECK_ARG(lmm_mode >= 1 && lmm_mode <= 4, "jb_lmm_prepare: lmm_mode must be 1..4");
    JB_CHECK_ARG(n > 0 && phi >= 1 && n_grid >= 2, "jb_lmm_prepare: bad sizes");
    JB_CHECK_ARG(n_cvt >= 1 && n_cvt <= kMaxCvt, "jb_lmm_prepare: n_cvt must be in 1..%d", kMaxCvt);
    JB_CHECK_ARG(n > n_cvt + 1, "jb_lmm_prepare: n must exceed n_cvt + 1");
    JB_CHECK_ARG(ldw >= n && ldy >= n, "jb_lmm_prepare: bad leading dimension");
    JB_CHECK_ARG(l_min > 0 && l_max > l_min, "jb_lmm_prepare: need 0 < l_min < l_max");
    JB_CHECK_ARG(lmm_mode == 1 || lam0, "jb_lmm_prepare: modes 2-4 need lam0");
    JB_CHECK_ARG(workspace_bytes >= jb_lmm_workspace_size(n, n_cvt, phi, n_grid),
                 "jb_lmm_prepare: workspace too small");
    JB_CHECK_ARG(phi <= 65535, "jb_lmm_prepare: too many phenotypes");
    JB_CHECK_ARG(precision == 0 || (l_min >= kDomainLo * (1 - 1e-12) && l_max <= kDomainHi * (1 + 1e-12)),
                 "jb_lmm_prepare: the series need 1e-5 <= l_min < l_max <= 1e5");
    cudaStream_t st = as_stream(stream);
    uint8_t* ws = static_cast<uint8_t*>(workspace);
    const double* l0 = lmm_mode == 1 ? nullptr : lam0;
    const bool series = precision != 0, sums_only = precision == 3 && lmm_mode == 3;
    switch (n_cvt) {
        case 1: return launch_prepare<1>(n, phi, n_grid, evals, UtW, ldw, Uty, ldy, l0, l_min, l_max, ws, st, series, sums_only);
        case 2: return launch_prepare<2>(n, phi, n_grid, evals, UtW, ldw, Uty, ldy, l0, l_min, l_max, ws, st, series, sums_only);
        case 3: return launch_prepare<3>(n, phi, n_grid, evals, UtW, ldw, Uty, ldy, l0, l_min, l_max, ws, st, series, sums_only);
        case 4: return launch_prepare<4>(n, phi, n_grid, evals, UtW, ldw, Uty, ldy, l0, l_min, l_max, ws, st, series, sums_only);
    }
    return JB_E_UNSUPPORTED;
}

int64_t jb_lmm_chunk_workspace_size(int64_t n, int32_t n_cvt, int32_t phi, int32_t n_grid,
                                    int64_t m) {
    if (n <= 0 || n_cvt < 1 || phi < 1 || n_grid < 1 || m < 0) return -1;
    return chunk_layout(n, n_cvt, phi, n_grid, m > 0 ? m : 1).total;
}

int32_t jb_lmm_series_rows(void) { return 1 + kChebG; }

int64_t jb_lmm_series_workspace_size(int64_t n, int32_t n_cvt, int32_t phi) {
    if (n <= 0 || n_cvt < 1 || n_cvt > kMaxCvt || phi < 1) return -1;
    return series_layout(n, n_cvt, phi).total;
}

int32_t jb_lmm_series_prepare(int64_t n, int32_t n_cvt, int32_t phi, int32_t n_grid,
                              const void* workspace, int64_t workspace_bytes, const double* U,
                              int64_t ldu, void* series_ws, int64_t series_bytes,
                              uintptr_t stream) {
    JB_CHECK_ARG(n > 0 && n_cvt >= 1 && n_cvt <= kMaxCvt && phi >= 1 && n_grid >= 2,
                 "jb_lmm_series_prepare: bad sizes");
    JB_CHECK_ARG(U && ldu >= n, "jb_lmm_series_prepare: bad eigenvector matrix");
    JB_CHECK_ARG(workspace && workspace_bytes >= jb_lmm_workspace_size(n, n_cvt, phi, n_grid),
                 "jb_lmm_series_prepare: workspace too small");
    const SeriesLayout SL = series_layout(n, n_cvt, phi);
    JB_CHECK_ARG(series_ws && series_bytes >= SL.total, "jb_lmm_series_prepare: series workspace too small");
    JB_CHECK_ARG(SL.rows_lin <= 65535, "jb_lmm_series_prepare: too many phenotypes");
    const WsLayout L = ws_layout(n, n_cvt, phi, n_grid);
    uint8_t* ws = const_cast<uint8_t*>(static_cast<const uint8_t*>(workspace));
    uint8_t* sws = static_cast<uint8_t*>(series_ws);
    cudaStream_t st = as_stream(stream);
    cublasHandle_t h = cublas_handle();
    if (!h) {
        set_error("cuBLAS handle creation failed");
        return JB_E_LIBRARY;
    }
    cublasStatus_t cs = bind_cublas(h, st, ws + L.blas, kCublasWorkspaceBytes);
    if (cs != CUBLAS_STATUS_SUCCESS) return cublas_status(cs, "cublasSetStream/Workspace");
    const double one = 1.0, zero = 0.0;
    double* V = reinterpret_cast<double*>(sws + SL.basis);
    // V (n x rows_lin) = U (n x n) * A_lin^T, A_lin stored as rows of n (column-major n x rows_lin)
    cs = cublasDgemm(h, CUBLAS_OP_N, CUBLAS_OP_N, (int)n, (int)SL.rows_lin, (int)n, &one, U, (int)ldu,
                     reinterpret_cast<const double*>(ws + L.alin), (int)n, &zero, V, (int)n);
    if (cs != CUBLAS_STATUS_SUCCESS) return cublas_status(cs, "cublasDgemm (series basis)");
    return tc::ozaki_split(V, n, SL.rows_lin, n, sws + SL.ozaki, st);
}

int32_t jb_lmm_chunk_series_i8(int64_t n, int32_t n_cvt, int32_t phi, int32_t n_grid, int64_t m,
                               const void* series_ws, int64_t series_bytes, const int8_t* codes,
                               int64_t ld_codes, const double* mean, int32_t has_missing,
                               void* rot_ws, int64_t rot_bytes, void* chunk_workspace,
                               int64_t chunk_bytes, uintptr_t stream) {
    JB_CHECK_ARG(n > 0 && n_cvt >= 1 && n_cvt <= kMaxCvt && phi >= 1 && n_grid >= 2 && m >= 0,
                 "jb_lmm_chunk_series_i8: bad sizes");
    if (m == 0) return JB_OK;
    const SeriesLayout SL = series_layout(n, n_cvt, phi);
    JB_CHECK_ARG(series_ws && series_bytes >= SL.total, "jb_lmm_chunk_series_i8: series workspace too small");
    const tc::RotChunkLayout RL = tc::rot_chunk_layout(n, m);
    JB_CHECK_ARG(rot_ws && rot_bytes >= RL.total, "jb_lmm_chunk_series_i8: rotation workspace too small");
    JB_CHECK_ARG(ceil_div(SL.rows_lin, 32) <= ceil_div(n, 32),
                 "jb_lmm_chunk_series_i8: more series rows than samples");
    JB_CHECK_ARG(codes && ld_codes >= n && (!has_missing || mean), "jb_lmm_chunk_series_i8: bad genotype input");
    const ChunkLayout CLy = chunk_layout(n, n_cvt, phi, n_grid, m);
    JB_CHECK_ARG(chunk_workspace && chunk_bytes >= CLy.total, "jb_lmm_chunk_series_i8: chunk workspace too small");
    uint8_t* rws = static_cast<uint8_t*>(rot_ws);
    double* CL = reinterpret_cast<double*>(static_cast<uint8_t*>(chunk_workspace) + CLy.cl);
    const uint8_t* ows = static_cast<const uint8_t*>(series_ws) + SL.ozaki;
    tc::Tile* tiles = reinterpret_cast<tc::Tile*>(rws + RL.tiles);
    int* status = reinterpret_cast<int*>(rws + RL.status);
    cudaStream_t st = as_stream(stream);
    if (has_missing) {  // the [calls | masks] pairs packed by jb_rotate_i8 for these codes
        const int64_t NB = ceil_div(m, 128);
        return tc::rotate_i8_gemm(ows, SL.rows_lin, n, reinterpret_cast<const int8_t*>(rws + RL.b_off),
                                  NB * 256, RL.ldb, true, m, mean, CL, SL.rows_lin, tiles, status, st);
    }
    return tc::rotate_i8_gemm(ows, SL.rows_lin, n, codes, m, ld_codes, false, m, nullptr, CL,
                              SL.rows_lin, tiles, status, st);
}

int32_t jb_lmm_chunk(int32_t lmm_mode, int32_t precision, int64_t n, int32_t n_cvt, int32_t phi,
                     int64_t m,
                     const double* evals, const double* UtW, int64_t ldw, const double* Uty,
                     int64_t ldy, const double* UtG, int64_t ldg, const double* lam0,
                     const double* logl0, double l_min, double l_max, int32_t n_grid,
                     int32_t n_iter, jb_lmm_out out, void* workspace, int64_t workspace_bytes,
                     void* chunk_workspace, int64_t chunk_bytes, uintptr_t stream) {
    JB_CHECK_ARG(lmm_mode >= 1 && lmm_mode <= 4, "jb_lmm_chunk: lmm_mode must be 1..4");
    JB_CHECK_ARG(n > 0 && phi >= 1 && m >= 0 && n_grid >= 2 && n_iter >= 0, "jb_lmm_chunk: bad sizes");
    JB_CHECK_ARG(n_cvt >= 1 && n_cvt <= kMaxCvt, "jb_lmm_chunk: n_cvt must be in 1..%d", kMaxCvt);
    JB_CHECK_ARG(n > n_cvt + 1, "jb_lmm_chunk: n must exceed n_cvt + 1");
    JB_CHECK_ARG(ldw >= n && ldy >= n && ldg >= n, "jb_lmm_chunk: bad leading dimension");
    JB_CHECK_ARG(l_min > 0 && l_max > l_min, "jb_lmm_chunk: need 0 < l_min < l_max");
    JB_CHECK_ARG(lmm_mode != 2 && lmm_mode != 4 ? true : logl0 != nullptr,
                 "jb_lmm_chunk: modes 2 and 4 need logl0");
    JB_CHECK_ARG(workspace_bytes >= jb_lmm_workspace_size(n, n_cvt, phi, n_grid),
                 "jb_lmm_chunk: workspace too small");
    if (m == 0) return JB_OK;
    const WsLayout L = ws_layout(n, n_cvt, phi, n_grid);
    uint8_t* ws = static_cast<uint8_t*>(workspace);
    Params p;
    p.mode = lmm_mode;
    p.n = n;
    p.phi = phi;
    p.m = m;
    p.evals = evals;
    p.W = UtW;
    p.ldw = ldw;
    p.Y = Uty;
    p.ldy = ldy;
    p.G = UtG;
    p.ldg = ldg;
    p.logl0 = logl0;
    p.n_grid = n_grid;
    p.n_iter = n_iter;
    p.loglam = reinterpret_cast<const double*>(ws + L.loglam);
    p.logdet = reinterpret_cast<const double*>(ws + L.logdet);
    p.H = reinterpret_cast<const double*>(ws + L.H);
    p.S = reinterpret_cast<const double*>(ws + L.S);
    const double df = (double)(n - n_cvt - 1);
    p.df = df;
    p.n_d = (double)n;
    p.c_reml = 0.5 * df * (std::log(df) - std::log(2 * M_PI) - 1.0);
    p.c_mle = 0.5 * (double)n * (std::log((double)n) - std::log(2 * M_PI) - 1.0);
    p.out = out;
    JB_CHECK_ARG(precision >= 0 && precision <= 3, "jb_lmm_chunk: precision must be 0 to 3");
    p.cheb = precision >= 1 ? reinterpret_cast<const double*>(ws + L.cheb) : nullptr;
    p.cheb_mid = reinterpret_cast<const double*>(ws + L.cmid);
    p.cheb_half = reinterpret_cast<const double*>(ws + L.chalf);
    p.tgrid = reinterpret_cast<const double*>(ws + L.tgrid);
    p.lam0 = lam0;
    JB_CHECK_ARG(precision != 3 || n_grid >= 16, "jb_lmm_chunk: precision 3 needs n_grid >= 16");
    JB_CHECK_ARG(precision == 0 || lmm_mode == 1 || lam0 != nullptr,
                 "jb_lmm_chunk: precision 1 to 3 needs lam0 in modes 2-4");
    JB_CHECK_ARG(precision == 0 || (l_min >= kDomainLo * (1 - 1e-12) && l_max <= kDomainHi * (1 + 1e-12)),
                 "jb_lmm_chunk: the series need 1e-5 <= l_min < l_max <= 1e5");
    {
        const double lo = std::log(kDomainLo), hi = std::log(kDomainHi);
        p.gmid = 0.5 * (lo + hi);
        p.ginv = 1.0 / (0.5 * (hi - lo));
    }
    cudaStream_t st = as_stream(stream);
    // chunk GEMMs: weighted x-sums of every table row (grid, ones, null) for all SNPs
    const ChunkLayout CLy = chunk_layout(n, n_cvt, phi, n_grid, m);
    JB_CHECK_ARG(chunk_workspace && chunk_bytes >= CLy.total, "jb_lmm_chunk: chunk workspace too small");
    uint8_t* cws = static_cast<uint8_t*>(chunk_workspace);
    double* CL = reinterpret_cast<double*>(cws + CLy.cl);
    double* CQ = reinterpret_cast<double*>(cws + CLy.cq);
    p.state = precision == 3 ? reinterpret_cast<SearchState*>(cws + CLy.state) : nullptr;
    p.open_count = reinterpret_cast<unsigned long long*>(cws + CLy.open);
    p.open_list = reinterpret_cast<int64_t*>(cws + CLy.open + 256);
    // FP64 form: grid rows, ones row, null rows (only when prepared); mixed: ones + series
    const int rows = precision >= 1 ? 1 + kChebG : n_grid + 1 + (lmm_mode == 1 ? 0 : phi);
    const int rows_lin = rows * (n_cvt + phi);
    if (precision != 3 || lmm_mode != 3) {  // the guided form's score test sums directly
        if (precision != 2) {  // precision 2: CL already formed by jb_lmm_chunk_series_i8
            cublasHandle_t h = cublas_handle();
            if (!h) {
                set_error("cuBLAS handle creation failed");
                return JB_E_LIBRARY;
            }
            cublasStatus_t cs = bind_cublas(h, st, cws + CLy.blas, kCublasWorkspaceBytes);
            if (cs != CUBLAS_STATUS_SUCCESS) return cublas_status(cs, "cublasSetStream/Workspace");
            const double one = 1.0, zero = 0.0;
            cs = cublasDgemm(h, CUBLAS_OP_T, CUBLAS_OP_N, rows_lin, (int)m, (int)n, &one,
                             reinterpret_cast<const double*>(ws + L.alin), (int)n, UtG, (int)ldg,
                             &zero, CL, rows_lin);
            if (cs != CUBLAS_STATUS_SUCCESS) return cublas_status(cs, "cublasDgemm (linear x-sums)");
        }
        const int32_t rc = launch_sq_sums(reinterpret_cast<const double*>(ws + L.asqt), rows, UtG,
                                          ldg, n, m, reinterpret_cast<double*>(cws + CLy.sqp), CQ,
                                          rows, st);
        if (rc) return rc;
    }
    p.CL = CL;
    p.ldcl = rows_lin;
    p.CQ = CQ;
    p.ldcq = rows;
    switch (n_cvt) {
        case 1: return launch_pairs<1>(p, st);
        case 2: return launch_pairs<2>(p, st);
        case 3: return launch_pairs<3>(p, st);
        case 4: return launch_pairs<4>(p, st);
    }
    return JB_E_UNSUPPORTED;
}

int32_t jb_null_mle(int64_t n, int32_t n_cvt, int32_t phi, const double* evals, const double* UtW,
                    int64_t ldw, const double* Uty, int64_t ldy, double l_min, double l_max,
                    int32_t n_grid, int32_t n_iter, double* lam0, double* logl0,
                    uintptr_t stream) {
    JB_CHECK_ARG(n > 0 && phi >= 1 && n_grid >= 2 && n_iter >= 0, "jb_null_mle: bad sizes");
    JB_CHECK_ARG(n_cvt >= 1 && n_cvt <= kMaxCvt, "jb_null_mle: n_cvt must be in 1..%d", kMaxCvt);
    JB_CHECK_ARG(ldw >= n && ldy >= n, "jb_null_mle: bad leading dimension");
    JB_CHECK_ARG(l_min > 0 && l_max > l_min, "jb_null_mle: need 0 < l_min < l_max");
    const double lo = std::log(l_min), hi = std::log(l_max);
    const double step = (hi - lo) / (double)(n_grid - 1);
    const double c_mle = 0.5 * (double)n * (std::log((double)n) - std::log(2 * M_PI) - 1.0);
    cudaStream_t st = as_stream(stream);
    switch (n_cvt) {
#define JB_NULL_CASE(CC)                                                                     \
    case CC:                                                                                 \
        null_mle_kernel<CC><<<phi * kNullCtas, kNullThreads, 0, st>>>(n, UtW, ldw, Uty, ldy, evals, lo, step,     \
                                                 n_grid, n_iter, hi, c_mle, lam0, logl0);    \
        JB_LAUNCH_CHECK("null_mle_kernel");                                                  \
        return JB_OK;
        JB_NULL_CASE(1)
        JB_NULL_CASE(2)
        JB_NULL_CASE(3)
        JB_NULL_CASE(4)
#undef JB_NULL_CASE
    }
    return JB_E_UNSUPPORTED;
}

}  // extern "C"
