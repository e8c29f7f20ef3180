// Series search of the lambda optima: one (SNP, phenotype) pair per group of LP lanes.
//
// The weighted sums of a pair at any log-lambda come from Chebyshev series (see jb_lmm.cu),
// so a probe costs a few hundred FP64 operations and no pass over the samples; the search is
// bound by FP64 issue.  A sum over the kChebG = 96 coefficients is defined as the butterfly
// sum of 32 virtual lanes, virtual lane l holding coefficients l, l + 32, l + 64.  Lane r of
// a group stands in for virtual lanes r, r + LP, r + 2 LP, ..., with the same values and the
// same order of every sum whatever LP is, so the group size only trades registers against
// repeated work: the coefficients of a pair take 3 (C + 2) 32 / LP doubles of each lane, and
// the per-probe scalar work (Pab recursion, golden-section steps) is repeated by every lane.
//   * LP = 4 for one covariate column (72 coefficient doubles, 8 pairs per warp) and 8 for
//     two to four (48 to 72 doubles, 4 pairs per warp) do the least work per pair; LP = 16
//     (12 to 36 doubles), 32 for three and four columns, has the shortest chain of steps per
//     pair, for chunks whose pairs cannot fill the GPU otherwise (search_lanes);
//   * offsets of the butterfly that stay within a lane need no shuffle;
//   * the logarithms of one likelihood are taken by different lanes of the group;
//   * grid points are shared out one per lane after their sums, so that their Pab recursions
//     and logarithms run once per group;
//   * the REML and MLE searches advance together and share the sums of a probe while every
//     pair of the warp has both at the same point (the first ten or so of the 22 probes).
// Measured against the earlier form (one pair per half-warp for one covariate column, per
// warp for more), the same results bit for bit: 2048 SNPs x 64 phenotypes, n = 20 000,
// every test 3.11 -> 1.38 ms; 8000 SNPs x 4 phenotypes, two columns, MLE 0.80 -> 0.40 ms;
// 8192 SNPs, one phenotype 0.26 -> 0.11 ms.
#pragma once

namespace jb {
namespace lmm {

constexpr int kSearchThreads = 128;  // 2 CTAs per SM: up to 255 registers

// Chebyshev values of a group: t[v] = T_{r + LP v}(x), m[v] = T_{LP - r + LP v}(x) (r the
// lane within the group), by the doubling identity T_{a+b} = 2 T_a T_b - T_{a-b} with a the
// largest power of two below the index.  Returns T_32(x).
template <int LP>
__device__ __forceinline__ double cheb_group(double x, int r, double (&t)[32 / LP],
                                             double (&m)[32 / LP]) {
    constexpr int V = 32 / LP;
    static_assert(LP == 4 || LP == 8 || LP == 16 || LP == 32, "group of 4, 8, 16 or 32 lanes");
    const double t2 = fma(2.0 * x, x, -1.0);
    const double t3 = fma(2.0 * t2, x, -x);
    double ta = fma(2.0 * t2, t2, -1.0);  // T_4
    const int q = r & 3;
    double lo = q == 0 ? 1.0 : (q == 1 ? x : (q == 2 ? t2 : t3));  // T_q
    double hi = q == 0 ? ta : (q == 1 ? t3 : (q == 2 ? t2 : x));   // T_{4-q}
#pragma unroll
    for (int a = 4; a < LP; a *= 2) {  // lo = T_{r mod 2a}, hi = T_{2a - r mod 2a}
        const bool up = (r & a) != 0;
        const double v = fma(2.0 * ta, up ? lo : hi, -(up ? hi : lo));
        lo = up ? v : lo;
        hi = up ? hi : v;
        ta = fma(2.0 * ta, ta, -1.0);
    }
    t[0] = lo;
    m[0] = hi;
#pragma unroll
    for (int a = 1; a < V; a *= 2) {
        const double two = 2.0 * ta;
#pragma unroll
        for (int v = a; v < 2 * a; ++v) {
            t[v] = fma(two, t[v - a], -m[2 * a - 1 - v]);
            m[v] = fma(two, m[v - a], -t[2 * a - 1 - v]);
        }
        ta = fma(two, ta, -1.0);
    }
    return ta;
}

// Butterfly sum of the 32 virtual lanes' values, p[v] the lane's own; the first step's
// products are never contracted into an FMA.
template <int LP>
__device__ __forceinline__ double group_sum(double (&p)[32 / LP]) {
#pragma unroll
    for (int h = 16 / LP; h > 0; h /= 2)
#pragma unroll
        for (int v = 0; v < h; ++v) p[v] = __dadd_rn(p[v], p[v + h]);
    double s = p[0];
#pragma unroll
    for (int o = LP / 2; o > 0; o >>= 1) s += __shfl_xor_sync(kFull, s, o);
    return s;
}

// Coefficients of the global x-sum series held by a lane, loaded once per pair.
template <int C, int LP>
struct PairCoef {
    double c[Lay<C>::NX][32 / LP][kCoefPerLane];
};
template <int C, int LP>
__device__ __forceinline__ void load_pair_coef(const Params& p, int64_t j, int f, int r,
                                               PairCoef<C, LP>& g) {
    const int64_t cp = C + p.phi;
#pragma unroll
    for (int v = 0; v < 32 / LP; ++v) {
#pragma unroll
        for (int i = 0; i < kCoefPerLane; ++i) {
            const int64_t row = 1 + r + LP * v + 32 * i;
            const double* rl = p.CL + j * p.ldcl + row * cp;
#pragma unroll
            for (int a = 0; a < C; ++a) g.c[a][v][i] = __ldg(rl + a);
            g.c[C][v][i] = __ldg(p.CQ + j * p.ldcq + row);
            g.c[C + 1][v][i] = __ldg(rl + C + f);
        }
    }
}

// The c+2 x-dependent sums at log-lambda s; identical bits in every lane of the group.
template <int C, int LP>
__device__ __forceinline__ void series_xsums(const Params& p, const PairCoef<C, LP>& g, double s,
                                             int r, double (&xs)[Lay<C>::NX]) {
    constexpr int V = 32 / LP;
    double t[V], m[V];
    const double t32 = cheb_group<LP>((s - p.gmid) * p.ginv, r, t, m);
    const double two = 2.0 * t32;
    double w[Lay<C>::NX][V];
#pragma unroll
    for (int v = 0; v < V; ++v) {
        const double t1 = fma(two, t[v], -m[V - 1 - v]);  // T_{l+32}, from T_{32-l}
        const double t2 = fma(two, t1, -t[v]);            // T_{l+64}
#pragma unroll
        for (int q = 0; q < Lay<C>::NX; ++q) {
            double u = __dmul_rn(g.c[q][v][0], t[v]);
            u = fma(g.c[q][v][1], t1, u);
            w[q][v] = fma(g.c[q][v][2], t2, u);
        }
    }
#pragma unroll
    for (int q = 0; q < Lay<C>::NX; ++q) xs[q] = group_sum<LP>(w[q]);
}

// The same sums at grid point k, its Chebyshev values from the table p.tgrid.
template <int C, int LP>
__device__ __forceinline__ void grid_xsums(const Params& p, const PairCoef<C, LP>& g, int k, int r,
                                           double (&xs)[Lay<C>::NX]) {
    constexpr int V = 32 / LP;
    const double* __restrict__ tg = p.tgrid + (int64_t)k * kChebG + r;
    double w[Lay<C>::NX][V];
#pragma unroll
    for (int v = 0; v < V; ++v) {
        const double t0 = __ldg(tg + LP * v), t1 = __ldg(tg + LP * v + 32), t2 = __ldg(tg + LP * v + 64);
#pragma unroll
        for (int q = 0; q < Lay<C>::NX; ++q)
            w[q][v] = fma(g.c[q][v][2], t2, fma(g.c[q][v][1], t1, __dmul_rn(g.c[q][v][0], t0)));
    }
#pragma unroll
    for (int q = 0; q < Lay<C>::NX; ++q) xs[q] = group_sum<LP>(w[q]);
}

// The same sums at four grid points k0 .. k0 + 3 at once, for groups of 16 or 32 lanes: each of
// the first two steps of the butterfly halves the points that a lane goes on with, so that four
// sums take 6 shuffles (32 lanes) in place of 20 (the grid was most of what one warp issues for
// a pair).  Lane r is left with point k0 + r / (LP / 4).  The additions are those of group_sum,
// bit for bit.
template <int C, int LP>
__device__ __forceinline__ void grid_xsums4(const Params& p, const PairCoef<C, LP>& g, int k0, int r,
                                            double (&xs)[Lay<C>::NX]) {
    constexpr int V = 32 / LP;
    static_assert(LP >= 16, "two steps of the butterfly between lanes");
    double w[Lay<C>::NX][4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const int k = k0 + e < p.n_grid ? k0 + e : p.n_grid - 1;
        const double* __restrict__ tg = p.tgrid + (int64_t)k * kChebG + r;
        double t[V][3];
#pragma unroll
        for (int v = 0; v < V; ++v)
#pragma unroll
            for (int i = 0; i < 3; ++i) t[v][i] = __ldg(tg + LP * v + 32 * i);
#pragma unroll
        for (int q = 0; q < Lay<C>::NX; ++q) {
            double u[V];
#pragma unroll
            for (int v = 0; v < V; ++v)
                u[v] = fma(g.c[q][v][2], t[v][2], fma(g.c[q][v][1], t[v][1],
                                                      __dmul_rn(g.c[q][v][0], t[v][0])));
            w[q][e] = V == 2 ? __dadd_rn(u[0], u[V - 1]) : u[0];
        }
    }
    const bool up1 = (r & (LP / 2)) != 0, up2 = (r & (LP / 4)) != 0;
#pragma unroll
    for (int q = 0; q < Lay<C>::NX; ++q) {
        double h[2];
#pragma unroll
        for (int e = 0; e < 2; ++e)
            h[e] = (up1 ? w[q][2 + e] : w[q][e]) +
                   __shfl_xor_sync(kFull, up1 ? w[q][e] : w[q][2 + e], LP / 2);
        double s = (up2 ? h[1] : h[0]) + __shfl_xor_sync(kFull, up2 ? h[0] : h[1], LP / 4);
#pragma unroll
        for (int o = LP / 8; o > 0; o >>= 1) s += __shfl_xor_sync(kFull, s, o);
        xs[q] = s;
    }
}

// log|H^-1| and the x-free sums of phenotype f at log-lambda s, from the expansions over the
// golden bracket of grid index `best` (degree 24, coefficients in virtual lanes 0..24).  With
// 16 or 32 lanes a pair's coefficients stay in registers; fewer lanes have none left and read them
// (through L1) at every probe.
template <int C, int LP>
struct Bracket {
    static constexpr int V = 32 / LP;
    static constexpr bool kHold = LP >= 16;
    double mid, inv_half;
    const double* __restrict__ cb;  // of this lane
    double c[kHold ? 1 + Lay<C>::NS : 1][V];
    __device__ __forceinline__ double coef(const Params& p, int f, int k, int v, int r) const {
        const bool in = LP * v + LP <= kChebN || r + LP * v < kChebN;
        const double* __restrict__ ck = cb + (k < 0 ? 0 : (int64_t)(1 + f * Lay<C>::NS + k) * kChebN);
        return LP * v < kChebN && in ? __ldg(ck + LP * v) : 0.0;
    }
    __device__ __forceinline__ void load(const Params& p, int best, int f, int r) {
        cb = p.cheb + (int64_t)best * (1 + (int64_t)p.phi * Lay<C>::NS) * kChebN + r;
        mid = __ldg(p.cheb_mid + best);
        inv_half = 1.0 / __ldg(p.cheb_half + best);
        if constexpr (kHold) {
#pragma unroll
            for (int k = -1; k < Lay<C>::NS; ++k)
#pragma unroll
                for (int v = 0; v < V; ++v) c[1 + k][v] = coef(p, f, k, v, r);
        }
    }
    __device__ __forceinline__ void sums(const Params& p, int f, double s, int r, double& logdet,
                                         double (&shared)[Lay<C>::NS]) const {
        double t[V], m[V];
        cheb_group<LP>((s - mid) * inv_half, r, t, m);
#pragma unroll
        for (int k = -1; k < Lay<C>::NS; ++k) {
            double w[V];
#pragma unroll
            for (int v = 0; v < V; ++v) {
                if constexpr (kHold)
                    w[v] = __dmul_rn(c[1 + k][v], t[v]);
                else
                    w[v] = __dmul_rn(coef(p, f, k, v, r), t[v]);
            }
            const double v = group_sum<LP>(w);
            if (k < 0)
                logdet = v;
            else
                shared[k] = v;
        }
    }
};

// REML and MLE log-likelihoods of one Pab result with the logarithms shared out: lane i <= C
// takes log of pivot i, lane C + 1 the one of P_yy; the sums are those of reml_logl / mle_logl.
template <int C, int LP>
__device__ __forceinline__ double group_reml(const PabOut<C>& pb, const double (&log_iab)[C + 1],
                                             double logdet_h, const Params& p, int r) {
    const double pyy = clamp_pyy(pb.yy1);
    double arg = pyy;
#pragma unroll
    for (int i = 0; i <= C; ++i) arg = r == i ? pb.diag[i] : arg;
    double lg = log(arg);
    if (r <= C && !(arg > 0)) lg = 0.0;
    double ldw = 0.0;
#pragma unroll
    for (int i = 0; i <= C; ++i) {
        ldw = __dadd_rn(ldw, __shfl_sync(kFull, lg, i, LP));
        ldw = __dsub_rn(ldw, log_iab[i]);
    }
    const double lpyy = __shfl_sync(kFull, lg, C + 1, LP);
    double f = __dsub_rn(p.c_reml, __dmul_rn(0.5, logdet_h));
    f = __dsub_rn(f, __dmul_rn(0.5, ldw));
    return __dsub_rn(f, __dmul_rn(__dmul_rn(0.5, p.df), lpyy));
}

// A golden section as the plain form's search leaves it (see lmm_open_kernel): bracket [a, b]
// before decision `step`, and the log-lambdas sc < sd of its two inner values.  step =
// n_iter: every decision is taken; step = -1: none, not even the grid's.
struct SearchState {
    double a, b, sc, sd, step;
};

// Where a search of the plain form reports: its state, and the list of searches left open.
struct SearchReport {
    SearchState* state = nullptr;  // null: this lane does not report
    int64_t id = 0;
    int64_t* list = nullptr;
    unsigned long long* count = nullptr;
    __device__ __forceinline__ void put(const SearchState& st, bool open) const {
        if (!state) return;
        *state = st;
        if (open) list[atomicAdd(count, 1ull)] = id;
    }
};

// One golden section (_golden_section_refine, likelihood_jax.py:419-488) as a sequence of
// probes: c, d, then one per step; probe number n_iter + 2 is the optimum (a + b) / 2.
// GUIDE: the probes are approximations of direct evaluations, their differences certain to
// GuideTau.  The first decision between values closer than that (or NaN) is left open: the
// state before it is reported, and the steps after it are without effect.
struct GuideTau {
    double whole;  // error of a probe's value
    double slope;  // of a difference, per unit of log-lambda between the probes
    double floor;  // the part that does not shrink with that distance (rounding)
    __device__ __forceinline__ double of(double dist) const {
        return floor + fmin(whole, slope * dist);
    }
};

template <bool GUIDE>
struct Golden {
    double a, b, c, d, fc, fd, s;  // s: the next probe
    bool left;                     // it replaces c (fc), else d (fd)
    double sc, sd;                 // GUIDE: where fc and fd were evaluated
    GuideTau tau;
    bool certain;
    __device__ __forceinline__ void start(const Params& p, int best) {
        const int lo = best - 1 > 0 ? best - 1 : 0;
        const int hi = best + 1 < p.n_grid - 1 ? best + 1 : p.n_grid - 1;
        a = p.loglam[lo];
        b = p.loglam[hi];
        inner();
        fc = fd = 0.0;
        s = c;
        left = true;
        sc = sd = 0.0;
        certain = true;
    }
    __device__ __forceinline__ void inner() {
        c = __dsub_rn(b, __dmul_rn(kPhi, __dsub_rn(b, a)));
        d = __dadd_rn(a, __dmul_rn(kPhi, __dsub_rn(b, a)));
    }
    // takes the value at probe `it` and sets the next one
    __device__ __forceinline__ void take(double f, int it, int n_iter, const SearchReport& out) {
        fc = left ? f : fc;
        fd = left ? fd : f;
        if (GUIDE) {
            sc = left ? s : sc;
            sd = left ? sd : s;
        }
        if (it == 0) {
            s = d;
            left = false;
            return;
        }
        if (it > n_iter) {
            s = __dmul_rn(__dadd_rn(a, b), 0.5);
            if (GUIDE && certain) out.put(SearchState{a, b, sc, sd, (double)n_iter}, false);
            return;
        }
        if (GUIDE && certain && !(fabs(fc - fd) > tau.of(fabs(sd - sc)))) {
            certain = false;
            out.put(SearchState{a, b, sc, sd, (double)(it - 1)}, true);
        }
        left = fc > fd;
        a = left ? a : c;
        b = left ? d : b;
        const double keep = left ? fc : fd;
        fc = keep;  // the one that the next probe replaces is overwritten
        fd = keep;
        if (GUIDE) {
            const double at = left ? sc : sd;
            sc = at;
            sd = at;
        }
        inner();
        s = left ? c : d;
    }
};

// GUIDE: how far a series log-likelihood can be from its direct evaluation, to first order.
// Two kinds of error enter the sums:
//   * the truncated series: every weight 1/(lambda e + 1) is off by at most kSeriesEps at any
//     log-lambda of the domain and any eigenvalue (the largest error over eigenvalues from
//     -5e-6 to 1e9 is 7.3e-12, at eigenvalues near 1), so a sum of x z terms is off by at most
//     kSeriesEps |x| |z|, with the unweighted norms: these stay what they are where the
//     weights have shrunk the sums themselves (to 1e-5 of their size at lambda = 1e5);
//   * rounding: `kappa` of the size of a sum's terms, weighted in the direct evaluations and
//     in the x-free expansions, unweighted for a series.
// Both are carried through the elimination of the covariates, whichever of them the sums
// cancel against: G holds the weighted products of the residuals, U their unweighted ones, q
// and q1 the sizes of the terms that make up a residual's square.  With x_r, y_r the residuals
// at level c and b = P_xy / P_xx,
//   |dP_xx| <= eps (|x_r|^2 + (|x| + |x_r|)^2) <= eps (3 |x_r|^2 + 2 |x|^2),
//   |dP_xy| <= eps |x| |y_r|,   |dP_yy'| <= 2 |b| |dP_xy| + b^2 |dP_xx|,
// and the log-likelihoods change by half of dP_xx / P_xx (REML) and n / 2 of dP_yy' / P_yy'.
// `whole` is the series' part, `floor` the rounding.  Compared with direct evaluations in
// double and in 80 bits, differences of probes stay below 0.15 of the bound that GuideTau
// makes of it (n = 400 to 4000, one to four covariate columns, spread and centred-kinship
// spectra, where the intercept keeps its weight at every lambda while all else shrinks, h2 = 0
// to 1, allele frequencies 0.01 to 0.99, phenotypes and covariates 0 to 100 standard
// deviations off zero).
constexpr double kSeriesEps = 1e-11;
struct GuideErr {
    double whole_mle, floor_mle, whole_reml, floor_reml;
};
template <int C>
__device__ __forceinline__ GuideErr guide_err(const Params& p, const double (&row0)[Lay<C>::NI],
                                              int64_t j, int f, double ldh) {
    using L = Lay<C>;
    constexpr int R = L::R;
    const double inf = __longlong_as_double(0x7ff0000000000000ll);
    const double kappa = 2.2e-16 * (4.0 + sqrt(p.n_d / 32.0));
    double G[L::NI], U[L::NI], xs[L::NX], q[R], q1[R];
    const double* cl = p.CL + j * p.ldcl;
#pragma unroll
    for (int a = 0; a < C; ++a) xs[a] = __ldg(cl + a);
    xs[C] = __ldg(p.CQ + j * p.ldcq);
    xs[C + 1] = __ldg(cl + C + f);
    assemble<C>(U, p.S + ((int64_t)p.n_grid * p.phi + f) * L::NS, xs);
    const double x1 = xs[C];  // |x|^2
#pragma unroll
    for (int k = 0; k < L::NI; ++k) G[k] = row0[k];
#pragma unroll
    for (int a = 0; a < R; ++a) {
        q[a] = fabs(G[L::idx(a, a)]);
        q1[a] = U[L::idx(a, a)];
    }
    double piv = 0.0;
    bool ok = true;
#pragma unroll
    for (int w = 0; w < C; ++w) {
        const double ww = G[L::idx(w, w)], inv = 1.0 / ww, uw = U[L::idx(w, w)];
        ok = ok && ww > 0.0;
        piv = fma(q[w], inv, piv);
        double l[R];
#pragma unroll
        for (int a = w + 1; a < R; ++a) l[a] = G[L::idx(a, w)] * inv;
#pragma unroll
        for (int a = w + 1; a < R; ++a) {
            q[a] = fma(l[a] * l[a], q[w], q[a]);
            q1[a] = fma(l[a] * l[a], q1[w], q1[a]);
#pragma unroll
            for (int b = a; b < R; ++b) {
                G[L::idx(a, b)] = fma(-l[a], G[L::idx(b, w)], G[L::idx(a, b)]);
                U[L::idx(a, b)] = fma(-l[a], U[L::idx(b, w)], fma(-l[b], fma(-l[a], uw, U[L::idx(a, w)]),
                                                                 U[L::idx(a, b)]));
            }
        }
    }
    const bool none = x1 == 0.0;  // a genotype of zeros: its sums are exact
    const double xx = none ? 1.0 : G[L::idx(C, C)], ix = 1.0 / xx;
    const double b = fabs(G[L::idx(C, C + 1)]) * ix;
    const double yy1 = fma(-b * b, xx, G[L::idx(C + 1, C + 1)]), ny = 0.5 * p.n_d / yy1;
    const double xr = fmax(U[L::idx(C, C)], 0.0) + kappa * q1[C];
    const double yr = fmax(U[L::idx(C + 1, C + 1)], 0.0) + kappa * q1[C + 1];
    const double exx = kSeriesEps * (3.0 * xr + 2.0 * x1), exy = kSeriesEps * sqrt(x1 * yr);
    const double fxx = kappa * sqrt(x1 * q1[C]), fxy = kappa * sqrt(x1 * q1[C + 1]);
    GuideErr e;
    e.whole_mle = ny * b * (2.0 * exy + b * exx);
    e.floor_mle = ny * (kappa * (q[C + 1] + b * b * q[C]) + b * (2.0 * fxy + b * fxx)) +
                  kappa * (p.n_d + fabs(ldh));
    e.whole_reml = e.whole_mle + 0.5 * exx * ix;
    e.floor_reml = e.floor_mle + 0.5 * (kappa * piv + fxx * ix);
    // first order needs errors well below what they are errors of
    if (!(ok && xx > 0.0 && yy1 > 0.0 && exx + fxx < 0.25 * xx)) e = GuideErr{inf, inf, inf, inf};
    return e;
}

// The bound over the golden bracket of grid index `best`, from the two at that point: across
// the bracket every weighted sum shrinks by at most exp(d), d the distance to its far end, so
// `whole` (through P_xx and P_yy') grows by at most exp(2 d) and `floor` by exp(d); both
// twice, for a difference of two probes.  The series' error is a combination of terms of degree
// 96 and up, so between close probes it cancels: its slope is at most 96 / 11.5 per unit of
// log-lambda within 0.95 of the domain (8.4 of the largest error, 68 at the ends, over the
// eigenvalues above), and 1 and 2 more for P_xx and P_yy' in the denominators.
__device__ __forceinline__ GuideTau guide_tau(const Params& p, int best, double whole, double floor) {
    const double s = p.loglam[best];
    const int lo = best - 1 > 0 ? best - 1 : 0;
    const int hi = best + 1 < p.n_grid - 1 ? best + 1 : p.n_grid - 1;
    const double d = fmax(p.loglam[hi] - s, s - p.loglam[lo]), f = exp(d);
    const double w = 2.0 * whole * f * f;
    return GuideTau{w, w * ((fabs(s - p.gmid) + d) * p.ginv < 0.95 ? 12.0 : 72.0), 2.0 * floor * f};
}

// Maximum of the grid's values, with the largest value that another point can have: each
// value comes with its error bound (the same at no two points: it grows with lambda).
struct ArgMaxLead {
    int idx = -1;
    double v = 0.0, e = 0.0, other = -INFINITY;
    bool nan = false;
    __device__ __forceinline__ void push(int i, double x, double err) {
        nan = nan || isnan(x + err) || isnan(x - err);
        if (idx >= 0) other = fmax(other, x > v ? v + e : x + err);
        if (idx < 0 || x > v) {
            idx = i;
            v = x;
            e = err;
        }
    }
    // the point is the one that exact values would give
    __device__ __forceinline__ bool certain() const { return !nan && v - e > other; }
    template <int GW>
    __device__ __forceinline__ void warp_reduce() {  // over groups of GW lanes
#pragma unroll
        for (int o = GW / 2; o > 0; o >>= 1) {
            const int oi = __shfl_xor_sync(kFull, idx, o);
            const double ov = __shfl_xor_sync(kFull, v, o), oe = __shfl_xor_sync(kFull, e, o);
            const double oo = __shfl_xor_sync(kFull, other, o);
            nan = __shfl_xor_sync(kFull, (int)nan, o) != 0 || nan;
            if (oi < 0) continue;
            const bool take = idx < 0 || ov > v || (ov == v && oi < idx);
            if (idx >= 0) other = fmax(other, take ? v + e : ov + oe);
            other = fmax(other, oo);
            v = take ? ov : v;
            e = take ? oe : e;
            idx = take ? oi : idx;
        }
    }
};

// What a kernel searches: by the mode, or one likelihood only.  The latter, for chunks that
// cannot fill the GPU, keeps the other search's state out of the registers.  With it and
// grid_xsums4, 200 pairs of the mixed form's likelihood-ratio test, one to four columns: 35.4,
// 40.6, 44.8, 69.6 -> 32.2, 33.0, 35.4, 41.1 us.
constexpr int kByMode = 0, kMleOnly = 1, kRemlOnly = 2;

// GUIDE = false: the mixed form, search and statistics.  GUIDE = true: the plain form's
// decisions, as far as they are certain (modes 1, 2 and 4); lmm_open_kernel and
// lmm_finish_kernel take over.
template <int C, int LP, bool GUIDE, int SEARCHES>
__global__ void __launch_bounds__(kSearchThreads, 2) lmm_search_kernel(const Params p) {
    using L = Lay<C>;
    const int64_t npairs = p.m * p.phi;
    const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if ((tid & ~31ll) / LP >= npairs) return;  // the whole warp is idle
    // a group past the last pair repeats the last pair and writes nothing
    const bool valid_pair = tid / LP < npairs;
    const int64_t wid = valid_pair ? tid / LP : npairs - 1;
    const int r = threadIdx.x & (LP - 1);
    const int64_t j = wid / p.phi;
    const int f = (int)(wid % p.phi);
    const bool need_reml = SEARCHES == kByMode ? p.mode == 1 || p.mode == 4 : SEARCHES == kRemlOnly;
    const bool need_mle = SEARCHES == kByMode ? p.mode == 2 || p.mode == 4 : SEARCHES == kMleOnly;
    const bool need_score = !GUIDE && SEARCHES == kByMode && (p.mode == 3 || p.mode == 4);
    const int64_t o = (int64_t)f * p.m + j;
    const int64_t srow = (int64_t)p.phi * L::NS;  // stride of one S row
    const bool writer = r == 0 && valid_pair;

    PairCoef<C, LP> g;
    load_pair_coef<C, LP>(p, j, f, r, g);

    // ---------------- H = 1 (Iab) and H = H0 (score)
    double log_iab[C + 1];
#pragma unroll
    for (int i = 0; i <= C; ++i) log_iab[i] = 0.0;
    if (need_reml) {
        double xs[L::NX], row0[L::NI];
        const double* cl = p.CL + j * p.ldcl;
#pragma unroll
        for (int a = 0; a < C; ++a) xs[a] = cl[a];
        xs[C] = p.CQ[j * p.ldcq];
        xs[C + 1] = cl[C + f];
        assemble<C>(row0, p.S + (int64_t)p.n_grid * srow + (int64_t)f * L::NS, xs);
        const PabOut<C> pb = pab_reduce<C>(row0);
#pragma unroll
        for (int i = 0; i <= C; ++i) log_iab[i] = pb.diag[i] > 0 ? log(pb.diag[i]) : 0.0;
    }
    if (need_score) {
        double xs[L::NX], row0[L::NI];
        series_xsums<C, LP>(p, g, log(p.lam0[f]), r, xs);
        assemble<C>(row0, p.S + (int64_t)(p.n_grid + 1 + f) * srow + (int64_t)f * L::NS, xs);
        const PabOut<C> pb = pab_reduce<C>(row0);
        bool valid;
        double beta, tau, se;
        beta_se<C>(pb, clamp_pyy(pb.yy1), p.df, valid, beta, tau, se);
        const double fstat = p.n_d * (pb.xy * pb.xy) / (pb.yy * (valid ? pb.xx : 1.0));
        if (writer) {
            // the F statistic (NaN: no test); lmm_fpvalue_kernel turns it into the p-value
            if (p.out.p_score) p.out.p_score[o] = valid ? fstat : jnan();
            if (p.mode == 3) {
                if (p.out.beta) p.out.beta[o] = beta;
                if (p.out.se) p.out.se[o] = se;
            }
        }
    }
    if (!GUIDE && !need_reml && !need_mle) {  // score only: the large-lambda rewrite
        double xs_m[L::NX], xs_r[L::NX];
        direct_fix<C, LP>(p, j, f, valid_pair, need_score, false, false, 0.0, 0.0, xs_m, xs_r);
        return;
    }

    // ---------------- shared lambda grid, LP points at a time
    std::conditional_t<GUIDE, ArgMaxLead, ArgMax> best_reml, best_mle;
#pragma unroll 1
    for (int g0 = 0; g0 < p.n_grid; g0 += LP) {
        double xs[L::NX];
        int k = g0 + r;
        if constexpr (LP >= 16) {
            // few pairs, so that the instructions of one warp set the time: four points at once
            constexpr int kPasses = LP / 4;
            const int mine = r & (kPasses - 1);
            k = g0 + 4 * mine + r / kPasses;
#pragma unroll 1
            for (int e = 0; e < kPasses; ++e) {
                if (e > 0 && g0 + 4 * e >= p.n_grid) break;
                double xe[L::NX];
                grid_xsums4<C, LP>(p, g, g0 + 4 * e, r, xe);
#pragma unroll
                for (int q = 0; q < L::NX; ++q) xs[q] = e == mine || e == 0 ? xe[q] : xs[q];
            }
        } else {
#pragma unroll 1
            for (int e = 0; e < LP; ++e) {
                double xe[L::NX];
                grid_xsums<C, LP>(p, g, g0 + e < p.n_grid ? g0 + e : p.n_grid - 1, r, xe);
#pragma unroll
                for (int q = 0; q < L::NX; ++q) xs[q] = e == r || e == 0 ? xe[q] : xs[q];
            }
        }
        if (k < p.n_grid) {
            double row0[L::NI];
            assemble<C>(row0, p.S + (int64_t)k * srow + (int64_t)f * L::NS, xs);
            const PabOut<C> pb = pab_reduce<C>(row0);
            const double ldh = p.logdet[k];
            if constexpr (GUIDE) {
                const GuideErr er = guide_err<C>(p, row0, j, f, ldh);
                if (need_reml)
                    best_reml.push(k, reml_logl<C>(pb, log_iab, ldh, p),
                                   2.0 * (er.whole_reml + er.floor_reml));
                if (need_mle)
                    best_mle.push(k, mle_logl<C>(pb, ldh, p), 2.0 * (er.whole_mle + er.floor_mle));
            } else {
                if (need_reml) best_reml.push(k, reml_logl<C>(pb, log_iab, ldh, p));
                if (need_mle) best_mle.push(k, mle_logl<C>(pb, ldh, p));
            }
        }
    }
    best_reml.template warp_reduce<LP>();
    best_mle.template warp_reduce<LP>();

    // ---------------- golden sections, both searches in step
    const int bm = need_mle ? best_mle.idx : best_reml.idx;
    const int br = need_reml ? best_reml.idx : best_mle.idx;
    Golden<GUIDE> gm, gr;
    gm.start(p, bm);
    gr.start(p, br);
    Bracket<C, LP> km, kr;
    km.load(p, bm, f, r);
    kr.load(p, br, f, r);
    SearchReport out_m, out_r;
    if constexpr (GUIDE) {
        if (writer) {
            out_m = SearchReport{p.state + 2 * wid, 2 * wid, p.open_list, p.open_count};
            out_r = SearchReport{p.state + 2 * wid + 1, 2 * wid + 1, p.open_list, p.open_count};
        }
        auto err_at = [&](int at) {
            double xs[L::NX], row0[L::NI];
            grid_xsums<C, LP>(p, g, at, r, xs);
            assemble<C>(row0, p.S + (int64_t)at * srow + (int64_t)f * L::NS, xs);
            return guide_err<C>(p, row0, j, f, p.logdet[at]);
        };
        auto settle = [&](Golden<GUIDE>& gs, const ArgMaxLead& best, int at, double whole,
                          double floor, const SearchReport& out) {
            gs.tau = guide_tau(p, at, whole, floor);
            gs.certain = best.certain();
            if (!gs.certain) out.put(SearchState{0.0, 0.0, 0.0, 0.0, -1.0}, true);
        };
        GuideErr e = err_at(bm);
        if (need_mle) settle(gm, best_mle, bm, e.whole_mle, e.floor_mle, out_m);
        if (__any_sync(kFull, bm != br)) e = err_at(br);
        if (need_reml) settle(gr, best_reml, br, e.whole_reml, e.floor_reml, out_r);
    }
    double xs_m[L::NX], xs_r[L::NX], sh_m[L::NS], sh_r[L::NS], ld_m = 0.0, ld_r = 0.0;
    PabOut<C> pb_m, pb_r;
#pragma unroll 1
    for (int it = 0;; ++it) {
        if (need_mle) {
            series_xsums<C, LP>(p, g, gm.s, r, xs_m);
            km.sums(p, f, gm.s, r, ld_m, sh_m);
        }
        if (need_reml) {
            if (!need_mle || __any_sync(kFull, gm.s != gr.s || bm != br)) {
                series_xsums<C, LP>(p, g, gr.s, r, xs_r);
                kr.sums(p, f, gr.s, r, ld_r, sh_r);
            } else {
#pragma unroll
                for (int q = 0; q < L::NX; ++q) xs_r[q] = xs_m[q];
#pragma unroll
                for (int q = 0; q < L::NS; ++q) sh_r[q] = sh_m[q];
                ld_r = ld_m;
            }
        }
        if (!GUIDE && it == p.n_iter + 2) break;
        double row0[L::NI];
        if (need_mle) {
            assemble<C>(row0, sh_m, xs_m);
            gm.take(mle_logl<C>(pab_reduce<C>(row0), ld_m, p), it, p.n_iter, out_m);
        }
        if (need_reml) {
            assemble<C>(row0, sh_r, xs_r);
            gr.take(group_reml<C, LP>(pab_reduce<C>(row0), log_iab, ld_r, p, r), it, p.n_iter, out_r);
        }
        if (GUIDE && it == p.n_iter + 1) return;
    }

    // ---------------- statistics at the optima; at large lambda from direct x-sums
    direct_fix<C, LP>(p, j, f, valid_pair, need_score, need_mle, need_reml, gm.s, gr.s, xs_m, xs_r);
    double row0[L::NI];
    if (need_mle) {
        assemble<C>(row0, sh_m, xs_m);
        const double logl = mle_logl<C>(pab_reduce<C>(row0), ld_m, p);
        if (writer) {
            if (p.out.lambda_mle) p.out.lambda_mle[o] = exp(gm.s);
            if (p.out.logl_mle) p.out.logl_mle[o] = logl;
            const double stat = jmax(2.0 * (logl - p.logl0[f]), 0.0);
            if (p.out.p_lrt) p.out.p_lrt[o] = chi2_1_sf(stat);
        }
    }
    if (need_reml) {
        assemble<C>(row0, sh_r, xs_r);
        const PabOut<C> pb = pab_reduce<C>(row0);
        write_wald<C>(p, pb, reml_logl<C>(pb, log_iab, ld_r, p), exp(gr.s), o, writer);
    }
}

// ---------------------------------------------------------------- plain form, guided
// The plain form's golden sections would take a direct FP64 pass over x per probe (46 passes
// with a logarithm and a reciprocal per sample and pair in mode 4), although nearly every
// decision is far from a tie.  So lmm_search_kernel<.., true> takes the decisions that its
// series approximations settle beyond their error (guide_err), lmm_open_kernel takes the few
// others by direct evaluations (lmm_close_kernel when they are many), and lmm_finish_kernel
// makes one direct pass per pair for the evaluations at the optima, whose sums the statistics
// use, and the score test.  All three form an evaluation's sums term by term in the order of
// eval_full, and the same values come out whichever kernel takes a search.  The decisions are
// those of a search of direct evaluations, but for two kinds that rounding settles: near-ties
// of grid points (lmm_pairs_kernel has their x-sums from a GEMM, in another order), and REML
// values closer than the rounding of their H = 1 determinant, whose sums (the chunk's ones row)
// come from GEMMs of different shapes.
// Measured, search of direct evaluations -> search + open + close + finish: 8192 SNPs, n =
// 1940, Wald 1976 -> 264 us; 2048 SNPs, three covariate columns, n = 10 000, every test 8294
// -> 796 us; 2048 SNPs, n = 20 000, every test 10 536 -> 832 us (and 0.4 ms more for the 97
// rows of series sums in place of 52 grid rows).  The gain shrinks where the likelihood is
// flat: lambda at its upper bound, n = 20 000: 19.7 -> 13 ms for 2000 SNPs x 2 phenotypes.

// One search by all threads of a CTA: tiles of kOpenTile samples staged in shared memory.
constexpr int kOpenThreads = 256, kOpenTile = 512;
template <int C>
struct OpenSmem {
    double col[Lay<C>::R][kOpenTile];  // W columns, x, y
    double h[kOpenTile], ld[kOpenTile];
    double sum[32];
};

// Log-likelihood at log-lambda s by all threads of the CTA, with eval_full's values: the
// weights and logarithms of a tile of samples are formed by all threads, then each warp adds
// up some of the NI + 1 sums over the tile as eval_full's one warp does.  The next tile's
// loads are in flight meanwhile.
template <int C, bool REML>
__device__ double block_logl(const Params& p, const double* __restrict__ x,
                             const double* __restrict__ y, double s,
                             const double (&log_iab)[C + 1], OpenSmem<C>& sm) {
    using L = Lay<C>;
    constexpr int kWarps = kOpenThreads / 32, kSlots = (L::NI + kWarps) / kWarps;
    constexpr int kPer = kOpenTile / kOpenThreads;  // samples of a tile per thread
    static_assert(L::NI + 1 <= 32, "sums of a pair");
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const double lam = exp(s);
    int ca[kSlots], cb[kSlots];  // this warp's sums: columns a <= b; log|H| is sum NI
    double acc[kSlots];
#pragma unroll
    for (int q = 0; q < kSlots; ++q) {
        acc[q] = 0.0;
        ca[q] = cb[q] = 0;
#pragma unroll
        for (int a = 0; a < L::R; ++a)
#pragma unroll
            for (int b = a; b < L::R; ++b)
                if (L::idx(a, b) == warp + q * kWarps) {
                    ca[q] = a;
                    cb[q] = b;
                }
    }
    double ev[kPer], col[kPer][L::R];
    auto fetch = [&](int64_t base) {
#pragma unroll
        for (int e = 0; e < kPer; ++e) {
            const int64_t i = base + threadIdx.x + e * kOpenThreads;
            if (i >= p.n) continue;
            ev[e] = __ldg(p.evals + i);
#pragma unroll
            for (int a = 0; a < C; ++a) col[e][a] = __ldg(p.W + a * p.ldw + i);
            col[e][C] = x[i];
            col[e][C + 1] = __ldg(y + i);
        }
    };
    fetch(0);
    for (int64_t base = 0; base < p.n; base += kOpenTile) {
        const int len = (int)(p.n - base < kOpenTile ? p.n - base : kOpenTile);
        __syncthreads();  // the previous tile (or call) has been read
#pragma unroll
        for (int e = 0; e < kPer; ++e) {
            const int i = threadIdx.x + e * kOpenThreads;
            if (i >= len) continue;
            const double v = __dadd_rn(__dmul_rn(lam, ev[e]), 1.0);
            sm.h[i] = __drcp_rn(v);
            sm.ld[i] = log(fabs(v));
#pragma unroll
            for (int a = 0; a < L::R; ++a) sm.col[a][i] = col[e][a];
        }
        __syncthreads();
        if (base + kOpenTile < p.n) fetch(base + kOpenTile);
#pragma unroll
        for (int q = 0; q < kSlots; ++q) {
            const int k = warp + q * kWarps;  // warp-uniform
            const double *pa = sm.col[ca[q]], *pb = sm.col[cb[q]];
            double t = acc[q];
            if (k < L::NI) {
#pragma unroll 8
                for (int i = lane; i < len; i += 32) t = fma(sm.h[i] * pa[i], pb[i], t);
            } else if (k == L::NI) {
#pragma unroll 8
                for (int i = lane; i < len; i += 32) t += sm.ld[i];
            }
            acc[q] = t;
        }
    }
#pragma unroll
    for (int q = 0; q < kSlots; ++q) {
        const double v = warp_sum(acc[q]);
        if (lane == 0 && warp + q * kWarps <= L::NI) sm.sum[warp + q * kWarps] = v;
    }
    __syncthreads();
    double row0[L::NI];
#pragma unroll
    for (int k = 0; k < L::NI; ++k) row0[k] = sm.sum[k];
    const PabOut<C> pb2 = pab_reduce<C>(row0);
    return REML ? reml_logl<C>(pb2, log_iab, sm.sum[L::NI], p) : mle_logl<C>(pb2, sm.sum[L::NI], p);
}

// Iab's logarithms of a pair (H = 1: the chunk's ones row).
template <int C>
__device__ __forceinline__ void pair_log_iab(const Params& p, int64_t j, int f,
                                             double (&log_iab)[C + 1]) {
    using L = Lay<C>;
    double xs[L::NX], row0[L::NI];
    const double* cl = p.CL + j * p.ldcl;
#pragma unroll
    for (int a = 0; a < C; ++a) xs[a] = cl[a];
    xs[C] = p.CQ[j * p.ldcq];
    xs[C + 1] = cl[C + f];
    assemble<C>(row0, p.S + ((int64_t)p.n_grid * p.phi + f) * L::NS, xs);
    const PabOut<C> pb = pab_reduce<C>(row0);
#pragma unroll
    for (int i = 0; i <= C; ++i) log_iab[i] = pb.diag[i] > 0 ? log(pb.diag[i]) : 0.0;
}

// Takes the open decisions of a search: `probe` evaluates a log-likelihood directly,
// `grid_best` picks the grid point.  Returns the optimum (a + b) / 2.
template <class Probe, class Grid>
__device__ __forceinline__ double close_golden(const Params& p, const SearchState& st, Probe probe,
                                               Grid grid_best) {
    double a = st.a, b = st.b, sc = st.sc, sd = st.sd;
    int it = (int)st.step;
    if (it < 0) {  // the grid as well
        const int best = grid_best();
        a = p.loglam[best - 1 > 0 ? best - 1 : 0];
        b = p.loglam[best + 1 < p.n_grid - 1 ? best + 1 : p.n_grid - 1];
        sc = __dsub_rn(b, __dmul_rn(kPhi, __dsub_rn(b, a)));
        sd = __dadd_rn(a, __dmul_rn(kPhi, __dsub_rn(b, a)));
        it = 0;
    }
    if (it < p.n_iter) {
        double c = __dsub_rn(b, __dmul_rn(kPhi, __dsub_rn(b, a)));
        double d = __dadd_rn(a, __dmul_rn(kPhi, __dsub_rn(b, a)));
        double fc = 0.0, fd = 0.0, s = sc;
        bool left = true;
        for (int e = 0;; ++e) {  // one copy of the evaluation: both inner values, then the steps
            const double f = probe(s);
            fc = left ? f : fc;
            fd = left ? fd : f;
            if (e == 0) {
                s = sd;
                left = false;
                continue;
            }
            left = fc > fd;
            a = left ? a : c;
            b = left ? d : b;
            if (++it == p.n_iter) break;
            const double keep = left ? fc : fd;
            fc = keep;
            fd = keep;
            c = __dsub_rn(b, __dmul_rn(kPhi, __dsub_rn(b, a)));
            d = __dadd_rn(a, __dmul_rn(kPhi, __dsub_rn(b, a)));
            s = left ? c : d;
        }
    }
    return __dmul_rn(__dadd_rn(a, b), 0.5);
}

// The best of a warp's share of the grid points (groups of kRun, one in `warps` from `warp` on)
// for a search whose grid decision is open, from the tabulated H rows.  A point's x-sums are
// added up by one warp in one order, whichever kernel takes the search and however many warps
// share the points.
template <int C, bool REML>
__device__ __forceinline__ ArgMax direct_grid(const Params& p, const double* __restrict__ x,
                                              const double* __restrict__ y, int f,
                                              const double (&log_iab)[C + 1], int warp, int warps) {
    using L = Lay<C>;
    constexpr int kRun = 4;
    ArgMax best;
#pragma unroll 1
    for (int g0 = kRun * warp; g0 < p.n_grid; g0 += kRun * warps) {
        double acc[kRun][L::NX];
#pragma unroll
        for (int e = 0; e < kRun; ++e)
#pragma unroll
            for (int q = 0; q < L::NX; ++q) acc[e][q] = 0.0;
        for (int64_t i = threadIdx.x & 31; i < p.n; i += 32) {
            const double xv = x[i], yv = __ldg(y + i);
            double w[C];
#pragma unroll
            for (int q = 0; q < C; ++q) w[q] = __ldg(p.W + q * p.ldw + i);
#pragma unroll
            for (int e = 0; e < kRun; ++e) {
                const int g = g0 + e < p.n_grid ? g0 + e : p.n_grid - 1;
                const double t = __ldg(p.H + (int64_t)g * p.n + i) * xv;
#pragma unroll
                for (int q = 0; q < C; ++q) acc[e][q] = fma(t, w[q], acc[e][q]);
                acc[e][C] = fma(t, xv, acc[e][C]);
                acc[e][C + 1] = fma(t, yv, acc[e][C + 1]);
            }
        }
#pragma unroll
        for (int e = 0; e < kRun; ++e) {
            double xs[L::NX], row0[L::NI];
#pragma unroll
            for (int q = 0; q < L::NX; ++q) xs[q] = warp_sum(acc[e][q]);
            if (g0 + e >= p.n_grid) continue;
            assemble<C>(row0, p.S + ((int64_t)(g0 + e) * p.phi + f) * L::NS, xs);
            const PabOut<C> pb = pab_reduce<C>(row0);
            const double ldh = p.logdet[g0 + e];
            best.push(g0 + e, REML ? reml_logl<C>(pb, log_iab, ldh, p) : mle_logl<C>(pb, ldh, p));
        }
    }
    return best;
}

// The same over all warps of a CTA.
template <int C, bool REML>
__device__ __forceinline__ int block_grid(const Params& p, const double* __restrict__ x,
                                          const double* __restrict__ y, int f,
                                          const double (&log_iab)[C + 1], OpenSmem<C>& sm) {
    constexpr int kWarps = kOpenThreads / 32;
    const int warp = threadIdx.x >> 5;
    ArgMax best = direct_grid<C, REML>(p, x, y, f, log_iab, warp, kWarps);
    if ((threadIdx.x & 31) == 0) {
        sm.sum[warp] = best.v;
        sm.sum[kWarps + warp] = best.idx;
    }
    __syncthreads();
    for (int w = 0; w < kWarps; ++w) best.merge((int)sm.sum[kWarps + w], sm.sum[w]);
    return best.idx;  // sum is next written after barriers of block_logl
}

// Few open searches (the usual chunk: a fraction of a percent): one CTA takes one at a time,
// so that they do not make a long tail of one warp each.  With more of them than
// kOpenPerSm per SM the CTAs' synchronisation costs more than it saves, and lmm_close_kernel
// takes them, one warp each.
constexpr int kOpenPerSm = 4;

template <int C, bool REML>
__device__ __noinline__ double open_search(const Params& p, int64_t wid, OpenSmem<C>& sm) {
    const int64_t j = wid / p.phi;
    const int f = (int)(wid % p.phi);
    const double* __restrict__ x = p.G + j * p.ldg;
    const double* __restrict__ y = p.Y + (int64_t)f * p.ldy;
    double log_iab[C + 1];
#pragma unroll
    for (int i = 0; i <= C; ++i) log_iab[i] = 0.0;
    if (REML) pair_log_iab<C>(p, j, f, log_iab);
    return close_golden(
        p, p.state[2 * wid + (REML ? 1 : 0)],
        [&](double s) { return block_logl<C, REML>(p, x, y, s, log_iab, sm); },
        [&] { return block_grid<C, REML>(p, x, y, f, log_iab, sm); });
}

template <int C>
__global__ void __launch_bounds__(kOpenThreads, 1) lmm_open_kernel(const Params p, int64_t most) {
    __shared__ OpenSmem<C> sm;
    const int64_t count = *p.open_count;
    if (count > most) return;
    for (int64_t e = blockIdx.x; e < count; e += gridDim.x) {
        const int64_t at = p.open_list[e];  // 2 pair + (1: REML)
        const double s = at & 1 ? open_search<C, true>(p, at >> 1, sm)
                                : open_search<C, false>(p, at >> 1, sm);
        __syncthreads();  // every thread has read the state
        if (threadIdx.x == 0) p.state[at] = SearchState{s, s, s, s, (double)p.n_iter};
    }
}

template <int C, bool REML>
__device__ __noinline__ double close_search(const Params& p, int64_t wid) {
    const int64_t j = wid / p.phi;
    const int f = (int)(wid % p.phi);
    const double* __restrict__ x = p.G + j * p.ldg;
    const double* __restrict__ y = p.Y + (int64_t)f * p.ldy;
    double log_iab[C + 1];
#pragma unroll
    for (int i = 0; i <= C; ++i) log_iab[i] = 0.0;
    if (REML) pair_log_iab<C>(p, j, f, log_iab);
    return close_golden(
        p, p.state[2 * wid + (REML ? 1 : 0)],
        [&](double s) { return eval_logl<C, REML>(p, x, y, s, log_iab, nullptr); },
        [&] { return direct_grid<C, REML>(p, x, y, f, log_iab, 0, 1).idx; });
}

template <int C>
__global__ void __launch_bounds__(kPairsThreads, PairsOccupancy<C>::kMinBlocks)
    lmm_close_kernel(const Params p, int64_t most) {
    const int64_t count = *p.open_count;
    if (count <= most) return;
    const int64_t nw = (int64_t)gridDim.x * kPairsThreads / 32;
    for (int64_t e = ((int64_t)blockIdx.x * kPairsThreads + threadIdx.x) / 32; e < count; e += nw) {
        const int64_t at = p.open_list[e];
        const double s = at & 1 ? close_search<C, true>(p, at >> 1) : close_search<C, false>(p, at >> 1);
        __syncwarp();  // every lane has read the state
        if ((threadIdx.x & 31) == 0) p.state[at] = SearchState{s, s, s, s, (double)p.n_iter};
    }
}

// One pass over x per pair, one warp each: the sums at the MLE and REML optima and the score
// test's sums at the null lambda (its H row is tabulated).  Bound by FP64 issue: a logarithm,
// a reciprocal and, with one covariate column, 9 multiply-adds per sample and optimum.
template <int C>
__global__ void __launch_bounds__(kPairsThreads, PairsOccupancy<C>::kMinBlocks)
    lmm_finish_kernel(const Params p) {
    using L = Lay<C>;
    constexpr int U = C <= 2 ? 4 : 2;  // samples in flight
    const int64_t wid = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / 32;
    if (wid >= p.m * p.phi) return;
    const int lane = threadIdx.x & 31;
    const int64_t j = wid / p.phi;
    const int f = (int)(wid % p.phi);
    const double* __restrict__ x = p.G + j * p.ldg;
    const double* __restrict__ y = p.Y + (int64_t)f * p.ldy;
    const double* __restrict__ h0 = p.H + (int64_t)(p.n_grid + f) * p.n;
    const int64_t o = (int64_t)f * p.m + j;
    const bool on[2] = {p.mode == 2 || p.mode == 4, p.mode == 1 || p.mode == 4};  // MLE, REML
    const bool score = p.mode == 3 || p.mode == 4;
    double s[2] = {0.0, 0.0}, lam[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        if (on[q]) s[q] = __dmul_rn(__dadd_rn(p.state[2 * wid + q].a, p.state[2 * wid + q].b), 0.5);
        lam[q] = exp(s[q]);
    }
    double acc[2][L::NI], ld[2] = {0.0, 0.0}, xs0[L::NX];
#pragma unroll
    for (int q = 0; q < 2; ++q)
#pragma unroll
        for (int k = 0; k < L::NI; ++k) acc[q][k] = 0.0;
#pragma unroll
    for (int k = 0; k < L::NX; ++k) xs0[k] = 0.0;
    for (int64_t i0 = lane; i0 < p.n; i0 += 32 * U) {
        double ev[U], hv[U], vec[U][L::R];
#pragma unroll
        for (int u = 0; u < U; ++u) {  // past the end: a sample without weight
            const int64_t i = i0 + 32 * u;
            const bool in = i < p.n;
            ev[u] = in ? __ldg(p.evals + i) : 0.0;
            hv[u] = in && score ? __ldg(h0 + i) : 0.0;
#pragma unroll
            for (int a = 0; a < C; ++a) vec[u][a] = in ? __ldg(p.W + a * p.ldw + i) : 0.0;
            vec[u][C] = in ? x[i] : 0.0;
            vec[u][C + 1] = in ? __ldg(y + i) : 0.0;
        }
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            if (!on[q]) continue;
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const double v = __dadd_rn(__dmul_rn(lam[q], ev[u]), 1.0);
                const double h = __drcp_rn(v);
                ld[q] += log(fabs(v));
#pragma unroll
                for (int a = 0; a < L::R; ++a) {
                    const double t = h * vec[u][a];
#pragma unroll
                    for (int b = a; b < L::R; ++b)
                        acc[q][L::idx(a, b)] = fma(t, vec[u][b], acc[q][L::idx(a, b)]);
                }
            }
        }
        if (score) {
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const double t = hv[u] * vec[u][C];
#pragma unroll
                for (int a = 0; a < C; ++a) xs0[a] = fma(t, vec[u][a], xs0[a]);
                xs0[C] = fma(t, vec[u][C], xs0[C]);
                xs0[C + 1] = fma(t, vec[u][C + 1], xs0[C + 1]);
            }
        }
    }
    if (score) {
        double row0[L::NI];
#pragma unroll
        for (int k = 0; k < L::NX; ++k) xs0[k] = warp_sum(xs0[k]);
        assemble<C>(row0, p.S + ((int64_t)(p.n_grid + 1 + f) * p.phi + f) * L::NS, xs0);
        const PabOut<C> pb = pab_reduce<C>(row0);
        bool valid;
        double beta, tau, se;
        beta_se<C>(pb, clamp_pyy(pb.yy1), p.df, valid, beta, tau, se);
        const double fstat = p.n_d * (pb.xy * pb.xy) / (pb.yy * (valid ? pb.xx : 1.0));
        if (lane == 0) {
            if (p.out.p_score) p.out.p_score[o] = valid ? fstat : jnan();
            if (p.mode == 3) {
                if (p.out.beta) p.out.beta[o] = beta;
                if (p.out.se) p.out.se[o] = se;
            }
        }
    }
    if (on[0]) {
        double row0[L::NI];
#pragma unroll
        for (int k = 0; k < L::NI; ++k) row0[k] = warp_sum(acc[0][k]);
        const double logl = mle_logl<C>(pab_reduce<C>(row0), warp_sum(ld[0]), p);
        if (lane == 0) {
            if (p.out.lambda_mle) p.out.lambda_mle[o] = lam[0];
            if (p.out.logl_mle) p.out.logl_mle[o] = logl;
            const double stat = jmax(2.0 * (logl - p.logl0[f]), 0.0);
            if (p.out.p_lrt) p.out.p_lrt[o] = chi2_1_sf(stat);
        }
    }
    if (on[1]) {
        double row0[L::NI], log_iab[C + 1];
        pair_log_iab<C>(p, j, f, log_iab);
#pragma unroll
        for (int k = 0; k < L::NI; ++k) row0[k] = warp_sum(acc[1][k]);
        const PabOut<C> pb = pab_reduce<C>(row0);
        write_wald<C>(p, pb, reml_logl<C>(pb, log_iab, warp_sum(ld[1]), p), lam[1], o, lane == 0);
    }
}

}  // namespace lmm
}  // namespace jb
