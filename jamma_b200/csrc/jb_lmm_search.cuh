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
//   * LP = 4 for one covariate column (72 coefficient doubles, 8 pairs per warp), LP = 8 for
//     two to four (48 to 72 doubles, 4 pairs per warp);
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

template <int C>
struct Search {
    static constexpr int LP = C == 1 ? 4 : 8;  // lanes per pair
    static constexpr int V = 32 / LP;          // virtual lanes per lane
    static constexpr int kThreads = 128;
    static constexpr int kMinBlocks = 2;       // up to 255 registers
};

// Chebyshev values of a group: t[v] = T_{r + LP v}(x), m[v] = T_{LP - r + LP v}(x) (r the
// lane within the group), by the doubling identity T_{a+b} = 2 T_a T_b - T_{a-b} with a the
// largest power of two below the index.  Returns T_32(x).
template <int LP>
__device__ __forceinline__ double cheb_group(double x, int r, double (&t)[32 / LP],
                                             double (&m)[32 / LP]) {
    constexpr int V = 32 / LP;
    static_assert(LP == 4 || LP == 8, "group of 4 or 8 lanes");
    const double t2 = fma(2.0 * x, x, -1.0);
    const double t3 = fma(2.0 * t2, x, -x);
    const double t4 = fma(2.0 * t2, t2, -1.0);
    const int q = r & 3;
    const double lo = q == 0 ? 1.0 : (q == 1 ? x : (q == 2 ? t2 : t3));  // T_q
    const double hi = q == 0 ? t4 : (q == 1 ? t3 : (q == 2 ? t2 : x));   // T_{4-q}
    double ta;
    if (LP == 4) {
        t[0] = lo;
        m[0] = hi;
        ta = t4;
    } else {
        const bool up = r >= 4;
        const double v = fma(2.0 * t4, up ? lo : hi, -(up ? hi : lo));
        t[0] = up ? v : lo;
        m[0] = up ? hi : v;
        ta = fma(2.0 * t4, t4, -1.0);
    }
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
template <int C>
struct PairCoef {
    double c[Lay<C>::NX][Search<C>::V][kCoefPerLane];
};
template <int C>
__device__ __forceinline__ void load_pair_coef(const Params& p, int64_t j, int f, int r,
                                               PairCoef<C>& g) {
    constexpr int LP = Search<C>::LP;
    const int64_t cp = C + p.phi;
#pragma unroll
    for (int v = 0; v < Search<C>::V; ++v) {
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
template <int C>
__device__ __forceinline__ void series_xsums(const Params& p, const PairCoef<C>& g, double s, int r,
                                             double (&xs)[Lay<C>::NX]) {
    constexpr int LP = Search<C>::LP, V = Search<C>::V;
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
template <int C>
__device__ __forceinline__ void grid_xsums(const Params& p, const PairCoef<C>& g, int k, int r,
                                           double (&xs)[Lay<C>::NX]) {
    constexpr int LP = Search<C>::LP, V = Search<C>::V;
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

// log|H^-1| and the x-free sums of phenotype f at log-lambda s, from the expansions over the
// golden bracket of grid index `best` (degree 24, coefficients in virtual lanes 0..24).
template <int C>
__device__ __forceinline__ void bracket_sums(const Params& p, int best, int f, double s, int r,
                                             double& logdet, double (&shared)[Lay<C>::NS]) {
    using L = Lay<C>;
    constexpr int LP = Search<C>::LP, V = Search<C>::V;
    const double* __restrict__ cb =
        p.cheb + (int64_t)best * (1 + (int64_t)p.phi * L::NS) * kChebN + r;
    double t[V], m[V];
    cheb_group<LP>((s - __ldg(p.cheb_mid + best)) * (1.0 / __ldg(p.cheb_half + best)), r, t, m);
#pragma unroll
    for (int k = -1; k < L::NS; ++k) {
        const double* __restrict__ ck = cb + (k < 0 ? 0 : (int64_t)(1 + f * L::NS + k) * kChebN);
        double w[V];
#pragma unroll
        for (int v = 0; v < V; ++v) {
            const bool in = LP * v + LP <= kChebN || r + LP * v < kChebN;
            w[v] = LP * v < kChebN && in ? __dmul_rn(__ldg(ck + LP * v), t[v]) : 0.0;
        }
        const double v = group_sum<LP>(w);
        if (k < 0)
            logdet = v;
        else
            shared[k] = v;
    }
}

// REML and MLE log-likelihoods of one Pab result with the logarithms shared out: lane i <= C
// takes log of pivot i, lane C + 1 the one of P_yy; the sums are those of reml_logl / mle_logl.
template <int C>
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
        ldw = __dadd_rn(ldw, __shfl_sync(kFull, lg, i, Search<C>::LP));
        ldw = __dsub_rn(ldw, log_iab[i]);
    }
    const double lpyy = __shfl_sync(kFull, lg, C + 1, Search<C>::LP);
    double f = __dsub_rn(p.c_reml, __dmul_rn(0.5, logdet_h));
    f = __dsub_rn(f, __dmul_rn(0.5, ldw));
    return __dsub_rn(f, __dmul_rn(__dmul_rn(0.5, p.df), lpyy));
}

// One golden section (_golden_section_refine, likelihood_jax.py:419-488) as a sequence of
// probes: c, d, then one per step; probe number n_iter + 2 is the optimum (a + b) / 2.
struct Golden {
    double a, b, c, d, fc, fd, s;  // s: the next probe
    bool left;                     // it replaces c (fc), else d (fd)
    __device__ __forceinline__ void start(const Params& p, int best) {
        const int lo = best - 1 > 0 ? best - 1 : 0;
        const int hi = best + 1 < p.n_grid - 1 ? best + 1 : p.n_grid - 1;
        a = p.loglam[lo];
        b = p.loglam[hi];
        inner();
        fc = fd = 0.0;
        s = c;
        left = true;
    }
    __device__ __forceinline__ void inner() {
        c = __dsub_rn(b, __dmul_rn(kPhi, __dsub_rn(b, a)));
        d = __dadd_rn(a, __dmul_rn(kPhi, __dsub_rn(b, a)));
    }
    // takes the value at probe `it` and sets the next one
    __device__ __forceinline__ void take(double f, int it, int n_iter) {
        fc = left ? f : fc;
        fd = left ? fd : f;
        if (it == 0) {
            s = d;
            left = false;
            return;
        }
        if (it > n_iter) {
            s = __dmul_rn(__dadd_rn(a, b), 0.5);
            return;
        }
        left = fc > fd;
        a = left ? a : c;
        b = left ? d : b;
        const double keep = left ? fc : fd;
        fc = keep;  // the one that the next probe replaces is overwritten
        fd = keep;
        inner();
        s = left ? c : d;
    }
};

template <int C>
__global__ void __launch_bounds__(Search<C>::kThreads, Search<C>::kMinBlocks)
    lmm_search_kernel(const Params p) {
    using L = Lay<C>;
    constexpr int LP = Search<C>::LP;
    const int64_t npairs = p.m * p.phi;
    const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if ((tid & ~31ll) / LP >= npairs) return;  // the whole warp is idle
    // a group past the last pair repeats the last pair and writes nothing
    const bool valid_pair = tid / LP < npairs;
    const int64_t wid = valid_pair ? tid / LP : npairs - 1;
    const int r = threadIdx.x & (LP - 1);
    const int64_t j = wid / p.phi;
    const int f = (int)(wid % p.phi);
    const bool need_reml = p.mode == 1 || p.mode == 4;
    const bool need_mle = p.mode == 2 || p.mode == 4;
    const bool need_score = p.mode == 3 || p.mode == 4;
    const int64_t o = (int64_t)f * p.m + j;
    const int64_t srow = (int64_t)p.phi * L::NS;  // stride of one S row
    const bool writer = r == 0 && valid_pair;

    PairCoef<C> g;
    load_pair_coef<C>(p, j, f, r, g);

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
        series_xsums<C>(p, g, log(p.lam0[f]), r, xs);
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
    if (!need_reml && !need_mle) {  // score only: the large-lambda rewrite happens here
        double xs_m[L::NX], xs_r[L::NX];
        direct_fix<C, LP>(p, j, f, valid_pair, need_score, false, false, 0.0, 0.0, xs_m, xs_r);
        return;
    }

    // ---------------- shared lambda grid, LP points at a time
    ArgMax best_reml, best_mle;
#pragma unroll 1
    for (int g0 = 0; g0 < p.n_grid; g0 += LP) {
        double xs[L::NX];
#pragma unroll 1
        for (int e = 0; e < LP; ++e) {
            double xe[L::NX];
            grid_xsums<C>(p, g, g0 + e < p.n_grid ? g0 + e : p.n_grid - 1, r, xe);
#pragma unroll
            for (int q = 0; q < L::NX; ++q) xs[q] = e == r || e == 0 ? xe[q] : xs[q];
        }
        const int k = g0 + r;
        if (k < p.n_grid) {
            double row0[L::NI];
            assemble<C>(row0, p.S + (int64_t)k * srow + (int64_t)f * L::NS, xs);
            const PabOut<C> pb = pab_reduce<C>(row0);
            const double ldh = p.logdet[k];
            if (need_reml) best_reml.push(k, reml_logl<C>(pb, log_iab, ldh, p));
            if (need_mle) best_mle.push(k, mle_logl<C>(pb, ldh, p));
        }
    }
    best_reml.warp_reduce<LP>();
    best_mle.warp_reduce<LP>();

    // ---------------- golden sections, both searches in step
    const int bm = need_mle ? best_mle.idx : best_reml.idx;
    const int br = need_reml ? best_reml.idx : best_mle.idx;
    Golden gm, gr;
    gm.start(p, bm);
    gr.start(p, br);
    double xs_m[L::NX], xs_r[L::NX], sh_m[L::NS], sh_r[L::NS], ld_m = 0.0, ld_r = 0.0;
    PabOut<C> pb_m, pb_r;
#pragma unroll 1
    for (int it = 0;; ++it) {
        if (need_mle) {
            series_xsums<C>(p, g, gm.s, r, xs_m);
            bracket_sums<C>(p, bm, f, gm.s, r, ld_m, sh_m);
        }
        if (need_reml) {
            if (!need_mle || __any_sync(kFull, gm.s != gr.s || bm != br)) {
                series_xsums<C>(p, g, gr.s, r, xs_r);
                bracket_sums<C>(p, br, f, gr.s, r, ld_r, sh_r);
            } else {
#pragma unroll
                for (int q = 0; q < L::NX; ++q) xs_r[q] = xs_m[q];
#pragma unroll
                for (int q = 0; q < L::NS; ++q) sh_r[q] = sh_m[q];
                ld_r = ld_m;
            }
        }
        if (it == p.n_iter + 2) break;
        double row0[L::NI];
        if (need_mle) {
            assemble<C>(row0, sh_m, xs_m);
            gm.take(mle_logl<C>(pab_reduce<C>(row0), ld_m, p), it, p.n_iter);
        }
        if (need_reml) {
            assemble<C>(row0, sh_r, xs_r);
            gr.take(group_reml<C>(pab_reduce<C>(row0), log_iab, ld_r, p, r), it, p.n_iter);
        }
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

}  // namespace lmm
}  // namespace jb
