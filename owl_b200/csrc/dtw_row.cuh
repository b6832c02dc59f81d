// dtw_row.cuh -- one candidate's predecessor search in a row of the
// dynamic-time-warping program (dtw.cu): the double-precision arithmetic of the
// program, each operation rounded by itself, and the single-precision screening
// that leaves it few predecessors to compare. Compiles for the host too
// (without contraction), where tests/dtw_row_host.cpp compares every decision
// with the unscreened program.
#pragma once

#include <cmath>

#ifdef __CUDACC__
#define DTW_HD __host__ __device__ __forceinline__
#else
#define DTW_HD inline
#endif

namespace owl {

constexpr double DTW_SMIN = 1.0e-8, DTW_SMAX = 1.0e2, DTW_ETA = 0.15, DTW_DELTA = 1.0e-10;
constexpr double DTW_HUGE = 1.7976931348623157e308;

#ifdef __CUDA_ARCH__
DTW_HD double dadd(double a, double b) { return __dadd_rn(a, b); }
DTW_HD double dsub(double a, double b) { return __dsub_rn(a, b); }
DTW_HD double dmul(double a, double b) { return __dmul_rn(a, b); }
#else
DTW_HD double dadd(double a, double b) { return a + b; }
DTW_HD double dsub(double a, double b) { return a - b; }
DTW_HD double dmul(double a, double b) { return a * b; }
#endif

// x / b, correctly rounded, for a divisor b used many times, with its reciprocal
// as rh + rl (rh = RN(1 / b), rl the rounded remainder): x rh + x rl lies within
// half an ulp and a little of the quotient, its remainder is exact in one
// multiply-add, and the last multiply-add rounds correctly (Markstein,
// Computation of elementary functions on the IBM RISC System/6000 processor,
// IBM J. Res. Dev. 34, 1990). For finite x whose quotient and remainder stay
// in the normal range, as the grid positions and slopes here do.
struct DivBy {
    double b, rh, rl;
    DTW_HD explicit DivBy(double b_) : b(b_), rh(1.0 / b_) { rl = dmul(fma(-b, rh, 1.0), rh); }
};
DTW_HD double ddivby(double x, const DivBy& d) {
    const double q = fma(x, d.rh, dmul(x, d.rl));
    return fma(fma(-d.b, q, x), d.rh, q);
}

// What the rows of a program share. A step x of position is allowed
// (s_min - delta <= RN(x / dt) <= s_max + delta) exactly for x_min <= x <= x_max
// (the products are off by an ulp at most; the searches are bounded all the same).
struct DtwSlopes {
    double dt, rinst, x_min, x_max;
    DivBy gdt;
    float rdt, cr;  // 1 / dt, dt rinst
    float dpos;     // slope error of rounded positions
    DTW_HD DtwSlopes(int n, double rinst_) : dt(1.0 / ((double)n - 1.0)), rinst(rinst_), gdt(dt) {
        x_max = dmul(DTW_SMAX + DTW_DELTA, dt);
        x_min = dmul(DTW_SMIN - DTW_DELTA, dt);
        for (int i = 0; i < 8 && above(x_max); ++i) x_max = nextafter(x_max, 0.0);
        for (int i = 0; i < 8 && !above(nextafter(x_max, DTW_HUGE)); ++i) x_max = nextafter(x_max, DTW_HUGE);
        for (int i = 0; i < 8 && below(x_min); ++i) x_min = nextafter(x_min, DTW_HUGE);
        for (int i = 0; i < 8 && !below(nextafter(x_min, 0.0)); ++i) x_min = nextafter(x_min, 0.0);
        rdt = (float)(1.0 / dt);
        cr = (float)dmul(dt, rinst);
        dpos = 1.0e-15f * rdt;
    }
    DTW_HD bool above(double x) const { return ddivby(x, gdt) > DTW_SMAX + DTW_DELTA; }
    DTW_HD bool below(double x) const { return ddivby(x, gdt) < DTW_SMIN - DTW_DELTA; }
};

// candidates per unit of position (0: a band too narrow to locate candidates in)
// and the slope's change per candidate, of a row whose band is du wide
struct DtwScale {
    float sc, c1;
};
DTW_HD DtwScale dtw_scale(double du, int m, double dt) {
    const double sc = du > 1.0e-9 ? (double)(m - 1) / du : 0.0;
    return DtwScale{(float)sc, sc > 0.0 ? (float)(1.0 / (sc * dt)) : 0.f};
}

// One lane's part of the search among the predecessors of a candidate at
// position tgk with node cost nu: G lanes share them, each of them taken by one
// lane, the same in both passes. First `screen` (the lane's least cost in single
// precision), then, with the least over the lanes, `resolve` (every predecessor
// of the lane whose cost lies within the error bound of the least one, in the
// program's double arithmetic); the least double cost over the lanes, ties to the
// lowest predecessor, is the program's (ascending order, strict improvement).
struct DtwLane {
    const DtwSlopes& w;
    const double *tc, *f;  // the row's positions and costs
    const float* f32;      // the costs in single precision
    int m, lane, G;
    double tgk, nu;
    DtwScale s;
    int jlo, jhi, in0, in1, na, ne;
    float s0, g1 = INFINITY, g2 = INFINITY;  // the least cost and the second least
    int j1 = 0;
    double best = DTW_HUGE;
    int bj = 0;

    DTW_HD DtwLane(const DtwSlopes& w_, const double* tc_, const double* f_, const float* f32_, int m_, int lane_, int G_,
                   double tgk_, double nu_, DtwScale s_)
        : w(w_), tc(tc_), f(f_), f32(f32_), m(m_), lane(lane_), G(G_), tgk(tgk_), nu(nu_), s(s_) {}

    DTW_HD bool allowed(int j) const {
        const double x = dsub(tgk, tc[j]);
        return x <= w.x_max && x >= w.x_min;
    }
    // (an unreachable predecessor, DTW_HUGE, never gives a lower cost)
    DTW_HD void exact(int j) {
        const double sl = ddivby(dsub(tgk, tc[j]), w.gdt);
        const double pc = dadd(f[j], dmul(w.dt, dadd(dmul(w.rinst, dmul(sl, sl)), nu)));
        if (pc < best || (pc == best && j < bj)) {
            best = pc;
            bj = j;
        }
    }
    // cost without the node's own term, in single precision: s falls by c1 per
    // candidate from its value at jlo
    DTW_HD float cost32(int j) const {
        const float sl = fmaf(-s.c1, (float)(j - jlo), s0);
        return fmaf(sl * sl, w.cr, f32[j]);
    }
    // the lane's predecessors, in the order of its first pass
    template <int UNROLL, typename F>
    DTW_HD void each(F&& take) {
#pragma unroll UNROLL
        for (int j = in0 + lane; j <= in1; j += G) take(j);
        for (int e = lane; e < ne; e += G) {
            const int j = e < na ? jlo + e : in1 + 1 + e - na;
            if (allowed(j)) take(j);
        }
    }
    // candidates of an allowed slope form one run (the slope falls as j grows): a
    // window [jlo, jhi] that holds it, two candidates to spare (the estimate is off
    // by less than one); all but its outer five at each end are allowed for certain
    DTW_HD void screen() {
        const float e0 = (float)(tgk - w.x_max - tc[0]) * s.sc, e1 = (float)(tgk - w.x_min - tc[0]) * s.sc;
        jlo = e0 <= 2.f ? 0 : (int)fminf(e0, (float)m) - 2;
        jhi = e1 >= (float)(m - 3) ? m - 1 : (int)fmaxf(e1, -3.f) + 2;
        in0 = jlo + 5;
        in1 = jhi - 5;
        na = in1 < in0 ? jhi - jlo + 1 : 5;
        ne = in1 < in0 ? na : 10;
        s0 = (float)dsub(tgk, tc[jlo < m ? jlo : m - 1]) * w.rdt;
        each<8>([&](int j) {
            const float v = cost32(j);
            g2 = fminf(g2, fmaxf(g1, v));
            if (v < g1) {
                g1 = v;
                j1 = j;
            }
        });
    }
    // g: the least g1 over the lanes. The bound is twice the error of a cost: 2 eps of
    // the cost (its predecessor's part and the sum) and 10 eps of the largest slope
    // term (s to 3 eps of s0, its square, the product), doubled; the positions' own
    // double rounding in the slope; costs too small for single precision; and the
    // double rounding of the program's own cost, the node's term included (five
    // roundings of 2^-53, twice: where the costs before are far below that term they
    // tie, and the lowest predecessor wins).
    DTW_HD void resolve(float g) {
        constexpr float EPS = 5.9604645e-8f;  // 2^-24
        const float sm = fabsf(s0) + s.c1;
        const float thr = g + EPS * (8.f * g + 40.f * (w.cr * (sm * sm))) +
                          4.f * w.cr * (2.f * sm * w.dpos + w.dpos * w.dpos) + 2.0e-15f * (float)dmul(w.dt, nu) + 1.0e-37f;
        if (!(thr < INFINITY)) {  // costs beyond single precision, none reachable, not a number
            each<1>([&](int j) { exact(j); });
        } else if (g1 <= thr) {
            exact(j1);
            if (g2 <= thr)  // more than one of the lane's
                each<1>([&](int j) {
                    if (cost32(j) <= thr) exact(j);
                });
        }
    }
    // every predecessor (a band too narrow to locate candidates in)
    DTW_HD void all() {
        for (int j = lane; j < m; j += G)
            if (allowed(j)) exact(j);
    }
};

}  // namespace owl
