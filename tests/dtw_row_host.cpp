// Host build of csrc/dtw_row.cuh: the screened predecessor search against the
// program as the reference writes it (ascending predecessors, strict improvement,
// true divisions), decision by decision, and the division by a fixed divisor
// against the division operator. Prints one line per check; exits 1 on a mismatch.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <vector>

#include "../owl_b200/csrc/dtw_row.cuh"

using namespace owl;

static long long division_mismatches() {
    long long bad = 0;
    std::mt19937_64 rng(1);
    std::uniform_real_distribution<double> u(-1.0, 1.0);
    for (int n = 3; n <= 16384; n += n < 300 ? 1 : 37) {
        const DivBy g((double)(n - 1));
        for (int i = 0; i < n; ++i) bad += ddivby((double)i, g) != (double)i / (double)(n - 1);
        const double dt = 1.0 / ((double)n - 1.0);
        const DivBy d(dt);
        for (int k = 0; k < 400; ++k) {
            const double x = u(rng) * std::pow(10.0, -12.0 * (k % 13) / 12.0);
            bad += ddivby(x, d) != x / dt;
        }
    }
    return bad;
}

struct Case {
    int n, m, niter;
    double rinst, rcuml, power, scale;
    int mute;  // leading samples without signal
    bool equal;  // obs = syn
};

// one trace: the program in double precision; at every row and candidate the
// screened search of every group size on the same costs must decide alike
static long long trace_mismatches(const Case& c, unsigned seed, long long& decisions) {
    const int n = c.n, m = c.m, jc = (m - 1) / 2;
    std::mt19937 rng(seed);
    std::normal_distribution<double> nd;
    std::uniform_real_distribution<double> ud(0.0, 1.0);
    std::vector<double> x(n), y(n);
    const double ctr = 0.2 + 0.6 * ud(rng), lag = 0.02 * ud(rng), wid = 0.02 + 0.1 * ud(rng);
    double nx = 0.0, ny = 0.0;
    for (int i = 0; i < n; ++i) {
        const double t = (double)i / (n - 1);
        auto pulse = [&](double q) { return std::exp(-q * q / (wid * wid)) * std::cos(3.0 * q / wid); };
        y[i] = pulse(t - ctr) + 1e-3 * nd(rng);
        x[i] = c.equal ? y[i] : 0.9 * pulse(t - ctr - lag) + 1e-3 * nd(rng);
        if (i < c.mute) x[i] = y[i] = 0.0;
        nx += x[i] * x[i];
        ny += y[i] * y[i];
    }
    for (int i = 0; i < n; ++i) {
        x[i] = c.scale * (float)(x[i] / std::sqrt(nx));
        y[i] = c.scale * (float)(y[i] / std::sqrt(ny));
    }
    const DtwSlopes w(n, c.rinst);
    const double dt = w.dt;
    std::vector<double> L(n), U(n), T(n), f(m), fn(m), tc(m), tn(m);
    std::vector<float> f32(m);
    std::vector<int> path((size_t)n * m);
    auto cost = [&](int i, double tg) {
        double q = std::fmin(std::fmax(tg, 0.0), 1.0) * (n - 1);
        const int i0 = std::min((int)q, n - 2);
        const double v = x[i0] + (q - i0) * (x[i0 + 1] - x[i0]), d = tg - (double)i / (n - 1);
        return std::pow(std::fabs(v - y[i]), c.power) + c.rcuml * (d * d);
    };
    auto positions = [&](int i, std::vector<double>& t) {
        for (int j = 0; j < m; ++j) t[j] = L[i] + (U[i] - L[i]) * ((double)j / (double)(m - 1));
    };
    long long bad = 0;
    for (int it = 0; it < c.niter; ++it) {
        for (int i = 0; i < n; ++i) {
            const double t = (double)i / (n - 1);
            const double u0 = std::fmin(std::fmin(DTW_SMAX * t, 1.0 - DTW_SMIN * (1.0 - t)), 1.0);
            const double l0 = std::fmax(std::fmax(DTW_SMIN * t, 1.0 - DTW_SMAX * (1.0 - t)), 0.0);
            const double r = it ? DTW_ETA * (U[i] - L[i]) / 2.0 : 0.0;
            U[i] = it ? std::fmin(T[i] + r, u0) : u0;
            L[i] = it ? std::fmax(T[i] - r, l0) : l0;
        }
        positions(0, tc);
        for (int k = 0; k < m; ++k) f[k] = k == jc ? cost(0, tc[k]) : DTW_HUGE;
        for (int i = 0; i + 1 < n; ++i) {
            positions(i, tc);
            positions(i + 1, tn);
            for (int k = 0; k < m; ++k) f32[k] = (float)f[k];
            const DtwScale sc = dtw_scale(U[i] - L[i], m, dt);
            for (int k = 0; k < m; ++k) {
                const double nu = cost(i + 1, tn[k]);
                double best = DTW_HUGE;
                int bj = 0;
                for (int j = 0; j < m; ++j) {
                    const double s = (tn[k] - tc[j]) / dt;
                    if (s < DTW_SMIN - DTW_DELTA || s > DTW_SMAX + DTW_DELTA || !(f[j] < DTW_HUGE)) continue;
                    const double pc = f[j] + dt * (c.rinst * (s * s) + nu);
                    if (pc < best) {
                        best = pc;
                        bj = j;
                    }
                }
                fn[k] = best;
                path[(size_t)(i + 1) * m + k] = bj;
                for (int G = 1; G <= 32; G *= 2) {
                    std::vector<DtwLane> ln;
                    float g = INFINITY;
                    for (int l = 0; l < G; ++l) {
                        ln.emplace_back(w, tc.data(), f.data(), f32.data(), m, l, G, tn[k], nu, sc);
                        if (sc.sc > 0.f) ln.back().screen();
                        g = std::fmin(g, ln.back().g1);
                    }
                    double b = DTW_HUGE;
                    int bb = 0;
                    for (DtwLane& q : ln) {
                        if (sc.sc > 0.f) q.resolve(g);
                        else q.all();
                        if (q.best < b || (q.best == b && q.bj < bb)) {
                            b = q.best;
                            bb = q.bj;
                        }
                    }
                    ++decisions;
                    bad += b != best || bb != bj;
                }
            }
            f.swap(fn);
        }
        int j = jc;
        for (int i = n - 1; i >= 0; --i) {
            T[i] = L[i] + (U[i] - L[i]) * ((double)j / (double)(m - 1));
            if (i) j = path[(size_t)i * m + j];
        }
    }
    return bad;
}

int main(int argc, char** argv) {
    const int traces = argc > 1 ? std::atoi(argv[1]) : 4;
    long long bad = division_mismatches();
    std::printf("divisions: %lld mismatches\n", bad);
    const Case cases[] = {
        {101, 101, 5, 0.1f, 1.0, 0.5, 1.0, 0, false},    // the defaults
        {61, 31, 5, 0.1f, 1.0, 0.5, 1.0, 20, false},     // muted samples
        {61, 31, 5, 0.1f, 1.0, 0.5, 1.0, 0, true},       // equal traces: no distance on the diagonal
        {47, 65, 20, 0.0, 1.0, 0.5, 1.0, 16, false},     // no slope cost, bands down to rounding
        {47, 33, 12, 0.1f, 0.0, 2.0, 1.0, 16, false},    // no position cost
        {47, 33, 4, 1e30, 1e30, 0.5, 1.0, 8, false},     // costs near the end of single precision
        {47, 33, 4, 3e38, 3e38, 1.0, 1.0, 8, false},     // and beyond
        {47, 33, 4, 0.1f, 1.0, 200.0, 3e2, 8, false},    // distances beyond single precision
        {47, 33, 4, 1e-38, 1e-38, 2.0, 1e-20, 8, false}, // costs below its normal range
        {9, 301, 5, 0.1f, 1.0, 0.5, 1.0, 0, false},      // many candidates, few rows
        {400, 5, 5, 0.1f, 1.0, 1.0, 1.0, 0, false},      // few candidates, many rows
    };
    for (const Case& c : cases) {
        long long b = 0, d = 0;
        for (int s = 0; s < traces; ++s) b += trace_mismatches(c, 100 * s + 7, d);
        std::printf("n %d m %d niter %d rinst %g rcuml %g power %g: %lld of %lld decisions differ\n", c.n, c.m, c.niter,
                    c.rinst, c.rcuml, c.power, b, d);
        bad += b;
    }
    return bad != 0;
}
