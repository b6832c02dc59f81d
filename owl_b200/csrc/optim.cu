// optim.cu -- search directions and gradient processing on the GPU.
//
// compute_search_direction (src/inverse/module_inversion_search_direction.f90:
// steepest descent, Polak-Ribiere conjugate gradient :38-86, two-loop L-BFGS
// :91-246) over fields that stay in device memory: every dot product is an FP64
// reduction in a fixed order (per-block partials, then one block), the vector
// updates are elementwise kernels, and s_i = x_{i+1} - x_i, y_i = g_{i+1} - g_i
// are formed on the fly from the models and gradients the caller keeps, as the
// reference reads them from its iteration directories.
//
// The gradient processing of process_model_single_parameter
// (src/inverse/2d/module_gradient.f90:733-892): Gaussian smoothing (separable,
// one pass per axis, edge samples replicated), Blackman taper ramps at the
// ends of each axis, mask, scale and max balance. FLIT's gauss_filt and taper
// are restated (a Gaussian of the given standard deviation in cells truncated
// at 3 sigma and normalised; Blackman ramps 0.42 - 0.5 cos(pi i / l) +
// 0.08 cos(2 pi i / l), i = 0..l-1, from each end).
#include <algorithm>
#include <cmath>
#include <vector>

#include "engine.cuh"
#include "workspace.cuh"

namespace owl {

namespace {

constexpr int RED_BLOCKS = 148 * 8;

// ---- search directions as a chain of launches without host round trips ----
//
// Each launch of the L-BFGS recursion finishes the dot products of the launch
// before (every block sums the per-block FP64 partials itself, in a fixed order,
// so no block waits for another), applies that pair's update to the direction
// and forms the partials of the next pair in the same pass: 2 np + 1 launches
// for np pairs, where a dot, a one-thread sum of its partials, a copy to the host
// and an update per pair were 6 np + 4 launches and 2 np + 1 host waits. A field
// of 80 k cells is latency bound: 401 x 201, six models, smoothing and taper
// included, takes 0.15 ms a pass against 2.1 ms (with the workspaces of workspace.cuh).
// A large field is bound by HBM, which needs some 40 KB of reads in flight per SM:
// a thread takes LB_CELLS cells at once, on up to four blocks of an SM. Six models of
// 12 / 40 / 85 million cells take 0.61 / 1.83 / 3.80 ms (6.1 TB/s), with one cell at a
// time on two blocks 1.65 / 5.2 / 11.0, with the launches that waited for the host
// 2.4 / 4.5 / 7.6; eight blocks gain 2 % there and lose 27 % on 361 k cells.
struct LbStep {
    long long n;
    int nparts;               // blocks of the launch before (its partials), 0: none
    const double* pin;        // nparts x 3 partials
    double* pout;             // gridDim x 3 partials
    double* sc;               // alpha[np], ys[np], gamma
    int np, prev;             // pairs; pair whose dot products pin holds
    const float* src;         // the direction so far
    float* r;                 // the direction
    const float *u1, *u0;     // update vector u1 - u0 of pair prev
    const float *x1, *x0, *g1, *g0;  // next pair: s = x1 - x0, y = g1 - g0
};
constexpr int LB_CELLS = 4;
enum { LB_FIRST = 0, LB_DOWN, LB_TURN, LB_UP, LB_LAST };

// sums of three values over the block (256 threads, fixed order), in every thread
__device__ __forceinline__ void block_sum3(double& a, double& b, double& c) {
    __shared__ double red[3][8];
    for (int o = 16; o; o >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, o);
        b += __shfl_xor_sync(0xffffffffu, b, o);
        c += __shfl_xor_sync(0xffffffffu, c, o);
    }
    __syncthreads();
    if ((threadIdx.x & 31) == 0) {
        red[0][threadIdx.x >> 5] = a;
        red[1][threadIdx.x >> 5] = b;
        red[2][threadIdx.x >> 5] = c;
    }
    __syncthreads();
    a = b = c = 0.0;
    for (int i = 0; i < 8; ++i) {
        a += red[0][i];
        b += red[1][i];
        c += red[2][i];
    }
}
__device__ __forceinline__ void sum_parts(const double* __restrict__ p, int n, double& a, double& b, double& c) {
    a = b = c = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        a += p[3 * i];
        b += p[3 * i + 1];
        c += p[3 * i + 2];
    }
    block_sum3(a, b, c);
}

// MODE: LB_FIRST dots of the newest pair; LB_DOWN q -= alpha y, dots of the next
// older pair; LB_TURN the oldest pair's q -= alpha y, the scaling gamma, y.r of the
// oldest pair; LB_UP r += s (alpha - beta), y.r of the next newer pair; LB_LAST the
// newest pair's update and the sign
template <int MODE>
__global__ void __launch_bounds__(256) k_lbfgs(const __grid_constant__ LbStep a) {
    pdl_prologue();
    double coef = 0.0, gamma = 0.0;
    if (MODE != LB_FIRST) {
        double d0, d1, d2;  // LB_DOWN / LB_TURN: s.q, y.s, y.y (newest pair); LB_UP / LB_LAST: y.r in d2
        sum_parts(a.pin, a.nparts, d0, d1, d2);
        double *alpha = a.sc, *ys = a.sc + a.np;
        if (MODE == LB_DOWN || MODE == LB_TURN) {
            const double al = d1 == 0.0 ? 0.0 : d0 / d1;
            coef = -al;
            if (MODE == LB_TURN) gamma = a.prev == a.np - 1 ? (d2 == 0.0 ? 0.0 : d1 / d2) : a.sc[2 * a.np];
            if (blockIdx.x == 0 && threadIdx.x == 0) {
                alpha[a.prev] = al;
                ys[a.prev] = d1;
                if (a.prev == a.np - 1) a.sc[2 * a.np] = d2 == 0.0 ? 0.0 : d1 / d2;
            }
        } else {
            const double y = ys[a.prev];
            coef = alpha[a.prev] - (y == 0.0 ? 0.0 : d2 / y);
        }
    }
    double p0 = 0.0, p1 = 0.0, p2 = 0.0;
    // LB_CELLS cells a thread at once, their reads ahead of their writes (r may be src)
    const long long step = (long long)gridDim.x * blockDim.x;
    for (long long i0 = (long long)blockIdx.x * blockDim.x + threadIdx.x; i0 < a.n; i0 += LB_CELLS * step) {
        float q[LB_CELLS], u1[LB_CELLS], u0[LB_CELLS], x1[LB_CELLS], x0[LB_CELLS], g1[LB_CELLS], g0[LB_CELLS];
#pragma unroll
        for (int e = 0; e < LB_CELLS; ++e) {
            const long long i = i0 + e * step;
            if (i >= a.n) continue;
            q[e] = a.src[i];
            if (MODE != LB_FIRST) {
                u1[e] = a.u1[i];
                u0[e] = a.u0[i];
            }
            if (MODE == LB_FIRST || MODE == LB_DOWN) {
                x1[e] = a.x1[i];
                x0[e] = a.x0[i];
            }
            if (MODE != LB_LAST) {
                g1[e] = a.g1[i];
                g0[e] = a.g0[i];
            }
        }
#pragma unroll
        for (int e = 0; e < LB_CELLS; ++e) {
            const long long i = i0 + e * step;
            if (i >= a.n) continue;
            if (MODE != LB_FIRST) {
                q[e] = (float)((double)q[e] + coef * ((double)u1[e] - (double)u0[e]));
                if (MODE == LB_TURN) q[e] = (float)(gamma * (double)q[e]);
                if (MODE == LB_LAST) q[e] = -q[e];
                a.r[i] = q[e];
            }
            if (MODE == LB_LAST) continue;
            const double y = (double)g1[e] - (double)g0[e];
            if (MODE == LB_FIRST || MODE == LB_DOWN) {
                const double s = (double)x1[e] - (double)x0[e];
                p0 += s * (double)q[e];
                p1 += y * s;
                if (MODE == LB_FIRST) p2 += y * y;
            } else {
                p2 += y * (double)q[e];
            }
        }
    }
    if (MODE == LB_LAST) return;
    block_sum3(p0, p1, p2);
    if (threadIdx.x == 0) {
        a.pout[(size_t)blockIdx.x * 3] = p0;
        a.pout[(size_t)blockIdx.x * 3 + 1] = p1;
        a.pout[(size_t)blockIdx.x * 3 + 2] = p2;
    }
}

// conjugate gradient: partials of gp.gp and (g - gp).g, then the direction
__global__ void __launch_bounds__(256) k_cg_dots(long long n, const float* __restrict__ g, const float* __restrict__ gp,
                                                 double* __restrict__ part) {
    double p0 = 0.0, p1 = 0.0, p2 = 0.0;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const double v = g[i], w = gp[i];
        p0 += w * w;
        p1 += (v - w) * v;
    }
    block_sum3(p0, p1, p2);
    if (threadIdx.x == 0) {
        part[(size_t)blockIdx.x * 3] = p0;
        part[(size_t)blockIdx.x * 3 + 1] = p1;
        part[(size_t)blockIdx.x * 3 + 2] = p2;
    }
}
__global__ void __launch_bounds__(256) k_cg_apply(long long n, const double* __restrict__ part, int nparts,
                                                  const float* g, const float* prev, float* srch) {
    pdl_prologue();
    double s1, s2, z;
    sum_parts(part, nparts, s1, s2, z);
    const double beta = s1 == 0.0 ? 0.0 : fmax(0.0, s2 / s1);
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        srch[i] = (float)(-(double)g[i] + beta * (double)prev[i]);
}

// (r may be g: LB_CELLS cells a thread at once, their reads ahead of their writes)
__global__ void __launch_bounds__(256) k_negate(long long n, const float* g, float* r) {
    const long long step = (long long)gridDim.x * blockDim.x;
    for (long long i0 = (long long)blockIdx.x * blockDim.x + threadIdx.x; i0 < n; i0 += LB_CELLS * step) {
        float v[LB_CELLS];
#pragma unroll
        for (int e = 0; e < LB_CELLS; ++e)
            if (i0 + e * step < n) v[e] = g[i0 + e * step];
#pragma unroll
        for (int e = 0; e < LB_CELLS; ++e)
            if (i0 + e * step < n) r[i0 + e * step] = -v[e];
    }
}

// one axis of a separable filter: field (n1, n2, n3), axis stride `st`, length `len`.
// The weights come in the kernel's parameters (every thread reads the same one:
// a constant operand), without an upload.
constexpr int SMOOTH_W = 513;
struct SmoothW {
    float w[SMOOTH_W];
};
template <typename I>
__device__ __forceinline__ void smooth_axis(const float* __restrict__ in, float* __restrict__ out, long long n, I st,
                                            int len, const float* w, int rad) {
    for (long long ii = (long long)blockIdx.x * blockDim.x + threadIdx.x; ii < n; ii += (long long)gridDim.x * blockDim.x) {
        const I i = (I)ii;
        const int p = (int)((i / st) % (I)len);
        const float* base = in + (ii - (long long)p * (long long)st);
        float acc = 0.f;
        for (int k = -rad; k <= rad; ++k) {
            const int q = min(max(p + k, 0), len - 1);
            acc += w[k + rad] * base[(long long)q * (long long)st];
        }
        out[ii] = acc;
    }
}
template <typename I>
__global__ void k_smooth_axis_p(const float* __restrict__ in, float* __restrict__ out, long long n, I st, int len,
                                const __grid_constant__ SmoothW w, int rad) {
    smooth_axis<I>(in, out, n, st, len, w.w, rad);
}
// weights of more taps than the parameters hold, from global memory
__global__ void k_smooth_axis(const float* __restrict__ in, float* __restrict__ out, long long n, long long st, int len,
                              const float* __restrict__ w, int rad) {
    smooth_axis<long long>(in, out, n, st, len, w, rad);
}

__global__ void k_taper(float* __restrict__ f, long long n, int n1, int n2, int n3, int a1, int b1, int a2, int b2,
                        int a3, int b3) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const int i1 = (int)(i % n1);
        const int i2 = (int)((i / n1) % n2);
        const int i3 = (int)(i / ((long long)n1 * n2));
        auto ramp = [](int j, int l) -> float {
            if (j >= l) return 1.f;
            const double t = (double)j / (double)l;
            return (float)(0.42 - 0.5 * cospi(t) + 0.08 * cospi(2.0 * t));
        };
        float w = 1.f;  // axes of one sample are left alone
        if (n1 > 1) w *= ramp(i1, a1) * ramp(n1 - 1 - i1, b1);
        if (n2 > 1) w *= ramp(i2, a2) * ramp(n2 - 1 - i2, b2);
        if (n3 > 1) w *= ramp(i3, a3) * ramp(n3 - 1 - i3, b3);
        f[i] *= w;
    }
}

__global__ void k_mul(float* __restrict__ f, long long n, const float* __restrict__ m, float c) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        f[i] = (m ? f[i] * m[i] : f[i]) * c;
}

__global__ void k_max_part(const float* __restrict__ f, long long n, float* __restrict__ part) {
    float m = -INFINITY;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        m = fmaxf(m, f[i]);
    for (int o = 16; o; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    __shared__ float red[8];
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        float t = red[0];
        for (int i = 1; i < 8; ++i) t = fmaxf(t, red[i]);
        part[blockIdx.x] = t;
    }
}

// sum of squares of each slice along an axis (one CTA per slice, FP64)
__global__ void k_slice_sumsq(const float* __restrict__ f, int n1, int n2, int n3, int axis, double* __restrict__ out) {
    const int j = blockIdx.x;
    const long long m = axis == 0 ? (long long)n2 * n3 : axis == 1 ? (long long)n1 * n3 : (long long)n1 * n2;
    double acc = 0.0;
    for (long long e = threadIdx.x; e < m; e += blockDim.x) {
        long long i1, i2, i3;
        if (axis == 0) { i1 = j; i2 = e % n2; i3 = e / n2; }
        else if (axis == 1) { i1 = e % n1; i2 = j; i3 = e / n1; }
        else { i1 = e % n1; i2 = e / n1; i3 = j; }
        const double v = f[(i3 * n2 + i2) * n1 + i1];
        acc += v * v;
    }
    __shared__ double red[256];
    red[threadIdx.x] = acc;
    __syncthreads();
    for (int o = blockDim.x / 2; o; o >>= 1) {
        if ((int)threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) out[j] = red[0];
}

// each element divided by the norm of its slice's window; NaN / Inf -> 0
__global__ void k_div_slice(float* __restrict__ f, long long n, int n1, int n2, int axis, const float* __restrict__ nrm) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const long long j = axis == 0 ? i % n1 : axis == 1 ? (i / n1) % n2 : i / ((long long)n1 * n2);
        const float v = f[i] / nrm[j];
        f[i] = isfinite(v) ? v : 0.f;
    }
}

// median of the (2 h1 + 1) x (2 h2 + 1) x (2 h3 + 1) window, truncated at the ends
__device__ float select_kth(float* a, int n, int k) {  // k-th smallest (0-based), a is reordered
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const float piv = a[(lo + hi) / 2];
        int i = lo, j = hi;
        while (i <= j) {
            while (a[i] < piv) ++i;
            while (a[j] > piv) --j;
            if (i <= j) {
                const float t = a[i]; a[i] = a[j]; a[j] = t;
                ++i; --j;
            }
        }
        if (k <= j) hi = j;
        else if (k >= i) lo = i;
        else return a[k];
    }
    return a[k];
}

__global__ void k_median(const float* __restrict__ in, float* __restrict__ out, int n1, int n2, int n3, int h1, int h2,
                         int h3) {
    const long long n = (long long)n1 * n2 * n3;
    float w[343];
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const int i1 = (int)(i % n1), i2 = (int)((i / n1) % n2), i3 = (int)(i / ((long long)n1 * n2));
        int c = 0;
        for (int a3 = max(0, i3 - h3); a3 <= min(n3 - 1, i3 + h3); ++a3)
            for (int a2 = max(0, i2 - h2); a2 <= min(n2 - 1, i2 + h2); ++a2)
                for (int a1 = max(0, i1 - h1); a1 <= min(n1 - 1, i1 + h1); ++a1)
                    w[c++] = in[((long long)a3 * n2 + a2) * n1 + a1];
        float v;
        if (c & 1) {
            v = select_kth(w, c, c / 2);
        } else {
            const float hi = select_kth(w, c, c / 2);
            float lo = w[0];  // after the selection, the largest of w[0 .. c/2 - 1] is the (c/2 - 1)-th
            for (int k = 1; k < c / 2; ++k) lo = fmaxf(lo, w[k]);
            v = 0.5f * (lo + hi);
        }
        out[i] = v;
    }
}

int blocks_for(long long n) { return (int)std::max<long long>(1, std::min<long long>((n + 255) / 256, RED_BLOCKS)); }

}  // namespace

// models[0..nm-1] oldest first, grads alike; srch written. All device pointers.
void search_direction(int method, long long n, int nm, const float* const* x, const float* const* g,
                      const float* prev_srch, float* srch, Workspace& ws) {
    cudaStream_t s = ws.s;
    const float* gk = g[nm - 1];
    // four blocks per SM at most: every launch sums the partials of the one before
    const int nb = (int)std::max<long long>(1, std::min<long long>((n + 255) / 256, 4 * 148));
    if (method == OWL_SEARCH_SD || nm < 2) {
        k_negate<<<nb, 256, 0, s>>>(n, gk, srch);
        OWL_LAUNCH_CHECK();
        return;
    }
    const int np = nm - 1;
    double* work = ws.take<double>((size_t)6 * nb + 2 * np + 1);  // two sets of partials, then alpha, ys, gamma
    if (method == OWL_SEARCH_CG) {
        // Polak-Ribiere: beta = max(0, g.(g - gp) / gp.gp), srch = -g + beta srch_prev
        OWL_CHECK(prev_srch, OWL_ERR_INVALID, "conjugate gradient needs the previous search direction");
        k_cg_dots<<<nb, 256, 0, s>>>(n, gk, g[nm - 2], work);
        launch_pdl(k_cg_apply, dim3(nb), dim3(256), 0, s, n, (const double*)work, nb, gk, prev_srch, srch);
        OWL_LAUNCH_CHECK();
        return;
    }
    // L-BFGS two-loop recursion over the pairs (x_{i+1} - x_i, g_{i+1} - g_i), newest first
    LbStep a{};
    a.n = n;
    a.nparts = nb;
    a.sc = work + (size_t)6 * nb;
    a.np = np;
    int flip = 0;
    auto next_pair = [&](int i) {
        a.x1 = x[i + 1]; a.x0 = x[i];
        a.g1 = g[i + 1]; a.g0 = g[i];
        a.pin = work + (size_t)3 * nb * flip;
        flip ^= 1;
        a.pout = work + (size_t)3 * nb * flip;
    };
    auto go = [&](void (*k)(LbStep)) { launch_pdl(k, dim3(nb), dim3(256), 0, s, a); };
    a.src = gk;
    a.r = srch;
    next_pair(np - 1);
    go(k_lbfgs<LB_FIRST>);
    for (int i = np - 1; i > 0; --i) {  // q -= alpha_i y_i; s.q and y.s of pair i - 1
        a.prev = i;
        a.u1 = g[i + 1]; a.u0 = g[i];
        next_pair(i - 1);
        go(k_lbfgs<LB_DOWN>);
        a.src = srch;
    }
    a.prev = 0;
    a.u1 = g[1]; a.u0 = g[0];
    next_pair(0);
    go(k_lbfgs<LB_TURN>);
    a.src = srch;
    for (int i = 0; i < np; ++i) {  // r += s_i (alpha_i - beta_i); y.r of pair i + 1
        a.prev = i;
        a.u1 = x[i + 1]; a.u0 = x[i];
        next_pair(std::min(i + 1, np - 1));
        go(i + 1 < np ? k_lbfgs<LB_UP> : k_lbfgs<LB_LAST>);
    }
    OWL_LAUNCH_CHECK();
}

void grad_process(int op, int n1, int n2, int n3, const float* param, const float* mask, float* f, Workspace& ws) {
    cudaStream_t s = ws.s;
    const long long n = (long long)n1 * n2 * n3;
    if (n == 0) return;
    const int nb = blocks_for(n);
    switch (op) {
        case OWL_GRAD_SMOOTH: {
            DevBuf<float> w;
            float* tmp = ws.take<float>(n);
            const int len[3] = {n1, n2, n3};
            const long long st[3] = {1, n1, (long long)n1 * n2};
            float *cur = f, *other = tmp;  // the axes' passes alternate between the two
            for (int ax = 0; ax < 3; ++ax) {
                const double sg = param[ax];
                if (!(sg > 0.0) || len[ax] < 2) continue;
                const int rad = std::max(1, (int)std::ceil(3.0 * sg));
                std::vector<float> hw(2 * rad + 1);
                double tot = 0.0;
                std::vector<double> dw(2 * rad + 1);
                for (int k = -rad; k <= rad; ++k) tot += dw[k + rad] = std::exp(-0.5 * (double)k * k / (sg * sg));
                for (int k = 0; k <= 2 * rad; ++k) hw[k] = (float)(dw[k] / tot);
                if (2 * rad + 1 <= SMOOTH_W) {
                    SmoothW wp;
                    std::copy(hw.begin(), hw.end(), wp.w);
                    const int nb1 = (int)std::max<long long>(1, std::min<long long>((n + 255) / 256, 148 * 32));
                    if (n < (1LL << 31))
                        k_smooth_axis_p<unsigned><<<nb1, 256, 0, s>>>(cur, other, n, (unsigned)st[ax], len[ax], wp, rad);
                    else
                        k_smooth_axis_p<long long><<<nb1, 256, 0, s>>>(cur, other, n, st[ax], len[ax], wp, rad);
                    OWL_LAUNCH_CHECK();
                } else {
                    w.upload(hw.data(), hw.size(), s);
                    k_smooth_axis<<<nb, 256, 0, s>>>(cur, other, n, st[ax], len[ax], w.p, rad);
                    OWL_LAUNCH_CHECK();
                    OWL_CUDA(cudaStreamSynchronize(s));  // w is reused by the next axis
                }
                std::swap(cur, other);
            }
            if (cur != f) OWL_CUDA(cudaMemcpyAsync(f, cur, n * sizeof(float), cudaMemcpyDeviceToDevice, s));
            break;
        }
        case OWL_GRAD_TAPER: {
            int l[6];
            for (int i = 0; i < 6; ++i) l[i] = std::max(0, (int)std::lround(param[i]));
            k_taper<<<nb, 256, 0, s>>>(f, n, n1, n2, n3, l[0], l[1], l[2], l[3], l[4], l[5]);
            OWL_LAUNCH_CHECK();
            break;
        }
        case OWL_GRAD_MASK:
            OWL_CHECK(mask, OWL_ERR_INVALID, "mask needs a mask field");
            k_mul<<<nb, 256, 0, s>>>(f, n, mask, 1.f);
            OWL_LAUNCH_CHECK();
            break;
        case OWL_GRAD_SCALE:
            k_mul<<<nb, 256, 0, s>>>(f, n, nullptr, param[0]);
            OWL_LAUNCH_CHECK();
            break;
        case OWL_GRAD_MAX_BALANCE: {
            float* part = ws.take<float>(nb);
            k_max_part<<<nb, 256, 0, s>>>(f, n, part);
            OWL_LAUNCH_CHECK();
            std::vector<float> hp(nb);
            OWL_CUDA(cudaMemcpyAsync(hp.data(), part, nb * sizeof(float), cudaMemcpyDeviceToHost, s));
            OWL_CUDA(cudaStreamSynchronize(s));
            const float m = *std::max_element(hp.begin(), hp.end());
            if (m != 0.f) {
                k_mul<<<nb, 256, 0, s>>>(f, n, nullptr, 1.f / m);
                OWL_LAUNCH_CHECK();
            }
            break;
        }
        case OWL_GRAD_RMS_BALANCE: {
            double* part = ws.take<double>(1);
            k_slice_sumsq<<<1, 256, 0, s>>>(f, 1, (int)n, 1, 0, part);  // the whole field as one slice
            OWL_LAUNCH_CHECK();
            double ss = 0.0;
            OWL_CUDA(cudaMemcpyAsync(&ss, part, sizeof(double), cudaMemcpyDeviceToHost, s));
            OWL_CUDA(cudaStreamSynchronize(s));
            const double rms = std::sqrt(ss / (double)n);
            if (rms != 0.0) {
                k_mul<<<nb, 256, 0, s>>>(f, n, nullptr, (float)(1.0 / rms));
                OWL_LAUNCH_CHECK();
            }
            break;
        }
        case OWL_GRAD_RMS_BALANCE_AXIS: {
            const int axis = (int)std::lround(param[0]) - 1;
            OWL_CHECK(axis >= 0 && axis <= 2, OWL_ERR_INVALID, "rms balance axis must be 1, 2 or 3");
            int wn = (int)std::lround(param[1]);
            if (wn % 2 == 0) --wn;
            OWL_CHECK(wn >= 1, OWL_ERR_INVALID, "rms balance window must be at least 1 cell");
            const int len[3] = {n1, n2, n3};
            const int L = len[axis];
            DevBuf<double> ss;
            ss.reserve(L);
            k_slice_sumsq<<<L, 256, 0, s>>>(f, n1, n2, n3, axis, ss.p);
            OWL_LAUNCH_CHECK();
            std::vector<double> hs(L);
            OWL_CUDA(cudaMemcpyAsync(hs.data(), ss.p, L * sizeof(double), cudaMemcpyDeviceToHost, s));
            OWL_CUDA(cudaStreamSynchronize(s));
            std::vector<float> hn(L);
            const int hw = (wn - 1) / 2;
            for (int j = 0; j < L; ++j) {
                double acc = 0.0;
                for (int k = std::max(0, j - hw); k <= std::min(L - 1, j + hw); ++k) acc += hs[k];
                hn[j] = (float)std::sqrt(acc);
            }
            DevBuf<float> dn;
            dn.upload(hn.data(), L, s);
            k_div_slice<<<nb, 256, 0, s>>>(f, n, n1, n2, axis, dn.p);
            OWL_LAUNCH_CHECK();
            OWL_CUDA(cudaStreamSynchronize(s));
            break;
        }
        case OWL_GRAD_MEDIAN: {
            int h[3];
            for (int i = 0; i < 3; ++i) h[i] = std::max(0, (int)std::lround(param[i]));
            if (n1 == 1) h[0] = 0;
            if (n2 == 1) h[1] = 0;
            if (n3 == 1) h[2] = 0;
            OWL_CHECK((2 * h[0] + 1) * (2 * h[1] + 1) * (2 * h[2] + 1) <= 343, OWL_ERR_INVALID,
                      "median window above 343 cells");
            float* tmp = ws.take<float>(n);
            k_median<<<nb, 256, 0, s>>>(f, tmp, n1, n2, n3, h[0], h[1], h[2]);
            OWL_LAUNCH_CHECK();
            OWL_CUDA(cudaMemcpyAsync(f, tmp, n * sizeof(float), cudaMemcpyDeviceToDevice, s));
            break;
        }
        default:
            throw OwlError(OWL_ERR_INVALID, "bad gradient processing op");
    }
    OWL_CUDA(cudaStreamSynchronize(s));
}

}  // namespace owl
