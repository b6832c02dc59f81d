// ac2d_res.cuh -- 2D acoustic segments with the state resident in shared memory
// (included by ac2d.cu after the step kernels, inside namespace owl).
//
// A step kernel reads and writes a shot's whole state through L2 twice a step
// and pays a launch boundary for each of its passes. Here one thread-block
// cluster owns one shot for all n steps of a launch: its C CTAs (C = 1,
// 2, 4, 8 or 16) hold consecutive rows of p, vx, vz and the CFS-PML memories in shared memory
// (with the coefficients about 3.1 MB for a 441 x 241 grid, 16 CTAs), each row
// whole, so that x neighbours are always local and only R boundary rows cross
// to the neighbouring CTAs, written into their halo rows (distributed shared
// memory) by the thread that computes them. A step is two phases, each ended by
// the cluster's hardware barrier (0.25 us; no polling):
//   P: the pending explosion taps of the step before, the receivers on one node, then
//      p -= dtbk (dx vx + dz vz)                      -> p rows to both neighbours
//   V: vx -= dtbx dx p, vz -= dtbz dz p               -> vz rows to both neighbours
//      and the receivers between nodes, from their window of 9 x 9 nodes
// Global memory sees only the traces, the stored stencil terms of the STORE
// variant, and the state and coefficients once a launch.
//
// A thread owns H rows x 4 cells: the z arms come from one column window of
// 2R - 1 + H float4 rows held in registers, the x arms from R / 2 + 1 float4
// loads per row, the arithmetic is packed two cells per instruction where the
// operands lie in pairs. What bounds it (counters of seven shots of 401 x 201, 16
// CTAs each): shared-memory wavefronts, 60 % of the cycles of the SMs in use and 66 %
// of the busiest; the barriers, a third of a warp's time (CTA barrier 19 %, the
// release before the cluster's 14 %); issue, 0.31 per cycle and scheduler. The storing
// variant adds its stores to HBM (1.17 TB/s). Measured on B200, us per step against
// the step launches (CUDA graph), 401 x 201: 8 shots 10.5 / 16.1, 32 26.0 / 34.5,
// 64 52.8 / 82.6; one shot of 151 x 101 2.4 / 8.5. Rows of the coefficients in
// registers or read through L2 each step (spills and L1 misses: 8.1 us a wave), and one
// code path with tests for the PML per row (5.1 us with a third more instructions),
// measured slower.
//
// Per cell the arithmetic is that of the one-cell step kernels (ac2d.cu), in the
// same order and rounding: traces, stored terms and states equal theirs to the bit.
#pragma once

constexpr int RES_MAXC = 16;     // CTAs of a cluster (above 8: non-portable size)
constexpr int RES_THREADS = 448;  // (128 registers a thread)
constexpr size_t RES_SMEM = 227 * 1024;

struct Ac2dRes {
    int C;            // CTAs per shot
    int n;            // steps of the launch
    int XG, XP;       // four-cell groups of a row; shared row pitch (4 XG + 2 R floats)
    int GL, GR, GN;   // groups g < GL or g >= GR hold x-PML cells; GN of them
    int zlo;          // storage row of the first resident row (the surface row with a free surface)
    int zb[RES_MAXC + 1];  // first resident row of each CTA, relative to zlo
    const int* inj_last;   // per shot: last step (1-based) with a nonzero amplitude
    const int2* org;       // traces of several taps: storage (x, z) of the window's first tap
    const float* fac;      // and the factors of its weights, [k][trace]: BOX_W along x, BOX_W along z, the trace's weight
                           // (null where no such trace is recorded)
};

__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned map_rank(unsigned addr, int rank) {
    unsigned o;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(o) : "r"(addr), "r"(rank));
    return o;
}
__device__ __forceinline__ void st_cluster4(unsigned addr, const float4& v) {
    // (no memory clobber: only the barrier that follows orders it, and loads of
    // the CTA's own rows may move across it)
    asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w));
}
// two packed floats: one instruction for two cells (each rounded as the scalar operation)
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float a, float b) {
    f32x2 v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b));
    return v;
}
__device__ __forceinline__ float2 unpack2(f32x2 v) {
    float2 f;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
    return f;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f32x2 sub2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
struct F4 {  // four cells as two pairs
    f32x2 a, b;
};
__device__ __forceinline__ F4 ldf4(const float* p) {
    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p);
    return F4{v.x, v.y};
}
__device__ __forceinline__ float4 to_float4(const F4& v) {
    const float2 a = unpack2(v.a), b = unpack2(v.b);
    return make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ float ld_cluster(unsigned addr) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
__device__ __forceinline__ int cluster_rank() {
    int r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// lanes q >= n set to zero (the cells past the right edge stay zero)
__device__ __forceinline__ void zero_tail(float4& v, int n) {
    if (n < 4) {
        v.w = 0.f;
        if (n < 3) v.z = 0.f;
        if (n < 2) v.y = 0.f;
    }
}

// one CTA's rows and its shared-memory arrays
template <int R>
struct ResCta {
    int rank, s, l0, nr;  // l0: first row relative to zlo
    float *p, *vz, *vx;   // p, vz: nr + 2 R rows (R halo rows on each side); vx: nr rows
    float *bk, *bx, *bz;  // coefficients dtbk, dtbx, dtbz: nr rows of 4 XG
    float4 *m1, *m3;      // x memories: [row][GN]
    float4 *m2, *m4;      // z memories: [z-PML row][XG]
    float4 *cxi, *cxh;    // x coefficients of the x-PML groups: a at [2 i], b at [2 i + 1]
    float2 *czi, *czh;    // z coefficients (a, b) of each row, 0 off the z-PML
    // z-PML rows: the first top_i (p) / top_h (v) rows and the rows from bot on
    int top_i, top_h, bot;
    __device__ int slot_i(int l) const { return l < top_i ? l : top_i + l - bot; }
    __device__ int slot_h(int l) const { return l < top_h ? l : top_h + l - bot; }
    __device__ bool pz_i(int l) const { return l < top_i || l >= bot; }
    __device__ bool pz_h(int l) const { return l < top_h || l >= bot; }
};

// floats of shared memory of a CTA of nr rows, of which npi / nph lie in the z-PML of p / v
inline size_t res_fwd_floats(int R, int XG, int XP, int GN, int nr, int npi, int nph) {
    return (size_t)(3 * nr + 4 * R) * XP + (size_t)12 * nr * XG + (size_t)8 * nr * GN + (size_t)4 * (npi + nph) * XG + (size_t)16 * GN +
           (size_t)4 * (nr + 4);
}

template <int R>
__device__ __forceinline__ void res_setup(const Ac2dDev& a, const Ac2dRes& q, float* sm, ResCta<R>& c) {
    c.rank = cluster_rank();
    c.s = blockIdx.y;
    c.l0 = q.zb[c.rank];
    c.nr = q.zb[c.rank + 1] - c.l0;
    const int z0 = q.zlo + c.l0;
    // rows with z < pr (p) / z <= pr (v) at the top (none with a free surface), z >= pr + nz at the bottom
    c.top_i = a.fsurf ? 0 : min(max(a.pr - z0, 0), c.nr);
    c.top_h = a.fsurf ? 0 : min(max(a.pr + 1 - z0, 0), c.nr);
    c.bot = min(max(a.pr + a.nz - z0, 0), c.nr);
    c.p = sm;
    c.vz = c.p + (size_t)(c.nr + 2 * R) * q.XP;
    c.vx = c.vz + (size_t)(c.nr + 2 * R) * q.XP;
    c.bk = c.vx + (size_t)c.nr * q.XP;
    c.bx = c.bk + (size_t)4 * c.nr * q.XG;
    c.bz = c.bx + (size_t)4 * c.nr * q.XG;
    c.m1 = reinterpret_cast<float4*>(c.bz + (size_t)4 * c.nr * q.XG);
    c.m3 = c.m1 + c.nr * q.GN;
    c.m2 = c.m3 + c.nr * q.GN;
    c.m4 = c.m2 + (c.top_i + c.nr - c.bot) * q.XG;
    c.cxi = c.m4 + (c.top_h + c.nr - c.bot) * q.XG;
    c.cxh = c.cxi + 2 * q.GN;
    c.czi = reinterpret_cast<float2*>(c.cxh + 2 * q.GN);
    c.czh = c.czi + c.nr + 4;
}

// whether group g holds x-PML cells, and its place among them
__device__ __forceinline__ bool res_xpml(const Ac2dRes& q, int g, int& i) {
    i = g < q.GL ? g : q.GL + g - q.GR;
    return g < q.GL || g >= q.GR;
}

// coefficient tables, 0 off the PML: there psi stays zero and D unchanged, as
// the step kernels leave them out
template <int R>
__device__ __forceinline__ void res_coefs(const Ac2dDev& a, const Ac2dRes& q, const ResCta<R>& c) {
    float4 *cxi = c.cxi, *cxh = c.cxh;
    for (int l = threadIdx.x; l < c.nr + 4; l += blockDim.x) {
        const int z = q.zlo + c.l0 + l;
        const bool pi = l < c.nr && c.pz_i(l), ph = l < c.nr && c.pz_h(l);
        c.czi[l] = pi ? make_float2(a.azi[z], a.bzi[z]) : make_float2(0.f, 0.f);
        c.czh[l] = ph ? make_float2(a.azh[z], a.bzh[z]) : make_float2(0.f, 0.f);
    }
    for (int i = threadIdx.x; i < q.GN; i += blockDim.x) {
        const int g = i < q.GL ? i : q.GR + i - q.GL;
        float4 ai, bi, ah, bh;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int x = a.x0 + 4 * g + e;
            const bool in = x < a.x1;
            const bool pi = in && pml_int(x, a.pr, a.nx), ph = in && pml_half(x, a.pr, a.nx);
            f4set(ai, e, pi ? a.axi[x] : 0.f);
            f4set(bi, e, pi ? a.bxi[x] : 0.f);
            f4set(ah, e, ph ? a.axh[x] : 0.f);
            f4set(bh, e, ph ? a.bxh[x] : 0.f);
        }
        cxi[2 * i] = ai; cxi[2 * i + 1] = bi;
        cxh[2 * i] = ah; cxh[2 * i + 1] = bh;
    }
}

// p at storage node (z, x) from the shared rows of its owner (0 outside the
// compute region; rows above a free surface mirror with a minus)
template <int R>
__device__ float res_read_p(const Ac2dDev& a, const Ac2dRes& q, const ResCta<R>& c, int z, int x) {
    float sg = 1.f;
    if (z < q.zlo) {
        if (!a.fsurf || z < a.pr - a.P) return 0.f;
        z = 2 * a.pr - z;
        sg = -1.f;
    }
    const int l = z - q.zlo;
    if (l >= q.zb[q.C] || x < a.x0 || x >= a.x1) return 0.f;
    int r = c.rank;
    while (l < q.zb[r]) --r;
    while (l >= q.zb[r + 1]) ++r;
    const float* f = c.p + (size_t)(l - q.zb[r] + R) * q.XP + (x - a.x0) + R;
    return sg * (r == c.rank ? *f : ld_cluster(map_rank(smem_addr(f), r)));
}

// one trace of the shot at step index cur (0-based): p plus the pending
// explosion taps, each trace a sequential sum over its taps
template <int R>
__device__ __noinline__ float res_sample(const Ac2dDev& a, const Ac2dRes& q, int r, bool pend, int cur) {
    extern __shared__ __align__(16) float res_sm[];
    ResCta<R> c;
    res_setup<R>(a, q, res_sm, c);
    float acc = 0.f;
    for (int j = a.pt.smp.ptr[r]; j < a.pt.smp.ptr[r + 1]; ++j) {
        const long long off = a.pt.smp.off[j];
        const int z = (int)(off / a.pitch), x = (int)(off - (long long)z * a.pitch);
        float v = res_read_p<R>(a, q, c, z, x);
        if (pend) v = ac2d_inj(a.pt, c.s, 0, x, z, cur, v);
        acc = acc + v * a.pt.smp.w[j];
    }
    return acc;
}

// The shot's injection items, one tap per thread. The first one's tap stays in
// registers for the launch, its amplitude read a phase ahead; further items are read
// per step, each while the one before is added.
struct ResTap {
    int o;    // shared offset of the thread's tap on the CTA's rows (-1: none)
    float w;
};
struct ResSrc {
    int last;     // last step (1-based) with a nonzero amplitude
    int it, nit;
    bool halo;    // the halo rows take the taps too
    ResTap t;
    float A;
};
template <int R>
__device__ __forceinline__ ResTap res_tap(const Ac2dDev& a, const Ac2dRes& q, const ResCta<R>& c, int it, bool halo) {
    ResTap t{-1, 0.f};
    if (threadIdx.x < BOX_W * BOX_W) {
        const int4 b = __ldg(a.pt.box + it);
        const int l = b.w + (int)threadIdx.x / BOX_W - q.zlo - c.l0, x = b.y + (int)threadIdx.x % BOX_W;
        const int h = halo ? R : 0;
        t.w = __ldg(a.pt.bw + (size_t)it * (BOX_W * BOX_W) + threadIdx.x);
        if (b.x == 0 && l >= -h && l < c.nr + h && x >= a.x0 && x < a.x1 && t.w != 0.f)
            t.o = (l + R) * q.XP + (x - a.x0) + R;
    }
    return t;
}
// items it0 and on of step index ti (0-based), in order
template <int R>
__device__ __noinline__ void res_inject_items(const Ac2dDev& a, const Ac2dRes& q, int it0, int ti, bool halo) {
    extern __shared__ __align__(16) float res_sm[];
    ResCta<R> c;
    res_setup<R>(a, q, res_sm, c);
    const int end = a.pt.item_ptr[c.s + 1], nt = a.pt.nt;
    const float* amp = a.pt.amp + ti;
    ResTap t = res_tap<R>(a, q, c, it0, halo);
    float A = __ldg(amp + (size_t)it0 * nt);
    for (int it = it0; it < end; ++it) {
        const ResTap cur = t;
        const float Ac = A;
        if (it + 1 < end) {
            t = res_tap<R>(a, q, c, it + 1, halo);
            A = __ldg(amp + (size_t)(it + 1) * nt);
        }
        if (cur.o >= 0 && Ac != 0.f) c.p[cur.o] = c.p[cur.o] + Ac * cur.w;
        __syncthreads();
    }
}
template <int R>
__device__ __forceinline__ void res_find_source(const Ac2dDev& a, const Ac2dRes& q, const ResCta<R>& c, bool halo,
                                                ResSrc& src) {
    const Ac2dPt& t = a.pt;
    src.last = q.inj_last[c.s];
    src.it = t.item_ptr[c.s];
    src.nit = t.item_ptr[c.s + 1] - src.it;
    src.halo = halo;
    src.t = ResTap{-1, 0.f};
    src.A = 0.f;
    if (src.nit > 0) src.t = res_tap<R>(a, q, c, src.it, halo);
}
// the taps of step index ti, whose amplitude of the first item is src.A; every
// thread of the CTA calls it, and the rows are complete after it
template <int R>
__device__ __forceinline__ void res_inject(const Ac2dDev& a, const Ac2dRes& q, const ResCta<R>& c, const ResSrc& src,
                                           int ti) {
    if (ti + 1 > src.last) return;
    if (src.t.o >= 0 && src.A != 0.f) c.p[src.t.o] = c.p[src.t.o] + src.A * src.t.w;
    __syncthreads();
    if (src.nit > 1) res_inject_items<R>(a, q, src.it + 1, ti, src.halo);
}

// Receivers of the CTA, up to two per thread, found once per launch (`list`:
// shared scratch of 1 + 2 blockDim ints). A trace of one tap belongs to the CTA of
// its row, one of several to the CTA of its window's middle row: the window then
// lies on the CTA's rows and its halo rows, which hold p of the same step from the
// end of the P phase on.
struct ResRec {  // a trace of one tap on the CTA's rows
    int r;       // trace
    int o;       // shared offset of the tap (-1: none)
    float w;
};
enum { RES_NONE = 0, RES_BOX, RES_NEAR, RES_SPAN };
struct ResWin {  // the others (by address: a step reads them only where there are some)
    int kind[2];  // a window on the CTA's own and halo rows / one that meets the taps of the shot's sources / taps
                  // beyond the CTA's rows
    int r[2];     // trace
    int o[2];     // shared offset of the window's first tap
};
enum { RES_HAS_TAPS = 1, RES_HAS_NEAR = 2 };
// halo rows of p below the CTA's last row that hold p
template <int R>
constexpr int RES_BELOW = R < BOX_W / 2 + 1 ? R : R - 1;
template <int R>
__device__ __forceinline__ int res_local(const Ac2dDev& a, const Ac2dRes& q, const ResCta<R>& c, long long off) {
    const int z = (int)(off / a.pitch), x = (int)(off - (long long)z * a.pitch), l = z - q.zlo - c.l0;
    return l >= 0 && l < c.nr && x >= a.x0 && x < a.x1 ? (l + R) * q.XP + (x - a.x0) + R : -1;
}
// (returns RES_HAS_*: some thread of the CTA has a trace of one tap / some window of
// the shot, on whichever CTA, meets the taps of its sources)
template <int R>
__device__ __noinline__ int res_find_receivers(const Ac2dDev& a, const Ac2dRes& q, ResRec* rec, ResWin* win) {
    extern __shared__ __align__(16) float res_sm[];
    ResCta<R> c;
    res_setup<R>(a, q, res_sm, c);
    int* list = reinterpret_cast<int*>(res_sm);
    if (threadIdx.x == 0) list[0] = 0;
    __syncthreads();
    const Ac2dPt& t = a.pt;
    bool near = false;
    for (int r = t.rec_ptr[c.s] + threadIdx.x; r < t.rec_ptr[c.s + 1]; r += blockDim.x) {
        const int j = t.smp.ptr[r], n = t.smp.ptr[r + 1] - j;
        if (n == 0) continue;  // no taps: the trace is zero
        const int2 g = n == 1 ? make_int2(0, 0) : q.org[r];
        near |= n > 1 && ac2d_inj_near(t, c.s, 1, g.x, g.x + BOX_W, g.y, g.y + BOX_W);
        int l = (n == 1 ? (int)(t.smp.off[j] / a.pitch) : g.y + BOX_W / 2) - q.zlo;
        l = min(max(l, 0), q.zb[q.C] - 1) - c.l0;
        if (l >= 0 && l < c.nr) {
            const int k = atomicAdd(list, 1);
            if (k < 2 * (int)blockDim.x) list[1 + k] = r;
        }
    }
    __syncthreads();
    const int count = list[0];
    for (int e = 0; e < 2; ++e) {
        const int k = threadIdx.x + e * blockDim.x;
        rec[e] = ResRec{0, -1, 0.f};
        win->kind[e] = RES_NONE;
        if (k < count) {
            const int r = list[1 + k], j = t.smp.ptr[r];
            win->r[e] = rec[e].r = r;
            if (t.smp.ptr[r + 1] == j + 1) {
                rec[e].w = t.smp.w[j];
                rec[e].o = res_local<R>(a, q, c, t.smp.off[j]);
                if (rec[e].o < 0) win->kind[e] = RES_SPAN;
            } else {
                const int2 g = q.org[r];
                const int l = g.y - q.zlo - c.l0, x = g.x - a.x0;
                win->o[e] = (l + R) * q.XP + x + R;
                win->kind[e] = l < -R || l + BOX_W > c.nr + RES_BELOW<R> || x < -R || x + BOX_W > 4 * q.XG + R ? RES_SPAN
                               : ac2d_inj_near(t, c.s, 1, g.x, g.x + BOX_W, g.y, g.y + BOX_W)                  ? RES_NEAR
                                                                                                               : RES_BOX;
            }
        }
    }
    const bool taps = __syncthreads_or(rec[0].o >= 0 || rec[1].o >= 0);
    near = __syncthreads_or(near);
    return (taps ? RES_HAS_TAPS : 0) | (near ? RES_HAS_NEAR : 0);
}
// a trace of several taps from the CTA's own and halo rows: the taps in order (z
// outer), weight by weight as the tables have them. The window's values lie at
// fixed offsets, the factors are read coalesced over the traces (19 floats each) and
// nothing goes through the kernel's parameters. A step of a one-shot 100 x 80 grid
// takes 2.5 us with traces on nodes, 3.2 us with 20 or 100 such ones and 4.8 us while
// sources that their windows meet are active; through the taps' own tables, one tap
// after another with its divisions, it took 61 us (13.8 us step by step).
__device__ __noinline__ float res_box(const float* __restrict__ f, int n, int XP, int o) {
    extern __shared__ __align__(16) float res_sm[];
    float fx[BOX_W], fz[BOX_W];
#pragma unroll
    for (int i = 0; i < BOX_W; ++i) {
        fx[i] = __ldg(f + (size_t)i * n);
        fz[i] = __ldg(f + (size_t)(BOX_W + i) * n);
    }
    const float wt = __ldg(f + (size_t)2 * BOX_W * n);
    float acc = 0.f;
#pragma unroll
    for (int k = 0; k < BOX_W; ++k) {
        float v[BOX_W];
#pragma unroll
        for (int i = 0; i < BOX_W; ++i) v[i] = res_sm[o + k * XP + i];
#pragma unroll
        for (int i = 0; i < BOX_W; ++i) {
            const float w = __fmul_rn(__fmul_rn(fx[i], fz[k]), wt);
            if (w != 0.f) acc = acc + v[i] * w;
        }
    }
    return acc;
}
// the thread's traces of several taps at row `row`: from the V phase's p (halo rows
// complete), except those that meet the taps of an active source (pend), and after
// the injection into own and halo rows (met) only those
template <int R>
__device__ __noinline__ void res_windows(const Ac2dDev& a, const Ac2dRes& q, const ResWin* win, int row, bool pend,
                                         bool met) {
    for (int e = 0; e < 2; ++e) {
        const int kind = win->kind[e], r = win->r[e];
        float* out = a.pt.rec + (size_t)row * a.pt.rtot + r;
        if (met ? kind == RES_NEAR : kind == RES_BOX || (kind == RES_NEAR && !pend))
            *out = res_box(q.fac + r, a.pt.rtot, q.XP, win->o[e]);
        else if (!met && kind == RES_SPAN)
            *out = res_sample<R>(a, q, r, pend, row - 1);
    }
}
// record the CTA's traces of one tap, from p with the step's injection, as trace
// row `row`; complete (for every thread) after it
__device__ __forceinline__ void res_record(const Ac2dDev& a, const float* p, const ResRec (&rec)[2], int row) {
#pragma unroll
    for (int e = 0; e < 2; ++e)
        if (rec[e].o >= 0) a.pt.rec[(size_t)row * a.pt.rtot + rec[e].r] = 0.f + p[rec[e].o] * rec[e].w;
    __syncthreads();
}

// four cells of a plane of the global state, the first n of them inside the grid
__device__ __forceinline__ float4 res_ld_plane(const float* f, int pitch, int z, int x, int n) {
    float4 v = ld4(f + (long long)z * pitch + x);
    zero_tail(v, n);
    return v;
}

template <int R>
__device__ __forceinline__ void res_load_state(const Ac2dDev& a, const Ac2dRes& q, const ResCta<R>& c) {
    const long long so = c.s * a.sst;
    const int z0 = q.zlo + c.l0, zend = q.zlo + q.zb[q.C];
    for (int i = threadIdx.x; i < (c.nr + 2 * R) * q.XP / 4; i += blockDim.x) {
        const int l = i / (q.XP / 4) - R, col = 4 * (i % (q.XP / 4)) - R;  // column relative to x0
        float4 p = make_float4(0.f, 0.f, 0.f, 0.f), v = p;
        if (col >= 0 && col < 4 * q.XG && z0 + l >= q.zlo && z0 + l < zend) {
            const int n = min(4, a.x1 - a.x0 - col);
            p = res_ld_plane(a.p + so, a.pitch, z0 + l, a.x0 + col, n);
            v = res_ld_plane(a.vz + so, a.pitch, z0 + l, a.x0 + col, n);
        }
        *reinterpret_cast<float4*>(c.p + (size_t)(l + R) * q.XP + col + R) = p;
        *reinterpret_cast<float4*>(c.vz + (size_t)(l + R) * q.XP + col + R) = v;
        if (l >= 0 && l < c.nr) {
            float4 w = make_float4(0.f, 0.f, 0.f, 0.f);
            if (col >= 0 && col < 4 * q.XG)
                w = res_ld_plane(a.vx + so, a.pitch, z0 + l, a.x0 + col, min(4, a.x1 - a.x0 - col));
            *reinterpret_cast<float4*>(c.vx + (size_t)l * q.XP + col + R) = w;
        }
    }
    for (int i = threadIdx.x; i < c.nr * q.XG; i += blockDim.x) {
        const int l = i / q.XG, g = i % q.XG, z = z0 + l, x = a.x0 + 4 * g, n = min(4, a.x1 - x);
        const long long o = (long long)z * a.pitch + x;
        *reinterpret_cast<float4*>(c.bk + 4 * i) = ldg4(a.dtbk + o);
        *reinterpret_cast<float4*>(c.bx + 4 * i) = ldg4(a.dtbx + o);
        *reinterpret_cast<float4*>(c.bz + 4 * i) = ldg4(a.dtbz + o);
        int gi;
        if (res_xpml(q, g, gi)) {
            c.m1[l * q.GN + gi] = res_ld_plane(a.m1 + so, a.pitch, z, x, n);
            c.m3[l * q.GN + gi] = res_ld_plane(a.m3 + so, a.pitch, z, x, n);
        }
        if (c.pz_i(l)) c.m2[c.slot_i(l) * q.XG + g] = res_ld_plane(a.m2 + so, a.pitch, z, x, n);
        if (c.pz_h(l)) c.m4[c.slot_h(l) * q.XG + g] = res_ld_plane(a.m4 + so, a.pitch, z, x, n);
    }
}

// the CTA's rows back to the global state; mirror: only the rows above a free
// surface (before the last injection, as the p kernel writes them)
template <int R>
__device__ __forceinline__ void res_save_mirror(const Ac2dDev& a, const Ac2dRes& q, const ResCta<R>& c) {
    const long long so = c.s * a.sst;
    for (int i = threadIdx.x; i < c.nr * q.XG; i += blockDim.x) {
        const int l = i / q.XG, g = i % q.XG, z = q.zlo + c.l0 + l, x = a.x0 + 4 * g;
        if (z <= a.pr || z > a.pr + a.P) continue;
        const float4 v = *reinterpret_cast<const float4*>(c.p + (size_t)(l + R) * q.XP + 4 * g + R);
        st4n(a.p + so + (long long)(2 * a.pr - z) * a.pitch + x, make_float4(-v.x, -v.y, -v.z, -v.w), min(4, a.x1 - x));
    }
}
template <int R>
__device__ __forceinline__ void res_save_state(const Ac2dDev& a, const Ac2dRes& q, const ResCta<R>& c) {
    const long long so = c.s * a.sst;
    for (int i = threadIdx.x; i < c.nr * q.XG; i += blockDim.x) {
        const int l = i / q.XG, g = i % q.XG, z = q.zlo + c.l0 + l, x = a.x0 + 4 * g, n = min(4, a.x1 - x);
        const long long o = so + (long long)z * a.pitch + x;
        st4n(a.p + o, *reinterpret_cast<const float4*>(c.p + (size_t)(l + R) * q.XP + 4 * g + R), n);
        st4n(a.vz + o, *reinterpret_cast<const float4*>(c.vz + (size_t)(l + R) * q.XP + 4 * g + R), n);
        st4n(a.vx + o, *reinterpret_cast<const float4*>(c.vx + (size_t)l * q.XP + 4 * g + R), n);
        int gi;
        if (res_xpml(q, g, gi)) {
            st4n(a.m1 + o, c.m1[l * q.GN + gi], n);
            st4n(a.m3 + o, c.m3[l * q.GN + gi], n);
        }
        if (c.pz_i(l)) st4n(a.m2 + o, c.m2[c.slot_i(l) * q.XG + g], n);
        if (c.pz_h(l)) st4n(a.m4 + o, c.m4[c.slot_h(l) * q.XG + g], n);
    }
}

// What a thread needs of its H rows x 4 cells: constant over the launch for a
// thread's only item, so that a step spends no instructions on it. `kind` says
// which form of the updates the item needs: each form is one basic block (its
// stores predicated), so that a row's reads are in flight during the row before.
enum { RI_X = 1, RI_Z = 2 };  // x-PML or ragged cells; z-PML, ragged or surface rows
template <int R, int H>
struct ResItem {
    int o;                // shared offset of (row lb, cell 4 g) in p and vz; vx: o - R XP
    int co;               // offset in the coefficients
    int go;               // offset in a plane of the global state
    int n;                // cells
    int xm, xc;           // x-PML group: its memories of row lb (float4; 0 off the x-PML), its coefficients (-1)
    int lb;               // first row
    int zi, zh;           // z memories of row lb (float4)
    unsigned rows, live;  // bit h: row lb + h exists; and is updated (not a surface row)
    unsigned pi, ph;      // bit h: the row lies in the z-PML of p / of vz
    unsigned up, dp, uv, dv;  // bit h: the row goes to the p halo of the CTA above / below, to its vz halo
    int kind;
};
template <int R, int H>
__device__ __forceinline__ ResItem<R, H> res_item(const Ac2dDev& a, const Ac2dRes& q, const ResCta<R>& c, int it) {
    ResItem<R, H> t;
    // items off the x-PML first, so that few warps hold x-PML work
    const int ni = q.XG - q.GN, ch = (c.nr + H - 1) / H;
    int g;
    if (it < ni * ch) {
        g = q.GL + it % ni;
        t.lb = it / ni * H;
    } else {
        const int i = (it - ni * ch) % q.GN;
        g = i < q.GL ? i : q.GR + i - q.GL;
        t.lb = (it - ni * ch) / q.GN * H;
    }
    const int x = a.x0 + 4 * g;
    t.n = min(4, a.x1 - x);
    t.o = (t.lb + R) * q.XP + 4 * g + R;
    t.co = 4 * (t.lb * q.XG + g);
    t.go = (q.zlo + c.l0 + t.lb) * a.pitch + x;
    int gi;
    const bool px = res_xpml(q, g, gi);
    t.xm = px ? t.lb * q.GN + gi : 0;
    t.xc = px ? gi : -1;
    // (the rows of one item never hold z-PML rows of both ends: the model has at least eight rows)
    t.zi = (t.lb < c.top_i ? t.lb : c.top_i + t.lb - c.bot) * q.XG + g;
    t.zh = (t.lb < c.top_h ? t.lb : c.top_h + t.lb - c.bot) * q.XG + g;
    t.rows = t.live = t.pi = t.ph = t.up = t.dp = t.uv = t.dv = 0;
#pragma unroll
    for (int h = 0; h < H; ++h) {
        const int l = t.lb + h;
        if (l >= c.nr) break;
        t.rows |= 1u << h;
        if (!(a.fsurf && c.rank == 0 && l == 0)) t.live |= 1u << h;
        if (c.pz_i(l)) t.pi |= 1u << h;
        if (c.pz_h(l)) t.ph |= 1u << h;
        // p: my rows 0 .. R - 2 follow the CTA above (where traces have windows, all rows that those may reach), my
        // last R rows precede the CTA below;
        // vz: my rows 0 .. R - 1 follow the CTA above, my last R - 1 rows precede the CTA below
        if (c.rank > 0 && l < (q.fac ? RES_BELOW<R> : R - 1)) t.up |= 1u << h;
        if (c.rank > 0 && l < R) t.uv |= 1u << h;
        if (c.rank + 1 < q.C && l >= c.nr - R) t.dp |= 1u << h;
        if (c.rank + 1 < q.C && l > c.nr - R) t.dv |= 1u << h;
    }
    t.kind = (px || t.n < 4 ? RI_X : 0) | (t.pi | t.ph || t.live != (1u << H) - 1 ? RI_Z : 0);
    return t;
}

// The updates keep the negated derivative (its scale is -1 / dx), so that the
// last operation is a plain multiply-add; negation changes no rounding.
// D' = D + psi with psi = a D + b psi_old for four cells, d = -D: rounded as
// the one-cell step kernels' expressions are.
__device__ __forceinline__ F4 res_pml4(const F4& d, const float4& a, const float4& b, float4& m) {
    const float4 v = to_float4(d);
    m.x = __fmaf_rn(b.x, m.x, -__fmul_rn(a.x, v.x));
    m.y = __fmaf_rn(b.y, m.y, -__fmul_rn(a.y, v.y));
    m.z = __fmaf_rn(b.z, m.z, -__fmul_rn(a.z, v.z));
    m.w = __fmaf_rn(b.w, m.w, -__fmul_rn(a.w, v.w));
    return F4{pack2(__fsub_rn(v.x, m.x), __fsub_rn(v.y, m.y)), pack2(__fsub_rn(v.z, m.z), __fsub_rn(v.w, m.w))};
}
// sums of c_k (f(+) - f(-)) along x: the cells' window w = f[x - R .. x + R + 3];
// S: 0 the nodes x + k, x + 1 - k, 1 the nodes x + k - 1, x - k
template <int R, int S>
__device__ __forceinline__ F4 res_arm_x(const float* w, const f32x2 (&ck)[R]) {
    F4 s{0ull, 0ull};
#pragma unroll
    for (int k = 1; k <= R; ++k) {
        float d[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) d[e] = w[R + e + k - S] - w[R + e + 1 - k - S];
        s.a = fma2(ck[k - 1], pack2(d[0], d[1]), s.a);
        s.b = fma2(ck[k - 1], pack2(d[2], d[3]), s.b);
    }
    return s;
}
// the same along z: rows hi + (k - 1) and lo - (k - 1) of the window
template <int R>
__device__ __forceinline__ F4 res_arm_z(const F4* hi, const F4* lo, const f32x2 (&ck)[R]) {
    F4 s{0ull, 0ull};
#pragma unroll
    for (int k = 1; k <= R; ++k) {
        s.a = fma2(ck[k - 1], sub2(hi[k - 1].a, lo[1 - k].a), s.a);
        s.b = fma2(ck[k - 1], sub2(hi[k - 1].b, lo[1 - k].b), s.b);
    }
    return s;
}
// c v, rounded by itself (a packed product followed by a packed sum would be
// contracted to one rounding; a multiply-add with zero is not)
__device__ __forceinline__ F4 res_scale(f32x2 c, const F4& v) { return F4{fma2(c, v.a, 0ull), fma2(c, v.b, 0ull)}; }
__device__ __forceinline__ void put4(float* w, const F4& v) {
    const float4 f = to_float4(v);
    w[0] = f.x; w[1] = f.y; w[2] = f.z; w[3] = f.w;
}
__device__ __forceinline__ float4 neg4(const F4& v) {
    const float4 f = to_float4(v);
    return make_float4(-f.x, -f.y, -f.z, -f.w);
}

// the item's rows that neighbouring CTAs read, into their halo rows
template <int R, int H>
__device__ __forceinline__ void res_push(const ResItem<R, H>& t, const float* f, int XP, unsigned ub, unsigned db,
                                         unsigned up, unsigned dn) {
#pragma unroll
    for (int h = 0; h < H; ++h) {
        const float4 v = ld4(f + t.o + h * XP);
        if (ub >> h & 1) st_cluster4(up + 4u * (unsigned)(t.o + h * XP), v);
        if (db >> h & 1) st_cluster4(dn + 4u * (unsigned)(t.o + h * XP), v);
    }
}

// p update of an item's rows (K: RI_* forms)
template <int R, int H, bool STORE, int K>
__device__ __forceinline__ void res_p_rows(const Ac2dDev& a, const Ac2dRes& q, const ResCta<R>& c,
                                           const ResItem<R, H>& t, const f32x2 (&ck)[R], long long slot,
                                           float* __restrict__ p, const float* __restrict__ vx,
                                           const float* __restrict__ vz, float4* __restrict__ m1,
                                           float4* __restrict__ m2) {
    const int XP = q.XP;
    const f32x2 nix = pack2(-a.idx, -a.idx), niz = pack2(-a.idz, -a.idz);
    float4 ax = make_float4(0.f, 0.f, 0.f, 0.f), bx = ax;
    if ((K & RI_X) && t.xc >= 0) {
        ax = c.cxi[2 * t.xc];
        bx = c.cxi[2 * t.xc + 1];
    }
    F4 w[2 * R - 1 + H];  // vz rows lb - R + 1 ..
#pragma unroll
    for (int j = 0; j < 2 * R - 1; ++j) w[j] = ldf4(vz + t.o + (j - R + 1) * XP);
#pragma unroll
    for (int h = 0; h < H; ++h) {
        // (rows past the CTA's last read rows that exist in shared memory; nothing of them is stored)
        const bool on = !(K & RI_Z) || (t.live >> h & 1);
        w[h + 2 * R - 1] = ldf4(vz + t.o + (h + R) * XP);
        float wx[2 * R + 4];
#pragma unroll
        for (int e = 0; e < R / 2 + 1; ++e) put4(wx + 4 * e, ldf4(vx + t.o + (h - R) * XP - R + 4 * e));
        const F4 p0 = ldf4(p + t.o + h * XP), bk = ldf4(c.bk + t.co + 4 * h * q.XG);
        F4 gx = res_scale(nix, res_arm_x<R, 0>(wx, ck));
        F4 gz = res_scale(niz, res_arm_z<R>(w + h + R, w + h + R - 1, ck));
        if (K & RI_X) {
            float4 m = m1[t.xm + h * q.GN];
            gx = res_pml4(gx, ax, bx, m);
            if (t.xc >= 0 && on) m1[t.xm + h * q.GN] = m;
        }
        if (K & RI_Z) {
            const bool pz = t.pi >> h & 1;
            const float2 cz = c.czi[t.lb + h];
            float4 m = make_float4(0.f, 0.f, 0.f, 0.f);
            if (pz) m = m2[t.zi + h * q.XG];
            gz = res_pml4(gz, make_float4(cz.x, cz.x, cz.x, cz.x), make_float4(cz.y, cz.y, cz.y, cz.y), m);
            if (pz) m2[t.zi + h * q.XG] = m;
        }
        const F4 gg{add2(gx.a, gz.a), add2(gx.b, gz.b)};
        float4 pn = to_float4(F4{fma2(bk.a, gg.a, p0.a), fma2(bk.b, gg.b, p0.b)});
        if (K & RI_X) zero_tail(pn, t.n);
        if (on) *reinterpret_cast<float4*>(p + t.o + h * XP) = pn;
        if (STORE && on) st4n_cs(a.Sp + slot + c.s * a.fs + t.go + h * a.pitch, neg4(gg), K & RI_X ? t.n : 4);
    }
}
template <int R, int H, bool STORE>
__device__ __forceinline__ void res_p_item(const Ac2dDev& a, const Ac2dRes& q, const ResCta<R>& c,
                                           const ResItem<R, H>& t, int kind, const f32x2 (&ck)[R], long long slot,
                                           unsigned up, unsigned dn) {
    if (kind == 0) res_p_rows<R, H, STORE, 0>(a, q, c, t, ck, slot, c.p, c.vx, c.vz, c.m1, c.m2);
    else if (kind == RI_X) res_p_rows<R, H, STORE, RI_X>(a, q, c, t, ck, slot, c.p, c.vx, c.vz, c.m1, c.m2);
    else if (kind == RI_Z) res_p_rows<R, H, STORE, RI_Z>(a, q, c, t, ck, slot, c.p, c.vx, c.vz, c.m1, c.m2);
    else res_p_rows<R, H, STORE, RI_X | RI_Z>(a, q, c, t, ck, slot, c.p, c.vx, c.vz, c.m1, c.m2);
    if (t.up | t.dp) res_push<R, H>(t, c.p, q.XP, t.up, t.dp, up, dn);
    if (a.fsurf && c.rank == 0 && t.lb <= R) {
        // rows above the surface mirror with a minus
#pragma unroll
        for (int h = 0; h < H; ++h) {
            const int l = t.lb + h;
            if (l < 1 || l > R) continue;
            const float4 v = ld4(c.p + t.o + h * q.XP);
            *reinterpret_cast<float4*>(c.p + t.o + (h - 2 * l) * q.XP) = make_float4(-v.x, -v.y, -v.z, -v.w);
        }
    }
}

// velocity update of an item's rows
template <int R, int H, bool STORE, int K>
__device__ __forceinline__ void res_v_rows(const Ac2dDev& a, const Ac2dRes& q, const ResCta<R>& c,
                                           const ResItem<R, H>& t, const f32x2 (&ck)[R], long long slot,
                                           const float* __restrict__ p, float* __restrict__ vx,
                                           float* __restrict__ vz, float4* __restrict__ m3,
                                           float4* __restrict__ m4) {
    const int XP = q.XP;
    const f32x2 nix = pack2(-a.idx, -a.idx), niz = pack2(-a.idz, -a.idz);
    float4 ax = make_float4(0.f, 0.f, 0.f, 0.f), bxx = ax;
    if ((K & RI_X) && t.xc >= 0) {
        ax = c.cxh[2 * t.xc];
        bxx = c.cxh[2 * t.xc + 1];
    }
    F4 w[2 * R - 1 + H];  // p rows lb - R ..
#pragma unroll
    for (int j = 0; j < 2 * R - 1; ++j) w[j] = ldf4(p + t.o + (j - R) * XP);
#pragma unroll
    for (int h = 0; h < H; ++h) {
        const bool row = !(K & RI_Z) || (t.rows >> h & 1), on = !(K & RI_Z) || (t.live >> h & 1);
        w[h + 2 * R - 1] = ldf4(p + t.o + (h + R - 1) * XP);
        float wx[2 * R + 4];
#pragma unroll
        for (int e = 0; e < R / 2 + 1; ++e)
            put4(wx + 4 * e, e == R / 4 ? w[h + R] : ldf4(p + t.o + h * XP - R + 4 * e));
        const F4 vx0 = ldf4(vx + t.o + (h - R) * XP), vz0 = ldf4(vz + t.o + h * XP);
        const F4 bx = ldf4(c.bx + t.co + 4 * h * q.XG), bz = ldf4(c.bz + t.co + 4 * h * q.XG);
        F4 gx = res_scale(nix, res_arm_x<R, 1>(wx, ck));
        F4 gz = res_scale(niz, res_arm_z<R>(w + h + R, w + h + R - 1, ck));
        if (K & RI_X) {
            float4 m = m3[t.xm + h * q.GN];
            gx = res_pml4(gx, ax, bxx, m);
            if (t.xc >= 0 && row) m3[t.xm + h * q.GN] = m;
        }
        if (K & RI_Z) {
            const bool pz = t.ph >> h & 1;
            const float2 cz = c.czh[t.lb + h];
            float4 m = make_float4(0.f, 0.f, 0.f, 0.f);
            if (pz) m = m4[t.zh + h * q.XG];
            gz = res_pml4(gz, make_float4(cz.x, cz.x, cz.x, cz.x), make_float4(cz.y, cz.y, cz.y, cz.y), m);
            if (pz) m4[t.zh + h * q.XG] = m;
        }
        float4 xn = to_float4(F4{fma2(bx.a, gx.a, vx0.a), fma2(bx.b, gx.b, vx0.b)});
        float4 zn = to_float4(F4{fma2(bz.a, gz.a, vz0.a), fma2(bz.b, gz.b, vz0.b)});
        if (K & RI_X) {
            zero_tail(xn, t.n);
            zero_tail(zn, t.n);
        }
        if (row) *reinterpret_cast<float4*>(vx + t.o + (h - R) * XP) = xn;
        if (on) *reinterpret_cast<float4*>(vz + t.o + h * XP) = zn;
        if (STORE) {
            const long long so = slot + c.s * a.fs + t.go + h * a.pitch;
            if (row) st4n_cs(a.Svx + so, neg4(gx), K & RI_X ? t.n : 4);
            if (on) st4n_cs(a.Svz + so, neg4(gz), K & RI_X ? t.n : 4);
        }
    }
}
template <int R, int H, bool STORE>
__device__ __forceinline__ void res_v_item(const Ac2dDev& a, const Ac2dRes& q, const ResCta<R>& c,
                                           const ResItem<R, H>& t, int kind, const f32x2 (&ck)[R], long long slot,
                                           unsigned up, unsigned dn) {
    if (kind == 0) res_v_rows<R, H, STORE, 0>(a, q, c, t, ck, slot, c.p, c.vx, c.vz, c.m3, c.m4);
    else if (kind == RI_X) res_v_rows<R, H, STORE, RI_X>(a, q, c, t, ck, slot, c.p, c.vx, c.vz, c.m3, c.m4);
    else if (kind == RI_Z) res_v_rows<R, H, STORE, RI_Z>(a, q, c, t, ck, slot, c.p, c.vx, c.vz, c.m3, c.m4);
    else res_v_rows<R, H, STORE, RI_X | RI_Z>(a, q, c, t, ck, slot, c.p, c.vx, c.vz, c.m3, c.m4);
    if (t.uv | t.dv) res_push<R, H>(t, c.vz, q.XP, t.uv, t.dv, up, dn);
}

// ONE: every item of the CTA has its own thread; SMP: traces are recorded
template <int R, int H, bool STORE, bool ONE, bool SMP>
__global__ void __launch_bounds__(RES_THREADS, 1) k_ac2d_fwd_res(const __grid_constant__ Ac2dDev a,
                                                                 const __grid_constant__ Ac2dRes q) {
    extern __shared__ __align__(16) float res_sm[];
    ResCta<R> c;
    res_setup<R>(a, q, res_sm, c);
    const int cur0 = *a.d_step;
    ResRec found[2];
    ResWin win;
    int has = 0;
    if (SMP) has = res_find_receivers<R>(a, q, found, &win);
    ResRec rec[2];
    if (SMP) {
        rec[0] = found[0];
        rec[1] = found[1];
    }
    const bool taps = has & RES_HAS_TAPS, near = has & RES_HAS_NEAR;
    const bool wins = SMP && (win.kind[0] != RES_NONE || win.kind[1] != RES_NONE);  // the thread has traces of several taps
    ResSrc src;
    res_find_source<R>(a, q, c, near, src);
    const float* amp = a.pt.amp + (size_t)src.it * a.pt.nt;
    res_coefs<R>(a, q, c);
    res_load_state<R>(a, q, c);
    // the neighbours' p and vz arrays (p first, then vz, as in res_setup)
    const int ru = max(c.rank - 1, 0), rd = min(c.rank + 1, q.C - 1);
    const int nup = q.zb[ru + 1] - q.zb[ru], ndn = q.zb[rd + 1] - q.zb[rd];
    const unsigned n_up = map_rank(smem_addr(res_sm), ru), n_dn = map_rank(smem_addr(res_sm), rd);
    // where row l of this CTA is row nup + l of the CTA above, l - nr of the one below
    const unsigned p_up = n_up + 4u * (unsigned)(nup * q.XP), p_dn = n_dn - 4u * (unsigned)(c.nr * q.XP);
    const unsigned v_up = p_up + 4u * (unsigned)((nup + 2 * R) * q.XP), v_dn = p_dn + 4u * (unsigned)((ndn + 2 * R) * q.XP);
    f32x2 ck[R];
#pragma unroll
    for (int k = 0; k < R; ++k) ck[k] = pack2(c_fd2[k], c_fd2[k]);
    // the thread's first item (further ones when the block has fewer threads)
    const int items = q.XG * ((c.nr + H - 1) / H);
    const ResItem<R, H> t0 = res_item<R, H>(a, q, c, threadIdx.x);
    // (decided per warp, so that a warp runs one form of the updates)
    const int kind = __reduce_or_sync(0xffffffffu, (int)threadIdx.x < items ? (unsigned)t0.kind : 0u);
    cluster_arrive();
    for (int i = 0; i < q.n; ++i) {
        const int cur = cur0 + i;
        const long long slot = STORE ? (long long)(cur % a.k) * a.sslot : 0;
        cluster_wait();
        // explosion sources, then receivers, of the step before; where windows meet the sources' taps, the taps go
        // into the halo rows too (each CTA adds the same), which the neighbours' next rows may replace only after that
        if (i > 0) {
            const bool meet = near && cur <= src.last;
            res_inject<R>(a, q, c, src, cur - 1);
            if (taps) res_record(a, c.p, rec, cur);
            if (meet) {
                if (wins) res_windows<R>(a, q, &win, cur, true, true);
                cluster_arrive();
                cluster_wait();
            }
        }
        if (ONE) {
            if ((int)threadIdx.x < items) res_p_item<R, H, STORE>(a, q, c, t0, kind, ck, slot, p_up, p_dn);
        } else {
            for (int it = threadIdx.x; it < items; it += blockDim.x) {
                const ResItem<R, H> t = res_item<R, H>(a, q, c, it);
                res_p_item<R, H, STORE>(a, q, c, t, t.kind, ck, slot, p_up, p_dn);
            }
        }
        cluster_arrive();
        if (cur + 1 <= src.last && src.nit > 0) src.A = __ldg(amp + cur);
        cluster_wait();
        if (SMP && wins && cur + 2 <= a.pt.nt) res_windows<R>(a, q, &win, cur + 1, cur + 1 <= src.last, false);
        if (ONE) {
            if ((int)threadIdx.x < items) res_v_item<R, H, STORE>(a, q, c, t0, kind, ck, slot, v_up, v_dn);
        } else {
            for (int it = threadIdx.x; it < items; it += blockDim.x) {
                const ResItem<R, H> t = res_item<R, H>(a, q, c, it);
                res_v_item<R, H, STORE>(a, q, c, t, t.kind, ck, slot, v_up, v_dn);
            }
        }
        cluster_arrive();
    }
    cluster_wait();
    if (a.fsurf) res_save_mirror<R>(a, q, c);
    __syncthreads();
    res_inject<R>(a, q, c, src, cur0 + q.n - 1);
    if (SMP && cur0 + q.n + 1 <= a.pt.nt) {
        if (taps) res_record(a, c.p, rec, cur0 + q.n);
        if (near && wins && cur0 + q.n <= src.last) res_windows<R>(a, q, &win, cur0 + q.n, true, true);
    }
    res_save_state<R>(a, q, c);
    tick_last_block(a.d_step, a.pt.d_done, q.n);
}
