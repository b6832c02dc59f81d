// common.cuh -- shared host/device utilities of the B200 SSG library.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <cstdio>
#include <cstring>
#include <stdexcept>
#include <string>
#include <vector>

#include "../../include/owl_ssg.h"

namespace owl {

// ----------------------------------------------------------------------------
// errors: every failure becomes an OwlError carrying an ABI status code; the
// C entry points catch it and return the code (never abort the process).
// ----------------------------------------------------------------------------
struct OwlError : std::runtime_error {
    int code;
    OwlError(int c, const std::string& m) : std::runtime_error(m), code(c) {}
};

void set_last_error(const std::string& msg);

#define OWL_CUDA(call)                                                                           \
    do {                                                                                         \
        cudaError_t e_ = (call);                                                                 \
        if (e_ != cudaSuccess) {                                                                 \
            int code_ = (e_ == cudaErrorMemoryAllocation) ? OWL_ERR_OOM : OWL_ERR_CUDA;          \
            throw ::owl::OwlError(code_, std::string(#call) + ": " + cudaGetErrorString(e_) +    \
                                             " (" __FILE__ ":" + std::to_string(__LINE__) + ")"); \
        }                                                                                        \
    } while (0)

#define OWL_CHECK(cond, code, msg)                              \
    do {                                                        \
        if (!(cond)) throw ::owl::OwlError((code), (msg));      \
    } while (0)

#define OWL_LAUNCH_CHECK() OWL_CUDA(cudaGetLastError())

// ----------------------------------------------------------------------------
// Programmatic dependent launch: a kernel launched with launch_pdl may start
// while the kernel before it on the stream drains; it must call pdl_prologue()
// before its first global read (griddepcontrol.wait returns once the previous
// grid has completed and its writes are visible), and the call also lets the
// next kernel be scheduled. OWL_NO_PDL=1 in the environment launches plainly.
// ----------------------------------------------------------------------------
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_prologue() {
    pdl_trigger();
    pdl_wait();
}

// barrier over the CTAs of a thread-block cluster: what every thread wrote
// before it (global or shared memory) is visible to every thread after it (not the
// .aligned form: the threads of a warp may come from loops of different lengths)
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}

bool pdl_enabled();

// cluster: dimensions of the thread-block clusters
template <typename... KArgs, typename... Args>
void launch_pdl_cluster(void (*k)(KArgs...), dim3 grid, dim3 block, dim3 cluster, size_t smem, cudaStream_t s,
                        Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (cluster.x * cluster.y * cluster.z > 1) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = cluster.x;
        attr[n].val.clusterDim.y = cluster.y;
        attr[n].val.clusterDim.z = cluster.z;
        ++n;
    }
    if (pdl_enabled()) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n].val.programmaticStreamSerializationAllowed = 1;
        ++n;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    OWL_CUDA(cudaLaunchKernelEx(&cfg, k, static_cast<KArgs>(args)...));
}
template <typename... KArgs, typename... Args>
void launch_pdl(void (*k)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, Args... args) {
    launch_pdl_cluster(k, grid, block, dim3(1, 1, 1), smem, s, args...);
}

// frees the idle workspaces of the current device (workspace.cu); the bytes they hold
void workspace_trim();
size_t workspace_idle_bytes();

// ----------------------------------------------------------------------------
// grow-only device buffer. Keeping the pointer stable across calls lets the
// captured CUDA graphs be replayed without re-instantiation.
// ----------------------------------------------------------------------------
template <typename T>
struct DevBuf {
    T* p = nullptr;
    size_t n = 0;  // capacity in elements
    DevBuf() = default;
    DevBuf(const DevBuf&) = delete;
    DevBuf& operator=(const DevBuf&) = delete;
    ~DevBuf() { release(); }
    void release() {
        if (p) cudaFree(p);
        p = nullptr;
        n = 0;
    }
    // returns true if the pointer changed
    bool reserve(size_t count) {
        if (count <= n && p) return false;
        release();
        size_t bytes = std::max<size_t>(count, 1) * sizeof(T);
        cudaError_t e = cudaMalloc(&p, bytes);
        if (e == cudaErrorMemoryAllocation) {
            (void)cudaGetLastError();
            workspace_trim();
            e = cudaMalloc(&p, bytes);
        }
        if (e != cudaSuccess) {
            // a failed allocation leaves the handle usable: clear the runtime's
            // last error so that the next launch check does not report it again
            p = nullptr;
            (void)cudaGetLastError();
            OWL_CUDA(e);
        }
        n = std::max<size_t>(count, 1);
        return true;
    }
    void zero(cudaStream_t s, size_t count) { OWL_CUDA(cudaMemsetAsync(p, 0, count * sizeof(T), s)); }
    void upload(const T* h, size_t count, cudaStream_t s) {
        reserve(count);
        if (count) OWL_CUDA(cudaMemcpyAsync(p, h, count * sizeof(T), cudaMemcpyHostToDevice, s));
    }
};

// ----------------------------------------------------------------------------
// point operators (source injection, receiver sampling, adjoint-source
// injection) in CSR form. Each item (a source of one shot, a receiver, a
// unique target cell) owns a contiguous run of taps (field slot, offset, w).
// ----------------------------------------------------------------------------
struct Tap {
    int field;   // field slot within the medium's state (e.g. 0 = p, 1 = vx, 2 = vz)
    int64_t off; // offset inside one shot's field (z * pitch + x)
    float w;     // weight
    int item;    // owning item for scatter tables (receiver / source index)
};

struct HostCSR {
    std::vector<int> ptr{0};
    std::vector<int> field, item;
    std::vector<long long> off;
    std::vector<float> w;
    void push(const Tap& t) {
        field.push_back(t.field);
        item.push_back(t.item);
        off.push_back(t.off);
        w.push_back(t.w);
    }
    void close_item() { ptr.push_back((int)field.size()); }
    int nitems() const { return (int)ptr.size() - 1; }
    int ntaps() const { return (int)field.size(); }
};

// a tap as the point kernels read it: one 16-byte load
struct alignas(16) TapRec {
    long long off;  // offset inside one shot's field
    int fi;         // field slot, or the item (trace) for scatter tables
    float w;
};

struct DevCSR {
    DevBuf<int> ptr, field, item;
    DevBuf<long long> off;
    DevBuf<float> w;
    DevBuf<TapRec> tap;
    int nitems = 0, ntaps = 0;
    // scatter: a scatter table, whose packed taps carry the item instead of the
    // field; split: the parts by themselves too, for point work inside stencil kernels
    void upload(const HostCSR& h, cudaStream_t s, bool scatter, bool split) {
        nitems = h.nitems();
        ntaps = h.ntaps();
        std::vector<TapRec> t(ntaps);
        for (int j = 0; j < ntaps; ++j) t[j] = TapRec{h.off[j], scatter ? h.item[j] : h.field[j], h.w[j]};
        tap.upload(t.data(), t.size(), s);
        ptr.upload(h.ptr.data(), h.ptr.size(), s);
        if (scatter) field.upload(h.field.data(), h.field.size(), s);
        if (!split) return;
        if (scatter) item.upload(h.item.data(), h.item.size(), s);
        off.upload(h.off.data(), h.off.size(), s);
        w.upload(h.w.data(), h.w.size(), s);
    }
};

// device view of a CSR table
struct CSRView {
    const int* ptr;
    const int* field;  // scatter tables
    const int* item;   // scatter tables, split
    const long long* off;  // split
    const float* w;        // split
    const TapRec* tap;
    int nitems;
};

inline CSRView view(const DevCSR& d) {
    return CSRView{d.ptr.p, d.field.p, d.item.p, d.off.p, d.w.p, d.tap.p, d.nitems};
}

// FD coefficients of the optimised staggered scheme (src/lib/module_fdcoef.f90:23-30, 59-62)
inline const float* fd_coefs(int half) {
    static const float c4[4] = {0.1217990e+1f, -0.9382142e-1f, 0.1507536e-1f, -0.1700324e-2f};
    static const float c8[8] = {0.1259312e+1f, -0.1280347e+0f, 0.3841945e-1f, -0.1473229e-1f,
                                0.5924913e-2f, -0.2248618e-2f, 0.7179226e-3f, -0.1400855e-3f};
    return half == 8 ? c8 : c4;
}

// CFS-PML coefficient of one node, damp_coef (src/solver/acoustic_iso_2d/module_cfspml.f90:37-56),
// evaluated in single precision in the reference's operation order.
void damp_coef(float bdvp, float d, float dist, int pml, float dt, float alphamax, float& a, float& b);

// 1D CFS-PML coefficients at integer and half nodes over the padded compute
// range [-pml+1, n+pml] (module_cfspml.f90:95-131), mapped to storage index
// i + pml + R - 1 with length `len`.
struct Pml1DHost {
    std::vector<float> ai, bi, ah, bh;
};
Pml1DHost build_pml_1d(int n, int pml, int R, int len, float d, float dt, float pmlvp, float alphamax);

int nint_f(float v);  // Fortran nint

// device-time measurement of a call
struct EventTimer {
    cudaEvent_t a = nullptr, b = nullptr;
    cudaStream_t s;
    explicit EventTimer(cudaStream_t st) : s(st) {
        OWL_CUDA(cudaEventCreate(&a));
        OWL_CUDA(cudaEventCreate(&b));
        OWL_CUDA(cudaEventRecord(a, s));
    }
    double stop_ms() {
        OWL_CUDA(cudaEventRecord(b, s));
        OWL_CUDA(cudaEventSynchronize(b));
        float ms = 0;
        OWL_CUDA(cudaEventElapsedTime(&ms, a, b));
        return ms;
    }
    ~EventTimer() {
        if (a) cudaEventDestroy(a);
        if (b) cudaEventDestroy(b);
    }
};

// simple cached CUDA graph of a launch sequence
struct GraphCache {
    cudaGraphExec_t exec = nullptr;
    std::vector<uintptr_t> sig;
    ~GraphCache() { reset(); }
    void reset() {
        if (exec) cudaGraphExecDestroy(exec);
        exec = nullptr;
        sig.clear();
    }
};

}  // namespace owl
