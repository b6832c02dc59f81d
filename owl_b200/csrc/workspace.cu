// workspace.cu -- the idle list of workspace.cuh.
#include "workspace.cuh"

#include <cudaTypedefs.h>

#include <mutex>

namespace owl {

namespace {

// (never destroyed: at process exit the driver takes the memory back, after
// which a destructor could no longer free it)
std::mutex& ws_lock() {
    static std::mutex* m = new std::mutex;
    return *m;
}
std::vector<Workspace*>& ws_idle() {
    static std::vector<Workspace*>* v = new std::vector<Workspace*>;
    return *v;
}

// identity of the current context, 0 where the driver does not tell
unsigned long long context_id() {
    static PFN_cuCtxGetId_v12000 get = [] {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult q{};
        if (cudaGetDriverEntryPoint("cuCtxGetId", &fn, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            fn = nullptr;
        return reinterpret_cast<PFN_cuCtxGetId_v12000>(fn);
    }();
    unsigned long long id = 0;
    if (get && get(nullptr, &id) != CUDA_SUCCESS) id = 0;
    return id;
}

}  // namespace

WorkspaceLease::WorkspaceLease() {
    int dev = 0;
    OWL_CUDA(cudaGetDevice(&dev));
    OWL_CUDA(cudaSetDevice(dev));  // the device's context exists and is this thread's from here on
    const unsigned long long ctx = context_id();
    {
        std::lock_guard<std::mutex> g(ws_lock());
        std::vector<Workspace*>& v = ws_idle();
        for (size_t i = v.size(); i-- > 0;) {
            if (v[i]->dev != dev) continue;
            Workspace* p = v[i];
            v.erase(v.begin() + (long)i);
            if (p->ctx == ctx) {
                w = p;
                break;
            }
            // its context is gone and its handles with it: forget the object, free nothing
        }
    }
    if (w) return;
    w = new Workspace;
    w->dev = dev;
    w->ctx = ctx;
    const cudaError_t e = cudaStreamCreateWithFlags(&w->s, cudaStreamNonBlocking);
    if (e != cudaSuccess) {
        w->s = nullptr;
        delete w;
        (void)cudaGetLastError();
        OWL_CUDA(e);
    }
}

WorkspaceLease::~WorkspaceLease() {
    if (ok && w->held() <= WS_BYTES) {
        std::lock_guard<std::mutex> g(ws_lock());
        int n = 0;
        for (const Workspace* p : ws_idle()) n += p->dev == w->dev;
        if (n < WS_IDLE) {
            ws_idle().push_back(w);
            return;
        }
    }
    if (!ok) cudaStreamSynchronize(w->s);  // nothing may still use the buffers
    delete w;
}

size_t workspace_idle_bytes() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    const unsigned long long ctx = context_id();
    std::lock_guard<std::mutex> g(ws_lock());
    size_t n = 0;
    for (const Workspace* p : ws_idle())
        if (p->dev == dev && p->ctx == ctx) n += p->held();
    return n;
}

void workspace_trim() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return;
    const unsigned long long ctx = context_id();
    std::vector<Workspace*> drop;
    {
        std::lock_guard<std::mutex> g(ws_lock());
        std::vector<Workspace*>& v = ws_idle();
        for (size_t i = v.size(); i-- > 0;)
            if (v[i]->dev == dev && v[i]->ctx == ctx) {
                drop.push_back(v[i]);
                v.erase(v.begin() + (long)i);
            }
    }
    for (Workspace* p : drop) delete p;
}

}  // namespace owl
