// workspace.cuh -- scratch of the stateless entry points (search directions,
// gradient processing, adjoint sources).
//
// Such a call needs a stream and a few device buffers for microseconds of work;
// creating and freeing them took most of its time (a small cudaMalloc and
// cudaFree about 0.6 ms, a stream 0.1 ms, against 30 us of kernels). A call
// borrows a Workspace for its own use alone and gives it back when its work on
// the stream has finished, so calls of several threads never share one. Idle
// workspaces are kept per device and context: at most WS_IDLE of them, each of at
// most WS_BYTES, and all are freed when a device allocation of the library runs
// out of memory.
#pragma once

#include "adjsrc.cuh"

namespace owl {

constexpr int WS_IDLE = 4;
constexpr size_t WS_BYTES = (size_t)256 << 20;

struct Workspace {
    int dev = 0;
    unsigned long long ctx = 0;  // the context it belongs to (a reset device starts another)
    cudaStream_t s = nullptr;
    DevBuf<unsigned char> buf;
    AdjointSource adj;
    ~Workspace() {
        if (s) cudaStreamDestroy(s);
    }
    size_t held() const { return buf.n + adj.held(); }
    template <typename T>
    T* take(size_t count) {
        buf.reserve(count * sizeof(T));
        return reinterpret_cast<T*>(buf.p);
    }
};

class WorkspaceLease {
public:
    WorkspaceLease();
    ~WorkspaceLease();
    WorkspaceLease(const WorkspaceLease&) = delete;
    WorkspaceLease& operator=(const WorkspaceLease&) = delete;
    Workspace* operator->() const { return w; }
    Workspace& operator*() const { return *w; }
    // the work on the stream has finished: the workspace may be kept (a call that
    // ends by an exception frees it instead)
    void done() { ok = true; }

private:
    Workspace* w = nullptr;
    bool ok = false;
};

}  // namespace owl
