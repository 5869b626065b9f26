// workspace.cuh -- device workspaces of single calls.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

namespace atmwfs {

// Stream-ordered allocation from the library's own memory pool of the current
// device.  The pool keeps up to kWorkspaceKeep bytes of what calls have freed,
// so that a call need not map and unmap its buffers (cudaMalloc / cudaFree, or
// the default pool, which returns everything at the next synchronisation: an
// 8192^2 transform waited 1.3 of 2.2 ms for that); what it keeps is given back
// when an engine context or a surrogate is destroyed, when an allocation of the
// library finds too little memory, and by atmwfs_release_workspaces.  Any thread
// and stream may allocate and free; a buffer is used on the stream it was
// allocated on.
constexpr size_t kWorkspaceKeep = size_t(1) << 30;
cudaError_t workspace_alloc(void** p, size_t bytes, cudaStream_t st);
void workspace_free(void* p, cudaStream_t st);          // p may be null
cudaError_t device_malloc(void** p, size_t bytes);      // cudaMalloc of what outlives a call
void workspace_release();                               // give back what the pools of all devices keep

// A workspace of one scope.
class Workspace {
public:
    Workspace(size_t bytes, cudaStream_t st) : st_(st) { err_ = workspace_alloc(&p_, bytes, st); }
    ~Workspace() { workspace_free(p_, st_); }
    Workspace(const Workspace&) = delete;
    Workspace& operator=(const Workspace&) = delete;
    cudaError_t error() const { return err_; }
    template <typename T> T* as() const { return static_cast<T*>(p_); }

private:
    void* p_ = nullptr;
    cudaStream_t st_;
    cudaError_t err_;
};

}  // namespace atmwfs
