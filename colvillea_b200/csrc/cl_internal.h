// Host-side internals shared by the library's translation units: device
// buffers, error propagation and the built acceleration structure.
#pragma once

#include "../../include/colvillea_b200.h"

#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstring>
#include <memory>
#include <string>
#include <utility>
#include <vector>

namespace clb
{
// Host milliseconds this thread has spent in cudaMalloc (the allocation share
// of a build's wall time).
double& allocMs();

// Fault injection for tests: of this thread's device allocations the next `after`
// are made and the `count` that follow report that memory ran out.
struct FailAlloc
{
    uint32_t after = 0, count = 0;
    bool     now()
    {
        if (count == 0u) return false;
        if (after > 0u)
        {
            --after;
            return false;
        }
        --count;
        return true;
    }
};
FailAlloc& failAlloc();

// Device allocation owned by one object (the reference's DeviceBuffer,
// src/core/devices/cudabuffer.h:39-96, with errors returned, not exit()), or
// page-locked host memory that kernels read in place.
struct DevBuf
{
    void*  p      = nullptr;
    size_t bytes  = 0;
    bool   pinned = false; // host memory; its owner waits for its readers before a release
    DevBuf()     = default;
    DevBuf(const DevBuf&) = delete;
    DevBuf& operator=(const DevBuf&) = delete;
    ~DevBuf() { release(); }
    void swap(DevBuf& o)
    {
        std::swap(p, o.p);
        std::swap(bytes, o.bytes);
        std::swap(pinned, o.pinned);
    }
    void release()
    {
        if (p) pinned ? cudaFreeHost(p) : cudaFree(p);
        p      = nullptr;
        bytes  = 0;
        pinned = false;
    }
    cl_status allocPinned(size_t n, std::string* err)
    {
        release();
        const cudaError_t e = cudaHostAlloc(&p, n, cudaHostAllocDefault);
        if (e != cudaSuccess)
        {
            p    = nullptr;
            *err = std::string("cudaHostAlloc(") + std::to_string(n) + ") failed: " + cudaGetErrorString(e);
            cudaGetLastError();
            return e == cudaErrorMemoryAllocation ? CL_ERR_OOM : CL_ERR_CUDA;
        }
        bytes  = n;
        pinned = true;
        return CL_OK;
    }
    cl_status alloc(size_t n, std::string* err)
    {
        release();
        if (n == 0) n = 16;
        const auto  t0 = std::chrono::steady_clock::now();
        cudaError_t e  = failAlloc().now() ? cudaErrorMemoryAllocation : cudaMalloc(&p, n);
        allocMs() += std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
        if (e != cudaSuccess)
        {
            p    = nullptr;
            *err = std::string("cudaMalloc(") + std::to_string(n) + ") failed: " + cudaGetErrorString(e);
            cudaGetLastError();
            return e == cudaErrorMemoryAllocation ? CL_ERR_OOM : CL_ERR_CUDA;
        }
        bytes = n;
        return CL_OK;
    }
    float*    f() const { return static_cast<float*>(p); }
    uint32_t* u() const { return static_cast<uint32_t*>(p); }
    template <class T> T* as() const { return static_cast<T*>(p); }
};

#define CL_TRY(expr)                                                                                                   \
    do                                                                                                                 \
    {                                                                                                                  \
        cl_status _s = (expr);                                                                                         \
        if (_s != CL_OK) return _s;                                                                                    \
    } while (0)

#define CL_CUDA(expr, errp)                                                                                            \
    do                                                                                                                 \
    {                                                                                                                  \
        cudaError_t _e = (expr);                                                                                       \
        if (_e != cudaSuccess)                                                                                         \
        {                                                                                                              \
            *(errp) = std::string(#expr) + ": " + cudaGetErrorString(_e);                                              \
            return CL_ERR_CUDA;                                                                                        \
        }                                                                                                              \
    } while (0)

// Part of a larger allocation, with DevBuf's accessors; it owns nothing.
struct ScratchBuf
{
    void*  p     = nullptr;
    size_t bytes = 0;
    float*    f() const { return static_cast<float*>(p); }
    uint32_t* u() const { return static_cast<uint32_t*>(p); }
    template <class T> T* as() const { return static_cast<T*>(p); }
};

// Lays out one allocation (a cudaMalloc or cudaFree takes 0.3 ms whatever its
// size): parts are taken at 256-byte boundaries, a rewind to a mark lets later
// parts share the memory of dead ones, and bind() gives the parts their places
// once the allocation of peak() bytes exists.
class Carver
{
public:
    void take(ScratchBuf& s, size_t bytes)
    {
        parts_.push_back({&s, off_});
        s.bytes = bytes;
        off_ += (bytes + 255) / 256 * 256;
        peak_ = std::max(peak_, off_);
    }
    size_t mark() const { return off_; }
    void   rewind(size_t m) { off_ = m; }
    size_t peak() const { return peak_; }
    void   bind(void* base) const
    {
        for (const auto& p : parts_) p.first->p = static_cast<char*>(base) + p.second;
    }

private:
    std::vector<std::pair<ScratchBuf*, size_t>> parts_;
    size_t                                      off_ = 0, peak_ = 0;
};

struct WideBvh
{
    DevBuf     mem;   // holds the four below
    ScratchBuf nodes; // 6 uint4 per node
    ScratchBuf tris;  // 3 float4 per triangle, leaf order
    ScratchBuf exact; // refit: 6 floats per node, the unquantised box of its triangles
    ScratchBuf scene; // scene bounds (6 ordered ints, refit); SAH sum (double at byte 32), copy of the root node (byte 48)
    // Nodes of tree level d are [levels[d], levels[d + 1]): the collapse
    // allocates each level's nodes in one launch.
    std::vector<uint32_t> levels;
    uint32_t numNodes = 0, depth = 0, numTris = 0;
    void     release()
    {
        mem.release();
        nodes = tris = exact = scene = ScratchBuf{};
        levels.clear();
        numNodes = depth = numTris = 0;
    }
};

// Grow-only device memory for a build's temporaries and for the device copy of
// its input, reused by the builds that share the arena (one per mesh of a
// two-level scene).
class BuildArena
{
public:
    cl_status reserve(size_t bytes, std::string* err)
    {
        return mem_.bytes < bytes ? mem_.alloc(bytes, err) : CL_OK;
    }
    void*     base() const { return mem_.p; }
    cl_status input(ScratchBuf& s, size_t bytes, std::string* err)
    {
        if (input_.bytes < bytes) CL_TRY(input_.alloc(bytes, err));
        s.p     = input_.p;
        s.bytes = bytes;
        return CL_OK;
    }

private:
    DevBuf mem_, input_;
};

// dTri9: 9 floats per triangle (world-space vertices), device memory.  The
// builder's temporaries come from `arena` (a local one when null).
cl_status buildWideBvh(const float* dTri9, uint32_t n, cudaStream_t st, WideBvh* out, std::string* err,
                       BuildArena* arena = nullptr);

// Refit after the vertices moved (same triangles, same vertex indices):
// rewrites the leaf triangles from vtx (3 float4 per vertex, position in the
// first) and triIdx (uint4 per triangle), then recomputes every node's child
// boxes level by level from the deepest, keeping the tree's topology and
// slot order.  Without moved vertices the nodes come out bit-identical to the
// build's.  Asynchronous on st.
cl_status refitWideBvh(WideBvh* bvh, const void* vtx, const void* triIdx, cudaStream_t st, std::string* err);

// Surface-area cost of the built tree: sum over child slots of the slot's
// quantised box area, times the triangle count for leaf slots, over the root
// box area (one unit per node visit and per triangle test).  Synchronises st.
cl_status wideBvhSahCost(WideBvh& bvh, cudaStream_t st, double* cost, std::string* err);

// Triangle positions (9 floats each, triangle order) gathered from vtx and
// triIdx, the input of buildWideBvh.  Asynchronous on st.
cl_status gatherTrianglePositions(const void* vtx, const void* triIdx, uint32_t n, float* tri9, cudaStream_t st,
                                  std::string* err);

// Thread-local last error message (cl_last_error).
void setLastError(const std::string& msg);

// Process-wide: set once a tensor-core kernel reported that its bounded
// mbarrier wait ran out.  Its tensor memory may then have been released under
// a matrix operation still in flight, so the context is suspect and every
// later call that would launch a network kernel is refused (CL_ERR_STATE).
bool tcSuspect();
void markTcSuspect();
cl_status refuseIfTcSuspect(std::string* err);

} // namespace clb
