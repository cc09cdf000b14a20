// Mesh uploads, vertex edits and the flattening of instances on the device.
//
// The meshes are copied to the device as the caller gives them and stay there;
// flattening (the reference's TLAS has no transforms, optix.cu:115), edits and
// the two-level scenes' pools and boxes read them from there.  The passes are
// bound by memory: each vertex reads 44 B and writes 48 B, each triangle reads
// 12 B and writes 16 B (0.1 ms for 1.17 M triangles; one host core took 47 ms
// for their copies and flattening), so an upload costs what its copies from
// pageable memory cost.  The arithmetic is in double and in a host loop's order.
// Where the meshes find no room on the device they lie in page-locked host
// memory, and the same kernels read them over PCIe.
#include "cl_geometry.h"

#include <cfloat>
#include <cmath>

namespace clb
{
namespace
{
constexpr int      kBlock  = 256;
constexpr uint32_t kNoMesh = 0xffffffffu;

// Edits of at most this many position floats are checked by the host, larger
// ones by a kernel, which costs a round trip of the device and a second copy.
// Whole edits by host and by kernel: 104 and 128 us for 16 vertices, 137 and 151
// for 4,096, 149 and 151 for 16,384, 189 and 166 for 32,400, 750 and 350 for
// 262,144.
constexpr size_t kHostCheckFloats = 32768;

// Ordered integer images of floats and doubles (their order is the numbers').
__device__ __forceinline__ uint32_t ordered(float f)
{
    const uint32_t b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ unsigned long long ordered(double d)
{
    const unsigned long long b = (unsigned long long)__double_as_longlong(d);
    return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}
float unordered(uint32_t v)
{
    const uint32_t b = (v & 0x80000000u) ? (v & 0x7fffffffu) : ~v;
    float          f;
    memcpy(&f, &b, 4);
    return f;
}
double unordered(unsigned long long v)
{
    const unsigned long long b = (v >> 63) ? (v & 0x7fffffffffffffffull) : ~v;
    double                   d;
    memcpy(&d, &b, 8);
    return d;
}

// Largest i with start(i) <= x, start non-decreasing, start(0) <= x.
template <class T, class F> __device__ __forceinline__ uint32_t lastAtMost(uint32_t n, T x, F start)
{
    uint32_t lo = 0u, hi = n;
    while (hi - lo > 1u)
    {
        const uint32_t mid = lo + (hi - lo) / 2u;
        if (start(mid) <= x)
            lo = mid;
        else
            hi = mid;
    }
    return lo;
}

// Smallest mesh id with a vertex index out of range.  tab: per mesh {first
// triangle, vertices} (meshes are not empty, so the bases increase).
__global__ void kCheckIndices(const uint32_t* __restrict__ idx, unsigned long long nt, const ulonglong2* __restrict__ tab,
                              uint32_t n, uint32_t* bad)
{
    const unsigned long long t = blockIdx.x * (unsigned long long)(blockDim.x) + threadIdx.x;
    if (t >= nt) return;
    const uint32_t  m  = lastAtMost(n, t, [&](uint32_t i) { return __ldg(&tab[i].x); });
    const uint32_t  nv = uint32_t(__ldg(&tab[m].y));
    const uint32_t* v  = idx + 3 * size_t(t);
    if (v[0] >= nv || v[1] >= nv || v[2] >= nv) atomicMin(bad, m);
}

// Smallest float index that is not finite.
__global__ void kCheckFinite(const float* __restrict__ x, size_t n, unsigned long long* bad)
{
    for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x)
        if (!isfinite(x[i])) atomicMin(bad, (unsigned long long)i);
}

struct PoolView
{
    const float* __restrict__ pos;
    const float* __restrict__ nrm;
    const float* __restrict__ tan;
    const float* __restrict__ uv;
    const uint32_t* __restrict__ idx;
};

// Vertex k of the copy I of its mesh.
__device__ __forceinline__ void flattenVertex(const PoolView& P, const FlatInst& I, uint32_t k, float4* __restrict__ vtx)
{
    const size_t   v     = I.srcVtx + size_t(k);
    const uint32_t flags = I.flags & 3u;
    float p[3], nn[3] = {0.0f, 0.0f, 0.0f}, t[3], uv[2] = {0.0f, 0.0f};
#pragma unroll
    for (int q = 0; q < 3; ++q)
    {
        p[q] = P.pos[3 * v + q];
        t[q] = P.tan[3 * v + q];
        if (flags & 1u) nn[q] = P.nrm[3 * v + q];
    }
    if (flags & 2u)
    {
        uv[0] = P.uv[2 * v];
        uv[1] = P.uv[2 * v + 1];
    }
    if (!(I.flags & 4u))
    {
        float p2[3], t2[3], n2[3];
#pragma unroll
        for (int r = 0; r < 3; ++r)
        {
            const double a = I.m[4 * r], b = I.m[4 * r + 1], c = I.m[4 * r + 2];
            p2[r] = float(a * p[0] + b * p[1] + c * p[2] + double(I.m[4 * r + 3]));
            t2[r] = float(a * t[0] + b * t[1] + c * t[2]);
            // n' = (inverse of the linear part)^T n
            n2[r] = float(I.it[3 * r] * nn[0] + I.it[3 * r + 1] * nn[1] + I.it[3 * r + 2] * nn[2]);
        }
#pragma unroll
        for (int q = 0; q < 3; ++q)
        {
            p[q]  = p2[q];
            t[q]  = t2[q];
            nn[q] = n2[q];
        }
    }
    float4* o = vtx + 3 * (I.dstVtx + size_t(k));
    o[0]      = make_float4(p[0], p[1], p[2], nn[0]);
    o[1]      = make_float4(nn[1], nn[2], t[0], t[1]);
    o[2]      = make_float4(t[2], uv[0], uv[1], __uint_as_float(flags));
}

// One thread per flattened vertex of copies inst[0, n) (base: the first one's dstVtx).
__global__ void __launch_bounds__(kBlock) kFlattenVertices(PoolView P, const FlatInst* __restrict__ inst, uint32_t n,
                                                           uint32_t base, uint32_t count, float4* __restrict__ vtx)
{
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= count) return;
    const uint32_t  dst = base + k;
    const FlatInst& I = inst[lastAtMost(n, dst, [&](uint32_t i) { return __ldg(&inst[i].dstVtx); })];
    flattenVertex(P, I, dst - I.dstVtx, vtx);
}

// One thread per vertex of one mesh's copies inst[list[..]], nv vertices each.
// An edit writes all copies in one launch, bound by its fixed costs up to
// about 100,000 vertices: whole edits of a 12-vertex mesh with 2,000 and 10,000
// copies took 8.3 and 41 ms with a launch for each copy, 0.14 and 0.15 ms so.
__global__ void __launch_bounds__(kBlock) kFlattenCopies(PoolView P, const FlatInst* __restrict__ inst,
                                                         const uint32_t* __restrict__ list, uint32_t nv, uint32_t total,
                                                         float4* __restrict__ vtx)
{
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= total) return;
    const uint32_t c = k / nv;
    flattenVertex(P, inst[__ldg(list + c)], k - c * nv, vtx);
}

__global__ void __launch_bounds__(kBlock) kFlattenTriangles(PoolView P, const FlatInst* __restrict__ inst, uint32_t n,
                                                            uint32_t count, uint4* __restrict__ triIdx)
{
    const uint32_t dst = blockIdx.x * blockDim.x + threadIdx.x;
    if (dst >= count) return;
    const FlatInst& I = inst[lastAtMost(n, dst, [&](uint32_t i) { return __ldg(&inst[i].dstTri); })];
    const uint32_t* x = P.idx + 3 * (I.srcTri + size_t(dst - I.dstTri));
    triIdx[dst]       = make_uint4(I.dstVtx + x[0], I.dstVtx + x[1], I.dstVtx + x[2], I.w);
}

// Box of each copy's mapped vertices: blocks (x, y) take chunk x of copy y;
// ordered 64-bit minima and (complemented) maxima, 6 words per copy.
__global__ void __launch_bounds__(kBlock) kInstanceBoxes(PoolView P, const FlatInst* __restrict__ inst,
                                                         unsigned long long* __restrict__ box)
{
    const FlatInst& I    = inst[blockIdx.y];
    double          l[3] = {1e300, 1e300, 1e300}, h[3] = {-1e300, -1e300, -1e300};
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < I.nv; v += gridDim.x * blockDim.x)
    {
        const float* p = P.pos + 3 * (I.srcVtx + size_t(v));
        const double x = p[0], y = p[1], z = p[2];
#pragma unroll
        for (int r = 0; r < 3; ++r)
        {
            const double c = double(I.m[4 * r]) * x + double(I.m[4 * r + 1]) * y + double(I.m[4 * r + 2]) * z +
                             double(I.m[4 * r + 3]);
            l[r] = c < l[r] ? c : l[r];
            h[r] = c > h[r] ? c : h[r];
        }
    }
#pragma unroll
    for (int r = 0; r < 3; ++r)
    {
        for (int o = 16; o > 0; o >>= 1)
        {
            const double a = __shfl_xor_sync(0xffffffffu, l[r], o), b = __shfl_xor_sync(0xffffffffu, h[r], o);
            l[r]           = a < l[r] ? a : l[r];
            h[r]           = b > h[r] ? b : h[r];
        }
        if ((threadIdx.x & 31u) == 0u && l[r] <= h[r])
        {
            atomicMin(box + 6 * size_t(blockIdx.y) + r, ordered(l[r]));
            atomicMin(box + 6 * size_t(blockIdx.y) + 3 + r, ~ordered(h[r]));
        }
    }
}

// Bounds of the flattened positions: ordered minima and (complemented) maxima.
__global__ void __launch_bounds__(kBlock) kVertexBounds(const float4* __restrict__ vtx, size_t n, uint32_t* bounds)
{
    float l[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, h[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
    for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x)
    {
        const float4 p = vtx[3 * i];
        const float  x[3] = {p.x, p.y, p.z};
#pragma unroll
        for (int r = 0; r < 3; ++r)
        {
            l[r] = fminf(l[r], x[r]);
            h[r] = fmaxf(h[r], x[r]);
        }
    }
#pragma unroll
    for (int r = 0; r < 3; ++r)
    {
        for (int o = 16; o > 0; o >>= 1)
        {
            l[r] = fminf(l[r], __shfl_xor_sync(0xffffffffu, l[r], o));
            h[r] = fmaxf(h[r], __shfl_xor_sync(0xffffffffu, h[r], o));
        }
        if ((threadIdx.x & 31u) == 0u)
        {
            atomicMin(bounds + r, ordered(l[r]));
            atomicMin(bounds + 3 + r, ~ordered(h[r]));
        }
    }
}

// Host arrays to consecutive places of one allocation.  Arrays below
// kPackBelow are gathered in a block of host memory first and copied together,
// since a copy call costs 3.5 us whatever its size.  cl_build_meshes on 2,000
// meshes of 12 vertices: 17 ms with a call for each array, 0.6 gathered; 1,000
// of 642: 11.4 and 4.4; 500 of 2,562: 13.1 and 9.3 (with a limit of 16 KB 13.7,
// of 256 KB 9.5); arrays of 120 KB and more: equal.  Blocks of 256, 128 and 64
// KB: 1,000 meshes of 642 in 4.6, 5.3 and 5.7 ms.
constexpr size_t kPackBelow = 65536, kPackBlock = size_t(1) << 20;
class PackedUpload
{
public:
    PackedUpload(const DevBuf& dst, size_t total, cudaStream_t st)
        : dst_(dst.as<char>()), host_(dst.pinned), cap_(std::min(kPackBlock, total)), block_(new char[cap_]), st_(st)
    {
    }
    // The next `bytes` of the allocation; src null: left as they are or written with zeros (nothing reads them).
    cl_status add(const void* src, size_t bytes, std::string* err)
    {
        if (host_ || bytes >= kPackBelow || bytes > cap_)
        {
            CL_TRY(flush(err));
            if (src && host_)
                memcpy(dst_ + at_, src, bytes);
            else if (src)
                CL_CUDA(cudaMemcpyAsync(dst_ + at_, src, bytes, cudaMemcpyHostToDevice, st_), err);
            at_ += bytes;
            return CL_OK;
        }
        if (fill_ + bytes > cap_) CL_TRY(flush(err));
        if (src)
            memcpy(block_.get() + fill_, src, bytes);
        else
            memset(block_.get() + fill_, 0, bytes);
        fill_ += bytes;
        return CL_OK;
    }
    // Copies what has been gathered (from pageable memory: the block is free again on return).
    cl_status flush(std::string* err)
    {
        if (fill_) CL_CUDA(cudaMemcpyAsync(dst_ + at_, block_.get(), fill_, cudaMemcpyHostToDevice, st_), err);
        at_ += fill_;
        fill_ = 0;
        return CL_OK;
    }

private:
    char*                   dst_;
    bool                    host_;
    size_t                  at_ = 0, fill_ = 0, cap_; // bytes placed; gathered behind them
    std::unique_ptr<char[]> block_;
    cudaStream_t            st_;
};

uint32_t blocksFor(size_t n) { return uint32_t((n + kBlock - 1) / kBlock); }
} // namespace

cl_status MeshPool::build(const cl_mesh_desc* meshes, uint32_t n, cudaStream_t st, std::string* err)
{
    std::vector<MeshInfo>   info(n);
    std::vector<ulonglong2> tab(n);
    size_t                  nv = 0, nt = 0;
    for (uint32_t m = 0; m < n; ++m)
    {
        const cl_mesh_desc& d = meshes[m];
        if (!d.positions || !d.indices || !d.tangents || d.num_vertices == 0 || d.num_triangles == 0)
        {
            *err = "mesh " + std::to_string(m) + ": positions, tangents and indices are required";
            return CL_ERR_INVALID_ARG;
        }
        info[m] = MeshInfo{d.num_vertices, d.num_triangles, nv, nt, d.normals != nullptr, d.uvs != nullptr};
        tab[m]  = make_ulonglong2(nt, d.num_vertices);
        nv += d.num_vertices;
        nt += d.num_triangles;
    }
    DevBuf mem;
    if (n)
    {
        const size_t words = 11 * nv + 3 * nt, tabAt = (words + 3) / 4 * 4; // 16-byte aligned table
        cl_status    s     = mem.alloc(4 * (tabAt + 4 * size_t(n) + 1), err);
        if (s == CL_ERR_OOM) s = mem.allocPinned(4 * words, err);
        if (s != CL_OK) return s;
        float*   f   = mem.f();
        uint32_t bad = kNoMesh;
        // The pool's five parts, mesh after mesh.
        PackedUpload up(mem, 4 * words, st);
        for (uint32_t m = 0; m < n; ++m) CL_TRY(up.add(meshes[m].positions, 12 * size_t(info[m].nv), err));
        for (uint32_t m = 0; m < n; ++m) CL_TRY(up.add(meshes[m].normals, 12 * size_t(info[m].nv), err));
        for (uint32_t m = 0; m < n; ++m) CL_TRY(up.add(meshes[m].tangents, 12 * size_t(info[m].nv), err));
        for (uint32_t m = 0; m < n; ++m) CL_TRY(up.add(meshes[m].uvs, 8 * size_t(info[m].nv), err));
        for (uint32_t m = 0; m < n; ++m) CL_TRY(up.add(meshes[m].indices, 12 * size_t(info[m].nt), err));
        CL_TRY(up.flush(err));
        if (mem.pinned)
        {
            for (uint32_t m = 0; m < n && bad == kNoMesh; ++m)
                for (size_t k = 0; k < 3 * size_t(info[m].nt); ++k)
                    if (meshes[m].indices[k] >= info[m].nv)
                    {
                        bad = m;
                        break;
                    }
        }
        else
        {
            auto* dTab = reinterpret_cast<ulonglong2*>(f + tabAt);
            auto* dBad = reinterpret_cast<uint32_t*>(dTab + n);
            CL_CUDA(cudaMemcpyAsync(dTab, tab.data(), 16 * size_t(n), cudaMemcpyHostToDevice, st), err);
            CL_CUDA(cudaMemsetAsync(dBad, 0xff, 4, st), err);
            kCheckIndices<<<blocksFor(nt), kBlock, 0, st>>>(mem.u() + 11 * nv, nt, dTab, n, dBad);
            CL_CUDA(cudaGetLastError(), err);
            CL_CUDA(cudaMemcpyAsync(&bad, dBad, 4, cudaMemcpyDeviceToHost, st), err);
        }
        CL_CUDA(cudaStreamSynchronize(st), err); // the caller's arrays are free again, and nothing reads the old pool
        if (bad != kNoMesh)
        {
            *err = "mesh " + std::to_string(bad) + ": vertex index out of range";
            return CL_ERR_INVALID_ARG;
        }
    }
    else
        CL_CUDA(cudaStreamSynchronize(st), err);
    mem_.swap(mem);
    info_.swap(info);
    nv_ = nv;
    return CL_OK;
}

bool MeshPool::spill(cudaStream_t st)
{
    std::string err;
    DevBuf      h;
    if (!mem_.p || mem_.pinned || h.allocPinned(mem_.bytes, &err) != CL_OK) return false;
    if (cudaMemcpyAsync(h.p, mem_.p, mem_.bytes, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess)
        return false;
    mem_.swap(h);
    edit_.release();
    return true;
}

// Into the pool; host memory is written at once (the stream has been synchronised).
cl_status MeshPool::put(float* dst, const float* src, size_t bytes, cudaStream_t st, std::string* err)
{
    if (mem_.pinned)
        memcpy(dst, src, bytes);
    else
        CL_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st), err);
    return CL_OK;
}

cl_status MeshPool::updateVertices(uint32_t mesh, const float* pos, const float* nrm, const float* tan, cudaStream_t st,
                                   std::string* err)
{
    MeshInfo&    i = info_[mesh];
    const size_t n = 3 * size_t(i.nv), b = 4 * n, at = 3 * i.vtxBase, errAt = (3 * n + 1) / 2 * 2;
    if (mem_.pinned || n <= kHostCheckFloats)
    {
        for (size_t k = 0; k < n; ++k)
            if (!std::isfinite(pos[k]))
            {
                *err = "vertex " + std::to_string(k / 3) + ": position is not finite";
                return CL_ERR_INVALID_ARG;
            }
        if (mem_.pinned) CL_CUDA(cudaStreamSynchronize(st), err);
        CL_TRY(put(this->pos() + at, pos, b, st, err));
        if (nrm) CL_TRY(put(this->nrm() + at, nrm, b, st, err));
        if (tan) CL_TRY(put(this->tan() + at, tan, b, st, err));
        if (nrm) i.hasN = true;
        return CL_OK;
    }
    if (edit_.bytes < 4 * errAt + 8) CL_TRY(edit_.alloc(4 * errAt + 8, err));
    float* e = edit_.f();
    auto*  dBad = reinterpret_cast<unsigned long long*>(e + errAt);
    CL_CUDA(cudaMemsetAsync(dBad, 0xff, 8, st), err);
    CL_CUDA(cudaMemcpyAsync(e, pos, b, cudaMemcpyHostToDevice, st), err);
    if (nrm) CL_CUDA(cudaMemcpyAsync(e + n, nrm, b, cudaMemcpyHostToDevice, st), err);
    if (tan) CL_CUDA(cudaMemcpyAsync(e + 2 * n, tan, b, cudaMemcpyHostToDevice, st), err);
    kCheckFinite<<<std::min<uint32_t>(blocksFor(n), 1184u), kBlock, 0, st>>>(e, n, dBad);
    CL_CUDA(cudaGetLastError(), err);
    unsigned long long bad = 0;
    CL_CUDA(cudaMemcpyAsync(&bad, dBad, 8, cudaMemcpyDeviceToHost, st), err);
    CL_CUDA(cudaStreamSynchronize(st), err); // the caller's arrays are free again
    if (bad != ~0ull)
    {
        *err = "vertex " + std::to_string(bad / 3) + ": position is not finite";
        return CL_ERR_INVALID_ARG;
    }
    CL_CUDA(cudaMemcpyAsync(this->pos() + at, e, b, cudaMemcpyDeviceToDevice, st), err);
    if (nrm)
    {
        CL_CUDA(cudaMemcpyAsync(this->nrm() + at, e + n, b, cudaMemcpyDeviceToDevice, st), err);
        i.hasN = true;
    }
    if (tan) CL_CUDA(cudaMemcpyAsync(this->tan() + at, e + 2 * n, b, cudaMemcpyDeviceToDevice, st), err);
    return CL_OK;
}

cl_status MeshPool::flatInst(uint32_t mesh, const float* M, uint32_t dstVtx, uint32_t dstTri, uint32_t w,
                             const std::string& what, FlatInst* out, std::string* err) const
{
    const MeshInfo& i = info_[mesh];
    FlatInst&       r = *out;
    const bool ident = M[0] == 1 && M[1] == 0 && M[2] == 0 && M[3] == 0 && M[4] == 0 && M[5] == 1 && M[6] == 0 &&
                       M[7] == 0 && M[8] == 0 && M[9] == 0 && M[10] == 1 && M[11] == 0;
    const double a = M[0], b = M[1], c = M[2], d = M[4], e = M[5], f = M[6], g = M[8], h = M[9], k = M[10];
    const double det = a * (e * k - f * h) - b * (d * k - f * g) + c * (d * h - e * g);
    if (!ident && std::fabs(det) < 1e-30)
    {
        *err = what + ": singular transform";
        return CL_ERR_INVALID_ARG;
    }
    // Inverse transpose of the linear part, row-major: it[3 r + c] = inverse[c][r].
    const double IT[9] = {(e * k - f * h) / det, -(d * k - f * g) / det, (d * h - e * g) / det,
                          -(b * k - c * h) / det, (a * k - c * g) / det,  -(a * h - b * g) / det,
                          (b * f - c * e) / det,  -(a * f - c * d) / det, (a * e - b * d) / det};
    memcpy(r.it, IT, sizeof(IT));
    memcpy(r.m, M, sizeof(r.m));
    r.srcVtx = i.vtxBase;
    r.dstVtx = dstVtx;
    r.nv     = i.nv;
    r.srcTri = i.triBase;
    r.dstTri = dstTri;
    r.nt     = i.nt;
    r.w      = w;
    r.flags  = (i.hasN ? 1u : 0u) | (i.hasUV ? 2u : 0u) | (ident ? 4u : 0u);
    return CL_OK;
}

cl_status MeshPool::flattenVertices(const DevBuf& inst, const FlatInst* host, uint32_t first, uint32_t count, void* vtx,
                                    cudaStream_t st, std::string* err) const
{
    const FlatInst& last = host[first + count - 1];
    const uint32_t  base = host[first].dstVtx, total = last.dstVtx + last.nv - base;
    kFlattenVertices<<<blocksFor(total), kBlock, 0, st>>>(PoolView{pos(), nrm(), tan(), uv(), idx()},
                                                          inst.as<const FlatInst>() + first, count, base, total,
                                                          static_cast<float4*>(vtx));
    CL_CUDA(cudaGetLastError(), err);
    return CL_OK;
}

cl_status MeshPool::flattenCopies(uint32_t mesh, const DevBuf& inst, const uint32_t* list, uint32_t count, void* vtx,
                                  cudaStream_t st, std::string* err) const
{
    if (count == 0) return CL_OK;
    const uint32_t nv = info_[mesh].nv, total = nv * count; // at most the scene's vertices
    kFlattenCopies<<<blocksFor(total), kBlock, 0, st>>>(PoolView{pos(), nrm(), tan(), uv(), idx()},
                                                        inst.as<const FlatInst>(), list, nv, total,
                                                        static_cast<float4*>(vtx));
    CL_CUDA(cudaGetLastError(), err);
    return CL_OK;
}

cl_status MeshPool::flattenTriangles(const DevBuf& inst, const FlatInst* host, uint32_t count, void* triIdx,
                                     cudaStream_t st, std::string* err) const
{
    const uint32_t total = host[count - 1].dstTri + host[count - 1].nt;
    kFlattenTriangles<<<blocksFor(total), kBlock, 0, st>>>(PoolView{pos(), nrm(), tan(), uv(), idx()},
                                                           inst.as<const FlatInst>(), count, total,
                                                           static_cast<uint4*>(triIdx));
    CL_CUDA(cudaGetLastError(), err);
    return CL_OK;
}

cl_status MeshPool::instanceBoxes(const DevBuf& inst, uint32_t first, uint32_t count, std::vector<double>* boxes, cudaStream_t st,
                                  std::string* err) const
{
    DevBuf d;
    CL_TRY(d.alloc(size_t(count) * 48, err));
    CL_CUDA(cudaMemsetAsync(d.p, 0xff, size_t(count) * 48, st), err);
    for (uint32_t y = 0; y < count; y += 65535u)
        kInstanceBoxes<<<dim3(16, std::min(65535u, count - y)), kBlock, 0, st>>>(
            PoolView{pos(), nrm(), tan(), uv(), idx()}, inst.as<const FlatInst>() + first + y,
            d.as<unsigned long long>() + 6 * size_t(y));
    CL_CUDA(cudaGetLastError(), err);
    std::vector<unsigned long long> h(size_t(count) * 6);
    CL_CUDA(cudaMemcpyAsync(h.data(), d.p, size_t(count) * 48, cudaMemcpyDeviceToHost, st), err);
    CL_CUDA(cudaStreamSynchronize(st), err);
    boxes->resize(size_t(count) * 6);
    for (size_t i = 0; i < h.size(); ++i)
    {
        // No vertex compared below or above the start values (all NaN): those values.
        const bool hi = i % 6 >= 3;
        (*boxes)[i]   = h[i] == ~0ull ? (hi ? -1e300 : 1e300) : unordered(hi ? ~h[i] : h[i]);
    }
    return CL_OK;
}

cl_status vertexBounds(const void* vtx, size_t n, cudaStream_t st, float lo[3], float hi[3], std::string* err)
{
    DevBuf d;
    CL_TRY(d.alloc(24, err));
    CL_CUDA(cudaMemsetAsync(d.p, 0xff, 24, st), err);
    kVertexBounds<<<std::min<uint32_t>(blocksFor(n), 296u), kBlock, 0, st>>>(static_cast<const float4*>(vtx), n, d.u());
    CL_CUDA(cudaGetLastError(), err);
    uint32_t h[6];
    CL_CUDA(cudaMemcpyAsync(h, d.p, 24, cudaMemcpyDeviceToHost, st), err);
    CL_CUDA(cudaStreamSynchronize(st), err);
    for (int a = 0; a < 3; ++a)
    {
        lo[a] = unordered(h[a]);
        hi[a] = unordered(~h[3 + a]);
    }
    return CL_OK;
}

} // namespace clb
