// Mesh data on the device and its flattening into the traced scene's vertex
// and triangle arrays.
#pragma once

#include "cl_internal.h"

#include <vector>

namespace clb
{
struct MeshInfo
{
    uint32_t nv = 0, nt = 0;           // vertices, triangles
    size_t   vtxBase = 0, triBase = 0; // the first ones in the pool
    bool     hasN = false, hasUV = false;
};

// One flattened copy of a mesh: vertices [srcVtx, srcVtx + nv) of the pool,
// mapped by `m` (3 x 4, row-major), go to [dstVtx, ..), triangles [srcTri,
// srcTri + nt) to [dstTri, ..).
struct FlatInst
{
    double   it[9];  // inverse transpose of the linear part (normals); unused when ident
    float    m[12];
    uint64_t srcVtx, srcTri;
    uint32_t dstVtx, nv, dstTri, nt;
    uint32_t w;      // 4th word of the triangles' index entries (the material)
    uint32_t flags;  // 1: normals, 2: uvs, 4: the transform is the identity
};

class MeshPool
{
public:
    // Uploads the meshes as given and checks their vertex indices.  On an
    // error the pool keeps what it held.  Without room on the device the pool is
    // page-locked host memory.
    cl_status build(const cl_mesh_desc* meshes, uint32_t n, cudaStream_t st, std::string* err);
    // New vertices of one mesh (normals, tangents: null keeps them).  Refuses
    // positions that are not finite before anything changes.  The arrays are
    // read until the stream has been synchronised.
    cl_status updateVertices(uint32_t mesh, const float* pos, const float* nrm, const float* tan, cudaStream_t st,
                             std::string* err);
    // Moves a pool on the device to page-locked host memory and releases the
    // edits' staging; false where there is nothing to release or no host memory.
    bool spill(cudaStream_t st);

    // The copy of `mesh` at (dstVtx, dstTri) under `M`; refuses a singular M.
    // `what` names it in the message.
    cl_status flatInst(uint32_t mesh, const float* M, uint32_t dstVtx, uint32_t dstTri, uint32_t w,
                       const std::string& what, FlatInst* out, std::string* err) const;
    // Writes the vertices (3 float4 each: {p, n.x} {n.yz, t.xy} {t.z, u, v,
    // flags}) of copies [first, first + count) of the table `inst` (`host`: the
    // same table in host memory).  The copies' destinations are consecutive.
    cl_status flattenVertices(const DevBuf& inst, const FlatInst* host, uint32_t first, uint32_t count, void* vtx,
                              cudaStream_t st, std::string* err) const;
    // The same for `count` copies of one mesh: entries list[0, count) (device) of the table.
    cl_status flattenCopies(uint32_t mesh, const DevBuf& inst, const uint32_t* list, uint32_t count, void* vtx,
                            cudaStream_t st, std::string* err) const;
    // Writes the index entries {3 vertex ids, w} of all `count` copies' triangles.
    cl_status flattenTriangles(const DevBuf& inst, const FlatInst* host, uint32_t count, void* triIdx, cudaStream_t st,
                               std::string* err) const;
    // World boxes of the vertices of copies [first, first + count), in double: 3 minima, 3 maxima per copy.
    cl_status instanceBoxes(const DevBuf& inst, uint32_t first, uint32_t count, std::vector<double>* boxes, cudaStream_t st,
                            std::string* err) const;

    size_t          size() const { return info_.size(); }
    const MeshInfo& operator[](size_t i) const { return info_[i]; }

private:
    float*    pos() const { return mem_.f(); }
    float*    nrm() const { return mem_.f() + 3 * nv_; }
    float*    tan() const { return mem_.f() + 6 * nv_; }
    float*    uv() const { return mem_.f() + 9 * nv_; }
    uint32_t* idx() const { return mem_.u() + 11 * nv_; }

    cl_status put(float* dst, const float* src, size_t bytes, cudaStream_t st, std::string* err);

    std::vector<MeshInfo> info_;
    DevBuf                mem_;    // positions | normals | tangents | uvs | triangle indices, mesh after mesh
    size_t                nv_ = 0; // vertices in the pool
    DevBuf                edit_;   // staging of an edit: 9 floats per vertex and an error word
};

// Bounds of n flattened vertices (ignoring NaN), FLT_MAX / -FLT_MAX where there are none.
cl_status vertexBounds(const void* vtx, size_t n, cudaStream_t st, float lo[3], float hi[3], std::string* err);

} // namespace clb
