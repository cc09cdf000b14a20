// Device build of the 8-wide compressed BVH (layout in cl_bvh.cuh).
//
// Replaces OptiX's BLAS/TLAS builds (owlGroupBuildAccel,
// src/core/devices/optixdevice.cpp:136-233) with a hand-written builder:
//   1. per-triangle boxes and centroid bounds;
//   2. 63-bit Morton codes of the centroids, sorted (CUB radix sort);
//   3. binary tree by PLOC clustering over the Morton order (Meister and
//      Bittner 2018), SAH-quality at LBVH speed; the binary radix tree of
//      Karras (HPG 2012) with bottom-up boxes is kept as a fallback;
//   4. surface-area-optimal collapse to 8-wide nodes (Ylitie, Karras and
//      Laine, HPG 2017): slot costs bottom up over the binary tree, then one
//      level of wide nodes per launch, each taking the children that the
//      costs' minima give it; subtrees of at most 3 triangles become leaf
//      slots; slots are assigned by octant; child boxes are quantised to
//      8 bits per plane, rounded outwards around a widened parent box.
#include "cl_bvh.cuh"
#include "cl_internal.h"

#include <cub/device/device_radix_sort.cuh>

#include <vector>

namespace clb
{
namespace
{
constexpr uint32_t kLeafFlag = 0x80000000u;

__device__ __forceinline__ uint32_t fordered(float f)
{
    uint32_t b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float funordered(uint32_t b)
{
    return __uint_as_float((b & 0x80000000u) ? (b & 0x7fffffffu) : ~b);
}

// Widening of every child box before quantisation: 2^-20 of the scene
// scale (the product is exact, so host and device agree bit for bit).
__host__ __device__ inline float sceneMargin(const float lo[3], const float hi[3])
{
    float scale = 0.0f;
    for (int a = 0; a < 3; ++a)
    {
        scale = fmaxf(scale, fmaxf(fabsf(lo[a]), fabsf(hi[a])));
        scale = fmaxf(scale, hi[a] - lo[a]);
    }
    return scale * 9.5367431640625e-07f + 1e-30f;
}

struct Bounds
{
    uint32_t clo[3], chi[3]; // centroid bounds (ordered ints)
    uint32_t slo[3], shi[3]; // scene bounds
};

// Grid-stride, reduced per block, one atomic per block and value (a warp's
// atomics on the 12 words cost 292 us for 1.17 M triangles, 18 us this way).
constexpr int kBoundsThreads = 256;
__global__ void __launch_bounds__(kBoundsThreads) kTriBounds(const float* __restrict__ tri9, uint32_t n,
                                                             float* __restrict__ lo, float* __restrict__ hi, Bounds* b)
{
    __shared__ uint32_t part[12][kBoundsThreads / 32];
    uint32_t            v[12]; // centroid min, max, box min, max (ordered), 3 axes each
    for (int k = 0; k < 12; ++k) v[k] = (k / 3) & 1 ? 0u : 0xffffffffu;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    {
        const float* t = tri9 + 9 * size_t(i);
        for (int a = 0; a < 3; ++a)
        {
            const float l = fminf(fminf(t[a], t[3 + a]), t[6 + a]), h = fmaxf(fmaxf(t[a], t[3 + a]), t[6 + a]);
            const uint32_t c = fordered(0.5f * l + 0.5f * h);
            lo[3 * size_t(i) + a] = l;
            hi[3 * size_t(i) + a] = h;
            v[a]                  = min(v[a], c);
            v[3 + a]              = max(v[3 + a], c);
            v[6 + a]              = min(v[6 + a], fordered(l));
            v[9 + a]              = max(v[9 + a], fordered(h));
        }
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int k = 0; k < 12; ++k)
    {
        for (int o = 16; o > 0; o >>= 1)
        {
            const uint32_t x = __shfl_xor_sync(0xffffffffu, v[k], o);
            v[k]             = (k / 3) & 1 ? max(v[k], x) : min(v[k], x);
        }
        if (lane == 0) part[k][warp] = v[k];
    }
    __syncthreads();
    if (threadIdx.x < 12)
    {
        const int  k   = threadIdx.x;
        const bool mx  = (k / 3) & 1;
        uint32_t   x   = part[k][0];
        uint32_t*  dst = k < 3 ? b->clo + k : k < 6 ? b->chi + (k - 3) : k < 9 ? b->slo + (k - 6) : b->shi + (k - 9);
        for (int w = 1; w < kBoundsThreads / 32; ++w) x = mx ? max(x, part[k][w]) : min(x, part[k][w]);
        if (mx)
            atomicMax(dst, x);
        else
            atomicMin(dst, x);
    }
}

__device__ __forceinline__ uint64_t expand21(uint32_t v)
{
    uint64_t x = v & 0x1fffffu;
    x          = (x | x << 32) & 0x1f00000000ffffull;
    x          = (x | x << 16) & 0x1f0000ff0000ffull;
    x          = (x | x << 8) & 0x100f00f00f00f00full;
    x          = (x | x << 4) & 0x10c30c30c30c30c3ull;
    x          = (x | x << 2) & 0x1249249249249249ull;
    return x;
}

__global__ void kMorton(const float* __restrict__ lo, const float* __restrict__ hi, uint32_t n, const Bounds* b,
                        uint64_t* __restrict__ keys, uint32_t* __restrict__ ids)
{
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint32_t q[3];
    for (int a = 0; a < 3; ++a)
    {
        float cmin = funordered(b->clo[a]), cmax = funordered(b->chi[a]);
        float c    = 0.5f * lo[3 * size_t(i) + a] + 0.5f * hi[3 * size_t(i) + a];
        float ext  = cmax - cmin;
        float u    = ext > 0.0f ? (c - cmin) / ext : 0.5f;
        u          = fminf(fmaxf(u, 0.0f), 1.0f);
        q[a]       = min(uint32_t(u * 2097152.0f), 2097151u);
    }
    keys[i] = expand21(q[0]) | (expand21(q[1]) << 1) | (expand21(q[2]) << 2);
    ids[i]  = i;
}

__device__ __forceinline__ int delta(const uint64_t* keys, int n, int i, int j)
{
    if (j < 0 || j > n - 1) return -1;
    uint64_t a = keys[i], b = keys[j];
    if (a == b) return 64 + __clz(uint32_t(i) ^ uint32_t(j));
    return __clzll(a ^ b);
}

__global__ void kRadixTree(const uint64_t* __restrict__ keys, int n, uint32_t* __restrict__ left,
                           uint32_t* __restrict__ right, uint32_t* __restrict__ parent)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n - 1) return;
    int d    = (delta(keys, n, i, i + 1) - delta(keys, n, i, i - 1)) >= 0 ? 1 : -1;
    int dmin = delta(keys, n, i, i - d);
    int lmax = 2;
    while (delta(keys, n, i, i + lmax * d) > dmin) lmax *= 2;
    int l = 0;
    for (int t = lmax / 2; t >= 1; t /= 2)
        if (delta(keys, n, i, i + (l + t) * d) > dmin) l += t;
    int j     = i + l * d;
    int dnode = delta(keys, n, i, j);
    int s     = 0;
    int t     = l;
    do
    {
        t = (t + 1) / 2;
        if (delta(keys, n, i, i + (s + t) * d) > dnode) s += t;
    } while (t > 1);
    int      g  = i + s * d + min(d, 0);
    uint32_t lc = (min(i, j) == g) ? (uint32_t(g) | kLeafFlag) : uint32_t(g);
    uint32_t rc = (max(i, j) == g + 1) ? (uint32_t(g + 1) | kLeafFlag) : uint32_t(g + 1);
    left[i]     = lc;
    right[i]    = rc;
    parent[(lc & kLeafFlag) ? (n - 1 + (lc & ~kLeafFlag)) : lc] = uint32_t(i);
    parent[(rc & kLeafFlag) ? (n - 1 + (rc & ~kLeafFlag)) : rc] = uint32_t(i);
}

__device__ __forceinline__ void refBox(uint32_t ref, const float* lo, const float* hi, const uint32_t* ids,
                                       const float* nlo, const float* nhi, float* l, float* h)
{
    if (ref & kLeafFlag)
    {
        uint32_t t = ids[ref & ~kLeafFlag];
        for (int a = 0; a < 3; ++a)
        {
            l[a] = lo[3 * size_t(t) + a];
            h[a] = hi[3 * size_t(t) + a];
        }
    }
    else
        for (int a = 0; a < 3; ++a)
        {
            l[a] = __ldcg(nlo + 3 * size_t(ref) + a);
            h[a] = __ldcg(nhi + 3 * size_t(ref) + a);
        }
}

__global__ void kBottomUp(int n, const float* __restrict__ lo, const float* __restrict__ hi, const uint32_t* __restrict__ ids,
                          const uint32_t* __restrict__ left, const uint32_t* __restrict__ right,
                          const uint32_t* __restrict__ parent, float* nlo, float* nhi, uint32_t* count,
                          uint32_t* arrive)
{
    int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    uint32_t node = parent[n - 1 + j];
    while (node != 0xffffffffu)
    {
        __threadfence();
        if (atomicAdd(&arrive[node], 1u) == 0u) return;
        __threadfence();
        float    l0[3], h0[3], l1[3], h1[3];
        uint32_t a = left[node], b = right[node];
        refBox(a, lo, hi, ids, nlo, nhi, l0, h0);
        refBox(b, lo, hi, ids, nlo, nhi, l1, h1);
        for (int k = 0; k < 3; ++k)
        {
            nlo[3 * size_t(node) + k] = fminf(l0[k], l1[k]);
            nhi[3 * size_t(node) + k] = fmaxf(h0[k], h1[k]);
        }
        uint32_t ca = (a & kLeafFlag) ? 1u : __ldcg(count + a);
        uint32_t cb = (b & kLeafFlag) ? 1u : __ldcg(count + b);
        count[node] = ca + cb;
        node        = parent[node];
    }
}

// ---------------------------------------------------------------------------
// PLOC (Meister and Bittner, "Parallel Locally-Ordered Clustering for
// Bounding Volume Hierarchy Construction", IEEE TVCG 2018).  Clusters start as
// the Morton-sorted triangles; each iteration finds every cluster's nearest
// neighbour (smallest merged surface area) within a window of +-kPlocRadius
// positions, merges mutual nearest neighbours into a new inner node and
// compacts the cluster list in order, until one cluster is left.
// ---------------------------------------------------------------------------
constexpr int kPlocRadius = 16;
constexpr int kPlocBlock  = 256;

__device__ __forceinline__ float mergedArea(float4 alo, float4 ahi, float4 blo, float4 bhi)
{
    float dx = fmaxf(ahi.x, bhi.x) - fminf(alo.x, blo.x);
    float dy = fmaxf(ahi.y, bhi.y) - fminf(alo.y, blo.y);
    float dz = fmaxf(ahi.z, bhi.z) - fminf(alo.z, blo.z);
    return dx * dy + dy * dz + dz * dx;
}

__global__ void kPlocInit(uint32_t n, const uint32_t* __restrict__ ids, const float* __restrict__ lo,
                          const float* __restrict__ hi, uint32_t* __restrict__ C, float4* __restrict__ blo,
                          float4* __restrict__ bhi)
{
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint32_t t = ids[i];
    C[i]       = i | kLeafFlag;
    blo[i]     = make_float4(lo[3 * size_t(t)], lo[3 * size_t(t) + 1], lo[3 * size_t(t) + 2], 0.0f);
    bhi[i]     = make_float4(hi[3 * size_t(t)], hi[3 * size_t(t) + 1], hi[3 * size_t(t) + 2], 0.0f);
}

// Iterations over many clusters take three launches: the nearest neighbours,
// the compaction's ranks (the last block to end adds up the blocks' counts, so
// no scan library call and no separate count kernel), and the merged list with
// its tree nodes.  The cluster count lives in device memory, so that
// iterations run without a host round trip; launches are sized for an upper
// bound and threads past the count return.  From kPlocFinish clusters on, one
// block does the remaining iterations (about 35 of 55) in shared memory.
// Before: six launches for each iteration; the clustering of 1.17 M triangles
// took 1.63 ms of kernels in 324 launches, now 0.89 ms in 73 (0.17 of it the one-block kernel).
constexpr int kPlocTile    = 1024; // clusters per block of the rank kernel
constexpr int kPlocMaxIter = 4098; // then the radix tree (many equal boxes merge one pair per iteration)

struct PlocState
{
    uint32_t m[2];        // clusters in this iteration's and the next one's list
    uint32_t nodeCounter; // inner nodes made
    uint32_t blocksDone;
};

struct PlocList
{
    uint32_t* C;   // cluster references
    float4*   lo;  // their boxes
    float4*   hi;
};

struct PlocTree
{
    uint32_t* left;
    uint32_t* right;
    float*    nlo;
    float*    nhi;
    uint32_t* count;
};

__device__ __forceinline__ void plocNode(const PlocTree& T, uint32_t k, uint32_t a, uint32_t b, float4 lo, float4 hi)
{
    T.left[k]                = a;
    T.right[k]               = b;
    T.nlo[3 * size_t(k)]     = lo.x;
    T.nlo[3 * size_t(k) + 1] = lo.y;
    T.nlo[3 * size_t(k) + 2] = lo.z;
    T.nhi[3 * size_t(k)]     = hi.x;
    T.nhi[3 * size_t(k) + 1] = hi.y;
    T.nhi[3 * size_t(k) + 2] = hi.z;
    const uint32_t ca = (a & kLeafFlag) ? 1u : T.count[a];
    const uint32_t cb = (b & kLeafFlag) ? 1u : T.count[b];
    T.count[k]        = ca + cb;
}

__global__ void __launch_bounds__(kPlocBlock) kPlocNearest(const PlocState* st, int cur, PlocList L, uint32_t* __restrict__ nn)
{
    const uint32_t m = st->m[cur];
    if (m <= 1u) return;
    __shared__ float4 slo[kPlocBlock + 2 * kPlocRadius], shi[kPlocBlock + 2 * kPlocRadius];
    const int b0 = int(blockIdx.x) * kPlocBlock - kPlocRadius;
    for (int k = threadIdx.x; k < kPlocBlock + 2 * kPlocRadius; k += kPlocBlock)
    {
        int g = b0 + k;
        if (g >= 0 && g < int(m))
        {
            slo[k] = L.lo[g];
            shi[k] = L.hi[g];
        }
    }
    __syncthreads();
    int i = int(blockIdx.x) * kPlocBlock + int(threadIdx.x);
    if (i >= int(m)) return;
    int    li = i - b0;
    float4 alo = slo[li], ahi = shi[li];
    float  best  = FLT_MAX;
    int    bestj = i == 0 ? 1 : i - 1;
    int    j0 = max(0, i - kPlocRadius), j1 = min(int(m) - 1, i + kPlocRadius);
    for (int j = j0; j <= j1; ++j)
    {
        if (j == i) continue;
        float c = mergedArea(alo, ahi, slo[j - b0], shi[j - b0]);
        if (c < best)
        {
            best  = c;
            bestj = j;
        }
    }
    nn[i] = uint32_t(bestj);
}

// Rank of each surviving cluster within its block's tile (~0: merged into an
// earlier one); the last block turns the tiles' counts into their bases.
__global__ void __launch_bounds__(kPlocBlock) kPlocRank(PlocState* st, int cur, const uint32_t* __restrict__ nn,
                                                        uint32_t* __restrict__ rank, uint32_t* tileBase)
{
    constexpr int       kWarps = kPlocBlock / 32, kPer = kPlocTile / kPlocBlock;
    __shared__ uint32_t wc[kPer * kWarps];
    __shared__ uint32_t sum[kPlocBlock];
    __shared__ bool     last;
    const uint32_t      m = st->m[cur], tiles = (m + kPlocTile - 1u) / kPlocTile;
    const uint32_t      w = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    if (blockIdx.x < tiles)
    {
        uint32_t local[kPer];
        for (int r = 0; r < kPer; ++r)
        {
            const uint32_t i    = blockIdx.x * uint32_t(kPlocTile) + uint32_t(r * kPlocBlock) + threadIdx.x;
            bool           keep = false;
            if (i < m)
            {
                const uint32_t j = m > 1u ? nn[i] : 0u;
                keep             = m <= 1u || !(j < i && nn[j] == i);
            }
            const uint32_t mask = __ballot_sync(0xffffffffu, keep);
            local[r]            = keep ? uint32_t(__popc(mask & ((1u << lane) - 1u))) : 0xffffffffu;
            if (lane == 0u) wc[r * kWarps + int(w)] = uint32_t(__popc(mask));
        }
        __syncthreads();
        if (threadIdx.x == 0)
        {
            uint32_t acc = 0u;
            for (int k = 0; k < kPer * kWarps; ++k)
            {
                const uint32_t x = wc[k];
                wc[k]            = acc;
                acc += x;
            }
            tileBase[blockIdx.x] = acc;
        }
        __syncthreads();
        for (int r = 0; r < kPer; ++r)
        {
            const uint32_t i = blockIdx.x * uint32_t(kPlocTile) + uint32_t(r * kPlocBlock) + threadIdx.x;
            if (i < m) rank[i] = local[r] == 0xffffffffu ? 0xffffffffu : wc[r * kWarps + int(w)] + local[r];
        }
    }
    if (threadIdx.x == 0)
    {
        __threadfence();
        last = atomicAdd(&st->blocksDone, 1u) == gridDim.x - 1u;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    // Exclusive scan of the tiles' counts: each thread a run of them.
    const uint32_t per = (tiles + kPlocBlock - 1u) / kPlocBlock, b = min(tiles, threadIdx.x * per), e = min(tiles, b + per);
    uint32_t       s   = 0u;
    for (uint32_t t = b; t < e; ++t) s += __ldcg(tileBase + t);
    sum[threadIdx.x] = s;
    __syncthreads();
    for (uint32_t o = 1u; o < uint32_t(kPlocBlock); o <<= 1)
    {
        const uint32_t x = threadIdx.x >= o ? sum[threadIdx.x - o] : 0u;
        __syncthreads();
        sum[threadIdx.x] += x;
        __syncthreads();
    }
    uint32_t acc = sum[threadIdx.x] - s;
    for (uint32_t t = b; t < e; ++t)
    {
        const uint32_t x = __ldcg(tileBase + t);
        tileBase[t]      = acc;
        acc += x;
    }
    if (threadIdx.x == kPlocBlock - 1)
    {
        st->m[cur ^ 1]  = sum[kPlocBlock - 1];
        st->blocksDone = 0u;
    }
}

// The next list: clusters move to their rank, mutual nearest neighbours become
// a new inner node.
__global__ void __launch_bounds__(kPlocBlock) kPlocEmit(PlocState* st, int cur, const uint32_t* __restrict__ nn,
                                                        const uint32_t* __restrict__ rank,
                                                        const uint32_t* __restrict__ tileBase, PlocList L, PlocList N,
                                                        PlocTree T, uint32_t maxInner)
{
    const uint32_t m = st->m[cur];
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t r = i < m ? rank[i] : 0xffffffffu;
    uint32_t       j = 0u;
    bool           merge = false;
    if (r != 0xffffffffu && m > 1u)
    {
        j     = nn[i];
        merge = nn[j] == i;
    }
    // One counter update per warp.
    const uint32_t mask = __ballot_sync(0xffffffffu, merge), lane = threadIdx.x & 31u;
    uint32_t       k    = 0u;
    if (mask)
    {
        if (lane == uint32_t(__ffs(mask) - 1)) k = atomicAdd(&st->nodeCounter, uint32_t(__popc(mask)));
        k = __shfl_sync(0xffffffffu, k, __ffs(mask) - 1) + uint32_t(__popc(mask & ((1u << lane) - 1u)));
    }
    if (r == 0xffffffffu) return;
    const uint32_t d  = tileBase[i / kPlocTile] + r;
    uint32_t       c  = L.C[i];
    float4         lo = L.lo[i], hi = L.hi[i];
    if (merge && k < maxInner)
    {
        const float4 l2 = L.lo[j], h2 = L.hi[j];
        lo = make_float4(fminf(lo.x, l2.x), fminf(lo.y, l2.y), fminf(lo.z, l2.z), 0.0f);
        hi = make_float4(fmaxf(hi.x, h2.x), fmaxf(hi.y, h2.y), fmaxf(hi.z, h2.z), 0.0f);
        plocNode(T, k, c, L.C[j], lo, hi);
        c = k;
    }
    N.C[d]  = c;
    N.lo[d] = lo;
    N.hi[d] = hi;
}

// The remaining iterations over at most kPlocFinish clusters, in one block:
// boxes in shared memory (one array per coordinate, so that a warp's window
// reads have no bank conflicts), compacted in place.  Leaves the root (or,
// after maxIter iterations, what is left) in the list and its count in st->m[cur].
constexpr int kPlocFinish        = 4096;
constexpr int kPlocFinishThreads = 1024;
constexpr size_t kPlocFinishSmem = size_t(kPlocFinish) * 32;
__global__ void __launch_bounds__(kPlocFinishThreads) kPlocFinishList(PlocState* st, int cur, PlocList L, PlocTree T,
                                                                      uint32_t maxInner, int maxIter)
{
    extern __shared__ float plocSmem[];
    constexpr int       kPer = kPlocFinish / kPlocFinishThreads;
    float* const        bx   = plocSmem; // 6 coordinate arrays
    uint32_t* const     C    = reinterpret_cast<uint32_t*>(plocSmem + 6 * kPlocFinish);
    uint32_t* const     nn   = C + kPlocFinish;
    __shared__ uint32_t wc[kPer * 32], wm[kPer * 32];
    __shared__ uint32_t mNext, nodes;
    const uint32_t      w = threadIdx.x >> 5, lane = threadIdx.x & 31u, lt = (1u << lane) - 1u;
    uint32_t            m = st->m[cur];
    if (m > uint32_t(kPlocFinish)) return; // not launched so; the host falls back
    for (uint32_t i = threadIdx.x; i < m; i += kPlocFinishThreads)
    {
        const float4 l = L.lo[i], h = L.hi[i];
        C[i]                   = L.C[i];
        bx[i]                  = l.x;
        bx[kPlocFinish + i]     = l.y;
        bx[2 * kPlocFinish + i] = l.z;
        bx[3 * kPlocFinish + i] = h.x;
        bx[4 * kPlocFinish + i] = h.y;
        bx[5 * kPlocFinish + i] = h.z;
    }
    if (threadIdx.x == 0) nodes = st->nodeCounter;
    __syncthreads();
    const auto box = [&](uint32_t i, float4* l, float4* h) {
        *l = make_float4(bx[i], bx[kPlocFinish + i], bx[2 * kPlocFinish + i], 0.0f);
        *h = make_float4(bx[3 * kPlocFinish + i], bx[4 * kPlocFinish + i], bx[5 * kPlocFinish + i], 0.0f);
    };
    for (int iter = 0; m > 1u && iter < maxIter; ++iter)
    {
        for (uint32_t i = threadIdx.x; i < m; i += kPlocFinishThreads)
        {
            float4 al, ah, bl, bh;
            box(i, &al, &ah);
            float    best  = FLT_MAX;
            uint32_t bestj = i == 0u ? 1u : i - 1u;
            const uint32_t j0 = i > uint32_t(kPlocRadius) ? i - kPlocRadius : 0u, j1 = min(m - 1u, i + kPlocRadius);
            for (uint32_t j = j0; j <= j1; ++j)
            {
                if (j == i) continue;
                box(j, &bl, &bh);
                const float c = mergedArea(al, ah, bl, bh);
                if (c < best)
                {
                    best  = c;
                    bestj = j;
                }
            }
            nn[i] = bestj;
        }
        __syncthreads();
        // Survivors and merges of this thread's clusters, ranked in list order.
        uint32_t keep[kPer], mrank[kPer];
        bool     merge[kPer];
#pragma unroll
        for (int r = 0; r < kPer; ++r)
        {
            const uint32_t i = uint32_t(r * kPlocFinishThreads) + threadIdx.x;
            bool           k = false;
            merge[r]         = false;
            if (i < m)
            {
                const uint32_t j = nn[i];
                const bool     mutual = nn[j] == i;
                k                = !(mutual && j < i);
                merge[r]         = mutual && j > i;
            }
            const uint32_t mk = __ballot_sync(0xffffffffu, k), mm = __ballot_sync(0xffffffffu, merge[r]);
            keep[r]  = k ? uint32_t(__popc(mk & lt)) : 0xffffffffu;
            mrank[r] = uint32_t(__popc(mm & lt));
            if (lane == 0u)
            {
                wc[r * 32 + int(w)] = uint32_t(__popc(mk));
                wm[r * 32 + int(w)] = uint32_t(__popc(mm));
            }
        }
        __syncthreads();
        if (w == 0u)
        {
            // Exclusive scans of the kPer * 32 warp counts: lane l adds entries [kPer l, kPer l + kPer).
            uint32_t a = 0u, b = 0u;
            for (int q = 0; q < kPer; ++q)
            {
                a += wc[kPer * int(lane) + q];
                b += wm[kPer * int(lane) + q];
            }
            uint32_t sa = a, sb = b;
            for (int o = 1; o < 32; o <<= 1)
            {
                const uint32_t xa = __shfl_up_sync(0xffffffffu, sa, o), xb = __shfl_up_sync(0xffffffffu, sb, o);
                if (int(lane) >= o)
                {
                    sa += xa;
                    sb += xb;
                }
            }
            if (lane == 31u) mNext = sa;
            uint32_t ea = sa - a, eb = sb - b + nodes;
            __syncwarp();
            if (lane == 31u) nodes += sb;
            for (int q = 0; q < kPer; ++q)
            {
                const uint32_t xa = wc[kPer * int(lane) + q], xb = wm[kPer * int(lane) + q];
                wc[kPer * int(lane) + q] = ea;
                wm[kPer * int(lane) + q] = eb;
                ea += xa;
                eb += xb;
            }
        }
        __syncthreads();
        uint32_t c[kPer];
        float4   lo[kPer], hi[kPer];
#pragma unroll
        for (int r = 0; r < kPer; ++r)
        {
            const uint32_t i = uint32_t(r * kPlocFinishThreads) + threadIdx.x;
            if (keep[r] == 0xffffffffu) continue;
            c[r] = C[i];
            box(i, &lo[r], &hi[r]);
            const uint32_t k = wm[r * 32 + int(w)] + mrank[r];
            if (merge[r] && k < maxInner)
            {
                float4 l2, h2;
                box(nn[i], &l2, &h2);
                lo[r] = make_float4(fminf(lo[r].x, l2.x), fminf(lo[r].y, l2.y), fminf(lo[r].z, l2.z), 0.0f);
                hi[r] = make_float4(fmaxf(hi[r].x, h2.x), fmaxf(hi[r].y, h2.y), fmaxf(hi[r].z, h2.z), 0.0f);
                plocNode(T, k, c[r], C[nn[i]], lo[r], hi[r]);
                c[r] = k;
            }
            keep[r] += wc[r * 32 + int(w)];
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < kPer; ++r)
        {
            if (keep[r] == 0xffffffffu) continue;
            const uint32_t d        = keep[r];
            C[d]                    = c[r];
            bx[d]                   = lo[r].x;
            bx[kPlocFinish + d]     = lo[r].y;
            bx[2 * kPlocFinish + d] = lo[r].z;
            bx[3 * kPlocFinish + d] = hi[r].x;
            bx[4 * kPlocFinish + d] = hi[r].y;
            bx[5 * kPlocFinish + d] = hi[r].z;
        }
        m = mNext;
        __syncthreads();
    }
    if (threadIdx.x == 0)
    {
        L.C[0]          = C[0];
        st->m[cur]      = m;
        st->nodeCounter = nodes;
    }
}

// ---------------------------------------------------------------------------
// Surface-area-optimal collapse (Ylitie, Karras and Laine, "Efficient
// incoherent ray traversal on GPUs through compressed wide BVHs", HPG 2017):
// cost(n, i), i = 1..8, is the smallest surface-area cost of representing the
// binary subtree of n with at most i slots of a wide node.
//   dist(n, j)  = min over k of cost(left, k) + cost(right, j - k)
//   cost(n, 1)  = A(n) c_tri |T(n)|          if |T(n)| <= 3 (a leaf slot)
//               = dist(n, 8) + A(n) c_node   otherwise (a wide node)
//   cost(n, i)  = min(cost(n, i - 1), dist(n, i))
// A triangle costs A(t) c_tri for any i.  Computed bottom up (the second
// child to arrive at a node computes it); kCollapse then distributes each
// wide node's 8 slots by the same minima.
// ---------------------------------------------------------------------------
constexpr float kCostNode = 1.0f; // a wide-node visit
constexpr float kCostTri  = 1.2f; // a triangle test, relative to a node visit (measured: 0.15-1.2)

__device__ __forceinline__ float halfArea(const float* l, const float* h)
{
    float dx = h[0] - l[0], dy = h[1] - l[1], dz = h[2] - l[2];
    return dx * dy + dy * dz + dz * dx;
}

__global__ void kDpParents(uint32_t ni, const uint32_t* __restrict__ left, const uint32_t* __restrict__ right,
                           uint32_t* __restrict__ parent, uint32_t* __restrict__ leafParent)
{
    uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= ni) return;
    uint32_t c[2] = {left[k], right[k]};
    for (int q = 0; q < 2; ++q)
    {
        if (c[q] & kLeafFlag)
            leafParent[c[q] & ~kLeafFlag] = k;
        else
            parent[c[q]] = k;
    }
}

// Slot costs of a child reference: a triangle's for every i, else cost[].
__device__ __forceinline__ void dpRefCosts(uint32_t r, const float* lo, const float* hi, const uint32_t* ids,
                                           const float* cost, float c[8])
{
    if (r & kLeafFlag)
    {
        uint32_t t = ids[r & ~kLeafFlag];
        float    a = halfArea(lo + 3 * size_t(t), hi + 3 * size_t(t)) * kCostTri;
        for (int i = 0; i < 8; ++i) c[i] = a;
    }
    else
    {
        const float4 a = __ldcg(reinterpret_cast<const float4*>(cost + 8 * size_t(r)));
        const float4 b = __ldcg(reinterpret_cast<const float4*>(cost + 8 * size_t(r)) + 1);
        c[0] = a.x, c[1] = a.y, c[2] = a.z, c[3] = a.w;
        c[4] = b.x, c[5] = b.y, c[6] = b.z, c[7] = b.w;
    }
}

__global__ void kDpCosts(uint32_t n, const uint32_t* __restrict__ leafParent, const uint32_t* __restrict__ parent,
                         const uint32_t* __restrict__ left, const uint32_t* __restrict__ right,
                         const float* __restrict__ lo, const float* __restrict__ hi, const uint32_t* __restrict__ ids,
                         const float* __restrict__ nlo, const float* __restrict__ nhi,
                         const uint32_t* __restrict__ count, float* cost, uint32_t* arrive)
{
    uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    uint32_t node = leafParent[j];
    while (node != 0xffffffffu)
    {
        __threadfence();
        if (atomicAdd(&arrive[node], 1u) == 0u) return;
        __threadfence();
        float cl[8], cr[8];
        dpRefCosts(left[node], lo, hi, ids, cost, cl);
        dpRefCosts(right[node], lo, hi, ids, cost, cr);
        float dist[9];
        for (int jj = 2; jj <= 8; ++jj)
        {
            float d = FLT_MAX;
            for (int k = 1; k < jj; ++k) d = fminf(d, cl[k - 1] + cr[jj - k - 1]);
            dist[jj] = d;
        }
        float    A   = halfArea(nlo + 3 * size_t(node), nhi + 3 * size_t(node));
        uint32_t cnt = count[node];
        float    c   = cnt <= 3u ? A * kCostTri * float(cnt) : dist[8] + A * kCostNode;
        float*   out = cost + 8 * size_t(node);
        out[0]       = c;
        for (int i = 2; i <= 8; ++i)
        {
            c          = fminf(c, dist[i]);
            out[i - 1] = c;
        }
        node = parent[node];
    }
}

struct CollapseArgs
{
    const float*    triPos; // 9 floats per triangle, original order
    const float*    lo;     // triangle boxes
    const float*    hi;
    const uint32_t* ids;    // sorted position -> triangle id
    const uint32_t* left;
    const uint32_t* right;
    const float*    nlo;
    const float*    nhi;
    const uint32_t* count;
    const float*    cost; // slot costs of the optimal collapse
    uint4*          nodes;
    float4*         tris;
    uint32_t*       nodeCounter;
    uint32_t*       triCounter;
    uint32_t*       nextCount;
    uint2*          nextTasks;
    float           margin;
    uint32_t        maxNodes;
    uint32_t        maxTris;
    uint32_t        maxTasks;
    uint32_t*       err;
};

__device__ __forceinline__ uint32_t refCount(const CollapseArgs& A, uint32_t r)
{
    return (r & kLeafFlag) ? 1u : A.count[r];
}

__device__ __forceinline__ uint32_t quantExp(float ext)
{
    // Smallest power of two e with 255 * e >= ext; returns its biased exponent.
    float    x  = ext / 255.0f;
    uint32_t b  = __float_as_uint(x);
    uint32_t ex = (b >> 23) & 0xffu;
    if (b & 0x7fffffu) ex += 1;
    if (ex < 1) ex = 1;
    if (ex > 254) ex = 254;
    float e = __uint_as_float(ex << 23);
    while (e * 255.0f < ext && ex < 254)
    {
        ++ex;
        e = __uint_as_float(ex << 23);
    }
    return ex;
}

// 8-bit planes of a child interval [lo, hi] in the frame (p, e), rounded
// outwards so that the dequantised box p + e * q contains the interval.
__device__ __forceinline__ void quantPlanes(float lo, float hi, float p, float e, uint32_t* ql, uint32_t* qh)
{
    int lo_ = int(floorf((lo - p) / e));
    int hi_ = int(ceilf((hi - p) / e));
    lo_     = max(0, min(255, lo_));
    hi_     = max(0, min(255, hi_));
    while (lo_ > 0 && p + e * float(lo_) > lo) --lo_;
    while (hi_ < 255 && p + e * float(hi_) < hi) ++hi_;
    *ql = uint32_t(lo_);
    *qh = uint32_t(hi_);
}

// One level of wide nodes, eight lanes per node.  Choosing the children is a
// chain of dependent loads (split after split), in which lane q holds the costs
// of budget q + 1, so a split takes two 32-byte loads and a few shuffles; then
// lane q boxes child q, the octant slots are handed out by an argmax over the
// lanes, and lane q quantises slot q and copies its triangles.  One thread per
// node did all of it in turn: 1.38 ms for the ten levels over 1.17 M triangles
// (31-80 us for each level of a few nodes), now 0.59 ms (17-33 us).
constexpr int kCollapseThreads = 128;
__global__ void __launch_bounds__(kCollapseThreads) kCollapse(CollapseArgs A, const uint2* __restrict__ tasks,
                                                              uint32_t ntasks)
{
    __shared__ uint32_t shCh[kCollapseThreads / 8][8], shN[kCollapseThreads / 8][16], shJ[kCollapseThreads / 8][16];
    __shared__ int      shAt[kCollapseThreads / 8][8];
    const uint32_t      ti = (blockIdx.x * blockDim.x + threadIdx.x) >> 3;
    if (ti >= ntasks) return; // whole groups of 8 lanes
    const uint32_t g = threadIdx.x >> 3, q = threadIdx.x & 7u;
    const uint32_t gs = threadIdx.x & 24u, gm = 0xffu << gs; // the group's lanes in its warp
    const uint32_t ref = tasks[ti].x, wide = tasks[ti].y;
    uint32_t *     ch = shCh[g], *sn = shN[g], *sj = shJ[g];

    // The children: (node, budget) pairs split until a budget of 1 or the cost
    // no longer needs the budget.
    uint32_t cnt = 0;
    if ((ref & kLeafFlag) || A.count[ref] <= 3u)
    {
        if (q == 0u) ch[0] = ref;
        cnt = 1;
    }
    else
    {
        uint32_t sp = 1;
        bool     root = true;
        uint32_t x = ref, j = 8u; // the pair on top of the stack
        while (cnt < 8u)
        {
            --sp;
            bool     leaf = !root && ((x & kLeafFlag) || j == 1u);
            uint32_t i    = j;
            if (!leaf && !root)
            {
                // Fewest slots with the same cost.
                const float    cx = __ldcg(A.cost + 8 * size_t(x) + q);
                const float    cj = __shfl_sync(gm, cx, int(j) - 1, 8);
                const uint32_t eq = (__ballot_sync(gm, cx == cj) >> gs) & 0xffu;
                while (i > 1u && ((eq >> (i - 2u)) & 1u)) --i;
                leaf = i == 1u;
            }
            root = false;
            if (leaf)
            {
                if (q == 0u) ch[cnt] = x;
                ++cnt;
            }
            else
            {
                const uint32_t l = A.left[x], r = A.right[x];
                const auto cost = [&](uint32_t c) {
                    if (!(c & kLeafFlag)) return __ldcg(A.cost + 8 * size_t(c) + q);
                    const uint32_t t = A.ids[c & ~kLeafFlag];
                    return halfArea(A.lo + 3 * size_t(t), A.hi + 3 * size_t(t)) * kCostTri;
                };
                const float cl = cost(l), cr = cost(r);
                // Lane q: budget k = q + 1 for the left child, i - k for the right one.
                const float other = __shfl_sync(gm, cr, (int(i) - 2 - int(q)) & 7, 8);
                float       c     = q + 1u < i ? cl + other : FLT_MAX;
                uint32_t    bk    = q + 1u;
                if (!(c < FLT_MAX)) c = FLT_MAX;
                for (int o = 1; o < 8; o <<= 1)
                {
                    const float    oc = __shfl_xor_sync(gm, c, o, 8);
                    const uint32_t ok = __shfl_xor_sync(gm, bk, o, 8);
                    if (oc < c || (oc == c && ok < bk))
                    {
                        c  = oc;
                        bk = ok;
                    }
                }
                if (q == 0u)
                {
                    sn[sp] = r, sj[sp] = i - bk;
                    sn[sp + 1] = l, sj[sp + 1] = bk;
                }
                sp += 2u;
            }
            __syncwarp(gm);
            if (sp == 0u) break;
            x = sn[sp - 1u];
            j = sj[sp - 1u];
            __syncwarp(gm);
        }
    }
    __syncwarp(gm);

    // Lane q: box of child q, widened by the margin; the parent box.
    const bool     have = q < cnt;
    const uint32_t mine = have ? ch[q] : 0u;
    float          clo[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, chi[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX}, plo[3], phi[3];
    if (have) refBox(mine, A.lo, A.hi, A.ids, A.nlo, A.nhi, clo, chi);
    for (int a = 0; a < 3; ++a)
    {
        if (have)
        {
            clo[a] -= A.margin;
            chi[a] += A.margin;
        }
        plo[a] = clo[a];
        phi[a] = chi[a];
        for (int o = 1; o < 8; o <<= 1)
        {
            plo[a] = fminf(plo[a], __shfl_xor_sync(gm, plo[a], o, 8));
            phi[a] = fmaxf(phi[a], __shfl_xor_sync(gm, phi[a], o, 8));
        }
    }

    // Octant slots: greedy on the alignment of child offset and slot direction
    // (the largest first, ties to the lower child, then the lower slot).
    if (q < 8u) shAt[g][q] = -1;
    __syncwarp(gm);
    const float dx = 0.5f * (clo[0] + chi[0]) - 0.5f * (plo[0] + phi[0]);
    const float dy = 0.5f * (clo[1] + chi[1]) - 0.5f * (plo[1] + phi[1]);
    const float dz = 0.5f * (clo[2] + chi[2]) - 0.5f * (plo[2] + phi[2]);
    uint32_t    used = 0u;
    bool        done = !have;
    for (uint32_t it = 0; it < cnt; ++it)
    {
        float    bc = -FLT_MAX;
        uint32_t bs = uint32_t(__ffs(~used) - 1), bk = done ? 8u : q;
        if (!done)
            for (uint32_t sl = 0; sl < 8u; ++sl)
            {
                const float c = ((sl & 1u) ? dx : -dx) + ((sl & 2u) ? dy : -dy) + ((sl & 4u) ? dz : -dz);
                if (!((used >> sl) & 1u) && c > bc)
                {
                    bc = c;
                    bs = sl;
                }
            }
        for (int o = 1; o < 8; o <<= 1)
        {
            const float    oc = __shfl_xor_sync(gm, bc, o, 8);
            const uint32_t os = __shfl_xor_sync(gm, bs, o, 8), ok = __shfl_xor_sync(gm, bk, o, 8);
            if (ok < 8u && (bk == 8u || oc > bc || (oc == bc && ok < bk)))
            {
                bc = oc;
                bs = os;
                bk = ok;
            }
        }
        used |= 1u << bs;
        if (bk == q)
        {
            done          = true;
            shAt[g][bs] = int(q);
        }
    }
    __syncwarp(gm);

    // Lane q: slot q.
    const int  k       = shAt[g][q];
    const bool present = k >= 0;
    float      slo[3], shi[3];
    for (int a = 0; a < 3; ++a)
    {
        slo[a] = __shfl_sync(gm, clo[a], k & 7, 8);
        shi[a] = __shfl_sync(gm, chi[a], k & 7, 8);
    }
    const uint32_t r      = present ? ch[k] : 0u;
    const uint32_t c      = present ? refCount(A, r) : 0u;
    const bool     inner  = c > 3u;
    const uint32_t leafN  = present && !inner ? c : 0u;
    const uint32_t lt     = (1u << q) - 1u;
    const uint32_t imask  = (__ballot_sync(gm, inner) >> gs) & 0xffu;
    const uint32_t m1     = (__ballot_sync(gm, leafN & 1u) >> gs) & 0xffu, m2 = (__ballot_sync(gm, leafN & 2u) >> gs) & 0xffu;
    const uint32_t nInner = __popc(imask), nTris = __popc(m1) + 2u * __popc(m2);
    const uint32_t triOff = __popc(m1 & lt) + 2u * __popc(m2 & lt), rank = __popc(imask & lt);
    uint32_t       base = 0u, tbase = 0u, tk = 0u;
    if (q == 0u)
    {
        if (nInner)
        {
            base = atomicAdd(A.nodeCounter, nInner);
            tk   = atomicAdd(A.nextCount, nInner);
        }
        tbase = atomicAdd(A.triCounter, nTris);
    }
    base  = __shfl_sync(gm, base, 0, 8);
    tk    = __shfl_sync(gm, tk, 0, 8);
    tbase = __shfl_sync(gm, tbase, 0, 8);
    if (base + nInner > A.maxNodes || tbase + nTris > A.maxTris || tk + nInner > A.maxTasks || wide >= A.maxNodes)
    {
        if (q == 0u) atomicOr(A.err, 2u);
        return;
    }
    if (inner) A.nextTasks[tk + rank] = make_uint2(r, base + rank);

    // Quantisation frame and this slot's planes.
    uint32_t ex[3], ql[3] = {255u, 255u, 255u}, qh[3] = {0u, 0u, 0u};
    for (int a = 0; a < 3; ++a)
    {
        ex[a] = quantExp(phi[a] - plo[a]);
        if (present) quantPlanes(slo[a], shi[a], plo[a], __uint_as_float(ex[a] << 23), &ql[a], &qh[a]);
    }
    uint32_t meta = 0u;
    if (leafN)
    {
        // The subtree's triangles (at most 3).
        uint32_t st[4];
        int      sp  = 0;
        uint32_t got = 0;
        st[sp++]     = r;
        while (sp > 0)
        {
            const uint32_t x = st[--sp];
            if (x & kLeafFlag)
            {
                const uint32_t tid = A.ids[x & ~kLeafFlag];
                const float*   tp  = A.triPos + 9 * size_t(tid);
                float4*        dst = A.tris + size_t(tbase + triOff + got) * kTriF4;
                dst[0]             = make_float4(tp[0], tp[1], tp[2], __uint_as_float(tid));
                dst[1]             = make_float4(tp[3], tp[4], tp[5], 0.0f);
                dst[2]             = make_float4(tp[6], tp[7], tp[8], 0.0f);
                ++got;
            }
            else
            {
                st[sp++] = A.right[x];
                st[sp++] = A.left[x];
            }
        }
        meta = (((1u << got) - 1u) << 5) | triOff;
    }
    // The slots' bytes: OR within each quad of lanes, then the second quad's words to lane 0.
    uint32_t wd[7] = {ql[0], ql[1], ql[2], qh[0], qh[1], qh[2], meta}, w1[7];
    for (int a = 0; a < 7; ++a)
    {
        wd[a] <<= 8u * (q & 3u);
        for (int o = 1; o < 4; o <<= 1) wd[a] |= __shfl_xor_sync(gm, wd[a], o, 8);
        w1[a] = __shfl_down_sync(gm, wd[a], 4, 8);
    }
    if (q == 0u)
    {
        uint4* np = A.nodes + size_t(wide) * kNodeU4;
        np[0]     = make_uint4(__float_as_uint(plo[0]), __float_as_uint(plo[1]), __float_as_uint(plo[2]),
                               ex[0] | (ex[1] << 8) | (ex[2] << 16) | (imask << 24));
        np[1]     = make_uint4(base, tbase, wd[6], w1[6]);
        np[2]     = make_uint4(wd[0], w1[0], wd[1], w1[1]);
        np[3]     = make_uint4(wd[2], w1[2], wd[3], w1[3]);
        np[4]     = make_uint4(wd[4], w1[4], wd[5], w1[5]);
    }
    // Leaf word and scales (n5).
    uint32_t lv = (meta >> 5) << (3u * q);
    for (int o = 1; o < 8; o <<= 1) lv |= __shfl_xor_sync(gm, lv, o, 8);
    if (q == 0u) A.nodes[size_t(wide) * kNodeU4 + 5] = make_uint4(lv, ex[0] << 23, ex[1] << 23, ex[2] << 23);
}

// Validation of a built tree (error bits: 1 exponent outside 1..254 or a scale
// that is not its power of two, 2 child index beyond the node count, 4 leaf
// word or leaf triangle range that is not the slots' or leaves the node's 24 or
// the triangle count, 8 triangle ids not a permutation of 0..n-1).  The
// traversal follows the leaf word (a hit slot's bits and the popcounts below
// them) and the float scales; the slots' metadata state the same.
__global__ void kValidateNodes(const uint4* __restrict__ nodes, uint32_t numNodes, uint32_t n, uint32_t* err)
{
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= numNodes) return;
    const uint4 n0 = nodes[size_t(i) * kNodeU4], n1 = nodes[size_t(i) * kNodeU4 + 1], n5 = nodes[size_t(i) * kNodeU4 + 5];
    uint32_t    imask = n0.w >> 24, bits = 0u;
    const uint32_t scale[3] = {n5.y, n5.z, n5.w};
    for (int a = 0; a < 3; ++a)
    {
        uint32_t e = (n0.w >> (8 * a)) & 0xffu;
        if (e < 1u || e > 254u || scale[a] != e << 23) bits |= 1u;
    }
    if (imask && uint64_t(n1.x) + __popc(imask) > numNodes) bits |= 2u;
    if (n5.x >> 24) bits |= 4u;
    for (int sl = 0; sl < 8; ++sl)
    {
        const uint32_t meta  = ((sl < 4 ? n1.z : n1.w) >> (8 * (sl & 3))) & 0xffu;
        const bool     leaf  = !(imask & (1u << sl)) && meta;
        const uint32_t unary = leaf ? meta >> 5 : 0u, word = (n5.x >> (3 * sl)) & 7u;
        if (word != unary) bits |= 4u;
        if (!leaf) continue;
        const uint32_t off = meta & 31u, cnt = unary == 1u ? 1u : unary == 3u ? 2u : unary == 7u ? 3u : 99u;
        if (cnt == 99u || off != __popc(n5.x & ((1u << (3 * sl)) - 1u)) || off + cnt > 24u || uint64_t(n1.y) + off + cnt > n)
            bits |= 4u;
    }
    if (bits) atomicOr(err, bits);
}

__global__ void kValidateTris(const float4* __restrict__ tris, uint32_t n, uint32_t* __restrict__ seen, uint32_t* err)
{
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint32_t id = __float_as_uint(tris[size_t(i) * kTriF4].w);
    if (id >= n)
    {
        atomicOr(err, 8u);
        return;
    }
    uint32_t bit = 1u << (id & 31u);
    if (atomicOr(seen + (id >> 5), bit) & bit) atomicOr(err, 8u);
}

// Error bits of a tree; seen: a bit per triangle, bits: one word (device).  Synchronises.
cl_status validateBvh(const uint4* nodes, uint32_t numNodes, const float4* tris, uint32_t n, uint32_t* seen,
                      uint32_t* bits, cudaStream_t st, uint32_t* out, std::string* err)
{
    CL_CUDA(cudaMemsetAsync(bits, 0, 4, st), err);
    CL_CUDA(cudaMemsetAsync(seen, 0, (size_t(n) + 31) / 32 * 4, st), err);
    kValidateNodes<<<(numNodes + 255) / 256, 256, 0, st>>>(nodes, numNodes, n, bits);
    kValidateTris<<<(n + 255) / 256, 256, 0, st>>>(tris, n, seen, bits);
    CL_CUDA(cudaGetLastError(), err);
    CL_CUDA(cudaMemcpyAsync(out, bits, 4, cudaMemcpyDeviceToHost, st), err);
    CL_CUDA(cudaStreamSynchronize(st), err);
    return CL_OK;
}

} // namespace

cl_status unitValidateBvh(const uint32_t* nodes, uint32_t numNodes, const float* tris, uint32_t n, uint32_t* bits,
                          std::string* err)
{
    if (!nodes || !tris || !bits || numNodes == 0 || n == 0)
    {
        *err = "a tree to validate needs nodes and triangles";
        return CL_ERR_INVALID_ARG;
    }
    const size_t nb = size_t(numNodes) * kNodeU4 * 16, tb = size_t(n) * kTriF4 * 16;
    DevBuf       d;
    ScratchBuf   dn, dt, seen, word;
    Carver       cv;
    cv.take(dn, nb);
    cv.take(dt, tb);
    cv.take(seen, (size_t(n) + 31) / 32 * 4);
    cv.take(word, 4);
    CL_TRY(d.alloc(cv.peak(), err));
    cv.bind(d.p);
    CL_CUDA(cudaMemcpy(dn.p, nodes, nb, cudaMemcpyHostToDevice), err);
    CL_CUDA(cudaMemcpy(dt.p, tris, tb, cudaMemcpyHostToDevice), err);
    return validateBvh(dn.as<const uint4>(), numNodes, dt.as<const float4>(), n, seen.u(), word.u(), nullptr, bits, err);
}

cl_status buildWideBvh(const float* dTri9, uint32_t n, cudaStream_t st, WideBvh* out, std::string* err,
                       BuildArena* arena)
{
    out->release();
    BuildArena  localArena;
    BuildArena& mem = arena ? *arena : localArena;
    if (n == 0)
    {
        *err = "cannot build a BVH over zero triangles";
        return CL_ERR_INVALID_ARG;
    }
    const size_t   nn = n, ni = nn > 1 ? nn - 1 : 1, taskCap = nn / 2 + 8;
    const uint32_t maxNodes = n + 1, blocks = (n + 255) / 256;

    // One allocation: what the whole build uses, then three phases (sort,
    // clustering, collapse) over the same memory.
    ScratchBuf lo, hi, keys, keys2, ids, ids2, left, right, parent, nlo, nhi, count, arrive, bounds, tmp, ctr, ploc;
    ScratchBuf listC[2], listLo[2], listHi[2], nnb, rank, tileBase;
    ScratchBuf dpCost, dpParent, dpLeafParent, tasksA, tasksB, nodes, tris, verr, seen;
    size_t     tmpBytes = 0;
    CL_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tmpBytes, (uint64_t*)nullptr, (uint64_t*)nullptr, (uint32_t*)nullptr,
                                            (uint32_t*)nullptr, int(n), 0, 63, st),
            err);
    Carver cv;
    cv.take(lo, nn * 12);
    cv.take(hi, nn * 12);
    cv.take(keys2, nn * 8);
    cv.take(ids2, nn * 4);
    cv.take(left, ni * 4);
    cv.take(right, ni * 4);
    cv.take(nlo, ni * 12);
    cv.take(nhi, ni * 12);
    cv.take(count, ni * 4);
    cv.take(bounds, sizeof(Bounds));
    cv.take(ctr, 16);
    cv.take(ploc, sizeof(PlocState));
    const size_t phase = cv.mark();
    cv.take(keys, nn * 8);
    cv.take(ids, nn * 4);
    cv.take(tmp, tmpBytes);
    cv.rewind(phase);
    for (int k = 0; k < 2; ++k)
    {
        cv.take(listC[k], nn * 4);
        cv.take(listLo[k], nn * 16);
        cv.take(listHi[k], nn * 16);
    }
    cv.take(nnb, nn * 4);
    cv.take(rank, nn * 4);
    cv.take(tileBase, (nn + kPlocTile - 1) / kPlocTile * 4);
    cv.take(parent, 2 * nn * 4);
    cv.rewind(phase);
    cv.take(arrive, ni * 4);
    cv.take(dpCost, ni * 32);
    cv.take(dpParent, ni * 4);
    cv.take(dpLeafParent, nn * 4);
    cv.take(tasksA, taskCap * 8);
    cv.take(tasksB, taskCap * 8);
    cv.take(nodes, size_t(maxNodes) * kNodeU4 * 16);
    cv.take(tris, nn * kTriF4 * 16);
    cv.take(verr, 4);
    cv.take(seen, (nn + 31) / 32 * 4);
    CL_TRY(mem.reserve(cv.peak(), err));
    cv.bind(mem.base());

    Bounds b0;
    for (int a = 0; a < 3; ++a)
    {
        b0.clo[a] = b0.slo[a] = 0xffffffffu;
        b0.chi[a] = b0.shi[a] = 0u;
    }
    CL_CUDA(cudaMemcpyAsync(bounds.p, &b0, sizeof(b0), cudaMemcpyHostToDevice, st), err);
    kTriBounds<<<std::min(blocks, 1184u), kBoundsThreads, 0, st>>>(dTri9, n, lo.f(), hi.f(), (Bounds*)bounds.p);
    kMorton<<<blocks, 256, 0, st>>>(lo.f(), hi.f(), n, (Bounds*)bounds.p, (uint64_t*)keys.p, ids.u());
    CL_CUDA(cudaGetLastError(), err);
    CL_CUDA(cub::DeviceRadixSort::SortPairs(tmp.p, tmpBytes, (uint64_t*)keys.p, (uint64_t*)keys2.p, ids.u(), ids2.u(),
                                            int(n), 0, 63, st),
            err);
    Bounds bh; // read back with the clustering's first count
    CL_CUDA(cudaMemcpyAsync(&bh, bounds.p, sizeof(bh), cudaMemcpyDeviceToHost, st), err);

    // Binary tree: PLOC over the Morton order (LBVH radix tree as fallback).
    uint32_t rootRef = kLeafFlag; // a single triangle: the root is a leaf
    if (n > 1)
    {
        PlocList  list[2] = {{listC[0].u(), listLo[0].as<float4>(), listHi[0].as<float4>()},
                             {listC[1].u(), listLo[1].as<float4>(), listHi[1].as<float4>()}};
        PlocTree  T{left.u(), right.u(), nlo.f(), nhi.f(), count.u()};
        PlocState s0{{n, 0u}, 0u, 0u};
        PlocState* ps = ploc.as<PlocState>();
        CL_CUDA(cudaMemcpyAsync(ps, &s0, sizeof(s0), cudaMemcpyHostToDevice, st), err);
        kPlocInit<<<blocks, 256, 0, st>>>(n, ids2.u(), lo.f(), hi.f(), list[0].C, list[0].lo, list[0].hi);
        // The host reads the cluster count every kPlocCheck iterations to size
        // the launches and to hand over to the one-block kernel.
        constexpr int kPlocCheck = 4;
        uint32_t      m   = n;
        int           cur = 0, iters = 0;
        while (m > uint32_t(kPlocFinish) && iters < kPlocMaxIter)
        {
            const uint32_t g = (m + kPlocBlock - 1) / kPlocBlock; // m: upper bound of the device count
            for (int k = 0; k < kPlocCheck; ++k)
            {
                kPlocNearest<<<g, kPlocBlock, 0, st>>>(ps, cur, list[cur], nnb.u());
                kPlocRank<<<(m + kPlocTile - 1) / kPlocTile, kPlocBlock, 0, st>>>(ps, cur, nnb.u(), rank.u(), tileBase.u());
                kPlocEmit<<<g, kPlocBlock, 0, st>>>(ps, cur, nnb.u(), rank.u(), tileBase.u(), list[cur], list[cur ^ 1], T,
                                                    n - 1);
                cur ^= 1;
                ++iters;
            }
            CL_CUDA(cudaGetLastError(), err);
            CL_CUDA(cudaMemcpyAsync(&m, ps->m + cur, 4, cudaMemcpyDeviceToHost, st), err);
            CL_CUDA(cudaStreamSynchronize(st), err);
        }
        if (m <= uint32_t(kPlocFinish))
        {
            CL_CUDA(cudaFuncSetAttribute(kPlocFinishList, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kPlocFinishSmem)),
                    err);
            kPlocFinishList<<<1, kPlocFinishThreads, kPlocFinishSmem, st>>>(ps, cur, list[cur], T, n - 1,
                                                                            kPlocMaxIter - iters);
            CL_CUDA(cudaGetLastError(), err);
            CL_CUDA(cudaMemcpyAsync(&m, ps->m + cur, 4, cudaMemcpyDeviceToHost, st), err);
            CL_CUDA(cudaMemcpyAsync(&rootRef, list[cur].C, 4, cudaMemcpyDeviceToHost, st), err);
            CL_CUDA(cudaStreamSynchronize(st), err);
        }
        if (m != 1)
        {
            // Fall back to the LBVH radix tree (Karras 2012) with bottom-up boxes
            // (rank: the arrival counters).
            CL_CUDA(cudaMemsetAsync(parent.p, 0xff, 2 * nn * 4, st), err);
            CL_CUDA(cudaMemsetAsync(rank.p, 0, ni * 4, st), err);
            kRadixTree<<<(n - 1 + 255) / 256, 256, 0, st>>>((uint64_t*)keys2.p, int(n), left.u(), right.u(),
                                                            parent.u());
            kBottomUp<<<blocks, 256, 0, st>>>(int(n), lo.f(), hi.f(), ids2.u(), left.u(), right.u(), parent.u(),
                                              nlo.f(), nhi.f(), count.u(), rank.u());
            CL_CUDA(cudaGetLastError(), err);
            rootRef = 0u;
        }
    }
    else
        CL_CUDA(cudaStreamSynchronize(st), err); // bh

    float margin;
    {
        auto unord = [](uint32_t v) {
            uint32_t bits = (v & 0x80000000u) ? (v & 0x7fffffffu) : ~v;
            float    f;
            memcpy(&f, &bits, 4);
            return f;
        };
        float l[3], h[3];
        for (int a = 0; a < 3; ++a)
        {
            l[a] = unord(bh.slo[a]);
            h[a] = unord(bh.shi[a]);
        }
        margin = sceneMargin(l, h);
    }

    // ctr: [0] node counter, [1] tri counter, [2] next task count, [3] error
    uint32_t c0[4] = {1u, 0u, 0u, 0u};
    CL_CUDA(cudaMemcpyAsync(ctr.p, c0, 16, cudaMemcpyHostToDevice, st), err);
    uint2 root = make_uint2(rootRef, 0u);
    CL_CUDA(cudaMemcpyAsync(tasksA.p, &root, 8, cudaMemcpyHostToDevice, st), err);

    // Slot costs of the optimal collapse, bottom up over the binary tree.
    if (n > 1)
    {
        CL_CUDA(cudaMemsetAsync(dpParent.p, 0xff, ni * 4, st), err);
        CL_CUDA(cudaMemsetAsync(dpLeafParent.p, 0xff, nn * 4, st), err);
        CL_CUDA(cudaMemsetAsync(arrive.p, 0, ni * 4, st), err);
        kDpParents<<<uint32_t((ni + 255) / 256), 256, 0, st>>>(uint32_t(n - 1), left.u(), right.u(), dpParent.u(),
                                                               dpLeafParent.u());
        kDpCosts<<<blocks, 256, 0, st>>>(n, dpLeafParent.u(), dpParent.u(), left.u(), right.u(), lo.f(), hi.f(),
                                         ids2.u(), nlo.f(), nhi.f(), count.u(), dpCost.f(), arrive.u());
        CL_CUDA(cudaGetLastError(), err);
    }

    CollapseArgs A;
    A.triPos      = dTri9;
    A.lo          = lo.f();
    A.hi          = hi.f();
    A.ids         = ids2.u();
    A.left        = left.u();
    A.right       = right.u();
    A.nlo         = nlo.f();
    A.nhi         = nhi.f();
    A.count       = count.u();
    A.cost        = n > 1 ? dpCost.f() : nullptr; // n == 1: the root is a leaf
    A.nodes       = nodes.as<uint4>();
    A.tris        = tris.as<float4>();
    A.nodeCounter = ctr.u() + 0;
    A.triCounter  = ctr.u() + 1;
    A.nextCount   = ctr.u() + 2;
    A.margin      = margin;
    A.maxNodes    = maxNodes;
    A.maxTris     = n;
    A.maxTasks    = uint32_t(taskCap);
    A.err         = ctr.u() + 3;

    uint32_t ntasks = 1, depth = 0;
    out->levels.assign({0u, 1u});
    ScratchBuf* cur = &tasksA;
    ScratchBuf* nxt = &tasksB;
    while (ntasks > 0)
    {
        ++depth;
        A.nextTasks = nxt->as<uint2>();
        CL_CUDA(cudaMemsetAsync(ctr.u() + 2, 0, 4, st), err);
        kCollapse<<<uint32_t((size_t(ntasks) * 8 + kCollapseThreads - 1) / kCollapseThreads), kCollapseThreads, 0, st>>>(
            A, cur->as<const uint2>(), ntasks);
        CL_CUDA(cudaGetLastError(), err);
        uint32_t hc[4];
        CL_CUDA(cudaMemcpyAsync(hc, ctr.p, 16, cudaMemcpyDeviceToHost, st), err);
        CL_CUDA(cudaStreamSynchronize(st), err);
        if (hc[3])
        {
            *err = "BVH collapse exceeded its node bound";
            return CL_ERR_STATE;
        }
        ntasks = hc[2];
        std::swap(cur, nxt);
        out->numNodes = hc[0];
        if (hc[0] > out->levels.back()) out->levels.push_back(hc[0]);
        if (hc[1] > n)
        {
            *err = "BVH collapse emitted too many triangles";
            return CL_ERR_STATE;
        }
    }
    out->depth   = depth;
    out->numTris = n;
    // The tree in memory of its own size (the collapse's bound is a node per
    // triangle; 1.17 M triangles make 0.15 M), with the refit's state (24 bytes
    // per node), so that a refit allocates nothing.
    {
        Carver keep;
        keep.take(out->nodes, size_t(out->numNodes) * kNodeU4 * 16);
        keep.take(out->tris, nn * kTriF4 * 16);
        keep.take(out->exact, size_t(out->numNodes) * 24);
        keep.take(out->scene, 128);
        CL_TRY(out->mem.alloc(keep.peak(), err));
        keep.bind(out->mem.p);
        CL_CUDA(cudaMemcpyAsync(out->nodes.p, nodes.p, out->nodes.bytes, cudaMemcpyDeviceToDevice, st), err);
        CL_CUDA(cudaMemcpyAsync(out->tris.p, tris.p, out->tris.bytes, cudaMemcpyDeviceToDevice, st), err);
    }
    // Validation of every index the traversal kernels will follow, on the
    // device; one error word comes back.
    {
        uint32_t bad = 0;
        CL_TRY(validateBvh(out->nodes.as<const uint4>(), out->numNodes, out->tris.as<const float4>(), n, seen.u(), verr.u(),
                           st, &bad, err));
        if (bad)
        {
            *err = (bad & 1u)   ? "BVH validation: bad exponent or scale"
                   : (bad & 2u) ? "BVH validation: child index out of range"
                   : (bad & 4u) ? "BVH validation: leaf triangle range out of bounds"
                                : "BVH validation: triangle ids are not a permutation";
            return CL_ERR_STATE;
        }
    }
    if (depth + 1 > uint32_t(kStackDepth))
    {
        *err = "BVH depth " + std::to_string(depth) + " exceeds the traversal stack";
        return CL_ERR_STATE;
    }
    return CL_OK;
}

namespace
{
constexpr int kRefitBlock = 128;

// Leaf triangles from the vertex array; scene bounds into bounds[0..5] as
// ordered ints (min x,y,z then max x,y,z): grid-stride, reduced per block,
// one atomic per block and value.
__global__ void __launch_bounds__(256) kRefitTris(float4* __restrict__ tris, uint32_t n, const float4* __restrict__ vtx,
                                                  const uint4* __restrict__ triIdx, uint32_t* __restrict__ bounds)
{
    __shared__ uint32_t part[6][8];
    uint32_t            ol[3] = {0xffffffffu, 0xffffffffu, 0xffffffffu}, oh[3] = {0u, 0u, 0u};
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    {
        float4*  t   = tris + kTriF4 * size_t(i);
        uint32_t tid = __float_as_uint(t[0].w);
        uint4    ix  = triIdx[tid];
        float4   a = vtx[3 * size_t(ix.x)], b = vtx[3 * size_t(ix.y)], c = vtx[3 * size_t(ix.z)];
        t[0]         = make_float4(a.x, a.y, a.z, __uint_as_float(tid));
        t[1]         = make_float4(b.x, b.y, b.z, 0.0f);
        t[2]         = make_float4(c.x, c.y, c.z, 0.0f);
        float l[3] = {fminf(fminf(a.x, b.x), c.x), fminf(fminf(a.y, b.y), c.y), fminf(fminf(a.z, b.z), c.z)};
        float h[3] = {fmaxf(fmaxf(a.x, b.x), c.x), fmaxf(fmaxf(a.y, b.y), c.y), fmaxf(fmaxf(a.z, b.z), c.z)};
        for (int k = 0; k < 3; ++k)
        {
            ol[k] = min(ol[k], fordered(l[k]));
            oh[k] = max(oh[k], fordered(h[k]));
        }
    }
    int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int k = 0; k < 3; ++k)
        for (int o = 16; o > 0; o >>= 1)
        {
            ol[k] = min(ol[k], __shfl_xor_sync(0xffffffffu, ol[k], o));
            oh[k] = max(oh[k], __shfl_xor_sync(0xffffffffu, oh[k], o));
        }
    if (lane == 0)
        for (int k = 0; k < 3; ++k)
        {
            part[k][warp]     = ol[k];
            part[3 + k][warp] = oh[k];
        }
    __syncthreads();
    if (threadIdx.x < 6)
    {
        int      k = threadIdx.x;
        uint32_t v = part[k][0];
        for (int w = 1; w < int(blockDim.x >> 5); ++w) v = k < 3 ? min(v, part[k][w]) : max(v, part[k][w]);
        if (k < 3)
        {
            if (v != 0xffffffffu) atomicMin(bounds + k, v);
        }
        else if (v != 0u)
            atomicMax(bounds + k, v);
    }
}

// One tree level, eight lanes per node (lane s = child slot s): each lane
// boxes its slot (the child's exact box from the level below, or its leaf
// triangles), the group reduces the node's exact and widened boxes, every
// lane quantises its own slot in the node's frame, and lane 0 writes the
// node.  Topology (imask, child and triangle bases, leaf metadata, slot
// order) is kept; the result equals kCollapse's for unchanged triangles.
__global__ void __launch_bounds__(128) kRefitLevel(uint4* __restrict__ nodes, const float4* __restrict__ tris,
                                                   float* __restrict__ exact, uint32_t first, uint32_t count,
                                                   const uint32_t* __restrict__ bounds)
{
    uint32_t g     = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t t     = g >> 3;
    int      s     = int(g & 7u);
    bool     valid = t < count;
    uint32_t node  = first + (valid ? t : 0u);
    float    sl[3], sh[3];
    for (int a = 0; a < 3; ++a)
    {
        sl[a] = funordered(bounds[a]);
        sh[a] = funordered(bounds[3 + a]);
    }
    float  margin = sceneMargin(sl, sh);
    uint4* np     = nodes + size_t(node) * kNodeU4;
    uint4  n0 = make_uint4(0, 0, 0, 0), n1 = make_uint4(0, 0, 0, 0);
    if (valid)
    {
        n0 = np[0];
        n1 = np[1];
    }
    uint32_t imask = n0.w >> 24;
    float    lo[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, hi[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
    bool     present = false;
    if (valid)
    {
        if (imask & (1u << s))
        {
            uint32_t     c = n1.x + __popc(imask & ((1u << s) - 1u));
            const float* x = exact + 6 * size_t(c);
            for (int a = 0; a < 3; ++a)
            {
                lo[a] = x[a];
                hi[a] = x[3 + a];
            }
            present = true;
        }
        else
        {
            uint32_t m = ((s < 4 ? n1.z : n1.w) >> (8 * (s & 3))) & 0xffu;
            if (m)
            {
                uint32_t off = m & 31u, cnt = __popc(m >> 5);
                for (uint32_t j = 0; j < cnt; ++j)
                {
                    const float4* tp = tris + size_t(n1.y + off + j) * kTriF4;
                    for (int v = 0; v < 3; ++v)
                    {
                        float4 p = tp[v];
                        lo[0] = fminf(lo[0], p.x);
                        lo[1] = fminf(lo[1], p.y);
                        lo[2] = fminf(lo[2], p.z);
                        hi[0] = fmaxf(hi[0], p.x);
                        hi[1] = fmaxf(hi[1], p.y);
                        hi[2] = fmaxf(hi[2], p.z);
                    }
                }
                present = true;
            }
        }
    }
    // Exact box of the node and its widened frame box (group of 8 lanes).
    float xlo[3], xhi[3], clo[3], chi[3], plo[3], phi[3];
    for (int a = 0; a < 3; ++a)
    {
        xlo[a] = lo[a];
        xhi[a] = hi[a];
        clo[a] = present ? lo[a] - margin : FLT_MAX;
        chi[a] = present ? hi[a] + margin : -FLT_MAX;
        plo[a] = clo[a];
        phi[a] = chi[a];
        for (int o = 1; o < 8; o <<= 1)
        {
            xlo[a] = fminf(xlo[a], __shfl_xor_sync(0xffffffffu, xlo[a], o, 8));
            xhi[a] = fmaxf(xhi[a], __shfl_xor_sync(0xffffffffu, xhi[a], o, 8));
            plo[a] = fminf(plo[a], __shfl_xor_sync(0xffffffffu, plo[a], o, 8));
            phi[a] = fmaxf(phi[a], __shfl_xor_sync(0xffffffffu, phi[a], o, 8));
        }
    }
    uint32_t ex[3], ql[3] = {255u, 255u, 255u}, qh[3] = {0u, 0u, 0u};
    for (int a = 0; a < 3; ++a)
    {
        ex[a] = quantExp(phi[a] - plo[a]);
        if (present) quantPlanes(clo[a], chi[a], plo[a], __uint_as_float(ex[a] << 23), &ql[a], &qh[a]);
    }
    // Pack the slot bytes: OR within each quad of lanes, then bring the
    // second quad's words to lane 0.
    uint32_t wl[3], wh[3];
    for (int a = 0; a < 3; ++a)
    {
        wl[a] = ql[a] << (8 * (s & 3));
        wh[a] = qh[a] << (8 * (s & 3));
        for (int o = 1; o < 4; o <<= 1)
        {
            wl[a] |= __shfl_xor_sync(0xffffffffu, wl[a], o, 8);
            wh[a] |= __shfl_xor_sync(0xffffffffu, wh[a], o, 8);
        }
    }
    uint32_t wl1[3], wh1[3];
    for (int a = 0; a < 3; ++a)
    {
        wl1[a] = __shfl_down_sync(0xffffffffu, wl[a], 4, 8);
        wh1[a] = __shfl_down_sync(0xffffffffu, wh[a], 4, 8);
    }
    if (valid && s == 0)
    {
        np[0] = make_uint4(__float_as_uint(plo[0]), __float_as_uint(plo[1]), __float_as_uint(plo[2]),
                           ex[0] | (ex[1] << 8) | (ex[2] << 16) | (imask << 24));
        np[2] = make_uint4(wl[0], wl1[0], wl[1], wl1[1]);
        np[3] = make_uint4(wl[2], wl1[2], wh[0], wh1[0]);
        np[4] = make_uint4(wh[1], wh1[1], wh[2], wh1[2]);
        np[5] = make_uint4(np[5].x, ex[0] << 23, ex[1] << 23, ex[2] << 23);
        float* x = exact + 6 * size_t(node);
        for (int a = 0; a < 3; ++a)
        {
            x[a]     = xlo[a];
            x[3 + a] = xhi[a];
        }
    }
}

__device__ __forceinline__ double boxArea(float lx, float ly, float lz, float hx, float hy, float hz)
{
    double dx = double(hx) - lx, dy = double(hy) - ly, dz = double(hz) - lz;
    return 2.0 * (dx * dy + dy * dz + dz * dx);
}

// Sum over all child slots of (dequantised box area) x (1 for an inner
// child, its triangle count for a leaf), into *sum; a copy of the root node
// goes behind it, so that the host reads both at once (each read of pageable
// memory waits for itself, 9 us).
__global__ void kSahSum(const uint4* __restrict__ nodes, uint32_t n, double* sum)
{
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    double   c = 0.0;
    if (i < 5u) reinterpret_cast<uint4*>(sum)[1 + i] = nodes[i];
    if (i < n)
    {
        const uint4* np = nodes + size_t(i) * kNodeU4;
        uint4        n0 = np[0], n1 = np[1], n2 = np[2], n3 = np[3], n4 = np[4];
        float        px = __uint_as_float(n0.x), py = __uint_as_float(n0.y), pz = __uint_as_float(n0.z);
        float        ex = __uint_as_float((n0.w & 0xffu) << 23), ey = __uint_as_float(((n0.w >> 8) & 0xffu) << 23),
              ez = __uint_as_float(((n0.w >> 16) & 0xffu) << 23);
        uint32_t imask = n0.w >> 24;
        for (int s = 0; s < 8; ++s)
        {
            int      w = s >> 2, sh = 8 * (s & 3);
            uint32_t lx = ((w ? n2.y : n2.x) >> sh) & 0xffu, ly = ((w ? n2.w : n2.z) >> sh) & 0xffu,
                     lz = ((w ? n3.y : n3.x) >> sh) & 0xffu;
            uint32_t hx = ((w ? n3.w : n3.z) >> sh) & 0xffu, hy = ((w ? n4.y : n4.x) >> sh) & 0xffu,
                     hz = ((w ? n4.w : n4.z) >> sh) & 0xffu;
            if (lx > hx) continue; // empty slot
            double weight;
            if (imask & (1u << s))
                weight = 1.0;
            else
            {
                uint32_t m = ((w ? n1.w : n1.z) >> sh) & 0xffu;
                weight     = double(__popc(m >> 5));
            }
            c += weight * boxArea(px + ex * float(lx), py + ey * float(ly), pz + ez * float(lz), px + ex * float(hx),
                                  py + ey * float(hy), pz + ez * float(hz));
        }
    }
    for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    if ((threadIdx.x & 31) == 0 && c != 0.0) atomicAdd(sum, c);
}

__global__ void kGatherTri9(const float4* __restrict__ vtx, const uint4* __restrict__ triIdx, uint32_t n,
                            float* __restrict__ tri9)
{
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint4 ix = triIdx[i];
    float4 a = vtx[3 * size_t(ix.x)], b = vtx[3 * size_t(ix.y)], c = vtx[3 * size_t(ix.z)];
    float* o = tri9 + 9 * size_t(i);
    o[0] = a.x; o[1] = a.y; o[2] = a.z;
    o[3] = b.x; o[4] = b.y; o[5] = b.z;
    o[6] = c.x; o[7] = c.y; o[8] = c.z;
}
} // namespace

cl_status refitWideBvh(WideBvh* bvh, const void* vtx, const void* triIdx, cudaStream_t st, std::string* err)
{
    if (!bvh->nodes.p || bvh->levels.size() < 2 || bvh->levels.back() != bvh->numNodes)
    {
        *err = "refit needs a built BVH";
        return CL_ERR_STATE;
    }
    if (bvh->exact.bytes < size_t(bvh->numNodes) * 24 || !bvh->scene.p)
    {
        *err = "refit buffers missing";
        return CL_ERR_STATE;
    }
    // Bounds start at (+inf ordered, -inf ordered): 0xff bytes for the
    // minima, zero bytes for the maxima.
    CL_CUDA(cudaMemsetAsync(bvh->scene.p, 0xff, 12, st), err);
    CL_CUDA(cudaMemsetAsync(bvh->scene.u() + 3, 0, 12, st), err);
    uint32_t n = bvh->numTris;
    static int sms = 0;
    if (!sms)
    {
        int dev = 0;
        CL_CUDA(cudaGetDevice(&dev), err);
        CL_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), err);
    }
    uint32_t blocks = std::min<uint32_t>((n + 255) / 256, uint32_t(sms) * 8u);
    kRefitTris<<<blocks, 256, 0, st>>>(bvh->tris.as<float4>(), n, static_cast<const float4*>(vtx),
                                       static_cast<const uint4*>(triIdx), bvh->scene.u());
    CL_CUDA(cudaGetLastError(), err);
    for (size_t d = bvh->levels.size() - 1; d-- > 0;)
    {
        uint32_t first = bvh->levels[d], count = bvh->levels[d + 1] - first;
        uint64_t lanes = uint64_t(count) * 8u;
        kRefitLevel<<<uint32_t((lanes + kRefitBlock - 1) / kRefitBlock), kRefitBlock, 0, st>>>(
            bvh->nodes.as<uint4>(), bvh->tris.as<const float4>(), bvh->exact.f(), first, count, bvh->scene.u());
        CL_CUDA(cudaGetLastError(), err);
    }
    return CL_OK;
}

cl_status wideBvhSahCost(WideBvh& bvh, cudaStream_t st, double* cost, std::string* err)
{
    if (!bvh.nodes.p || bvh.numNodes == 0)
    {
        *err = "no BVH";
        return CL_ERR_STATE;
    }
    double* sum = reinterpret_cast<double*>(bvh.scene.as<char>() + 32);
    CL_CUDA(cudaMemsetAsync(sum, 0, 8, st), err);
    kSahSum<<<(bvh.numNodes + 255) / 256, 256, 0, st>>>(bvh.nodes.as<const uint4>(), bvh.numNodes, sum);
    CL_CUDA(cudaGetLastError(), err);
    uint32_t back[24]; // the sum, 8 unused bytes, the root node
    CL_CUDA(cudaMemcpyAsync(back, sum, sizeof(back), cudaMemcpyDeviceToHost, st), err);
    CL_CUDA(cudaStreamSynchronize(st), err);
    double          total;
    const uint32_t* h = back + 4;
    memcpy(&total, back, 8);
    // Root box extent per axis: e * (largest qhi - smallest qlo) over the
    // root's present slots (qlo words at h[8 + 2a + w], qhi at h[14 + 2a + w]).
    double ext[3];
    for (int a = 0; a < 3; ++a)
    {
        uint32_t eb = ((h[3] >> (8 * a)) & 0xffu) << 23;
        float    e;
        memcpy(&e, &eb, 4);
        uint32_t qlo = 255, qhi = 0;
        for (int sl = 0; sl < 8; ++sl)
        {
            int      w = sl >> 2, sh = 8 * (sl & 3);
            uint32_t lo = (h[8 + 2 * a + w] >> sh) & 0xffu, hi = (h[14 + 2 * a + w] >> sh) & 0xffu;
            if (lo > hi) continue;
            qlo = std::min(qlo, lo);
            qhi = std::max(qhi, hi);
        }
        ext[a] = qhi >= qlo ? double(e) * double(qhi - qlo) : 0.0;
    }
    double rootArea = 2.0 * (ext[0] * ext[1] + ext[1] * ext[2] + ext[2] * ext[0]);
    *cost           = rootArea > 0.0 ? 1.0 + total / rootArea : 0.0;
    return CL_OK;
}

cl_status gatherTrianglePositions(const void* vtx, const void* triIdx, uint32_t n, float* tri9, cudaStream_t st,
                                  std::string* err)
{
    kGatherTri9<<<(n + 255) / 256, 256, 0, st>>>(static_cast<const float4*>(vtx), static_cast<const uint4*>(triIdx),
                                                  n, tri9);
    CL_CUDA(cudaGetLastError(), err);
    return CL_OK;
}

} // namespace clb
