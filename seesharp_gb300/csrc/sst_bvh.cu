// GPU BVH construction (replaces the Embree build behind Raytracer.CommitScene, Scene.cs:108-113).
//
// Linear BVH after Karras, "Maximizing Parallelism in the Construction of BVHs, Octrees, and k-d
// Trees" (HPG 2012):
//   1. centroid bounds (atomic min/max on order-preserving integer images of the floats)
//   2. 63-bit Morton keys of the triangle centroids, radix-sorted with CUB
//   3. one thread per internal node finds its key range and split (longest common prefix, ties
//      broken by the sorted index)
//   4. bottom-up refit: the second child to arrive computes the parent's box, leaf count and the
//      surface-area cost C(n) = min(Ci N A(n) [N <= kMaxLeafSize], Ct A(n) + C(l) + C(r)), which
//      decides where subtrees collapse into multi-triangle leaves
//   5. kept inner nodes are numbered by a prefix sum and written in the traversal layout (both
//      child boxes in the parent, 64-byte nodes); a collapsed subtree becomes one leaf reference
//      to its contiguous range of sorted triangles.
#include <cub/cub.cuh>
#include <thrust/iterator/counting_iterator.h>
#include <thrust/iterator/transform_iterator.h>
#include <math_constants.h>
#include <algorithm>
#include <cstdlib>
#include <cuda_runtime.h>

#include "sst_bvh.h"
#include "sst_types.h"

namespace sst {

namespace {

// Traversal cost relative to one triangle test.  0.25 keeps most leaves at one triangle: on the
// 1M-triangle scene it traverses 3.4% faster than 1.0 (and 1.0 17% faster than 3.0).
constexpr float kCt = 0.25f;
constexpr float kCi = 1.0f;
// PLOC rounds between two looks at the cluster count.  A round leaves 70 to 80% of the clusters, so the
// third one's grid is at most twice what it needs.  Commits of 10K / 102K / 614K / 1M / 2M triangles with a
// look after every round: 1.11 / 2.35 / 4.68 / 6.49 / 11.17 ms, every second: 1.09 / 2.20 / 4.51 / 6.29 / 10.94,
// every third: 1.07 / 2.17 / 4.48 / 6.25 / 10.88, every fourth: 1.07 / 2.16 / 4.44 / 6.18 / 10.84, every sixth:
// 1.08 / 2.16 / 4.39 / 6.14 / 10.80.  (With four read-backs and a wait after each of the 61 rounds, no block
// that does the last half of them and a read-back per level of the wide tree: 614K triangles 8.8 ms.)
constexpr int kPlocRounds = 3;

__device__ __forceinline__ int floatOrd(float f) {
    int i = __float_as_int(f);
    return i >= 0 ? i : i ^ 0x7FFFFFFF;
}
__device__ __forceinline__ float ordFloat(int i) { return __int_as_float(i >= 0 ? i : i ^ 0x7FFFFFFF); }

__global__ void k_centroid_bounds(const float4* tri, int n, int* bounds /* 6: min xyz, max xyz (ordered ints) */) {
    __shared__ int smin[3], smax[3];
    if (threadIdx.x < 3) { smin[threadIdx.x] = 0x7FFFFFFF; smax[threadIdx.x] = (int)0x80000000; }
    __syncthreads();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        float4 a = tri[3 * (size_t)i], b = tri[3 * (size_t)i + 1], c = tri[3 * (size_t)i + 2];
        float cx = 0.5f * (fminf(a.x, fminf(b.x, c.x)) + fmaxf(a.x, fmaxf(b.x, c.x)));
        float cy = 0.5f * (fminf(a.y, fminf(b.y, c.y)) + fmaxf(a.y, fmaxf(b.y, c.y)));
        float cz = 0.5f * (fminf(a.z, fminf(b.z, c.z)) + fmaxf(a.z, fmaxf(b.z, c.z)));
        atomicMin(&smin[0], floatOrd(cx)); atomicMin(&smin[1], floatOrd(cy)); atomicMin(&smin[2], floatOrd(cz));
        atomicMax(&smax[0], floatOrd(cx)); atomicMax(&smax[1], floatOrd(cy)); atomicMax(&smax[2], floatOrd(cz));
    }
    __syncthreads();
    if (threadIdx.x < 3) {
        atomicMin(&bounds[threadIdx.x], smin[threadIdx.x]);
        atomicMax(&bounds[3 + threadIdx.x], smax[threadIdx.x]);
    }
}

__device__ __forceinline__ unsigned long long spread21(unsigned int v) {
    unsigned long long x = v & 0x1FFFFFu;
    x = (x | x << 32) & 0x1F00000000FFFFull;
    x = (x | x << 16) & 0x1F0000FF0000FFull;
    x = (x | x << 8) & 0x100F00F00F00F00Full;
    x = (x | x << 4) & 0x10C30C30C30C30C3ull;
    x = (x | x << 2) & 0x1249249249249249ull;
    return x;
}

__global__ void k_morton(const float4* tri, int n, const int* bounds, unsigned long long* keys, int* vals) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float lo[3] = {ordFloat(bounds[0]), ordFloat(bounds[1]), ordFloat(bounds[2])};
    float hi[3] = {ordFloat(bounds[3]), ordFloat(bounds[4]), ordFloat(bounds[5])};
    float4 a = tri[3 * (size_t)i], b = tri[3 * (size_t)i + 1], c = tri[3 * (size_t)i + 2];
    float cc[3] = {0.5f * (fminf(a.x, fminf(b.x, c.x)) + fmaxf(a.x, fmaxf(b.x, c.x))),
                   0.5f * (fminf(a.y, fminf(b.y, c.y)) + fmaxf(a.y, fmaxf(b.y, c.y))),
                   0.5f * (fminf(a.z, fminf(b.z, c.z)) + fmaxf(a.z, fmaxf(b.z, c.z)))};
    unsigned int q[3];
    for (int k = 0; k < 3; ++k) {
        float ext = hi[k] - lo[k];
        float t = ext > 0.0f ? (cc[k] - lo[k]) / ext : 0.5f;
        q[k] = (unsigned int)fminf(fmaxf(t * 2097152.0f, 0.0f), 2097151.0f);
    }
    keys[i] = (spread21(q[0]) << 2) | (spread21(q[1]) << 1) | spread21(q[2]);
    vals[i] = i;
}

// Longest common prefix of sorted keys i and j (-1 outside [0, n)); equal keys compare indices.
__device__ __forceinline__ int delta(const unsigned long long* k, int n, int i, int j) {
    if (j < 0 || j >= n) return -1;
    unsigned long long a = k[i], b = k[j];
    if (a == b) return 64 + __clz((unsigned)(i ^ j));
    return __clzll(a ^ b);
}

// Internal node i covers sorted leaves [first, last]; children encoded >= 0 internal, < 0 leaf ~idx.
__global__ void k_karras(const unsigned long long* k, int n, int2* range, int2* child, int* parentInner, int* parentLeaf) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n - 1) return;
    int d = (delta(k, n, i, i + 1) - delta(k, n, i, i - 1)) >= 0 ? 1 : -1;
    int dmin = delta(k, n, i, i - d);
    int lmax = 2;
    while (delta(k, n, i, i + lmax * d) > dmin) lmax <<= 1;
    int l = 0;
    for (int t = lmax >> 1; t >= 1; t >>= 1)
        if (delta(k, n, i, i + (l + t) * d) > dmin) l += t;
    int j = i + l * d;
    int dnode = delta(k, n, i, j);
    int s = 0;
    int div = 2;
    for (int t = (l + 1) / 2; ; t = (l + div - 1) / div) {
        if (delta(k, n, i, i + (s + t) * d) > dnode) s += t;
        if (t == 1) break;
        div <<= 1;
    }
    int gamma = i + s * d + min(d, 0);
    int first = min(i, j), last = max(i, j);
    int left = (first == gamma) ? ~gamma : gamma;
    int right = (last == gamma + 1) ? ~(gamma + 1) : gamma + 1;
    range[i] = make_int2(first, last);
    child[i] = make_int2(left, right);
    if (left < 0) parentLeaf[~left] = i; else parentInner[left] = i;
    if (right < 0) parentLeaf[~right] = i; else parentInner[right] = i;
}

struct NodeFit {
    float lo[3], hi[3];
};

__device__ __forceinline__ float areaOf(const float* lo, const float* hi) {
    float dx = fmaxf(0.0f, hi[0] - lo[0]), dy = fmaxf(0.0f, hi[1] - lo[1]), dz = fmaxf(0.0f, hi[2] - lo[2]);
    return dx * dy + dy * dz + dz * dx;
}

// Bottom-up refit from every leaf.  boxes: 6 floats per inner node; cost: per inner node;
// collapse[i] = 1 when the subtree is cheaper as one leaf.
__global__ void k_refit(const float4* tri, const int* order, int n, const int2* range, const int2* child, const int* parentInner,
                        const int* parentLeaf, int* visits, float* boxes, float* cost, int* collapse, float ct, int maxLeaf) {
    int li = blockIdx.x * blockDim.x + threadIdx.x;
    if (li >= n) return;
    int node = parentLeaf[li];
    while (node >= 0) {
        __threadfence();
        if (atomicAdd(&visits[node], 1) == 0) return;  // the other child is not done yet
        __threadfence();
        int2 c = child[node];
        float lo[3] = {1e30f, 1e30f, 1e30f}, hi[3] = {-1e30f, -1e30f, -1e30f};
        float cs = 0.0f;
        for (int s = 0; s < 2; ++s) {
            int ch = s == 0 ? c.x : c.y;
            float clo[3], chi[3], ccost;
            if (ch < 0) {
                int t = order[~ch];
                float4 a = tri[3 * (size_t)t], b = tri[3 * (size_t)t + 1], d = tri[3 * (size_t)t + 2];
                clo[0] = fminf(a.x, fminf(b.x, d.x)); chi[0] = fmaxf(a.x, fmaxf(b.x, d.x));
                clo[1] = fminf(a.y, fminf(b.y, d.y)); chi[1] = fmaxf(a.y, fmaxf(b.y, d.y));
                clo[2] = fminf(a.z, fminf(b.z, d.z)); chi[2] = fmaxf(a.z, fmaxf(b.z, d.z));
                ccost = kCi * areaOf(clo, chi);
            } else {
                const volatile float* bx = boxes + 6 * (size_t)ch;
                for (int k = 0; k < 3; ++k) { clo[k] = bx[k]; chi[k] = bx[3 + k]; }
                ccost = ((const volatile float*)cost)[ch];
            }
            for (int k = 0; k < 3; ++k) { lo[k] = fminf(lo[k], clo[k]); hi[k] = fmaxf(hi[k], chi[k]); }
            cs += ccost;
        }
        float A = areaOf(lo, hi);
        int2 r = range[node];
        int cnt = r.y - r.x + 1;
        float split = ct * A + cs;
        float leaf = kCi * cnt * A;
        bool col = cnt <= maxLeaf && leaf <= split;
        float* bo = boxes + 6 * (size_t)node;
        for (int k = 0; k < 3; ++k) { bo[k] = lo[k]; bo[3 + k] = hi[k]; }
        cost[node] = col ? leaf : split;
        collapse[node] = col ? 1 : 0;
        node = parentInner[node];
    }
}

// kept[i] = 1 when inner node i is not inside a collapsed subtree (and is not collapsed itself);
// depth[i] = number of kept ancestors.  Walks to the root (depth bounded by the key length).
__global__ void k_kept(const int* parentInner, const int* collapse, int n, int* kept, int* maxDepth) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n - 1) return;
    int k = (i == 0 || !collapse[i]) ? 1 : 0;
    int depth = 0;
    int p = parentInner[i];
    for (int guard = 0; p >= 0 && guard < 4096; ++guard) {
        if (collapse[p] && p != 0) k = 0;
        ++depth;
        p = parentInner[p];
    }
    kept[i] = k;
    if (k) atomicMax(maxDepth, depth);
}

// ---------------------------------------------------------------------------------------------
// PLOC topology (Meister and Bittner, "Parallel Locally-Ordered Clustering for Bounding Volume
// Hierarchy Construction", 2018): the clusters start as the Morton-sorted leaves; in each round
// every cluster finds the cluster within a radius of positions whose union box has the smallest
// surface area, mutual nearest neighbours merge into a new inner node, and the cluster list is
// compacted in order.  The resulting tree is then given a depth-first leaf order so that every
// subtree covers a contiguous range, and the LBVH's refit / collapse / emit stages finish it.
// ---------------------------------------------------------------------------------------------

__device__ __forceinline__ float unionArea(const float* a, const float* b) {
    float lo[3], hi[3];
    for (int k = 0; k < 3; ++k) { lo[k] = fminf(a[k], b[k]); hi[k] = fmaxf(a[3 + k], b[3 + k]); }
    return areaOf(lo, hi);
}

// clusters = sorted leaves ~i with their triangle boxes
__global__ void k_ploc_init(const float4* tri, const int* order, int n, int* clus, float* cbox) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int t = order[i];
    float4 a = tri[3 * (size_t)t], b = tri[3 * (size_t)t + 1], d = tri[3 * (size_t)t + 2];
    float* o = cbox + 6 * (size_t)i;
    o[0] = fminf(a.x, fminf(b.x, d.x)); o[3] = fmaxf(a.x, fmaxf(b.x, d.x));
    o[1] = fminf(a.y, fminf(b.y, d.y)); o[4] = fmaxf(a.y, fmaxf(b.y, d.y));
    o[2] = fminf(a.z, fminf(b.z, d.z)); o[5] = fmaxf(a.z, fmaxf(b.z, d.z));
    clus[i] = ~i;
}

// Nearest neighbour within `radius` positions (ties: the smaller index).  A block keeps its clusters'
// boxes and those of `radius` positions on both sides in shared memory (every box is read up to
// 2 radius + 1 times).  Blocks past the *nc clusters have nothing to do.
constexpr int kNnThreads = 256;
constexpr int kPlocMaxRadius = 256;
__global__ void __launch_bounds__(kNnThreads) k_ploc_nn(const float* cbox, const int* nc, int radius, int* nn) {
    __shared__ float box[6][kNnThreads + 2 * kPlocMaxRadius];
    const int n = *nc, first = blockIdx.x * kNnThreads;
    if (first >= n) return;
    const int lo = max(0, first - radius), hi = min(n, first + kNnThreads + radius);
    for (int e = threadIdx.x; e < 6 * (hi - lo); e += kNnThreads) box[e % 6][e / 6] = cbox[6 * (size_t)lo + e];
    __syncthreads();
    const int i = first + threadIdx.x;
    if (i >= n) return;
    float me[6];
    for (int k = 0; k < 6; ++k) me[k] = box[k][i - lo];
    float best = CUDART_INF_F;
    int bj = -1;
    const int j0 = max(0, i - radius), j1 = min(n - 1, i + radius);
    for (int j = j0; j <= j1; ++j) {
        if (j == i) continue;
        const float o[6] = {box[0][j - lo], box[1][j - lo], box[2][j - lo], box[3][j - lo], box[4][j - lo], box[5][j - lo]};
        float a = unionArea(me, o);
        if (a < best) { best = a; bj = j; }
    }
    nn[i] = bj;
}

// What becomes of cluster i, as one 64-bit item for a single scan of both: bit 0: it stays in the list
// (possibly merged), bit 32: it merges with its mutual nearest neighbour (it is the lower of the two).
// Items past the *nc clusters are zero, so that a scan over a larger count gives the same sums.
struct PlocFlags {
    const int* nn;
    const int* nc;
    __device__ __forceinline__ unsigned long long operator()(int i) const {
        if (i >= *nc) return 0ull;
        const int j = nn[i];
        const bool mutual = j >= 0 && nn[j] == i;
        return ((mutual && i < j) ? (1ull << 32) : 0ull) | ((!mutual || i < j) ? 1ull : 0ull);
    }
};

// Merged clusters become inner nodes in creation order: so far n - *nc of them, since every merge leaves
// one cluster less.  The last cluster's thread writes the new count.
__global__ void k_ploc_compact(const int* clus, const float* cbox, const int* nn, const int* nc, int n, const unsigned long long* before, int* clusOut,
                               float* cboxOut, int* ncOut, int2* child) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int m = *nc;
    if (i >= m) return;
    const unsigned long long f = PlocFlags{nn, nc}(i), at = before[i];
    const int out = (int)(uint32_t)at;
    if (i == m - 1) *ncOut = out + (int)(f & 1u);
    if (!(f & 1u)) return;
    float b[6];
    for (int k = 0; k < 6; ++k) b[k] = cbox[6 * (size_t)i + k];
    if (f >> 32) {
        const int j = nn[i], id = n - m + (int)(at >> 32);
        child[id] = make_int2(clus[i], clus[j]);
        for (int k = 0; k < 3; ++k) {
            b[k] = fminf(b[k], cbox[6 * (size_t)j + k]);
            b[3 + k] = fmaxf(b[3 + k], cbox[6 * (size_t)j + 3 + k]);
        }
        clusOut[out] = id;
    } else {
        clusOut[out] = clus[i];
    }
    for (int k = 0; k < 6; ++k) cboxOut[6 * (size_t)out + k] = b[k];
}

// The remaining rounds of at most kTailClusters clusters in one block, boxes and references in shared
// memory: the same searches, merges and numbering.  About half of all rounds run on so few clusters, and
// as separate launches each costs tens of microseconds of launches and a wait for a few thousand items.
// Leaves the cluster count in *nc: 1 when the tree is complete, more when no pair merges (NaN boxes).
constexpr int kTailThreads = 1024, kTailPer = 4, kTailClusters = kTailThreads * kTailPer;
constexpr int kTailSlices = kTailClusters / 32;
constexpr size_t kTailSmem = sizeof(float) * 6 * kTailClusters + sizeof(int) * 2 * kTailClusters;
__global__ void __launch_bounds__(kTailThreads) k_ploc_tail(const int* clusIn, const float* cboxIn, int* nc, int n, int radius, int2* child) {
    extern __shared__ float tailMem[];
    float* const box = tailMem;                                              // [6][kTailClusters]
    int* const clus = reinterpret_cast<int*>(box + 6 * kTailClusters);
    int* const nn = clus + kTailClusters;
    __shared__ int2 before[kTailSlices];  // (kept, created) in the slices of 32 clusters before
    __shared__ int2 total;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned below = (1u << lane) - 1u;
    int m = *nc;
    if (m > kTailClusters) return;
    for (int e = tid; e < 6 * m; e += kTailThreads) box[(e % 6) * kTailClusters + e / 6] = cboxIn[e];
    for (int i = tid; i < m; i += kTailThreads) clus[i] = clusIn[i];
    __syncthreads();
    while (m > 1) {
        for (int i = tid; i < m; i += kTailThreads) {
            float me[6];
            for (int k = 0; k < 6; ++k) me[k] = box[k * kTailClusters + i];
            float best = CUDART_INF_F;
            int bj = -1;
            const int j0 = max(0, i - radius), j1 = min(m - 1, i + radius);
            for (int j = j0; j <= j1; ++j) {
                if (j == i) continue;
                float o[6];
                for (int k = 0; k < 6; ++k) o[k] = box[k * kTailClusters + j];
                const float a = unionArea(me, o);
                if (a < best) { best = a; bj = j; }
            }
            nn[i] = bj;
        }
        __syncthreads();
        unsigned keep[kTailPer], make[kTailPer];
        int ref[kTailPer];
        float nb[kTailPer][6];
        int2 pair[kTailPer];
#pragma unroll
        for (int q = 0; q < kTailPer; ++q) {
            const int i = q * kTailThreads + tid;
            bool kp = false, mk = false;
            if (i < m) {
                const int j = nn[i];
                const bool mutual = j >= 0 && nn[j] == i;
                mk = mutual && i < j;
                kp = !mutual || i < j;
                if (kp) {
                    for (int k = 0; k < 6; ++k) nb[q][k] = box[k * kTailClusters + i];
                    ref[q] = clus[i];
                    if (mk) {
                        for (int k = 0; k < 3; ++k) {
                            nb[q][k] = fminf(nb[q][k], box[k * kTailClusters + j]);
                            nb[q][3 + k] = fmaxf(nb[q][3 + k], box[(3 + k) * kTailClusters + j]);
                        }
                        pair[q] = make_int2(ref[q], clus[j]);
                    }
                }
            }
            keep[q] = __ballot_sync(0xffffffffu, kp);
            make[q] = __ballot_sync(0xffffffffu, mk);
            if (lane == 0) before[q * (kTailThreads / 32) + warp] = make_int2(__popc(keep[q]), __popc(make[q]));
        }
        __syncthreads();
        if (warp == 0) {
            constexpr int per = kTailSlices / 32;
            int2 own[per], sum = make_int2(0, 0);
            for (int k = 0; k < per; ++k) {
                own[k] = before[lane * per + k];
                sum.x += own[k].x;
                sum.y += own[k].y;
            }
            int2 inc = sum;
            for (int o = 1; o < 32; o <<= 1) {
                const int x = __shfl_up_sync(0xffffffffu, inc.x, o), y = __shfl_up_sync(0xffffffffu, inc.y, o);
                if (lane >= o) { inc.x += x; inc.y += y; }
            }
            int2 at = make_int2(inc.x - sum.x, inc.y - sum.y);
            for (int k = 0; k < per; ++k) {
                before[lane * per + k] = at;
                at.x += own[k].x;
                at.y += own[k].y;
            }
            if (lane == 31) total = inc;
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < kTailPer; ++q) {
            if (!(keep[q] >> lane & 1u)) continue;
            const int2 at = before[q * (kTailThreads / 32) + warp];
            const int out = at.x + __popc(keep[q] & below);
            if (make[q] >> lane & 1u) {
                const int id = n - m + at.y + __popc(make[q] & below);
                child[id] = pair[q];
                ref[q] = id;
            }
            clus[out] = ref[q];
            for (int k = 0; k < 6; ++k) box[k * kTailClusters + out] = nb[q][k];
        }
        const int2 t = total;
        __syncthreads();
        m = t.x;
        if (t.y == 0) break;  // no mutual pair: boxes that are not numbers
    }
    if (tid == 0) *nc = m;
}

// creation ids -> final ids (root = 0: reversed creation order); parent pointers
__global__ void k_ploc_renumber(const int2* childC, int n, int2* child, int* parentInner, int* parentLeaf) {
    int id = blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= n - 1) return;
    int nid = (n - 2) - id;
    int2 c = childC[id];
    int a = c.x >= 0 ? (n - 2) - c.x : c.x;
    int b = c.y >= 0 ? (n - 2) - c.y : c.y;
    child[nid] = make_int2(a, b);
    if (a < 0) parentLeaf[~a] = nid; else parentInner[a] = nid;
    if (b < 0) parentLeaf[~b] = nid; else parentInner[b] = nid;
}

// subtree leaf counts, bottom-up from every leaf (the second child to arrive continues)
__global__ void k_ploc_sizes(const int2* child, const int* parentLeaf, const int* parentInner, int n, int* visits, int* size) {
    int li = blockIdx.x * blockDim.x + threadIdx.x;
    if (li >= n) return;
    int node = parentLeaf[li];
    while (node >= 0) {
        __threadfence();
        if (atomicAdd(&visits[node], 1) == 0) return;
        __threadfence();
        int2 c = child[node];
        int sa = c.x < 0 ? 1 : ((const volatile int*)size)[c.x];
        int sb = c.y < 0 ? 1 : ((const volatile int*)size)[c.y];
        size[node] = sa + sb;
        node = parentInner[node];
    }
}

// depth-first offsets: a node's first leaf is the number of leaves left of it, summed over the
// ancestors of which it lies in the right subtree.  Inner nodes get their leaf range; leaves their
// position in the new order.
__global__ void k_ploc_offsets(const int2* child, const int* parentInner, const int* parentLeaf, const int* size, int n, int2* range,
                               int* leafPos) {
    int x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= 2 * n - 1) return;
    bool leaf = x >= n - 1;
    int self = leaf ? ~(x - (n - 1)) : x;
    int p = leaf ? parentLeaf[x - (n - 1)] : parentInner[x];
    int off = 0, cur = self;
    for (int guard = 0; p >= 0 && guard < 1 << 20; ++guard) {
        int2 c = child[p];
        if (c.y == cur) off += c.x < 0 ? 1 : size[c.x];
        cur = p;
        p = parentInner[p];
    }
    if (leaf) leafPos[x - (n - 1)] = off;
    else range[x] = make_int2(off, off + size[x] - 1);
}

__global__ void k_ploc_leaf_parents(const int2* child, int n, int* parentLeaf) {
    int x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= n - 1) return;
    int2 c = child[x];
    if (c.x < 0) parentLeaf[~c.x] = x;
    if (c.y < 0) parentLeaf[~c.y] = x;
}

// leaves re-encoded by their depth-first position; the triangle order follows
__global__ void k_ploc_reorder(int2* child, const int* leafPos, const int* sortedOrder, int n, int* order) {
    int x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x < n) order[leafPos[x]] = sortedOrder[x];
    if (x < n - 1) {
        int2 c = child[x];
        if (c.x < 0) c.x = ~leafPos[~c.x];
        if (c.y < 0) c.y = ~leafPos[~c.y];
        child[x] = c;
    }
}

__device__ __forceinline__ uint32_t leafRef(int first, int count) {
    return kLeafFlag | ((uint32_t)(count - 1) << kLeafCountShift) | (uint32_t)first;
}

__global__ void k_emit(const float4* tri, const int* order, int n, const int2* range, const int2* child, const int* collapse, const int* kept,
                       const int* newIdx, const float* boxes, float4* nodes) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n - 1 || !kept[i]) return;
    int2 c = child[i];
    float4* out = nodes + 4 * (size_t)newIdx[i];
    float4 o0, o1, o2, o3;
    uint32_t refs[2];
    float b[2][6];
    for (int s = 0; s < 2; ++s) {
        int ch = s == 0 ? c.x : c.y;
        if (ch < 0) {
            int t = order[~ch];
            float4 a = tri[3 * (size_t)t], bb = tri[3 * (size_t)t + 1], d = tri[3 * (size_t)t + 2];
            b[s][0] = fminf(a.x, fminf(bb.x, d.x)); b[s][3] = fmaxf(a.x, fmaxf(bb.x, d.x));
            b[s][1] = fminf(a.y, fminf(bb.y, d.y)); b[s][4] = fmaxf(a.y, fmaxf(bb.y, d.y));
            b[s][2] = fminf(a.z, fminf(bb.z, d.z)); b[s][5] = fmaxf(a.z, fmaxf(bb.z, d.z));
            refs[s] = leafRef(~ch, 1);
        } else {
            for (int k = 0; k < 6; ++k) b[s][k] = boxes[6 * (size_t)ch + k];
            if (collapse[ch]) {
                int2 r = range[ch];
                refs[s] = leafRef(r.x, r.y - r.x + 1);
            } else {
                refs[s] = (uint32_t)newIdx[ch];
            }
        }
    }
    o0 = make_float4(b[0][0], b[0][3], b[0][1], b[0][4]);
    o1 = make_float4(b[1][0], b[1][3], b[1][1], b[1][4]);
    o2 = make_float4(b[0][2], b[0][5], b[1][2], b[1][5]);
    o3 = make_float4(__uint_as_float(refs[0]), __uint_as_float(refs[1]), 0.0f, 0.0f);
    out[0] = o0; out[1] = o1; out[2] = o2; out[3] = o3;
}

// Single-triangle scene: root with the same one-triangle leaf in both slots.
__global__ void k_emit_single(const float4* tri, float4* nodes) {
    float4 a = tri[0], b = tri[1], c = tri[2];
    float lo[3] = {fminf(a.x, fminf(b.x, c.x)), fminf(a.y, fminf(b.y, c.y)), fminf(a.z, fminf(b.z, c.z))};
    float hi[3] = {fmaxf(a.x, fmaxf(b.x, c.x)), fmaxf(a.y, fmaxf(b.y, c.y)), fmaxf(a.z, fmaxf(b.z, c.z))};
    uint32_t r = leafRef(0, 1);
    nodes[0] = make_float4(lo[0], hi[0], lo[1], hi[1]);
    nodes[1] = make_float4(lo[0], hi[0], lo[1], hi[1]);
    nodes[2] = make_float4(lo[2], hi[2], lo[2], hi[2]);
    nodes[3] = make_float4(__uint_as_float(r), __uint_as_float(r), 0.0f, 0.0f);
}

template <class T> T* carve(char*& p, size_t n) {
    size_t off = (reinterpret_cast<size_t>(p) + 255) & ~size_t(255);
    T* r = reinterpret_cast<T*>(off);
    p = reinterpret_cast<char*>(off + n * sizeof(T));
    return r;
}

}  // namespace

// CUB temporary storage shared by the radix sort and the prefix sum.
static size_t cubTempBytes(int n) {
    size_t sortBytes = 0, scanBytes = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, sortBytes, (unsigned long long*)nullptr, (unsigned long long*)nullptr, (int*)nullptr, (int*)nullptr, n,
                                    0, 63);
    cub::DeviceScan::ExclusiveSum(nullptr, scanBytes, (int*)nullptr, (int*)nullptr, n > 1 ? n - 1 : 1);
    size_t plocBytes = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, plocBytes, thrust::make_transform_iterator(thrust::make_counting_iterator<int>(0), PlocFlags{nullptr, nullptr}),
                                  (unsigned long long*)nullptr, n);
    return std::max(std::max(sortBytes, scanBytes), plocBytes);
}

size_t lbvhScratchBytes(int n) {
    size_t tmp = cubTempBytes(n);
    size_t s = 0;
    s += 2 * sizeof(unsigned long long) * n + 2 * sizeof(int) * n;  // keys, values (double buffer)
    s += sizeof(int2) * n * 2;                                       // range, child
    s += sizeof(int) * n * 2;                                        // parents
    s += sizeof(int) * n * 4;                                        // visits, collapse, kept, newIdx
    s += sizeof(float) * n * 7;                                      // boxes, cost
    s += sizeof(int) * n * 6 + sizeof(unsigned long long) * n + sizeof(float) * n * 12 + sizeof(int2) * n + 4096;  // PLOC clusters, positions, boxes, sizes
    s += tmp + 64 * 256 + 64;
    return s;
}

int buildLbvh(const float4* tri, int n, float4* nodesOut, int* orderOut, void* scratch, size_t scratchBytes, int* hostNodeCount, int* hostMaxDepth,
              cudaStream_t st, int method) {
    if (n <= 0) { *hostNodeCount = 0; *hostMaxDepth = 0; return 0; }
    if (n == 1) {
        k_emit_single<<<1, 1, 0, st>>>(tri, nodesOut);
        int zero = 0;
        cudaMemcpyAsync(orderOut, &zero, sizeof(int), cudaMemcpyHostToDevice, st);
        *hostNodeCount = 1;
        *hostMaxDepth = 0;
        return cudaStreamSynchronize(st) == cudaSuccess ? 0 : -1;
    }
    char* p = static_cast<char*>(scratch);
    unsigned long long* keysA = carve<unsigned long long>(p, n);
    unsigned long long* keysB = carve<unsigned long long>(p, n);
    int* valsA = carve<int>(p, n);
    int* valsB = carve<int>(p, n);
    int2* range = carve<int2>(p, n);
    int2* child = carve<int2>(p, n);
    int* parentInner = carve<int>(p, n);
    int* parentLeaf = carve<int>(p, n);
    int* visits = carve<int>(p, n);
    int* collapse = carve<int>(p, n);
    int* kept = carve<int>(p, n);
    int* newIdx = carve<int>(p, n);
    float* boxes = carve<float>(p, 6 * size_t(n));
    float* cost = carve<float>(p, n);
    int* small = carve<int>(p, 16);  // 0..5 centroid bounds, 6 max depth, 7 kept total
    size_t tmpBytes = cubTempBytes(n);
    void* tmp = carve<char>(p, tmpBytes);
    if (size_t(p - static_cast<char*>(scratch)) > scratchBytes) return -2;

    int init[8] = {0x7FFFFFFF, 0x7FFFFFFF, 0x7FFFFFFF, (int)0x80000000, (int)0x80000000, (int)0x80000000, 0, 0};
    cudaMemcpyAsync(small, init, sizeof(init), cudaMemcpyHostToDevice, st);
    int grid = (n + 255) / 256;
    k_centroid_bounds<<<std::min(grid, 1024), 256, 0, st>>>(tri, n, small);
    k_morton<<<grid, 256, 0, st>>>(tri, n, small, keysA, valsA);
    cub::DeviceRadixSort::SortPairs(tmp, tmpBytes, keysA, keysB, valsA, valsB, n, 0, 63, st);
    cudaMemsetAsync(parentInner, 0xFF, sizeof(int) * n, st);
    cudaMemsetAsync(visits, 0, sizeof(int) * n, st);
    const int* order = valsB;
    if (method == 1 && n > 2) {
        // PLOC topology in place of the radix tree
        const char* re = getenv("SST_PLOC_RADIUS");
        const int plocRadius = re ? std::max(1, std::min(256, atoi(re))) : 16;
        int* clus = carve<int>(p, n);
        int* clus2 = carve<int>(p, n);
        float* cbox = carve<float>(p, 6 * size_t(n));
        float* cbox2 = carve<float>(p, 6 * size_t(n));
        int* nn = carve<int>(p, n);
        unsigned long long* before = carve<unsigned long long>(p, n);
        int* nc = carve<int>(p, 4);
        int2* childC = carve<int2>(p, n);
        int* size = carve<int>(p, n);
        int* leafPos = carve<int>(p, n);
        int* order2 = carve<int>(p, n);
        if (size_t(p - static_cast<char*>(scratch)) > scratchBytes) return -2;
        k_ploc_init<<<grid, 256, 0, st>>>(tri, valsB, n, clus, cbox);
        // Every round reads the cluster count on the device; the host's figure only bounds the grids and
        // the scan, so it is read back once every few rounds, until one block can do the rest.
        int ncH = n, cur = 0;
        cudaMemcpyAsync(nc, &ncH, sizeof(int), cudaMemcpyHostToDevice, st);
        static_assert(kTailSmem <= 200 * 1024, "shared memory of the tail block");
        if (cudaFuncSetAttribute(k_ploc_tail, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kTailSmem)) != cudaSuccess) return -1;
        while (ncH > kTailClusters) {
            for (int r = 0; r < kPlocRounds; ++r) {
                const int* ncIn = nc + cur;
                k_ploc_nn<<<(ncH + kNnThreads - 1) / kNnThreads, kNnThreads, 0, st>>>(cbox, ncIn, plocRadius, nn);
                auto flags = thrust::make_transform_iterator(thrust::make_counting_iterator<int>(0), PlocFlags{nn, ncIn});
                size_t scanBytes = tmpBytes;
                if (cub::DeviceScan::ExclusiveSum(tmp, scanBytes, flags, before, ncH, st) != cudaSuccess) return -2;
                k_ploc_compact<<<(ncH + 255) / 256, 256, 0, st>>>(clus, cbox, nn, ncIn, n, before, clus2, cbox2, nc + (1 - cur), childC);
                cur = 1 - cur;
                std::swap(clus, clus2);
                std::swap(cbox, cbox2);
            }
            int left = 0;
            cudaMemcpyAsync(&left, nc + cur, sizeof(int), cudaMemcpyDeviceToHost, st);
            if (cudaStreamSynchronize(st) != cudaSuccess) return -1;
            if (left >= ncH || left < 1) return -3;  // every round merges at least the closest pair: degenerate boxes
            ncH = left;
        }
        k_ploc_tail<<<1, kTailThreads, kTailSmem, st>>>(clus, cbox, nc + cur, n, plocRadius, childC);
        cudaMemcpyAsync(&ncH, nc + cur, sizeof(int), cudaMemcpyDeviceToHost, st);
        if (cudaStreamSynchronize(st) != cudaSuccess) return -1;
        if (ncH != 1) return -3;
        k_ploc_renumber<<<grid, 256, 0, st>>>(childC, n, child, parentInner, parentLeaf);
        cudaMemsetAsync(size, 0, sizeof(int) * n, st);
        k_ploc_sizes<<<grid, 256, 0, st>>>(child, parentLeaf, parentInner, n, visits, size);
        cudaMemsetAsync(visits, 0, sizeof(int) * n, st);
        k_ploc_offsets<<<(2 * n - 1 + 255) / 256, 256, 0, st>>>(child, parentInner, parentLeaf, size, n, range, leafPos);
        k_ploc_reorder<<<grid, 256, 0, st>>>(child, leafPos, valsB, n, order2);
        // the leaves' parents in the new order
        cudaMemsetAsync(parentLeaf, 0xFF, sizeof(int) * n, st);
        k_ploc_leaf_parents<<<grid, 256, 0, st>>>(child, n, parentLeaf);
        order = order2;
    } else {
        k_karras<<<grid, 256, 0, st>>>(keysB, n, range, child, parentInner, parentLeaf);
    }
    // SAH constants: traversal cost relative to one triangle test and the largest leaf
    // (SST_BVH_CT / SST_BVH_LEAF override them for experiments)
    const char* ctEnv = getenv("SST_BVH_CT");
    const char* leafEnv = getenv("SST_BVH_LEAF");
    const float ct = ctEnv ? (float)atof(ctEnv) : kCt;
    const int maxLeaf = leafEnv ? std::max(1, std::min(kMaxLeafSize, atoi(leafEnv))) : kMaxLeafSize;
    k_refit<<<grid, 256, 0, st>>>(tri, order, n, range, child, parentInner, parentLeaf, visits, boxes, cost, collapse, ct, maxLeaf);
    k_kept<<<grid, 256, 0, st>>>(parentInner, collapse, n, kept, small + 6);
    size_t scanBytes = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, scanBytes, kept, newIdx, n - 1, st);
    if (scanBytes > tmpBytes) return -2;
    cub::DeviceScan::ExclusiveSum(tmp, scanBytes, kept, newIdx, n - 1, st);
    int hs[2];
    cudaMemcpyAsync(&hs[0], newIdx + (n - 2), sizeof(int), cudaMemcpyDeviceToHost, st);
    cudaMemcpyAsync(&hs[1], kept + (n - 2), sizeof(int), cudaMemcpyDeviceToHost, st);
    int md = 0;
    cudaMemcpyAsync(&md, small + 6, sizeof(int), cudaMemcpyDeviceToHost, st);
    if (cudaStreamSynchronize(st) != cudaSuccess) return -1;
    *hostNodeCount = hs[0] + hs[1];
    *hostMaxDepth = md;
    k_emit<<<grid, 256, 0, st>>>(tri, order, n, range, child, collapse, kept, newIdx, boxes, nodesOut);
    cudaMemcpyAsync(orderOut, order, sizeof(int) * n, cudaMemcpyDeviceToDevice, st);
    return cudaStreamSynchronize(st) == cudaSuccess ? 0 : -1;
}

}  // namespace sst

namespace sst {
namespace {
__global__ void k_leaf_gather(const int* order, int n, const float4* trivG, const float4* triNG, const int4* auxG, const int4* vtxG, float4* triv,
                              float4* triN, int4* aux, int4* vtx) {
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    int g = order[t];
    float4 a = trivG[3 * (size_t)g];
    a.w = __int_as_float(g);
    triv[3 * (size_t)t] = a;
    triv[3 * (size_t)t + 1] = trivG[3 * (size_t)g + 1];
    triv[3 * (size_t)t + 2] = trivG[3 * (size_t)g + 2];
    triN[t] = triNG[g];
    aux[t] = auxG[g];
    vtx[t] = vtxG[g];
}
}  // namespace

void launch_leaf_gather(const int* order, int n, const float4* trivG, const float4* triNG, const int4* auxG, const int4* vtxG, float4* triv,
                        float4* triN, int4* aux, int4* vtx, cudaStream_t st) {
    if (n <= 0) return;
    k_leaf_gather<<<(n + 255) / 256, 256, 0, st>>>(order, n, trivG, triNG, auxG, vtxG, triv, triN, aux, vtx);
}
}  // namespace sst

// =============================================================================================
// 4-wide BVH from the binary one.  Each 4-wide node is made from a binary inner node by opening
// its inner children with the largest surface area until it has four children (or only leaves
// remain); leaves are shared unchanged.  Level-synchronous: one launch per level of the 4-wide
// tree, the frontier holds the level's binary nodes in the order of their 4-wide slots.
// Node layout (8 float4, 128 bytes): lo.x[4], hi.x[4], lo.y[4], hi.y[4], lo.z[4], hi.z[4],
// child references[4] (a 4-wide node index or a leaf reference), one unused float4 (a node is one
// 128-byte line).  Nodes with fewer children have inside-out boxes in the other places.
// =============================================================================================
namespace sst {
namespace {
struct Child4 {
    uint32_t ref;
    float lo[3], hi[3];
};
__device__ float halfArea(const Child4& c) {
    float dx = c.hi[0] - c.lo[0], dy = c.hi[1] - c.lo[1], dz = c.hi[2] - c.lo[2];
    return dx * dy + dy * dz + dz * dx;
}
__device__ void readChildren(const float4* nodes2, uint32_t b, Child4& c0, Child4& c1) {
    const float4* nd = nodes2 + 4 * (size_t)b;
    float4 n0 = nd[0], n1 = nd[1], n2 = nd[2], n3 = nd[3];
    c0.lo[0] = n0.x; c0.hi[0] = n0.y; c0.lo[1] = n0.z; c0.hi[1] = n0.w; c0.lo[2] = n2.x; c0.hi[2] = n2.y;
    c1.lo[0] = n1.x; c1.hi[0] = n1.y; c1.lo[1] = n1.z; c1.hi[1] = n1.w; c1.lo[2] = n2.z; c1.hi[2] = n2.w;
    c0.ref = __float_as_uint(n3.x);
    c1.ref = __float_as_uint(n3.y);
}
// The levels of a wide build: the number of nodes in a level and the slot of its first node, for three
// levels in turn (one being read, the next being filled, the one after zeroed), and the depth so far.
struct Levels {
    int count[3], first[3], depth;
};
// Starts a level's launch: false when the level is empty for the calling block.  Every launch empties
// the counter of the level after the next, so a launch past the last level finds nothing and harms
// nothing, and the host need not wait for the count of each level.
__device__ __forceinline__ bool beginLevel(Levels* lv, int level) {
    const int n = lv->count[level % 3];
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        lv->count[(level + 2) % 3] = 0;
        if (n > 0) {
            lv->first[(level + 1) % 3] = lv->first[level % 3] + n;
            lv->depth = level + 1;
        }
    }
    return (int)(blockIdx.x * blockDim.x) < n;
}
// Places of this lane's `inner` children in the next level (whole warps call it; one addition per warp).
__device__ __forceinline__ int placeChildren(Levels* lv, int level, int inner) {
    const int lane = threadIdx.x & 31;
    int sum = inner;
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, sum, o);
        if (lane >= o) sum += v;
    }
    int base = 0;
    if (lane == 31 && sum > 0) base = atomicAdd(&lv->count[(level + 1) % 3], sum);
    return __shfl_sync(0xffffffffu, base, 31) + sum - inner;
}
__global__ void k_collapse4(const float4* nodes2, const int* frontier, Levels* lv, int level, float4* nodes4, int* next) {
    if (!beginLevel(lv, level)) return;
    const int n = lv->count[level % 3], first = lv->first[level % 3];
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool valid = i < n;
    const int item = valid ? frontier[i] : 0;
    Child4 c[4];
    int cnt = 2;
    readChildren(nodes2, (uint32_t)item, c[0], c[1]);
    while (cnt < 4) {
        int best = -1;
        float bestA = -1.0f;
        for (int k = 0; k < cnt; ++k)
            if (!(c[k].ref & kLeafFlag)) {
                float a = halfArea(c[k]);
                if (a > bestA) { bestA = a; best = k; }
            }
        if (best < 0) break;
        Child4 a, b;
        readChildren(nodes2, c[best].ref, a, b);
        c[best] = a;
        c[cnt++] = b;
    }
    int inner = 0;
    for (int k = 0; k < cnt; ++k) inner += (c[k].ref & kLeafFlag) ? 0 : 1;
    int at = placeChildren(lv, level, valid ? inner : 0);
    if (!valid) return;
    float4* out = nodes4 + 8 * (size_t)(first + i);
    float v[6][4];
    uint32_t refs[4];
    for (int k = 0; k < 4; ++k) {
        if (k < cnt) {
            for (int a = 0; a < 3; ++a) { v[2 * a][k] = c[k].lo[a]; v[2 * a + 1][k] = c[k].hi[a]; }
            uint32_t r = c[k].ref;
            if (!(r & kLeafFlag)) {
                next[at] = (int)r;
                r = (uint32_t)(first + n + at++);  // the next level's slots follow this level's
            }
            refs[k] = r;
        } else {
            // an inside-out box: its near planes lie at +inf and its far ones at -inf for every direction
            for (int a = 0; a < 6; ++a) v[a][k] = (a & 1) ? -CUDART_INF_F : CUDART_INF_F;
            refs[k] = 0u;
        }
    }
    for (int a = 0; a < 6; ++a) out[a] = make_float4(v[a][0], v[a][1], v[a][2], v[a][3]);
    out[6] = make_float4(__uint_as_float(refs[0]), __uint_as_float(refs[1]), __uint_as_float(refs[2]), __uint_as_float(refs[3]));
    out[7] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
}
__global__ void k_collapse_root(int* frontier, Levels* lv) {
    *lv = Levels{{1, 0, 0}, {0, 1, 0}, 0};
    frontier[0] = 0;
}

// Runs launch(level, bound, ...) for every level.  A level has at most width times the nodes of the one
// before and at most the binary nodes; the counts are looked at once those bounds meet and then after
// every third level.
template <class Launch>
int buildLevels(int nNodes2, int width, void* scratch, int* hostNodeCount, int* hostDepth, cudaStream_t st, Launch launch) {
    *hostNodeCount = 0;
    *hostDepth = 0;
    if (nNodes2 <= 0) return 0;
    Levels* lv = static_cast<Levels*>(scratch);
    int* fr[2] = {reinterpret_cast<int*>(static_cast<char*>(scratch) + 256), reinterpret_cast<int*>(static_cast<char*>(scratch) + 256) + nNodes2};
    k_collapse_root<<<1, 1, 0, st>>>(fr[0], lv);
    long long bound = 1;
    int sinceLook = 0;
    bool looking = false;
    for (int level = 0; level < 4 * kMaxBvhDepth; ++level) {
        launch(level, int(bound), lv, fr[level & 1], fr[1 - (level & 1)]);
        bound = std::min<long long>(bound * width, nNodes2);
        looking |= bound == nNodes2;
        if (!looking || ++sinceLook < 3) continue;
        sinceLook = 0;
        Levels h;
        if (cudaMemcpyAsync(&h, lv, sizeof(Levels), cudaMemcpyDeviceToHost, st) != cudaSuccess) return -1;
        if (cudaStreamSynchronize(st) != cudaSuccess) return -1;
        bound = h.count[(level + 1) % 3];
        if (bound == 0) {
            *hostDepth = h.depth;
            *hostNodeCount = h.first[h.depth % 3];
            return 0;
        }
    }
    return -2;
}
}  // namespace

size_t bvh4ScratchBytes(int nNodes2) { return 2 * sizeof(int) * (size_t)std::max(1, nNodes2) + 1024; }

int buildBvh4(const float4* nodes2, int nNodes2, float4* nodes4, void* scratch, int* hostNodeCount, int* hostDepth, cudaStream_t st) {
    return buildLevels(nNodes2, 4, scratch, hostNodeCount, hostDepth, st, [&](int level, int bound, Levels* lv, int* frontier, int* next) {
        k_collapse4<<<(bound + 127) / 128, 128, 0, st>>>(nodes2, frontier, lv, level, nodes4, next);
    });
}
}  // namespace sst

// =============================================================================================
// 8-wide BVH from the binary one, its children in octant slots.  Each node is made from a
// binary inner node by opening its inner children, largest surface area first, until it has eight
// children (or only leaves remain); leaves are the binary tree's leaves, unchanged.  The children
// are then placed in the eight slots by the octant of their box centre relative to the node's
// (slot bit 0: +x side, bit 1: +y, bit 2: +z), greedily, best-aligned (child, slot) pair first,
// as in the octant ordering of Ylitie, Karras and Laine, "Efficient Incoherent Ray Traversal on
// GPUs Through Compressed Wide BVHs" (HPG 2017).  A ray whose direction has the sign bits o
// (bit set for a negative component) then visits the slots in the order s ^ o ascending, which
// puts the children that lie first along its direction first, without a per-node sort.
// Node layout (15 float4, 240 bytes): lo.x[8], hi.x[8], lo.y[8], hi.y[8], lo.z[8], hi.z[8] (two
// float4 each), child references[8] (an 8-wide node index or a leaf reference), and
// (valid-slot mask | inner-slot mask << 8, -, -, -).  Level-synchronous like the 4-wide build.
// =============================================================================================
namespace sst {
namespace {
__global__ void k_collapse8(const float4* nodes2, const int* frontier, Levels* lv, int level, float4* nodes8, int* next) {
    if (!beginLevel(lv, level)) return;
    const int n = lv->count[level % 3], first = lv->first[level % 3];
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool valid = i < n;
    const int item = valid ? frontier[i] : 0;
    Child4 c[8];
    int cnt = 2;
    readChildren(nodes2, (uint32_t)item, c[0], c[1]);
    while (cnt < 8) {
        int best = -1;
        float bestA = -1.0f;
        for (int k = 0; k < cnt; ++k)
            if (!(c[k].ref & kLeafFlag)) {
                float a = halfArea(c[k]);
                if (a > bestA) { bestA = a; best = k; }
            }
        if (best < 0) break;
        Child4 a, b;
        readChildren(nodes2, c[best].ref, a, b);
        c[best] = a;
        c[cnt++] = b;
    }
    // node centre and the children's offsets from it
    float lo[3] = {CUDART_INF_F, CUDART_INF_F, CUDART_INF_F}, hi[3] = {-CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F};
    for (int k = 0; k < cnt; ++k)
        for (int a = 0; a < 3; ++a) { lo[a] = fminf(lo[a], c[k].lo[a]); hi[a] = fmaxf(hi[a], c[k].hi[a]); }
    float off[8][3];
    for (int k = 0; k < cnt; ++k)
        for (int a = 0; a < 3; ++a) off[k][a] = 0.5f * (c[k].lo[a] + c[k].hi[a]) - 0.5f * (lo[a] + hi[a]);
    // greedy assignment: repeatedly the (child, slot) pair of largest alignment between the child's
    // offset and the slot's octant direction among the unassigned ones (ties: lower child, slot)
    int slotOf[8], childIn[8];
    for (int k = 0; k < 8; ++k) { slotOf[k] = -1; childIn[k] = -1; }
    for (int n = 0; n < cnt; ++n) {
        float bestV = -CUDART_INF_F;
        int bc = -1, bs = -1;
        for (int k = 0; k < cnt; ++k) {
            if (slotOf[k] >= 0) continue;
            for (int s = 0; s < 8; ++s) {
                if (childIn[s] >= 0) continue;
                float v = ((s & 1) ? off[k][0] : -off[k][0]) + ((s & 2) ? off[k][1] : -off[k][1]) + ((s & 4) ? off[k][2] : -off[k][2]);
                if (v > bestV) { bestV = v; bc = k; bs = s; }
            }
        }
        slotOf[bc] = bs;
        childIn[bs] = bc;
    }
    int numInner = 0;
    for (int k = 0; k < cnt; ++k) numInner += (c[k].ref & kLeafFlag) ? 0 : 1;
    int at = placeChildren(lv, level, valid ? numInner : 0);
    if (!valid) return;
    float v[6][8];
    uint32_t refs[8];
    uint32_t slots = 0, inner = 0;
    for (int s = 0; s < 8; ++s) {
        const int k = childIn[s];
        if (k >= 0) {
            for (int a = 0; a < 3; ++a) { v[2 * a][s] = c[k].lo[a]; v[2 * a + 1][s] = c[k].hi[a]; }
            uint32_t r = c[k].ref;
            slots |= 1u << s;
            if (!(r & kLeafFlag)) {
                next[at] = (int)r;
                r = (uint32_t)(first + n + at++);
                inner |= 1u << s;
            }
            refs[s] = r;
        } else {
            for (int a = 0; a < 6; ++a) v[a][s] = 0.0f;
            refs[s] = 0u;
        }
    }
    float4* out = nodes8 + 15 * (size_t)(first + i);
    for (int a = 0; a < 6; ++a) {
        out[2 * a] = make_float4(v[a][0], v[a][1], v[a][2], v[a][3]);
        out[2 * a + 1] = make_float4(v[a][4], v[a][5], v[a][6], v[a][7]);
    }
    out[12] = make_float4(__uint_as_float(refs[0]), __uint_as_float(refs[1]), __uint_as_float(refs[2]), __uint_as_float(refs[3]));
    out[13] = make_float4(__uint_as_float(refs[4]), __uint_as_float(refs[5]), __uint_as_float(refs[6]), __uint_as_float(refs[7]));
    out[14] = make_float4(__uint_as_float(slots | (inner << 8)), 0.0f, 0.0f, 0.0f);
}
}  // namespace

size_t bvh8ScratchBytes(int nNodes2) { return bvh4ScratchBytes(nNodes2); }

int buildBvh8(const float4* nodes2, int nNodes2, float4* nodes8, void* scratch, int* hostNodeCount, int* hostDepth, cudaStream_t st) {
    return buildLevels(nNodes2, 8, scratch, hostNodeCount, hostDepth, st, [&](int level, int bound, Levels* lv, int* frontier, int* next) {
        k_collapse8<<<(bound + 127) / 128, 128, 0, st>>>(nodes2, frontier, lv, level, nodes8, next);
    });
}
}  // namespace sst
