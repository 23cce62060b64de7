// Scene construction on the GPU: vertex normals, scene AABB, primitive
// precomputation and the LBVH (Morton codes, radix sort, Karras hierarchy,
// bottom-up refit, breadth-first node order) and the walk kernels' search tree.
//
// Replaces the reference's host Scene<N>::configure_normal / configure
// (include/scene.cuh:368-453), which did the AABB on the host and the BVH in
// the third-party lbvh library.  Everything here is deterministic: vertex
// normals are summed per vertex in (face, slot) order, the tree is a pure
// function of the sorted (morton << 32 | prim) keys, and boxes are min/max.
#include <cub/cub.cuh>

#include <vector>

#include "scene_impl.h"
#include "wos_device.cuh"

namespace wosd {

#define WOS_TRY(x)                                    \
    do {                                              \
        cudaError_t _e = (x);                         \
        if (_e != cudaSuccess) return fail_cuda(_e, #x); \
    } while (0)

// ------------------------------------------------------------------ kernels
__device__ __forceinline__ int ordered_int(float f) {
    int i = __float_as_int(f);
    return i >= 0 ? i : i ^ 0x7fffffff;
}
__device__ __forceinline__ float from_ordered_int(int i) { return __int_as_float(i >= 0 ? i : i ^ 0x7fffffff); }

// out[0]: whether an index is out of range; out[1] (2D): segments f whose end
// vertex starts segment f + 1, cyclically.
__global__ void k_check_indices(const int *F, int nF, int dim, int nV, int *out) {
    int bad = 0, chain = 0;
    for (long long f = blockIdx.x * (long long)blockDim.x + threadIdx.x; f < nF; f += (long long)gridDim.x * blockDim.x) {
        for (int k = 0; k < dim; ++k) bad |= F[f * dim + k] < 0 || F[f * dim + k] >= nV;
        if (dim == 2) chain += F[2 * f + 1] == F[2 * (f + 1 < nF ? f + 1 : 0)];
    }
    if (bad) atomicOr(&out[0], 1);
    if (chain) atomicAdd(&out[1], chain);
}

// Start of a build's counters: [0, 6) the bounding box's ordered ints, [6] the
// deepest node, [7, 9) floats: the order's cost (k_tree_bounds).
constexpr int BUILD_COUNTERS = 9;
__global__ void k_build_init(int *c) {
    if (threadIdx.x < BUILD_COUNTERS)
        c[threadIdx.x] = threadIdx.x < 3 ? 0x7fffffff : threadIdx.x < 6 ? (int)0x80000000 : 0;
}

__global__ void k_aabb(const float *V, int nV, int dim, int *lohi) {
    // lohi[0..2] = ordered min, lohi[3..5] = ordered max
    __shared__ int smin[3], smax[3];
    if (threadIdx.x < 3) {
        smin[threadIdx.x] = 0x7fffffff;
        smax[threadIdx.x] = (int)0x80000000;
    }
    __syncthreads();
    int lmin[3] = {0x7fffffff, 0x7fffffff, 0x7fffffff}, lmax[3] = {(int)0x80000000, (int)0x80000000, (int)0x80000000};
    for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < nV; v += gridDim.x * blockDim.x)
        for (int k = 0; k < dim; ++k) {
            const int o = ordered_int(V[(size_t)v * dim + k]);
            lmin[k] = min(lmin[k], o);
            lmax[k] = max(lmax[k], o);
        }
    for (int k = 0; k < dim; ++k) {
        atomicMin(&smin[k], lmin[k]);
        atomicMax(&smax[k], lmax[k]);
    }
    __syncthreads();
    if (threadIdx.x < dim) {
        atomicMin(&lohi[threadIdx.x], smin[threadIdx.x]);
        atomicMax(&lohi[3 + threadIdx.x], smax[threadIdx.x]);
    }
}

// Per (face, slot) normal contribution.
template <int D>
__global__ void k_face_normals(const float *V, const int *F, int nF, float *contrib) {
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= nF) return;
    if (D == 2) {
        const int i0 = F[2 * f], i1 = F[2 * f + 1];
        const float dx = V[2 * i1] - V[2 * i0], dy = V[2 * i1 + 1] - V[2 * i0 + 1];
        float nx = dy, ny = -dx;
        const float len = sqrtf(dot2(nx, ny, nx, ny));
        if (len > 0.0f) {
            nx = nx / len;
            ny = ny / len;
        } else {
            nx = ny = 0.0f;
        }
        for (int s = 0; s < 2; ++s) {
            contrib[(size_t)(2 * f + s) * 2] = nx;
            contrib[(size_t)(2 * f + s) * 2 + 1] = ny;
        }
    } else {
        const int i0 = F[3 * f], i1 = F[3 * f + 1], i2 = F[3 * f + 2];
        const float *p0 = V + 3 * (size_t)i0, *p1 = V + 3 * (size_t)i1, *p2 = V + 3 * (size_t)i2;
        float e10[3], e20[3], e21[3], e01[3], e02[3], e12[3];
        for (int k = 0; k < 3; ++k) {
            e10[k] = p1[k] - p0[k];
            e20[k] = p2[k] - p0[k];
            e21[k] = p2[k] - p1[k];
            e01[k] = p0[k] - p1[k];
            e02[k] = p0[k] - p2[k];
            e12[k] = p1[k] - p2[k];
        }
        float n[3];
        cross3(e10[0], e10[1], e10[2], e20[0], e20[1], e20[2], n[0], n[1], n[2]);
        const float len = sqrtf(dot3(n[0], n[1], n[2], n[0], n[1], n[2]));
        if (len > 0.0f) {
            for (int k = 0; k < 3; ++k) n[k] = n[k] / len;
        } else {
            n[0] = n[1] = n[2] = 0.0f;
        }
        auto angle = [](const float *a, const float *b) {
            float c[3];
            cross3(a[0], a[1], a[2], b[0], b[1], b[2], c[0], c[1], c[2]);
            return wosm::atan2_(sqrtf(dot3(c[0], c[1], c[2], c[0], c[1], c[2])), dot3(a[0], a[1], a[2], b[0], b[1], b[2]));
        };
        const float ang[3] = {angle(e10, e20), angle(e21, e01), angle(e02, e12)};
        for (int s = 0; s < 3; ++s) {
            for (int k = 0; k < 3; ++k) contrib[(size_t)(3 * f + s) * 3 + k] = ang[s] * n[k];
        }
    }
}

__global__ void k_iota(int *x, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) x[i] = i;
}

// First slot of each vertex in the sorted slots, first[nV] = n: vertices without
// faces have an empty range.  A search per vertex: filling the vertices between two
// neighbours' from the slots leaves a long run of them to one thread (20 million
// vertices of which the first 1,000 have faces: 74 ms a scene, 17 where those are
// spread).
__global__ void k_vertex_ranges(const int *verts, int n, int nV, int *first) {
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v > nV) return;
    int lo = 0, hi = n;
    while (lo < hi) {
        const int mid = lo + (hi - lo) / 2;
        if (verts[mid] < v)
            lo = mid + 1;
        else
            hi = mid;
    }
    first[v] = lo;
}

template <int D>
__global__ void k_vertex_normals(const int *slots, const int *first, const float *contrib, int nV, float *N) {
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= nV) return;
    float s[3] = {0.0f, 0.0f, 0.0f};
    const int end = first[v + 1];
    for (int i = first[v]; i < end; ++i) {
        const int slot = slots[i];
        for (int k = 0; k < D; ++k) s[k] += contrib[(size_t)slot * D + k];
    }
    const float len = sqrtf(D == 2 ? dot2(s[0], s[1], s[0], s[1]) : dot3(s[0], s[1], s[2], s[0], s[1], s[2]));
    for (int k = 0; k < D; ++k) N[(size_t)v * D + k] = len > 0.0f ? s[k] / len : 0.0f;
}

__device__ __forceinline__ uint32_t spread2(uint32_t x) {
    x &= 0xffffu;
    x = (x | (x << 8)) & 0x00ff00ffu;
    x = (x | (x << 4)) & 0x0f0f0f0fu;
    x = (x | (x << 2)) & 0x33333333u;
    x = (x | (x << 1)) & 0x55555555u;
    return x;
}
__device__ __forceinline__ uint32_t spread3(uint32_t x) {
    x &= 0x3ffu;
    x = (x | (x << 16)) & 0x030000ffu;
    x = (x | (x << 8)) & 0x0300f00fu;
    x = (x | (x << 4)) & 0x030c30c3u;
    x = (x | (x << 2)) & 0x09249249u;
    return x;
}

// Hilbert index of a 3D cell (10 bits per axis), by Skilling's transpose
// method ("Programming the Hilbert curve", AIP Conf. Proc. 707, 2004): undo
// the excess work of the axes, Gray-encode, then interleave the transposed
// bits, axis 0 most significant.  Consecutive indices are face-adjacent
// cells, so runs of primitives sorted by it are more compact than Morton
// runs, whose curve jumps between octants.
__device__ __forceinline__ uint32_t hilbert3(uint32_t x0, uint32_t x1, uint32_t x2) {
    uint32_t X[3] = {x0, x1, x2};
    const uint32_t M = 1u << 9;
    for (uint32_t Q = M; Q > 1; Q >>= 1) {
        const uint32_t P = Q - 1;
        for (int i = 0; i < 3; ++i) {
            if (X[i] & Q) {
                X[0] ^= P;
            } else {
                const uint32_t t = (X[0] ^ X[i]) & P;
                X[0] ^= t;
                X[i] ^= t;
            }
        }
    }
    X[1] ^= X[0];
    X[2] ^= X[1];
    uint32_t t = 0;
    for (uint32_t Q = M; Q > 1; Q >>= 1)
        if (X[2] & Q) t ^= Q - 1;
    for (int i = 0; i < 3; ++i) X[i] ^= t;
    return (spread3(X[0]) << 2) | (spread3(X[1]) << 1) | spread3(X[2]);
}

// Primitive precomputation, primitive boxes and sort keys: Morton (order 0),
// the input index (order 1) or Hilbert (order 2) of the box centre.
template <int D>
__global__ void k_prims(const float *V, const int *F, int nF, const int *lohi, float4 *seg, float *seginv,
                        float4 *tri, float *pbox, unsigned long long *keys, int order) {
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= nF) return;
    float slo[3], shi[3];
    for (int k = 0; k < D; ++k) {
        slo[k] = from_ordered_int(lohi[k]);
        shi[k] = from_ordered_int(lohi[3 + k]);
    }
    float bl[3], bh[3];
    if (D == 2) {
        const int i0 = F[2 * f], i1 = F[2 * f + 1];
        const float ax = V[2 * i0], ay = V[2 * i0 + 1], bx = V[2 * i1], by = V[2 * i1 + 1];
        const float bax = bx - ax, bay = by - ay;
        const float len2 = dot2(bax, bay, bax, bay);
        seg[f] = make_float4(ax, ay, bax, bay);
        seginv[f] = len2 > 0.0f ? 1.0f / len2 : 0.0f;
        bl[0] = fminf(ax, bx);
        bh[0] = fmaxf(ax, bx);
        bl[1] = fminf(ay, by);
        bh[1] = fmaxf(ay, by);
    } else {
        const int i0 = F[3 * f], i1 = F[3 * f + 1], i2 = F[3 * f + 2];
        float a[3], b[3], c[3];
        for (int k = 0; k < 3; ++k) {
            a[k] = V[3 * (size_t)i0 + k];
            b[k] = V[3 * (size_t)i1 + k];
            c[k] = V[3 * (size_t)i2 + k];
        }
        float ab[3], ac[3];
        for (int k = 0; k < 3; ++k) {
            ab[k] = b[k] - a[k];
            ac[k] = c[k] - a[k];
        }
        tri[3 * f] = make_float4(a[0], a[1], a[2], dot3(ab[0], ab[1], ab[2], ab[0], ab[1], ab[2]));
        tri[3 * f + 1] = make_float4(ab[0], ab[1], ab[2], dot3(ab[0], ab[1], ab[2], ac[0], ac[1], ac[2]));
        tri[3 * f + 2] = make_float4(ac[0], ac[1], ac[2], dot3(ac[0], ac[1], ac[2], ac[0], ac[1], ac[2]));
        for (int k = 0; k < 3; ++k) {
            bl[k] = fminf(fminf(a[k], b[k]), c[k]);
            bh[k] = fmaxf(fmaxf(a[k], b[k]), c[k]);
        }
    }
    uint32_t q[3];
    const float scale = D == 2 ? 65536.0f : 1024.0f;
    for (int k = 0; k < D; ++k) {
        pbox[(size_t)f * 2 * D + k] = bl[k];
        pbox[(size_t)f * 2 * D + D + k] = bh[k];
        const float c = (bl[k] + bh[k]) * 0.5f;
        const float ext = shi[k] - slo[k];
        const float u = ext > 0.0f ? (c - slo[k]) / ext : 0.0f;
        q[k] = (uint32_t)fminf(fmaxf(u * scale, 0.0f), scale - 1.0f);
    }
    uint32_t m;
    if (order == 1)
        m = (uint32_t)f;
    else if (D == 3 && order == 2)
        m = hilbert3(q[0], q[1], q[2]);
    else
        m = D == 2 ? (spread2(q[0]) | (spread2(q[1]) << 1))
                   : (spread3(q[0]) | (spread3(q[1]) << 1) | (spread3(q[2]) << 2));
    keys[f] = ((unsigned long long)m << 32) | (unsigned)f;
}

__device__ __forceinline__ int kdelta(const unsigned long long *k, int n, int i, int j) {
    if (j < 0 || j >= n) return -1;
    return __clzll(k[i] ^ k[j]);
}

// Karras 2012, one thread per internal node.
__global__ void k_karras(const unsigned long long *k, int n, int2 *child, int *parent_int, int *parent_leaf) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n - 1) return;
    const int d = (kdelta(k, n, i, i + 1) - kdelta(k, n, i, i - 1)) >= 0 ? 1 : -1;
    const int dmin = kdelta(k, n, i, i - d);
    int lmax = 2;
    while (kdelta(k, n, i, i + lmax * d) > dmin) lmax *= 2;
    int l = 0;
    for (int t = lmax / 2; t >= 1; t /= 2)
        if (kdelta(k, n, i, i + (l + t) * d) > dmin) l += t;
    const int j = i + l * d;
    const int dnode = kdelta(k, n, i, j);
    int s = 0;
    for (int div = 2;; div *= 2) {
        const int t = (l + div - 1) / div;
        if (kdelta(k, n, i, i + (s + t) * d) > dnode) s += t;
        if (t == 1) break;
    }
    const int gamma = i + s * d + min(d, 0);
    int2 c;
    if (min(i, j) == gamma) {
        c.x = ~gamma;
        parent_leaf[gamma] = i;
    } else {
        c.x = gamma;
        parent_int[gamma] = i;
    }
    if (max(i, j) == gamma + 1) {
        c.y = ~(gamma + 1);
        parent_leaf[gamma + 1] = i;
    } else {
        c.y = gamma + 1;
        parent_int[gamma + 1] = i;
    }
    child[i] = c;
}

// Bottom-up boxes: the second thread to reach a node merges its children.
template <int D>
__global__ void k_refit(const unsigned long long *keys, int n, const float *pbox, const int2 *child,
                        const int *parent_int, const int *parent_leaf, int *flags, float *nbox) {
    const int leaf = blockIdx.x * blockDim.x + threadIdx.x;
    if (leaf >= n) return;
    int v = parent_leaf[leaf];
    while (v >= 0) {
        __threadfence();
        if (atomicAdd(&flags[v], 1) == 0) return;
        __threadfence();
        const int2 c = child[v];
        float lo[3], hi[3];
        for (int side = 0; side < 2; ++side) {
            const int r = side == 0 ? c.x : c.y;
            const float *b;
            if (r < 0) {
                const unsigned prim = (unsigned)keys[~r];
                b = pbox + (size_t)prim * 2 * D;
            } else {
                b = nbox + (size_t)r * 2 * D;
            }
            for (int k = 0; k < D; ++k) {
                const float l = __ldcg(b + k), h = __ldcg(b + D + k);
                lo[k] = side == 0 ? l : fminf(lo[k], l);
                hi[k] = side == 0 ? h : fmaxf(hi[k], h);
            }
        }
        for (int k = 0; k < D; ++k) {
            __stcg(nbox + (size_t)v * 2 * D + k, lo[k]);
            __stcg(nbox + (size_t)v * 2 * D + D + k, hi[k]);
        }
        v = parent_int[v];
    }
}

__global__ void k_depth(const int *parent_int, int nInt, unsigned long long *dkeys, int *maxdepth) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nInt) return;
    int d = 0, v = i;
    while (v > 0 && d < 4096) {
        v = parent_int[v];
        ++d;
    }
    dkeys[i] = ((unsigned long long)d << 32) | (unsigned)i;
    atomicMax(maxdepth, d);
}

__global__ void k_bfs_rank(const unsigned long long *sorted, int nInt, int *new_of_old) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= nInt) return;
    new_of_old[(unsigned)sorted[r]] = r;
}

template <int D>
__global__ void k_write_nodes(const unsigned long long *keys, int nInt, const float *pbox, const float *nbox,
                              const int2 *child, const int *new_of_old, float4 *node) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nInt) return;
    const int2 c = child[i];
    float lo[2][3], hi[2][3];
    int ref[2];
    for (int side = 0; side < 2; ++side) {
        const int r = side == 0 ? c.x : c.y;
        const float *b;
        if (r < 0) {
            b = pbox + (size_t)(unsigned)keys[~r] * 2 * D;
            ref[side] = r;
        } else {
            b = nbox + (size_t)r * 2 * D;
            ref[side] = new_of_old[r];
        }
        for (int k = 0; k < D; ++k) {
            lo[side][k] = b[k];
            hi[side][k] = b[D + k];
        }
    }
    const int o = new_of_old[i];
    if (D == 2) {
        node[3 * o] = make_float4(lo[0][0], lo[0][1], hi[0][0], hi[0][1]);
        node[3 * o + 1] = make_float4(lo[1][0], lo[1][1], hi[1][0], hi[1][1]);
        node[3 * o + 2] = make_float4(__int_as_float(ref[0]), __int_as_float(ref[1]), 0.0f, 0.0f);
    } else {
        node[4 * o] = make_float4(lo[0][0], lo[0][1], lo[0][2], hi[0][0]);
        node[4 * o + 1] = make_float4(hi[0][1], hi[0][2], lo[1][0], lo[1][1]);
        node[4 * o + 2] = make_float4(lo[1][2], hi[1][0], hi[1][1], hi[1][2]);
        node[4 * o + 3] = make_float4(__int_as_float(ref[0]), __int_as_float(ref[1]), 0.0f, 0.0f);
    }
}

template <int D>
__global__ void k_leaf_data(const unsigned long long *keys, int n, const float4 *seg, const float *seginv,
                            const float4 *tri, float4 *lseg, float *lseginv, float4 *ltri, int *lorig) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    const int f = (int)(unsigned)keys[s];
    lorig[s] = f;
    if (D == 2) {
        lseg[s] = seg[f];
        lseginv[s] = seginv[f];
    } else {
        ltri[3 * s] = tri[3 * f];
        ltri[3 * s + 1] = tri[3 * f + 1];
        ltri[3 * s + 2] = tri[3 * f + 2];
    }
}

// Leaf blocks of the search tree (SceneView::prims) in the tree's order: torig,
// or, where `keys` is given, the order of those sorted keys, stored to torig.  The
// last leaf repeats the last primitive.
template <int D>
__global__ void k_tree_prims(int nF, int n_leaf, const unsigned long long *keys, const float4 *seg,
                             const float *seginv, const float4 *tri, float4 *prims, int *torig) {
    constexpr int N = Tree<D>::LEAF, W = Tree<D>::LEAF_W;
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n_leaf * N) return;
    const int s = min(p, nF - 1), leaf = p / N, c = p % N;
    const int f = keys != nullptr ? (int)(unsigned)keys[s] : torig[s];
    if (keys != nullptr || p >= nF) torig[p] = f;
    float4 *b = prims + (size_t)leaf * W;
    if (D == 2) {
        b[c] = seg[f];
        reinterpret_cast<float *>(b + 4)[c] = seginv[f];
    } else {
        for (int k = 0; k < 3; ++k) b[3 * c + k] = tri[3 * (size_t)f + k];
    }
}

// ------------------------------------------------------------------ tree order
// Order of a mesh's triangles in its search tree: recursive median splits.  From
// one segment of `cap` positions (a power of two times the leaf size, covering the
// mesh) down to leaves, each segment is sorted along the longest axis of its
// triangles' centres and cut in the middle, so that every node of the implicit
// tree is a compact patch.  Runs of a Hilbert curve, whose cells cut a surface
// anywhere, take 28 node and 5.7 leaf visits per query on 81,920 triangles where
// these take 20 and 4.5.  Segments above SPLIT_SMALL positions are sorted by one
// radix sort per level (keys: segment, then the coordinate in 16 bits, or what is left
// of 32 above 134 million triangles); one block takes each smaller segment through all of
// its levels in shared memory.
constexpr int SPLIT_SMALL = 1024;

__device__ __forceinline__ float box_centre(const float *pbox, int f, int k) {
    return (pbox[6 * (size_t)f + k] + pbox[6 * (size_t)f + 3 + k]) * 0.5f;
}

__global__ void k_split_init(int *bounds, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) bounds[i] = i % 6 < 3 ? 0x7fffffff : (int)0x80000000;
}

// Bounds of the segments' centres, ordered ints: 3 minima, 3 maxima each.
// cap: a multiple of the block's size.
__global__ void __launch_bounds__(256) k_split_bounds(const float *pbox, const int *ord, int nF, int cap, int *bounds) {
    __shared__ int red[6];
    if (threadIdx.x < 6) red[threadIdx.x] = threadIdx.x < 3 ? 0x7fffffff : (int)0x80000000;
    __syncthreads();
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    for (int k = 0; k < 3; ++k) {
        const bool on = p < nF;
        const int c = on ? ordered_int(box_centre(pbox, ord[p], k)) : 0;
        const int lo = __reduce_min_sync(0xffffffffu, on ? c : 0x7fffffff);
        const int hi = __reduce_max_sync(0xffffffffu, on ? c : (int)0x80000000);
        if ((threadIdx.x & 31) == 0) {
            atomicMin(&red[k], lo);
            atomicMax(&red[3 + k], hi);
        }
    }
    __syncthreads();
    int *b = bounds + 6 * ((blockIdx.x * blockDim.x) / cap);
    if (threadIdx.x < 3) atomicMin(&b[threadIdx.x], red[threadIdx.x]);
    else if (threadIdx.x < 6) atomicMax(&b[threadIdx.x], red[threadIdx.x]);
}

__device__ __forceinline__ int longest_axis(const int *b, float &lo, float &ext) {
    int a = 0;
    ext = -1.0f;
    for (int k = 0; k < 3; ++k) {
        const float l = from_ordered_int(b[k]), e = from_ordered_int(b[3 + k]) - l;
        if (e > ext) {
            a = k;
            ext = e;
            lo = l;
        }
    }
    if (!(ext >= 0.0f)) lo = 0.0f;
    return a;
}

__global__ void k_split_keys(const float *pbox, const int *ord, int nF, int cap, int bits, const int *bounds,
                             unsigned *keys) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= nF) return;
    const int seg = p / cap;
    float lo, ext;
    const int a = longest_axis(bounds + 6 * seg, lo, ext);
    const float u = ext > 0.0f ? (box_centre(pbox, ord[p], a) - lo) / ext : 0.0f;
    const float n = (float)(1 << bits);
    keys[p] = (unsigned)seg << bits | (unsigned)fminf(fmaxf(u * n, 0.0f), n - 1.0f);
}

__global__ void __launch_bounds__(SPLIT_SMALL) k_split_small(const float *pbox, int nF, int leaf, int *ord) {
    __shared__ float cen[3][SPLIT_SMALL];
    __shared__ int ids[SPLIT_SMALL];
    __shared__ unsigned long long buf[SPLIT_SMALL];
    __shared__ int bounds[SPLIT_SMALL / 32][6];
    const unsigned FULL = 0xffffffffu;
    const int t = threadIdx.x, p = blockIdx.x * SPLIT_SMALL + t;
    const bool on = p < nF;  // the last positions stay last: their keys are the largest
    ids[t] = on ? ord[p] : -1;
    for (int k = 0; k < 3; ++k) cen[k][t] = on ? box_centre(pbox, ids[t], k) : 0.0f;
    __syncthreads();
    for (int cap = SPLIT_SMALL; cap > leaf; cap >>= 1) {
        // bounds of each segment's centres
        const int seg = t / cap;
        int b[6];
        for (int k = 0; k < 3; ++k) {
            const int c = ordered_int(cen[k][t]);
            b[k] = on ? c : 0x7fffffff;
            b[3 + k] = on ? c : (int)0x80000000;
            for (int o = 1; o < min(cap, 32); o <<= 1) {
                b[k] = min(b[k], __shfl_xor_sync(FULL, b[k], o));
                b[3 + k] = max(b[3 + k], __shfl_xor_sync(FULL, b[3 + k], o));
            }
        }
        if (cap > 32) {
            if (t < SPLIT_SMALL / 32)
                for (int k = 0; k < 6; ++k) bounds[t][k] = k < 3 ? 0x7fffffff : (int)0x80000000;
            __syncthreads();
            if ((t & 31) == 0)
                for (int k = 0; k < 3; ++k) {
                    atomicMin(&bounds[seg][k], b[k]);
                    atomicMax(&bounds[seg][3 + k], b[3 + k]);
                }
            __syncthreads();
            for (int k = 0; k < 6; ++k) b[k] = bounds[seg][k];
            __syncthreads();
        }
        float lo, ext;
        const int a = longest_axis(b, lo, ext);
        // ascending bitonic sort of the segment: coordinate, then place
        unsigned long long key =
            (unsigned long long)(on ? (unsigned)ordered_int(cen[a][t]) ^ 0x80000000u : 0xffffffffu) << 32 | (unsigned)t;
        for (int k = 2; k <= cap; k <<= 1)
            for (int j = k >> 1; j > 0; j >>= 1) {
                unsigned long long other;
                if (j >= 32) {
                    buf[t] = key;
                    __syncthreads();
                    other = buf[t ^ j];
                    __syncthreads();
                } else {
                    other = __shfl_xor_sync(FULL, key, j);
                }
                const bool up = ((t & (cap - 1)) & k) == 0, first = (t & j) == 0;
                if ((key > other) == (up == first)) key = other;
            }
        const int from = (int)(unsigned)key;
        const float x = cen[0][from], y = cen[1][from], z = cen[2][from];
        const int id = ids[from];
        __syncthreads();
        cen[0][t] = x;
        cen[1][t] = y;
        cen[2][t] = z;
        ids[t] = id;
        __syncthreads();
    }
    if (on) ord[p] = ids[t];
}

// Eigenvectors of a symmetric 3 x 3 matrix by cyclic Jacobi rotations: on
// return the columns of v are orthonormal to float accuracy and a is (nearly)
// diagonal, a[k][k] the eigenvalue of column k.
__device__ void sym3_eigen(float a[3][3], float v[3][3]) {
    for (int r = 0; r < 3; ++r)
        for (int c = 0; c < 3; ++c) v[r][c] = r == c ? 1.0f : 0.0f;
    for (int sweep = 0; sweep < 8; ++sweep) {
        const float off = a[0][1] * a[0][1] + a[0][2] * a[0][2] + a[1][2] * a[1][2];
        const float dia = a[0][0] * a[0][0] + a[1][1] * a[1][1] + a[2][2] * a[2][2];
        if (!(off > 1e-14f * dia)) break;
        for (int p = 0; p < 2; ++p) {
            for (int q = p + 1; q < 3; ++q) {
                if (a[p][q] == 0.0f) continue;
                // rotation in the (p, q) plane that zeroes a[p][q]: A <- J^T A J
                const float th = (a[q][q] - a[p][p]) / (2.0f * a[p][q]);
                const float t = (th >= 0.0f ? 1.0f : -1.0f) / (fabsf(th) + sqrtf(th * th + 1.0f));
                const float c = 1.0f / sqrtf(t * t + 1.0f), s = t * c;
                for (int k = 0; k < 3; ++k) {
                    const float akp = a[k][p], akq = a[k][q];
                    a[k][p] = c * akp - s * akq;
                    a[k][q] = s * akp + c * akq;
                }
                for (int k = 0; k < 3; ++k) {
                    const float apk = a[p][k], aqk = a[q][k];
                    a[p][k] = c * apk - s * aqk;
                    a[q][k] = s * apk + c * aqk;
                }
                for (int k = 0; k < 3; ++k) {
                    const float vkp = v[k][p], vkq = v[k][q];
                    v[k][p] = c * vkp - s * vkq;
                    v[k][q] = s * vkp + c * vkq;
                }
            }
        }
    }
}

// Sum / minimum / maximum of x over the TPN threads of one node (1, a warp or
// the block); every thread gets the result.
template <int TPN, class Op>
__device__ __forceinline__ float node_reduce(float x, Op op, float *red) {
    if constexpr (TPN > 1) {
        for (int o = 16; o > 0; o >>= 1) x = op(x, __shfl_xor_sync(0xffffffffu, x, o));
    }
    if constexpr (TPN > 32) {
        __syncthreads();
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = x;
        __syncthreads();
        x = red[threadIdx.x & 31];
        for (int o = 16; o > 0; o >>= 1) x = op(x, __shfl_xor_sync(0xffffffffu, x, o));
    }
    return x;
}

// Vertices, relative to o, of the primitive at the tree's position s as the
// distance code sees them: a and a + d of a segment; a, a + ab and a + ac of a
// triangle.
template <int D>
__device__ __forceinline__ void prim_vertices(const float4 *prims, int s, const float *o, float y[3][3]) {
    const float4 *b = prims + (size_t)(s / Tree<D>::LEAF) * Tree<D>::LEAF_W;
    const int i = s % Tree<D>::LEAF;
    if (D == 2) {
        const float4 g = b[i];
        y[0][0] = g.x - o[0];
        y[0][1] = g.y - o[1];
        y[1][0] = y[0][0] + g.z;
        y[1][1] = y[0][1] + g.w;
    } else {
        const float4 a = b[3 * i], ab = b[3 * i + 1], ac = b[3 * i + 2];
        const float p[3] = {a.x, a.y, a.z}, e[3] = {ab.x, ab.y, ab.z}, f[3] = {ac.x, ac.y, ac.z};
        for (int k = 0; k < 3; ++k) {
            y[0][k] = p[k] - o[k];
            y[1][k] = y[0][k] + e[k];
            y[2][k] = y[0][k] + f[k];
        }
    }
}

// Bound of a node of `np` primitives from position s0, by TPN threads, all of
// which call.  The axes are the principal axes of the vertices, eigenvectors of
// their covariance, made orthonormal, shrunk a little and rounded (2D: to float,
// 3D: to multiples of 2^-15) so that the rounded axes -- with the third 3D axis
// evaluated in float exactly as the query does (obb_axis2) -- form a matrix of
// norm at most 1.  The centre is the middle of the projections on the axes.  The
// extents bound the vertices about the rounded centre along the rounded axes,
// widened by 4e-6 of the node's diameter d.  That covers the query's float
// rounding of q - c and of the products with it (relative 2^-22 of |q - c| <=
// |q - y| + |y - c|: 1e-6 d for the latter) and the float evaluation here:
// vertices relative to the node's first one (2 x 2^-24 of at most 2 d each),
// their products with the axes (3.1e-7 d) and the centre's (3.7e-7 d), in all
// 2.2e-6 d.
//   2D: out = (u0, c, e0, e1).
//   3D: out = (c, u0, u1, e) with the axes in units of 2^-15.
template <int D, int TPN>
__device__ __forceinline__ void node_bound(const float4 *prims, int s0, int np, int t, float *red, float *out) {
    constexpr int NV = D == 2 ? 2 : 3;
    auto add = [](float a, float b) { return a + b; };
    auto lower = [](float a, float b) { return fminf(a, b); };
    auto upper = [](float a, float b) { return fmaxf(a, b); };
    // moments about the first vertex
    float y0[3] = {0.0f, 0.0f, 0.0f}, y[3][3], m[3] = {0.0f, 0.0f, 0.0f};
    float cv[6] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    prim_vertices<D>(prims, s0, y0, y);
    for (int k = 0; k < D; ++k) y0[k] = y[0][k];
    for (int i = t; i < np; i += TPN) {
        prim_vertices<D>(prims, s0 + i, y0, y);
        for (int j = 0; j < NV; ++j) {
            const float *w = y[j];
            for (int k = 0; k < D; ++k) m[k] += w[k];
            cv[0] = fmaf(w[0], w[0], cv[0]);
            cv[1] = fmaf(w[0], w[1], cv[1]);
            cv[3] = fmaf(w[1], w[1], cv[3]);
            if (D == 3) {
                cv[2] = fmaf(w[0], w[2], cv[2]);
                cv[4] = fmaf(w[1], w[2], cv[4]);
                cv[5] = fmaf(w[2], w[2], cv[5]);
            }
        }
    }
    const float n = (float)np * NV;
    for (int k = 0; k < D; ++k) m[k] = node_reduce<TPN>(m[k], add, red) / n;
    for (int k = 0; k < 6; ++k)
        if (D == 3 || k < 2 || k == 3) cv[k] = node_reduce<TPN>(cv[k], add, red) / n;
    cv[0] -= m[0] * m[0];
    cv[1] -= m[0] * m[1];
    cv[3] -= m[1] * m[1];
    // orthogonal axes u[0], u[1] (and u[2]: the normal)
    // 3D: rounding moves an axis by up to 2.7e-5 and two axes' product by 5.3e-5
    const double shrink = D == 2 ? 1.0 - 0x1p-20 : (1.0 - 6e-5) * 32768.0;
    const float unit[3] = {D == 2 ? 1.0f : 0x1p-15f, D == 2 ? 1.0f : 0x1p-15f, 0x1p-30f};  // of u[k]
    float u[3][3];
    if (D == 2) {
        double th = 0.5 * atan2(2.0 * (double)cv[1], (double)cv[0] - (double)cv[3]);
        if (!(fabs(th) <= 2.0)) th = 0.0;  // overflow of the moments: any axes do
        u[0][0] = (float)(cos(th) * shrink);
        u[0][1] = (float)(sin(th) * shrink);
        u[1][0] = -u[0][1];
        u[1][1] = u[0][0];
    } else {
        cv[2] -= m[0] * m[2];
        cv[4] -= m[1] * m[2];
        cv[5] -= m[2] * m[2];
        // scaled so that squares of tiny nodes' entries stay normal floats; the
        // coordinate axes where the moments leave the range of float
        const float tr = cv[0] + cv[3] + cv[5];
        const bool scaled = tr > 1e-36f && tr < INFINITY;
        float A[3][3] = {{0.0f, 0.0f, 0.0f}, {0.0f, 0.0f, 0.0f}, {0.0f, 0.0f, 0.0f}};
        if (scaled) {
            const float sc = 1.0f / tr;
            A[0][0] = cv[0] * sc;
            A[1][1] = cv[3] * sc;
            A[2][2] = cv[5] * sc;
            A[0][1] = A[1][0] = cv[1] * sc;
            A[0][2] = A[2][0] = cv[2] * sc;
            A[1][2] = A[2][1] = cv[4] * sc;
        }
        float vec[3][3];
        sym3_eigen(A, vec);
        int o[3] = {0, 1, 2};  // by falling variance
        for (int a = 0; a < 2; ++a)
            for (int b = a + 1; b < 3; ++b)
                if (A[o[b]][o[b]] > A[o[a]][o[a]]) {
                    const int w = o[a];
                    o[a] = o[b];
                    o[b] = w;
                }
        double p[3], w[3], lp = 0.0, lw = 0.0, pw = 0.0;
        for (int k = 0; k < 3; ++k) lp += (double)vec[k][o[0]] * vec[k][o[0]];
        lp = 1.0 / sqrt(lp);
        for (int k = 0; k < 3; ++k) {
            p[k] = vec[k][o[0]] * lp;
            pw += p[k] * vec[k][o[1]];
        }
        for (int k = 0; k < 3; ++k) {
            w[k] = vec[k][o[1]] - pw * p[k];
            lw += w[k] * w[k];
        }
        lw = shrink / sqrt(lw);
        for (int k = 0; k < 3; ++k) {
            u[0][k] = (float)rint(p[k] * shrink);
            u[1][k] = (float)rint(w[k] * lw);
        }
        obb_axis2(u[0], u[1], u[2]);
    }
    // ranges of u_k.(y - y0), and the centre in the middle of them
    float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    for (int i = t; i < np; i += TPN) {
        prim_vertices<D>(prims, s0 + i, y0, y);
        for (int j = 0; j < NV; ++j)
            for (int k = 0; k < D; ++k) {
                const float p = D == 2 ? dot2(u[k][0], u[k][1], y[j][0], y[j][1])
                                       : dot3(u[k][0], u[k][1], u[k][2], y[j][0], y[j][1], y[j][2]) * unit[k];
                lo[k] = fminf(lo[k], p);
                hi[k] = fmaxf(hi[k], p);
            }
    }
    float d2 = 0.0f;
    for (int k = 0; k < D; ++k) {
        lo[k] = node_reduce<TPN>(lo[k], lower, red);
        hi[k] = node_reduce<TPN>(hi[k], upper, red);
        d2 = fmaf(hi[k] - lo[k], hi[k] - lo[k], d2);
    }
    float cf[3], ef[3], w[3];
    for (int c = 0; c < D; ++c) {
        float x = 0.0f;
        for (int k = 0; k < D; ++k) x = fmaf(0.5f * (lo[k] + hi[k]) * unit[k], u[k][c], x);
        cf[c] = y0[c] + x;
        w[c] = cf[c] - y0[c];
    }
    // the axes are orthonormal to 3e-4, so the diameter is at most this
    const float pad = 4.01e-6f * sqrtf(d2);
    for (int k = 0; k < D; ++k) {
        const float off =
            D == 2 ? dot2(u[k][0], u[k][1], w[0], w[1]) : dot3(u[k][0], u[k][1], u[k][2], w[0], w[1], w[2]) * unit[k];
        ef[k] = __fadd_ru(fmaxf(hi[k] - off, off - lo[k]), pad);
    }
    if (D == 2) {
        out[0] = u[0][0];
        out[1] = u[0][1];
        out[2] = cf[0];
        out[3] = cf[1];
        out[4] = ef[0];
        out[5] = ef[1];
    } else {
        auto pair = [](float lo16, float hi16) {
            return __uint_as_float((unsigned)((int)lo16 + 32768) | (unsigned)((int)hi16 + 32768) << 16);
        };
        // the upper half of a float not below x > 0
        auto up = [](float x) { return (__float_as_uint(x) + 0xffffu) >> 16; };
        for (int k = 0; k < 3; ++k) out[k] = cf[k];
        out[3] = pair(u[0][0], u[0][1]);
        out[4] = pair(u[0][2], u[1][0]);
        out[5] = pair(u[1][1], u[1][2]);
        out[6] = __uint_as_float(up(ef[0]) | up(ef[1]) << 16);
        out[7] = ef[2];
    }
}

// Store the bound of node i of depth `depth` in its parent's block.
template <int D>
__device__ __forceinline__ void write_bound(float4 *tree, int depth, int i, const float *o) {
    float4 *b = tree + (size_t)tree_block(depth - 1, (unsigned)i >> 2) * Tree<D>::NODE_W;
    const int c = i & 3;
    if (D == 2) {
        b[c] = make_float4(o[0], o[1], o[2], o[3]);
        reinterpret_cast<float2 *>(b + 4)[c] = make_float2(o[4], o[5]);
    } else {
        b[2 * c] = make_float4(o[0], o[1], o[2], o[3]);
        b[2 * c + 1] = make_float4(o[4], o[5], o[6], o[7]);
    }
}

// Bounds of the tree's nodes.  A node of up to TREE_LANE_PRIMS primitives takes a
// thread, of up to TREE_WARP_PRIMS a warp, a larger one a block; the large ones
// (k_tree_bounds with LARGE) are few and each long, so their blocks are big.
constexpr int TREE_THREADS = 256, TREE_LARGE_THREADS = 1024;
constexpr int TREE_LANE_PRIMS = 16, TREE_WARP_PRIMS = 512;
struct TreePlan {
    int depth, nF;
    int first[TREE_MAX_DEPTH + 2];  // first block of depth d's nodes, d = d0..d1; [d1 + 1]: blocks in all
    int count[TREE_MAX_DEPTH + 1];  // nodes of depth d
    int d0, d1;
};
__host__ __device__ inline long long node_prims(int leaf, int height) { return (long long)leaf << (2 * height); }
__host__ __device__ inline int nodes_per_block(long long prims) {
    return prims <= TREE_LANE_PRIMS ? TREE_THREADS : prims <= TREE_WARP_PRIMS ? TREE_THREADS / 32 : 1;
}

// Area of a node's box (an eighth of its surface) and of np triangles from position s0
// (twice theirs), lengths times inv.
__device__ __forceinline__ float box_area(const float *o, float inv) {
    const unsigned e01 = __float_as_uint(o[6]);
    const float e0 = __uint_as_float(e01 << 16) * inv, e1 = __uint_as_float(e01 & 0xffff0000u) * inv, e2 = o[7] * inv;
    return fmaf(e0, e1, fmaf(e0, e2, e1 * e2));
}
__device__ __forceinline__ float triangle_area(const float4 *prims, int s0, int np, float inv) {
    float a = 0.0f;
    for (int s = s0; s < s0 + np; ++s) {
        const float4 *b = prims + (size_t)(s / Tree<3>::LEAF) * Tree<3>::LEAF_W + 3 * (s % Tree<3>::LEAF);
        const float4 ab = b[1], ac = b[2];
        float n[3];
        cross3(ab.x * inv, ab.y * inv, ab.z * inv, ac.x * inv, ac.y * inv, ac.z * inv, n[0], n[1], n[2]);
        a += sqrtf(dot3(n[0], n[1], n[2], n[0], n[1], n[2]));
    }
    return a;
}

// cost (3D): adds the areas of all boxes to [0] and of all triangles to [1], in units of
// the scene's largest extent (of its box, lohi).
template <int D, bool LARGE>
__global__ void __launch_bounds__(LARGE ? TREE_LARGE_THREADS : TREE_THREADS) k_tree_bounds(
    TreePlan P, const float4 *prims, float4 *tree, const int *lohi, float *cost) {
    __shared__ float red[32];
    int d = P.d0;
    while (d < P.d1 && (int)blockIdx.x >= P.first[d + 1]) ++d;
    const long long cap = node_prims(Tree<D>::LEAF, P.depth - d);
    const int per = nodes_per_block(cap), base = ((int)blockIdx.x - P.first[d]) * per;
    const int i = base + (LARGE ? 0 : per == TREE_THREADS ? (int)threadIdx.x : (int)threadIdx.x >> 5);
    const bool there = i < P.count[d];
    // a node beyond the last still takes part in its warp's reductions
    const long long s0 = (there ? i : P.count[d] - 1) * cap;
    const int np = (int)min(cap, (long long)P.nF - s0);
    float o[8];
    bool writer = there;
    if (LARGE) {
        node_bound<D, TREE_LARGE_THREADS>(prims, (int)s0, np, threadIdx.x, red, o);
        writer = writer && threadIdx.x == 0;
    } else if (per == TREE_THREADS) {
        node_bound<D, 1>(prims, (int)s0, np, 0, red, o);
    } else {
        node_bound<D, 32>(prims, (int)s0, np, threadIdx.x & 31, red, o);
        writer = writer && (threadIdx.x & 31) == 0;
    }
    if (D == 3) {
        float ext = 0.0f, area[2] = {0.0f, 0.0f};
        for (int k = 0; k < 3; ++k) ext = fmaxf(ext, from_ordered_int(lohi[3 + k]) - from_ordered_int(lohi[k]));
        const float inv = ext > 0.0f ? 1.0f / ext : 0.0f;
        if (writer) {
            area[0] = box_area(o, inv);
            if (d == P.depth) area[1] = triangle_area(prims, (int)s0, np, inv);
        }
        for (int k = 0; k < 2; ++k) {
            if (!(area[k] < INFINITY)) area[k] = 0.0f;  // vertices that are not finite
            for (int x = 16; x > 0; x >>= 1) area[k] += __shfl_xor_sync(0xffffffffu, area[k], x);
            if ((threadIdx.x & 31) == 0 && area[k] != 0.0f) atomicAdd(&cost[k], area[k]);
        }
    }
    if (!writer) return;
    write_bound<D>(tree, d, i, o);
    if (i == P.count[d] - 1) {
        // the last node also fills its parent's block with infinitely far children
        float far[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
        if (D == 2)
            far[4] = -INFINITY;
        else
            far[6] = __uint_as_float(0xff800000u >> 16);  // e0 = -inf
        for (int k = i + 1; (k & 3) != 0; ++k) write_bound<D>(tree, d, k, far);
    }
}

// ------------------------------------------------------------------ host
static inline int nblk(long long n, int b) { return (int)((n + b - 1) / b); }

// How much farther than a triangle's closest point the one that tri_closest finds may
// be, for query points up to R from the triangle's vertex a.  Its barycentric
// coordinates are quotients of differences of products: with A = |ab|, B = |ac|, s the
// sine between them and M = R + A + B, the products are below A B M^2 and carry up to
// 16 x 2^-24 of that (and a few steps of the denormal floats), the quotients' denominator
// is A^2 B^2 s^2, and the coordinates move the point along ab and ac.  A region taken
// for its neighbour moves it by no more, and twice that is allowed for; the point always
// lies on the triangle.  2e-6 of an edge for an even triangle near by, more than its
// length for a needle of aspect 1e-4, whose coordinates are noise.  (96 million random
// triangles and points, aspects 1 to 1e-7: at most 0.011 of this, never off the triangle.)
// -1 where there is no telling: the products overflow, or their sum, that denominator, is
// so small that its reciprocal does, and the distance may be NaN at some points.
__device__ __forceinline__ float closest_error(float4 t1, float4 t2, float ab2, float R) {
    const float A = sqrtf(ab2), B = sqrtf(t2.w), M = R + A + B, m = A * B * M * M;
    const float p = ab2 * t2.w, det = p - t1.w * t1.w;
    if (!(m < 1e37f && (p > 1e-24f || (det > 1e-36f && det > 1e-5f * p)))) return -1.0f;
    return det > 0.0f ? 0x1p-19f * m * (A + B) / det : INFINITY;
}

// Upper bound of the computed distance to the nearest of a leaf's primitives from any
// point within h of x, less h; infinite where none is known.  2D: the computed distance
// at x, as distances to a segment are exact to search_bound's slack.  3D: a triangle's is
// that at x and the error above, or the distance to its farthest vertex.
template <int D>
__device__ __forceinline__ float leaf_reach(const SceneView &S, unsigned leaf, const float *x, float h) {
    constexpr int N = Tree<D>::LEAF;
    float d2[N], u = INFINITY;
    leaf_distances<D>(S, leaf, x, d2);
    if constexpr (D == 2) {
        for (int c = 0; c < N; ++c) u = fminf(u, d2[c]);
        return sqrtf(u);
    } else {
        const float4 *b = S.prims + (size_t)leaf * Tree<3>::LEAF_W;
        for (int c = 0; c < N; ++c) {
            const float4 t0 = b[3 * c], t1 = b[3 * c + 1], t2 = b[3 * c + 2];
            const float v[3] = {x[0] - t0.x, x[1] - t0.y, x[2] - t0.z};
            const float b0 = v[0] - t1.x, b1 = v[1] - t1.y, b2 = v[2] - t1.z;
            const float c0 = v[0] - t2.x, c1 = v[1] - t2.y, c2 = v[2] - t2.z;
            const float ra = dot3(v[0], v[1], v[2], v[0], v[1], v[2]);
            const float far = fmaxf(ra, fmaxf(dot3(b0, b1, b2, b0, b1, b2), dot3(c0, c1, c2, c0, c1, c2)));
            const float e = closest_error(t1, t2, t0.w, sqrtf(ra) + h);
            if (e >= 0.0f && d2[c] < INFINITY) u = fminf(u, fminf(sqrtf(d2[c]) + e, sqrtf(far)));
        }
        return u;
    }
}

// Entry grid of the search tree (SceneView::grid), a thread per cell.  U + h (leaf_reach),
// for the leaf found by going to the nearest child at each depth from the cell's centre x
// and h the cell's half diagonal, bounds the computed distance from every point q of the
// cell to its nearest primitive, so all its nearest primitives lie within U + 2 h of x:
// nodes farther than that are left out.  Distances take search_bound's slack wherever a
// computed one stands for a true one or the reverse; h that of the rounding of a point's
// cell and of x.  The cell's nodes are the root's children, replaced by their own children
// as long as four are enough.  The cell of the points outside has the root's children.
// (At most 128 registers: 56 us for the 32^3 cells of 81,920 triangles, 65 without the bound.)
template <int D>
__global__ void __launch_bounds__(128, 4) k_entry_grid(SceneView S, const int *lohi, uint4 *node, float4 *box) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x, bits = S.grid_bits, G = 1 << bits;
    const int cells = 1 << (D * bits);
    if (i > cells) return;
    float lo[3] = {0.0f, 0.0f, 0.0f}, ext[3], ext_max = 0.0f, abs_max = 0.0f, x[3];
    for (int k = 0; k < D; ++k) {
        lo[k] = from_ordered_int(lohi[k]);
        const float hi = from_ordered_int(lohi[3 + k]);
        ext[k] = hi - lo[k];
        ext_max = fmaxf(ext_max, ext[k]);
        abs_max = fmaxf(abs_max, fmaxf(fabsf(lo[k]), fabsf(hi)));
    }
    const float unit = fmaxf(ext_max, FLT_MIN);
    float h2 = 0.0f, inv[3] = {0.0f, 0.0f, 0.0f};
    for (int k = 0; k < D; ++k) {
        ext[k] = fmaxf(ext[k], ext_max * 0x1p-20f);  // flat
        const float cell = ext[k] / (float)G;
        inv[k] = (float)G / ext[k];
        x[k] = lo[k] + ((float)(i >> (k * bits) & (G - 1)) + 0.5f) * cell;
        h2 = fmaf(cell / unit, cell / unit, h2);
    }
    const float h = 0.5005f * sqrtf(h2) * unit + 1e-6f * ext_max + 1e-6f * abs_max + TOL_MIN;
    const float e = (1.0f + 0.5f * D) * 0x1.02p-20f * ext_max + TOL_MIN;  // prune_tol's largest in the box
    auto widen = [&](float d) { return sqrtf(search_bound<D>((d * d) * (1.0f + 0x1p-20f), search_tol<D>(e))); };

    auto distances = [&](unsigned block, float *dd) {
        block_distances<D>(S.tree + (size_t)block * Tree<D>::NODE_W, x, dd);
    };
    // A vertex that is not finite, or an extent that overflows, leaves no centre to
    // descend from (children that do not exist are infinitely far from finite points
    // only): such a cell has the root's children.
    bool finite = true;
    for (int k = 0; k < D; ++k) finite = finite && fabsf(x[k]) <= FLT_MAX;
    for (int k = 0; k < D; ++k) x[k] = finite ? x[k] : 0.0f;
    float d[4];
    unsigned idx = 0;
    for (int dep = 0; dep < S.tree_depth; ++dep) {
        distances(tree_block(dep, idx), d);
        int near = 0;
        for (int c = 1; c < 4; ++c)
            if (d[c] < d[near]) near = c;
        idx = 4u * idx + near;
    }
    const float r = h + widen(widen(widen(leaf_reach<D>(S, idx, x, h)) + h));
    const float r2 = finite ? (r * r) * (1.0f + 0x1p-20f) : INFINITY;

    unsigned n[4] = {0u, 1u, 2u, 3u};
    int count = 4;
    if (r2 <= FLT_MAX && i < cells) {
        auto drop = [&](const float *dd, unsigned first, unsigned *out, int at) {
            for (int c = 0; c < 4; ++c)
                if (dd[c] <= r2) {
                    if (at < 4) out[at] = first + c;
                    ++at;
                }
            return at;
        };
        distances(0u, d);
        count = drop(d, 0u, n, 0);
        for (bool more = true; more;) {
            for (int c = count; c < 4; ++c) n[c] = GRID_NONE;
            sort4(n);  // the highest nodes first
            more = false;
            for (int c = 0; c < count && !more; ++c) {
                int dep;
                unsigned j, kids[4];
                tree_place(n[c], dep, j);
                if (dep == S.tree_depth) break;
                distances(tree_block(dep, j), d);
                const int nk = drop(d, tree_node(dep + 1, 4u * j), kids, 0);
                if (count - 1 + nk > 4) continue;
                n[c] = n[--count];
                for (int k = 0; k < nk; ++k) n[count++] = kids[k];
                more = true;
            }
        }
    }
    for (int c = count; c < 4; ++c) n[c] = GRID_NONE;
    node[i] = make_uint4(n[0], n[1], n[2], n[3]);
    float4 *b = box + (size_t)i * Tree<D>::NODE_W;
    for (int c = 0; c < 4; ++c) {
        const float4 *from = S.tree + (size_t)(n[c] >> 2) * Tree<D>::NODE_W;
        const int k = n[c] & 3;
        const bool is = n[c] != GRID_NONE;
        if (D == 2) {
            b[c] = is ? from[k] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            reinterpret_cast<float2 *>(b + 4)[c] =
                is ? reinterpret_cast<const float2 *>(from + 4)[k] : make_float2(-INFINITY, 0.0f);
        } else {
            b[2 * c] = is ? from[2 * k] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            b[2 * c + 1] =
                is ? from[2 * k + 1] : make_float4(0.0f, 0.0f, __uint_as_float(0xff800000u >> 16), 0.0f);
        }
    }
    if (i == 0) {
        float4 *head = reinterpret_cast<float4 *>(node) - 2;
        head[0] = make_float4(lo[0], lo[1], lo[2], 0.0f);
        head[1] = make_float4(inv[0], inv[1], inv[2], 0.0f);
    }
}
// Cells per axis, as a power of two: 16 cells per primitive up to 128^2 (1.8 MB:
// 112 bytes each) or 32^3 (4.7 MB: 144 bytes each).  Finer cells save node steps
// -- 2D, 4,096 segments: 5.9 per query without a grid, 3.2, 2.8, 2.3 with 64, 128,
// 256 cells per axis; 3D, 20,480 triangles: 14.2 without, 11.4, 9.9, 8.3 with 16,
// 32, 64 -- but take memory and time to build.  256^2 against 128^2: the 2D
// gradient of 80,222 x 256 walks on 4,096 segments 98.8 and 100.8 ms; 64^3 against
// 32^3: the 3D solve of 20,000 x 64 on 20,480 triangles 8.3 and 8.9 ms, but a
// moved mesh of 81,920 and 10,007 closest points on it 0.95 and 0.81 ms.
static int entry_grid_bits(int dim, int nF) {
    int bits = 1;
    while (bits < (dim == 2 ? 7 : 5) && (1LL << (dim * bits)) < 16LL * nF) ++bits;
    return bits;
}

template <typename T>
static cudaError_t dalloc(T **p, size_t count, cudaStream_t st) {
    if (count == 0) count = 1;
    return cudaMallocAsync((void **)p, count * sizeof(T), st);
}

void SceneImpl::release(cudaStream_t st) {
    void *ptrs[] = {V, F, N, g, seg, seginv, tri, node, lseg, lseginv, ltri, lorig, cdf, tree, prims, torig, vslot, vfirst, grid, guide};
    for (void *p : ptrs)
        if (p) cudaFreeAsync(p, st);
    V = nullptr;
    F = nullptr;
    N = nullptr;
    g = nullptr;
    seg = nullptr;
    seginv = nullptr;
    tri = nullptr;
    node = nullptr;
    lseg = nullptr;
    lseginv = nullptr;
    ltri = nullptr;
    lorig = nullptr;
    cdf = nullptr;
    tree = nullptr;
    prims = nullptr;
    torig = nullptr;
    vslot = nullptr;
    grid = nullptr;
    vfirst = nullptr;
    tree_ordered = false;
    guide = nullptr;
}

// Normalised CDF of pmf_i ~ r_i log(1/r_i), r_i = (i + 0.5)/n, built in
// double on the host (include/tabulated_G_cdf.cuh:5-8 regenerated from its
// formula, wos/wos_with_source.py:17-23).
void build_g_cdf(std::vector<float> &cdf, int n) {
    std::vector<double> pmf(n);
    double total = 0.0;
    for (int i = 0; i < n; ++i) {
        const double r = (i + 0.5) / n;
        pmf[i] = r * std::log(1.0 / r) / (2.0 * 3.14159265358979323846);
        total += pmf[i];
    }
    cdf.resize(n);
    double acc = 0.0;
    for (int i = 0; i < n; ++i) {
        acc += pmf[i];
        cdf[i] = (float)(acc / total);
    }
    cdf[n - 1] = 1.0f;
}

void build_g_guide(const std::vector<float> &cdf, int ng, std::vector<unsigned short> &guide) {
    const int n = (int)cdf.size();
    guide.resize(ng + 1);
    int l = 0;
    for (int k = 0; k <= ng; ++k) {
        const float u = (float)k / (float)ng;
        while (l < n - 1 && !(u < cdf[l])) ++l;
        guide[k] = (unsigned short)l;
    }
}

// Temporaries: one allocation, carved up; freed on the stream when its scope is left.
struct Arena {
    cudaStream_t st = nullptr;
    char *base = nullptr;
    size_t used = 0;
    explicit Arena(cudaStream_t s) : st(s) {}
    Arena(const Arena &) = delete;
    ~Arena() {
        if (base) cudaFreeAsync(base, st);
    }
    template <typename T>
    T *take(size_t n) {
        T *p = reinterpret_cast<T *>(base + used);
        used += (std::max<size_t>(n, 1) * sizeof(T) + 255) & ~(size_t)255;
        return p;
    }
};

__global__ void k_key_order(const unsigned long long *keys, int n, int *ord) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) ord[i] = (int)(unsigned)keys[i];
}

// S.torig: the median-split order of the triangles, from the boxes pbox; starts
// from the sorted keys' order, which only settles ties.
static int median_order(SceneImpl &S, const float *pbox, const unsigned long long *skeys, cudaStream_t st) {
    const int nF = S.nF, TB = 256;
    k_key_order<<<nblk(nF, TB), TB, 0, st>>>(skeys, nF, S.torig);
    long long cap = SPLIT_SMALL;
    while (cap < nF) cap *= 2;
    if (cap > SPLIT_SMALL) {
        const int max_seg = nblk(nF, 2 * SPLIT_SMALL);
        // at most 2^20 segments, as nF is an int
        int seg_bits = 0;
        while ((1LL << seg_bits) < max_seg) ++seg_bits;
        const int bits = std::min(16, 32 - seg_bits);
        int *bounds = nullptr, *ord2 = nullptr;
        unsigned *keys = nullptr, *keys2 = nullptr;
        size_t tmp_bytes = 0;
        cub::DeviceRadixSort::SortPairs(nullptr, tmp_bytes, keys, keys2, S.torig, ord2, nF, 0, bits + seg_bits, st);
        void *tmp = nullptr;
        Arena A(st);
        for (int pass = 0; pass < 2; ++pass) {  // sizes, then the buffers
            A.used = 0;
            bounds = A.take<int>((size_t)6 * max_seg);
            ord2 = A.take<int>(nF);
            keys = A.take<unsigned>(nF);
            keys2 = A.take<unsigned>(nF);
            tmp = A.take<char>(tmp_bytes);
            if (pass == 0) WOS_TRY(cudaMallocAsync((void **)&A.base, A.used, st));
        }
        int *cur = S.torig, *alt = ord2;
        for (; cap > SPLIT_SMALL; cap /= 2) {
            const int n_seg = nblk(nF, (int)std::min<long long>(cap, 1LL << 30));
            k_split_init<<<nblk(6 * n_seg, TB), TB, 0, st>>>(bounds, 6 * n_seg);
            const int c = (int)std::min<long long>(cap, 1LL << 30);
            k_split_bounds<<<nblk(nF, TB), TB, 0, st>>>(pbox, cur, nF, c, bounds);
            k_split_keys<<<nblk(nF, TB), TB, 0, st>>>(pbox, cur, nF, c, bits, bounds, keys);
            int used = bits;
            while ((1LL << (used - bits)) < n_seg) ++used;
            WOS_TRY(cub::DeviceRadixSort::SortPairs(tmp, tmp_bytes, keys, keys2, cur, alt, nF, 0, used, st));
            std::swap(cur, alt);
        }
        if (cur != S.torig)
            WOS_TRY(cudaMemcpyAsync(S.torig, cur, sizeof(int) * nF, cudaMemcpyDeviceToDevice, st));
    }
    k_split_small<<<nblk(nF, SPLIT_SMALL), SPLIT_SMALL, 0, st>>>(pbox, nF, Tree<3>::LEAF, S.torig);
    WOS_TRY(cudaGetLastError());
    return 0;
}

// Whether a mesh has moved too far for the order of its triangles: the areas of the
// tree's boxes have grown by a third since the order was made, in units of the scene's
// extent or of the triangles' own area, or that area is another one altogether (the
// scene was made from vertices that only held a place: flat, collapsed, shuffled).
//   Search steps of the kept order over those of a new one, and the boxes' growth:
// 20,480 loose triangles on a unit sphere displaced by up to 0.02, 0.05, 0.1, 0.5 take
// 1.05, 1.26, 1.77, 16.4 times the steps at 1.11, 1.53, 2.5, 15.4; 20,000 in a box by
// 0.1 2.15 at 1.6; a sphere twisted by 3 radians 2.5 at 1.75.  Spheres displaced by up
// to 15 or 40 % in waves, rotated, squashed or stretched: 0.84 to 1.01 at up to 1.11.
static bool order_worn(const float *then, const float *now) {
    return now[0] > 1.3f * then[0] || now[0] * then[1] > 1.3f * then[0] * now[1] || now[1] > 4.0f * then[1] ||
           now[1] < 0.25f * then[1];
}

// The Green's function tables, the same for every scene, computed once.
struct GTables {
    std::vector<float> cdf;
    std::vector<unsigned short> guide;
};
static const GTables &g_tables() {
    static const GTables t = [] {
        GTables x;
        build_g_cdf(x.cdf, 10000);
        build_g_guide(x.cdf, 2048, x.guide);
        return x;
    }();
    return t;
}

static int index_bits(long long n) {
    int b = 1;
    while (b < 32 && (1LL << b) < n) ++b;
    return b;
}

// Slots (face, corner) by vertex, in face order: vslot, and vfirst[v] the first
// of vertex v.  They depend on the faces alone, so once per scene.
static int build_vertex_slots(SceneImpl &S, cudaStream_t st) {
    const int n = S.nF * S.dim, TB = 256, bits = index_bits(S.nV);
    int *ids = nullptr, *verts = nullptr;
    size_t tmp_bytes = 0;
    WOS_TRY(dalloc(&S.vslot, n, st));
    WOS_TRY(dalloc(&S.vfirst, (size_t)S.nV + 1, st));
    cub::DeviceRadixSort::SortPairs(nullptr, tmp_bytes, S.F, verts, ids, S.vslot, n, 0, bits, st);
    void *tmp = nullptr;
    Arena A(st);
    for (int pass = 0; pass < 2; ++pass) {
        A.used = 0;
        ids = A.take<int>(n);
        verts = A.take<int>(n);
        tmp = A.take<char>(tmp_bytes);
        if (pass == 0) WOS_TRY(cudaMallocAsync((void **)&A.base, A.used, st));
    }
    k_iota<<<nblk(n, TB), TB, 0, st>>>(ids, n);
    WOS_TRY(cub::DeviceRadixSort::SortPairs(tmp, tmp_bytes, S.F, verts, ids, S.vslot, n, 0, bits, st));
    k_vertex_ranges<<<nblk((long long)S.nV + 1, TB), TB, 0, st>>>(verts, n, S.nV, S.vfirst);
    WOS_TRY(cudaGetLastError());
    return 0;
}

// The search tree of the primitives in the order torig (or that of `keys`), in the
// buffers of the first build (their sizes depend on nF alone): device views held
// elsewhere -- batch plans, captured graphs, launches on other streams -- keep pointing
// at live memory.
template <int D>
static int build_tree(SceneImpl &S, const unsigned long long *keys, int *counters, cudaStream_t st) {
    constexpr int N = Tree<D>::LEAF;
    const int nF = S.nF, TB = 256, n_leaf = (nF + N - 1) / N;
    TreePlan P{};
    P.depth = S.tree_depth;
    P.nF = nF;
    for (int d = 1; d <= P.depth; ++d) {
        const long long cap = node_prims(N, P.depth - d);
        P.count[d] = (int)((nF + cap - 1) / cap);
    }
    k_tree_prims<D><<<nblk((long long)n_leaf * N, TB), TB, 0, st>>>(nF, n_leaf, keys, S.seg, S.seginv, S.tri, S.prims,
                                                                S.torig);
    // the depths of large nodes, then the others
    int split = 1;
    while (split <= P.depth && node_prims(N, P.depth - split) > TREE_WARP_PRIMS) ++split;
    float *cost = reinterpret_cast<float *>(counters + 7);
    for (int part = 0; part < 2; ++part) {
        P.d0 = part == 0 ? 1 : split;
        P.d1 = part == 0 ? split - 1 : P.depth;
        int blocks = 0;
        for (int d = P.d0; d <= P.d1; ++d) {
            P.first[d] = blocks;
            blocks += nblk(P.count[d], nodes_per_block(node_prims(N, P.depth - d)));
        }
        if (blocks == 0) continue;
        P.first[P.d1 + 1] = blocks;
        if (part == 0)
            k_tree_bounds<D, true><<<blocks, TREE_LARGE_THREADS, 0, st>>>(P, S.prims, S.tree, counters, cost);
        else
            k_tree_bounds<D, false><<<blocks, TREE_THREADS, 0, st>>>(P, S.prims, S.tree, counters, cost);
    }
    const int cells = (1 << (D * S.grid_bits)) + 1;
    k_entry_grid<D><<<nblk(cells, 128), 128, 0, st>>>(S.view(), counters, S.grid_node(), S.grid_box());
    WOS_TRY(cudaGetLastError());
    return 0;
}

template <int D>
static int build_geometry(SceneImpl &S, cudaStream_t st) {
    const int nV = S.nV, nF = S.nF, nInt = nF - 1;
    const int TB = 256;
    if (S.vslot == nullptr)
        if (int rc = build_vertex_slots(S, st)) return rc;
    // Sorts are stable and start in index order, so keys sort by their upper
    // half alone: the Morton code or Hilbert index, and the node's depth.
    const int key_bits = D == 2 ? 32 : 30, depth_bits = 12;
    size_t tmp_bytes = 0, t2 = 0;
    unsigned long long *none = nullptr;
    if (S.prim_order != 1)
        cub::DeviceRadixSort::SortKeys(nullptr, tmp_bytes, none, none, nF, 32, 32 + key_bits, st);
    if (nInt > 0) cub::DeviceRadixSort::SortKeys(nullptr, t2, none, none, nInt, 32, 32 + depth_bits, st);
    tmp_bytes = std::max(tmp_bytes, t2);
    Arena A(st);
    int *counters = nullptr, *pint = nullptr, *pleaf = nullptr, *flags = nullptr, *new_of_old = nullptr;
    float *contrib = nullptr, *pbox = nullptr, *nbox = nullptr;
    unsigned long long *mkeys = nullptr, *skeys = nullptr, *dkeys = nullptr, *dkeys2 = nullptr;
    int2 *child = nullptr;
    void *tmp = nullptr;
    for (int pass = 0; pass < 2; ++pass) {  // sizes, then the buffers
        A.used = 0;
        counters = A.take<int>(BUILD_COUNTERS);
        contrib = A.take<float>((size_t)nF * D * D);
        pbox = A.take<float>((size_t)nF * 2 * D);
        mkeys = A.take<unsigned long long>(nF);
        skeys = S.prim_order == 1 ? mkeys : A.take<unsigned long long>(nF);
        tmp = A.take<char>(tmp_bytes);
        child = A.take<int2>(nInt);
        pint = A.take<int>(nInt);
        pleaf = A.take<int>(nF);
        flags = A.take<int>(nInt);
        new_of_old = A.take<int>(nInt);
        nbox = A.take<float>((size_t)nInt * 2 * D);
        dkeys = A.take<unsigned long long>(nInt);
        dkeys2 = A.take<unsigned long long>(nInt);
        if (pass == 0) WOS_TRY(cudaMallocAsync((void **)&A.base, A.used, st));
    }
    // ---- bounding box and vertex normals
    k_build_init<<<1, 32, 0, st>>>(counters);
    k_aabb<<<std::min(nblk(nV, TB), 1024), TB, 0, st>>>(S.V, nV, D, counters);
    k_face_normals<D><<<nblk(nF, TB), TB, 0, st>>>(S.V, S.F, nF, contrib);
    k_vertex_normals<D><<<nblk(nV, TB), TB, 0, st>>>(S.vslot, S.vfirst, contrib, nV, S.N);

    // ---- primitives and sort keys: a polyline whose segments follow each other
    // keeps its input order (its leaves are then arcs of the curve, the most
    // compact runs; the keys are sorted as they are); other polylines sort by
    // Morton code, meshes by Hilbert index
    k_prims<D><<<nblk(nF, TB), TB, 0, st>>>(S.V, S.F, nF, counters, S.seg, S.seginv, S.tri, pbox, mkeys, S.prim_order);
    if (S.prim_order != 1)
        WOS_TRY(cub::DeviceRadixSort::SortKeys(tmp, tmp_bytes, mkeys, skeys, nF, 32, 32 + key_bits, st));
    k_leaf_data<D><<<nblk(nF, TB), TB, 0, st>>>(skeys, nF, S.seg, S.seginv, S.tri, S.lseg, S.lseginv, S.ltri, S.lorig);

    // ---- search tree
    const bool new_order = D == 3 && !S.tree_ordered;
    if (new_order)
        if (int rc = median_order(S, pbox, skeys, st)) return rc;
    if (int rc = build_tree<D>(S, D == 2 ? skeys : nullptr, counters, st)) return rc;
    S.tree_ordered = true;

    // ---- hierarchy
    S.nNodes = nInt;
    if (nInt > 0) {
        WOS_TRY(cudaMemsetAsync(pint, 0xff, sizeof(int) * nInt, st));
        WOS_TRY(cudaMemsetAsync(pleaf, 0xff, sizeof(int) * nF, st));
        WOS_TRY(cudaMemsetAsync(flags, 0, sizeof(int) * nInt, st));
        k_karras<<<nblk(nInt, TB), TB, 0, st>>>(skeys, nF, child, pint, pleaf);
        k_refit<D><<<nblk(nF, TB), TB, 0, st>>>(skeys, nF, pbox, child, pint, pleaf, flags, nbox);
        k_depth<<<nblk(nInt, TB), TB, 0, st>>>(pint, nInt, dkeys, counters + 6);
        WOS_TRY(cub::DeviceRadixSort::SortKeys(tmp, tmp_bytes, dkeys, dkeys2, nInt, 32, 32 + depth_bits, st));
        k_bfs_rank<<<nblk(nInt, TB), TB, 0, st>>>(dkeys2, nInt, new_of_old);
        k_write_nodes<D><<<nblk(nInt, TB), TB, 0, st>>>(skeys, nInt, pbox, nbox, child, new_of_old, S.node);
    }
    WOS_TRY(cudaGetLastError());
    int host[BUILD_COUNTERS];
    WOS_TRY(cudaMemcpyAsync(host, counters, sizeof(host), cudaMemcpyDeviceToHost, st));
    WOS_TRY(cudaStreamSynchronize(st));
    float cost[2];
    memcpy(cost, host + 7, sizeof(cost));
    if (D == 3 && !new_order && order_worn(S.order_cost, cost)) {
        WOS_TRY(cudaMemsetAsync(counters + 7, 0, sizeof(cost), st));
        if (int rc = median_order(S, pbox, skeys, st)) return rc;
        if (int rc = build_tree<D>(S, nullptr, counters, st)) return rc;
        WOS_TRY(cudaMemcpyAsync(cost, counters + 7, sizeof(cost), cudaMemcpyDeviceToHost, st));
        WOS_TRY(cudaStreamSynchronize(st));
        memcpy(S.order_cost, cost, sizeof(cost));
    } else if (new_order) {
        memcpy(S.order_cost, cost, sizeof(cost));
    }
    auto from_ord = [](int i) {
        int b = i >= 0 ? i : i ^ 0x7fffffff;
        float f;
        memcpy(&f, &b, 4);
        return f;
    };
    for (int k = 0; k < 3; ++k) {
        S.lo[k] = k < D ? from_ord(host[k]) : 0.0f;
        S.hi[k] = k < D ? from_ord(host[3 + k]) : 0.0f;
    }
    float ext = INFINITY;
    for (int k = 0; k < D; ++k) ext = fminf(ext, fabsf(S.hi[k] - S.lo[k]));
    S.half_min_extent = ext * 0.5f;
    S.depth = host[6];
    return 0;
}

int SceneImpl::allocate(cudaStream_t st) {
    const int D = dim;
    WOS_TRY(dalloc(&V, (size_t)nV * D, st));
    WOS_TRY(dalloc(&F, (size_t)nF * D, st));
    WOS_TRY(dalloc(&N, (size_t)nV * D, st));
    WOS_TRY(dalloc(&g, nV, st));
    if (D == 2) {
        WOS_TRY(dalloc(&seg, nF, st));
        WOS_TRY(dalloc(&seginv, nF, st));
        WOS_TRY(dalloc(&lseg, nF, st));
        WOS_TRY(dalloc(&lseginv, nF, st));
        WOS_TRY(dalloc(&node, (size_t)std::max(nF - 1, 1) * 3, st));
    } else {
        WOS_TRY(dalloc(&tri, (size_t)nF * 3, st));
        WOS_TRY(dalloc(&ltri, (size_t)nF * 3, st));
        WOS_TRY(dalloc(&node, (size_t)std::max(nF - 1, 1) * 4, st));
    }
    const int N = D == 2 ? Tree<2>::LEAF : Tree<3>::LEAF;
    const long long n_leaf = ((long long)nF + N - 1) / N;
    WOS_TRY(dalloc(&lorig, nF, st));
    WOS_TRY(dalloc(&torig, (size_t)n_leaf * N, st));
    tree_depth = 1;
    while ((1LL << (2 * tree_depth)) < n_leaf) ++tree_depth;
    if (tree_depth > TREE_MAX_DEPTH) return fail(WOS_ERR_UNSUPPORTED, "scene too large for the search tree");
    // blocks: those of the depths above the leaves' parents, then the parents
    const size_t blocks = (size_t)tree_block(tree_depth - 1, 0) + (size_t)((n_leaf + 3) / 4);
    WOS_TRY(dalloc(&tree, blocks * (D == 2 ? Tree<2>::NODE_W : Tree<3>::NODE_W), st));
    WOS_TRY(dalloc(&prims, (size_t)n_leaf * (D == 2 ? Tree<2>::LEAF_W : Tree<3>::LEAF_W), st));
    grid_bits = entry_grid_bits(dim, nF);
    const size_t cells = ((size_t)1 << (dim * grid_bits)) + 1;
    WOS_TRY(dalloc(&grid, 2 + (cells + 1) + cells * (dim == 2 ? Tree<2>::NODE_W : Tree<3>::NODE_W), st));
    const GTables &tables = g_tables();
    const std::vector<float> &c = tables.cdf;
    const std::vector<unsigned short> &gd = tables.guide;
    n_cdf = (int)c.size();
    n_guide = (int)gd.size() - 1;
    WOS_TRY(dalloc(&cdf, c.size(), st));
    WOS_TRY(dalloc(&guide, gd.size(), st));
    WOS_TRY(cudaMemcpyAsync(cdf, c.data(), c.size() * sizeof(float), cudaMemcpyHostToDevice, st));
    WOS_TRY(cudaMemcpyAsync(guide, gd.data(), gd.size() * sizeof(unsigned short), cudaMemcpyHostToDevice, st));
    return 0;
}

// Checks the faces and decides the primitives' order.
int SceneImpl::check_indices(cudaStream_t st) {
    Arena A(st);
    WOS_TRY(cudaMallocAsync((void **)&A.base, 2 * sizeof(int), st));
    int *out = A.take<int>(2);
    WOS_TRY(cudaMemsetAsync(out, 0, 2 * sizeof(int), st));
    k_check_indices<<<std::min(nblk(nF, 256), 4096), 256, 0, st>>>(F, nF, dim, nV, out);
    int host[2] = {0, 0};
    WOS_TRY(cudaMemcpyAsync(host, out, sizeof(host), cudaMemcpyDeviceToHost, st));
    WOS_TRY(cudaStreamSynchronize(st));
    if (host[0]) return fail(WOS_ERR_INVALID_ARGUMENT, "face index out of range [0, nV)");
    // a polyline of which at least 90 % of the segments follow each other
    prim_order = dim == 3 ? 2 : nF >= 2 && host[1] >= nF - nF / 10 ? 1 : 0;
    return 0;
}

int SceneImpl::build(cudaStream_t st) {
    const int rc = dim == 2 ? build_geometry<2>(*this, st) : build_geometry<3>(*this, st);
    ++generation;
    return rc;
}

SceneView SceneImpl::view() const {
    SceneView v{};
    v.dim = dim;
    v.nV = nV;
    v.nF = nF;
    v.V = V;
    v.F = F;
    v.N = N;
    v.g = g;
    v.seg = seg;
    v.seginv = seginv;
    v.tri = tri;
    v.nNodes = nNodes;
    v.node = node;
    v.lseg = lseg;
    v.lseginv = lseginv;
    v.ltri = ltri;
    v.lorig = lorig;
    for (int k = 0; k < 3; ++k) {
        v.lo[k] = lo[k];
        v.hi[k] = hi[k];
    }
    v.half_min_extent = half_min_extent;
    v.max_extent = 0.0f;
    for (int k = 0; k < dim; ++k) {
        v.max_extent = fmaxf(v.max_extent, hi[k] - lo[k]);
        v.centre[k] = (lo[k] + hi[k]) * 0.5f;
    }
    for (int k = dim; k < 3; ++k) v.centre[k] = 0.0f;
    v.src_type = src_type;
    for (int k = 0; k < 5; ++k) v.src[k] = src[k];
    v.cdf = cdf;
    v.n_cdf = n_cdf;
    v.guide = guide;
    v.n_guide = n_guide;
    v.tree_depth = tree_depth;
    v.tree = tree;
    v.prims = prims;
    v.torig = torig;
    v.grid_bits = grid_bits;
    v.grid = grid_box();
    v.grid_node = grid_node();
    return v;
}

}  // namespace wosd
