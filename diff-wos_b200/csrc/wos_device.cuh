// Device-side scene view, geometry, nearest-primitive queries and samplers
// for the walk-on-spheres kernels (sm_100a).
//
// Arithmetic is written with explicit fmaf() and compiled with -fmad=false,
// so each function returns the same bits as the CPU oracle's restatement of
// the same reference function (cited per function).
#pragma once

#include <cuda_runtime.h>
#include <float.h>
#include <limits.h>
#include <stdint.h>

#include "wos_math.h"

namespace wosd {

// ------------------------------------------------------------------ status
// Bits of the device status word (OR-ed by kernels, read by the host).
enum StatusBits : int {
    ST_STACK_OVERFLOW = 1,   // BVH traversal stack ran out (result may be wrong)
    ST_BAD_PRIM       = 2,   // a query returned no primitive
    ST_NONFINITE      = 4,   // a walk produced a non-finite value
    ST_QUEUE_LIMIT    = 8,   // a persistent loop hit its iteration limit
};

// ------------------------------------------------------------------ layout
// Scene data in HBM.  Primitive data is precomputed once per scene:
//   2D segment f:   seg[f]  = (a.x, a.y, (b-a).x, (b-a).y), seginv[f] = 1/|b-a|^2
//   3D triangle f:  tri[3f] = (a.xyz, |ab|^2), tri[3f+1] = (ab.xyz, ab.ac),
//                   tri[3f+2] = (ac.xyz, |ac|^2)
// The LBVH (Karras, leaf size 1) is stored breadth-first; node k holds the
// boxes of both children and the two child references:
//   2D: node[3k] = (L.lo, L.hi), node[3k+1] = (R.lo, R.hi), node[3k+2].xy = refs
//   3D: node[4k..4k+2] = (L.lo.xyz, L.hi.xyz, R.lo.xyz, R.hi.xyz) packed,
//       node[4k+3].xy = refs
// A reference r >= 0 is an internal node, r < 0 is leaf ~r in the order of the
// tree's sort keys (meshes: Hilbert, polylines: Morton or, where chained, the input's);
// leaf data is copied into that order (lseg/lseginv/ltri) with the original
// primitive index in lorig.
struct SceneView {
    int dim, nV, nF;
    const float *V;    // nV x dim
    const int *F;      // nF x dim
    const float *N;    // vertex normals, nV x dim
    const float *g;    // Dirichlet values, nV
    const float4 *seg;
    const float *seginv;
    const float4 *tri;
    int nNodes;
    const float4 *node;
    const float4 *lseg;
    const float *lseginv;
    const float4 *ltri;
    const int *lorig;
    float lo[3], hi[3];
    float half_min_extent;  // min_k (hi_k - lo_k) / 2
    float max_extent;       // max_k (hi_k - lo_k)
    float centre[3];        // (lo + hi) / 2
    int src_type;
    float src[5];
    const float *cdf;  // G CDF table (n_cdf entries)
    int n_cdf;
    // guide[k] = first index l with cdf[l] > k / n_guide (k = 0..n_guide):
    // brackets the CDF search to a few entries
    const unsigned short *guide;
    int n_guide;
    // Search tree of the walk kernels: an implicit 4-ary tree over the
    // primitives in an order of its own (torig: position -> original index).
    // Leaf i holds the primitives at positions [LEAF i, LEAF i + LEAF); the root is at
    // depth 0, the leaves at depth tree_depth, and node i of depth d has the children
    // [4 i, 4 i + 4) of depth d + 1.
    // Every node is bounded by an oriented box (k_tree_bounds): orthonormal axes
    // u_k, a centre c and half-extents e_k with |u_k.(y - c)| <= e_k for every
    // point y of its primitives.  A node's four child boxes are one block of
    // `tree`, block (4^d - 1) / 3 + i (tree_block):
    //   2D, 6 float4: (u0.xy, c.xy) per child, then (e0, e1) of two children
    //       each, with u1 = (-u0.y, u0.x);
    //   3D, 8 float4, 32 bytes per child: c as 3 floats, u0 and u1 as six
    //       16-bit integers in units of 2^-15 (offset by 32768), e0 and e1 as the
    //       upper halves of floats, e2 as a float; u2 = u0 x u1.
    // A child that does not exist is infinitely far (e0 = -inf).  A leaf's
    // primitives are one block of `prims`: 2D 5 float4, the segments
    // (a, b - a) and their 1/|b - a|^2; 3D 3 float4 per triangle, as in `tri`.
    // The last leaf repeats the last primitive (and its original index).
    int tree_depth;
    const float4 *tree;
    const float4 *prims;
    const int *torig;
    // Entry grid of the search tree over the bounding box, 2^grid_bits cells per
    // axis and one more for all points outside.  A cell is a node block of its
    // own, in `grid`: the boxes of up to four nodes whose subtrees hold, for
    // every point of the cell, all its nearest primitives; their numbers
    // (tree_node) are in grid_node.  Two float4 before those: the grid's corner
    // and its cells per unit length.
    int grid_bits;
    const float4 *grid;
    const uint4 *grid_node;
};

// Shape of the search tree: primitives per leaf, float4 per node block and per
// leaf block.
template <int D>
struct Tree;
template <>
struct Tree<2> {
    static constexpr int LEAF = 4, NODE_W = 6, LEAF_W = 5;
};
template <>
struct Tree<3> {
    static constexpr int LEAF = 2, NODE_W = 8, LEAF_W = 3 * LEAF;
};
constexpr int TREE_MAX_DEPTH = 15;  // a stack entry holds the depth in 4 bits
// Most entries on a search's stack: three siblings at each depth.
__host__ __device__ constexpr int tree_stack_entries(int depth) { return 3 * depth; }
// Block of the node i at depth d: the blocks of the depths above come first.
__host__ __device__ __forceinline__ unsigned tree_block(int d, unsigned i) {
    return i + (0x55555555u & ((1u << (2 * d)) - 1u));
}

// Number of the node i at depth d >= 1: the child boxes of `tree` counted in
// their order.  tree_place is the inverse.
__host__ __device__ __forceinline__ unsigned tree_node(int d, unsigned i) {
    return i + (0x55555554u & ((1u << (2 * d)) - 1u));
}
__device__ __forceinline__ void tree_place(unsigned node, int &d, unsigned &i) {
    d = (31 - __clz(3u * node + 4u)) >> 1;
    i = node - (0x55555554u & ((1u << (2 * d)) - 1u));
}
constexpr unsigned GRID_NONE = 0xffffffffu;

template <int D>
struct NodeWords;
template <>
struct NodeWords<2> {
    static constexpr int K = 3;
};
template <>
struct NodeWords<3> {
    static constexpr int K = 4;
};

// ------------------------------------------------------------------ Philox
// Philox-4x32-10 (Salmon et al., SC 2011); counter = (point, walk, step, role).
struct Rng {
    uint32_t k0, k1;
};

__host__ __device__ inline Rng make_rng(uint64_t seed) {
    return Rng{(uint32_t)seed, (uint32_t)(seed >> 32) ^ 0x5bd1e995u};
}

__device__ __forceinline__ uint4 philox(Rng key, uint32_t c0, uint32_t c1, uint32_t c2, uint32_t c3) {
    uint32_t k0 = key.k0, k1 = key.k1;
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        const uint32_t lo0 = 0xD2511F53u * c0, hi0 = __umulhi(0xD2511F53u, c0);
        const uint32_t lo1 = 0xCD9E8D57u * c2, hi1 = __umulhi(0xCD9E8D57u, c2);
        const uint32_t n0 = hi1 ^ c1 ^ k0, n2 = hi0 ^ c3 ^ k1;
        c0 = n0;
        c1 = lo1;
        c2 = n2;
        c3 = lo0;
        k0 += 0x9E3779B9u;
        k1 += 0xBB67AE85u;
    }
    return make_uint4(c0, c1, c2, c3);
}

enum { ROLE_PRIMAL = 0, ROLE_ANTI_A = 1, ROLE_ANTI_B = 2, ROLE_EXTRA = 3, ROLE_JITTER = 4, ROLE_BOUNDARY = 5 };

// ------------------------------------------------------------------ vectors
__device__ __forceinline__ float dot2(float ax, float ay, float bx, float by) { return fmaf(ax, bx, ay * by); }
__device__ __forceinline__ float dot3(float ax, float ay, float az, float bx, float by, float bz) {
    return fmaf(ax, bx, fmaf(ay, by, az * bz));
}
__device__ __forceinline__ void cross3(float ax, float ay, float az, float bx, float by, float bz, float &ox,
                                       float &oy, float &oz) {
    ox = ay * bz - az * by;
    oy = az * bx - ax * bz;
    oz = ax * by - ay * bx;
}

// ------------------------------------------------------------------ geometry
// Squared distance from p to a segment (include/util.cuh:108-114), with the
// clamped parameter h.
__device__ __forceinline__ float seg_d2(float4 s, float inv, float px, float py, float &h) {
    const float pax = px - s.x, pay = py - s.y;
    float t = dot2(pax, pay, s.z, s.w) * inv;
    t = fminf(fmaxf(t, 0.0f), 1.0f);
    const float vx = fmaf(-s.z, t, pax), vy = fmaf(-s.w, t, pay);
    h = t;
    return dot2(vx, vy, vx, vy);
}

// Closest point on a triangle (include/util.cuh:22-106, Ericson's Voronoi
// regions), in terms of a, ab, ac and the precomputed dot products.
// Returns the squared distance; (v, w) weight b and c; (dx, dy, dz) = x - pt.
__device__ __forceinline__ float tri_closest(float4 t0, float4 t1, float4 t2, float x, float y, float z, float &v,
                                             float &w, float &dx, float &dy, float &dz) {
    const float axx = x - t0.x, axy = y - t0.y, axz = z - t0.z;
    const float ab2 = t0.w, abac = t1.w, ac2 = t2.w;
    const float d1 = dot3(t1.x, t1.y, t1.z, axx, axy, axz);
    const float d2 = dot3(t2.x, t2.y, t2.z, axx, axy, axz);
    if (d1 <= 0.0f && d2 <= 0.0f) {
        v = 0.0f;
        w = 0.0f;
    } else {
        const float d3 = d1 - ab2, d4 = d2 - abac;
        if (d3 >= 0.0f && d4 <= d3) {
            v = 1.0f;
            w = 0.0f;
        } else {
            const float d5 = d1 - abac, d6 = d2 - ac2;
            if (d6 >= 0.0f && d5 <= d6) {
                v = 0.0f;
                w = 1.0f;
            } else {
                const float vc = d1 * d4 - d3 * d2;
                if (vc <= 0.0f && d1 >= 0.0f && d3 <= 0.0f) {
                    v = d1 / (d1 - d3);
                    w = 0.0f;
                } else {
                    const float vb = d5 * d2 - d1 * d6;
                    if (vb <= 0.0f && d2 >= 0.0f && d6 <= 0.0f) {
                        v = 0.0f;
                        w = d2 / (d2 - d6);
                    } else {
                        const float va = d3 * d6 - d5 * d4;
                        const float e43 = d4 - d3, e56 = d5 - d6;
                        if (va <= 0.0f && e43 >= 0.0f && e56 >= 0.0f) {
                            w = e43 / (e43 + e56);
                            v = 1.0f - w;
                        } else {
                            const float sum = va + vb + vc;
                            if (sum > 0.0f) {
                                const float denom = 1.0f / sum;
                                v = vb * denom;
                                w = vc * denom;
                            } else {
                                v = 0.0f;
                                w = 0.0f;
                            }
                        }
                    }
                }
            }
        }
    }
    dx = fmaf(-t2.x, w, fmaf(-t1.x, v, axx));
    dy = fmaf(-t2.y, w, fmaf(-t1.y, v, axy));
    dz = fmaf(-t2.z, w, fmaf(-t1.z, v, axz));
    return dot3(dx, dy, dz, dx, dy, dz);
}

// Squared distance to a triangle for the search tree's leaves: a branch-free
// form of tri_closest's region cascade.  Every region test is evaluated with
// the cascade's own expressions, the first region that holds
// picks the result, and the one division the edge and face regions need is
// issued once with the selected numerator and denominator.  Each value is the
// same IEEE operation on the same operands as in the cascade, so the results
// are identical to tri_closest's, but the lanes of a warp testing different
// triangles do not diverge (and run one division instead of up to four in
// turn).  Brute force and the LBVH keep the cascade, which skips work per lane.
__device__ __forceinline__ float tri_d2_uniform(float4 t0, float4 t1, float4 t2, float x, float y, float z) {
    const float axx = x - t0.x, axy = y - t0.y, axz = z - t0.z;
    const float ab2 = t0.w, abac = t1.w, ac2 = t2.w;
    const float d1 = dot3(t1.x, t1.y, t1.z, axx, axy, axz);
    const float d2 = dot3(t2.x, t2.y, t2.z, axx, axy, axz);
    const float d3 = d1 - ab2, d4 = d2 - abac;
    const float d5 = d1 - abac, d6 = d2 - ac2;
    const float vc = d1 * d4 - d3 * d2;
    const float vb = d5 * d2 - d1 * d6;
    const float va = d3 * d6 - d5 * d4;
    const float e43 = d4 - d3, e56 = d5 - d6;
    const float sum = va + vb + vc;
    const bool rA = d1 <= 0.0f && d2 <= 0.0f;                  // vertex a
    const bool rB = d3 >= 0.0f && d4 <= d3;                    // vertex b
    const bool rC = d6 >= 0.0f && d5 <= d6;                    // vertex c
    const bool rAB = vc <= 0.0f && d1 >= 0.0f && d3 <= 0.0f;   // edge ab
    const bool rAC = vb <= 0.0f && d2 >= 0.0f && d6 <= 0.0f;   // edge ac
    const bool rBC = va <= 0.0f && e43 >= 0.0f && e56 >= 0.0f; // edge bc
    // numerator / denominator of the first edge region that holds, else the face
    float num = 1.0f, den = sum;
    if (rBC) {
        num = e43;
        den = e43 + e56;
    }
    if (rAC) {
        num = d2;
        den = d2 - d6;
    }
    if (rAB) {
        num = d1;
        den = d1 - d3;
    }
    const float q = num / den;
    float v = 0.0f, w = 0.0f;
    if (rA) {
    } else if (rB) {
        v = 1.0f;
    } else if (rC) {
        w = 1.0f;
    } else if (rAB) {
        v = q;
    } else if (rAC) {
        w = q;
    } else if (rBC) {
        w = q;
        v = 1.0f - q;
    } else if (sum > 0.0f) {
        v = vb * q;
        w = vc * q;
    }
    const float dx = fmaf(-t2.x, w, fmaf(-t1.x, v, axx));
    const float dy = fmaf(-t2.y, w, fmaf(-t1.y, v, axy));
    const float dz = fmaf(-t2.z, w, fmaf(-t1.z, v, axz));
    return dot3(dx, dy, dz, dx, dy, dz);
}

__device__ __forceinline__ float tri_d2(float4 t0, float4 t1, float4 t2, float x, float y, float z) {
    float v, w, dx, dy, dz;
    return tri_closest(t0, t1, t2, x, y, z, v, w, dx, dy, dz);
}

// ------------------------------------------------------------------ queries
struct Hit {
    int prim;
    float d2;
};

// Per-thread LBVH work counters: queries, node visits (two child boxes each),
// primitive distance evaluations.
struct Work {
    unsigned nq, nb, np;
};

// The same interface counting nothing: the query functions take either type,
// and the hot kernels run with NoWork unless work accounting is switched on
// (the counters' registers and adds cost 1-3 % of a step).
struct NoCount {
    __device__ __forceinline__ NoCount &operator+=(unsigned) { return *this; }
};
struct NoWork {
    NoCount nq, nb, np;
};

// Pruning slack of the LBVH: a box is skipped only when its squared distance exceeds
// (1 + 2^-10) best + 1025 (s 2^-20)^2, where s bounds the coordinates' magnitude around
// the scene (the search tree's: search_bound).  s 2^-20 is at least 1e-22, whose square is 7 steps of the
// denormal floats: squared distances that small are only exact to a few steps.
constexpr float TOL_MIN = 1e-22f;
template <int D>
__device__ __forceinline__ float prune_tol(const SceneView &S, const float *p) {
    float s = S.max_extent;
#pragma unroll
    for (int k = 0; k < D; ++k) s += fabsf(p[k] - S.centre[k]);
    return fmaf(s, 0x1p-20f, TOL_MIN);
}
template <int D>
__device__ __forceinline__ float prune_tol2(const SceneView &S, const float *p) {
    const float e = prune_tol<D>(S, p);
    return 1025.0f * (e * e);
}
__device__ __forceinline__ float prune_bound(float best, float tol2) { return fmaf(best, 1.0009765625f, tol2); }

// Brute-force nearest over the original primitive order, ties to the lowest
// index (include/scene.cuh:102-128).  Bound by the latency of the primitives' loads
// where few lanes search: eight are in flight (one walk on 8,192 segments 1.80 ms, 2.36
// with the compiler's four).
template <int D, class WK>
__device__ __forceinline__ Hit nearest_brute(const SceneView &S, const float *p, WK &wk) {
    Hit h{-1, INFINITY};
    wk.nq += 1;
    wk.np += (unsigned)S.nF;
    if (D == 2) {
#pragma unroll 8
        for (int f = 0; f < S.nF; ++f) {
            float t;
            const float d2 = seg_d2(__ldg(&S.seg[f]), __ldg(&S.seginv[f]), p[0], p[1], t);
            if (d2 < h.d2) {
                h.d2 = d2;
                h.prim = f;
            }
        }
    } else {
#pragma unroll 8
        for (int f = 0; f < S.nF; ++f) {
            const float d2 = tri_d2(__ldg(&S.tri[3 * f]), __ldg(&S.tri[3 * f + 1]), __ldg(&S.tri[3 * f + 2]), p[0],
                                    p[1], p[2]);
            if (d2 < h.d2) {
                h.d2 = d2;
                h.prim = f;
            }
        }
    }
    return h;
}

template <int D>
__device__ __forceinline__ float box_d2(const float *lo, const float *hi, const float *p) {
    float d[3];
#pragma unroll
    for (int k = 0; k < D; ++k) d[k] = fmaxf(fmaxf(lo[k] - p[k], p[k] - hi[k]), 0.0f);
    return D == 2 ? fmaf(d[0], d[0], d[1] * d[1]) : fmaf(d[0], d[0], fmaf(d[1], d[1], d[2] * d[2]));
}

template <int D>
__device__ __forceinline__ void load_node(const float4 *base, int k, float (*lo)[3], float (*hi)[3], int &c0,
                                          int &c1) {
    if (D == 2) {
        const float4 a = base[3 * k], b = base[3 * k + 1], c = base[3 * k + 2];
        lo[0][0] = a.x;
        lo[0][1] = a.y;
        hi[0][0] = a.z;
        hi[0][1] = a.w;
        lo[1][0] = b.x;
        lo[1][1] = b.y;
        hi[1][0] = b.z;
        hi[1][1] = b.w;
        c0 = __float_as_int(c.x);
        c1 = __float_as_int(c.y);
    } else {
        const float4 a = base[4 * k], b = base[4 * k + 1], c = base[4 * k + 2], e = base[4 * k + 3];
        lo[0][0] = a.x;
        lo[0][1] = a.y;
        lo[0][2] = a.z;
        hi[0][0] = a.w;
        hi[0][1] = b.x;
        hi[0][2] = b.y;
        lo[1][0] = b.z;
        lo[1][1] = b.w;
        lo[1][2] = c.x;
        hi[1][0] = c.y;
        hi[1][1] = c.z;
        hi[1][2] = c.w;
        c0 = __float_as_int(e.x);
        c1 = __float_as_int(e.y);
    }
}

#ifndef WOS_STACK
#define WOS_STACK 64
#endif

// LBVH nearest: nearest-first descent with a per-thread stack, conservative
// pruning, ties to the lowest original index.
template <int D, class WK>
__device__ __forceinline__ Hit nearest_bvh(const SceneView &S, const float *p, int *status, WK &wk) {
    Hit h{-1, INFINITY};
    wk.nq += 1;
    if (S.nF == 1) {
        wk.np += 1;
        h.prim = 0;
        if (D == 2) {
            float t;
            h.d2 = seg_d2(__ldg(&S.seg[0]), __ldg(&S.seginv[0]), p[0], p[1], t);
        } else {
            h.d2 = tri_d2(__ldg(&S.tri[0]), __ldg(&S.tri[1]), __ldg(&S.tri[2]), p[0], p[1], p[2]);
        }
        return h;
    }
    const float tol2 = prune_tol2<D>(S, p);
    int stn[WOS_STACK];
    float std2[WOS_STACK];
    int sp = 1;
    stn[0] = 0;
    std2[0] = 0.0f;
    while (sp > 0) {
        --sp;
        const int v = stn[sp];
        if (std2[sp] > prune_bound(h.d2, tol2)) continue;
        wk.nb += 1;
        float lo[2][3], hi[2][3];
        int ch[2];
        load_node<D>(S.node, v, lo, hi, ch[0], ch[1]);
        float bd[2];
        bd[0] = box_d2<D>(lo[0], hi[0], p);
        bd[1] = box_d2<D>(lo[1], hi[1], p);
        const int nr = bd[1] < bd[0] ? 1 : 0;
        const int cn = nr ? ch[1] : ch[0], cf = nr ? ch[0] : ch[1];
        const float dn = nr ? bd[1] : bd[0], df = nr ? bd[0] : bd[1];
#pragma unroll
        for (int pass = 0; pass < 2; ++pass) {
            const int c = pass == 0 ? cn : cf;
            const float bdc = pass == 0 ? dn : df;
            if (c < 0 && bdc <= prune_bound(h.d2, tol2)) {
                const int leaf = ~c;
                wk.np += 1;
                float d2;
                if (D == 2) {
                    float t;
                    d2 = seg_d2(__ldg(&S.lseg[leaf]), __ldg(&S.lseginv[leaf]), p[0], p[1], t);
                } else {
                    d2 = tri_d2(__ldg(&S.ltri[3 * leaf]), __ldg(&S.ltri[3 * leaf + 1]), __ldg(&S.ltri[3 * leaf + 2]),
                                p[0], p[1], p[2]);
                }
                if (d2 <= h.d2) {
                    const int orig = __ldg(&S.lorig[leaf]);
                    if (d2 < h.d2 || orig < h.prim) {
                        h.d2 = d2;
                        h.prim = orig;
                    }
                }
            }
        }
        if (cf >= 0 && df <= prune_bound(h.d2, tol2)) {
            if (sp < WOS_STACK) {
                stn[sp] = cf;
                std2[sp] = df;
                ++sp;
            } else {
                atomicOr(status, ST_STACK_OVERFLOW);
            }
        }
        if (cn >= 0 && dn <= prune_bound(h.d2, tol2)) {
            if (sp < WOS_STACK) {
                stn[sp] = cn;
                std2[sp] = dn;
                ++sp;
            } else {
                atomicOr(status, ST_STACK_OVERFLOW);
            }
        }
    }
    return h;
}

// Squared distance to primitive f in the original order.
template <int D>
__device__ __forceinline__ float prim_d2(const SceneView &S, int f, const float *q) {
    if (D == 2) {
        float t;
        return seg_d2(__ldg(&S.seg[f]), __ldg(&S.seginv[f]), q[0], q[1], t);
    }
    return tri_d2(__ldg(&S.tri[3 * f]), __ldg(&S.tri[3 * f + 1]), __ldg(&S.tri[3 * f + 2]), q[0], q[1], q[2]);
}

// ------------------------------------------------------------------ ball test
// One bisection step of the inscribed-ball search accepts the radius m when
// |d - m| <= 1e-5f for the nearest distance d from the candidate centre
// (wosm::ball_accepts).  Since fl(sqrtf(d2) - m) is non-decreasing in d2, the
// step rejects exactly when some primitive "blocks" the ball,
// sqrtf(d2) - m < -1e-5f, or when even the nearest distance is above
// m + 1e-5f; the caller rules the second case out with the ball's own
// primitive.  So a step needs no nearest search: it may stop at the first
// blocking primitive.
__device__ __forceinline__ bool ball_blocks(float d2, float m) { return sqrtf(d2) - m < -1e-5f; }

// ------------------------------------------------------------------ tree search
// Nearest-primitive search with one lane per query: a depth-first descent of
// the 4-ary tree, nearest child first, that can be left after any step and
// taken up again.  The 32 lanes of a warp are at different places of different
// searches; per step the warp votes which kind runs, a node (four box bounds)
// or a leaf (four exact distances), and the lanes at the other kind wait
// (search_run).  A lane whose search ends waits only until enough others have
// ended too, while the rest keep their state: no lane waits for the slowest
// search of its warp.
//
// Why lanes and not the warp or a group per query: a query needs few boxes (24
// in 2D at 4,096 segments, about 105 in 3D at 81,920 triangles) and the step
// overhead -- reductions across lanes, loop control, the walk's own work -- is
// paid per lane and not per warp.  Random 16-byte loads that hit L1 cost the SM
// 11 cycles per warp load against 4.2 when consecutive, so 32 lanes at 32
// places are affordable.  Measured against a warp per query on a 32-ary tree:
// forward solve of 14,592 points x 64 walks on 1,024 segments 1.64 -> 0.74 ms, 2D
// gradient of 80,222 x 256 on 4,096 segments 187 -> 106 ms, 3D solve of 20,000 x
// 64 on 20,480 triangles 21.4 -> 16.2 ms, 3D gradient of 100,000 x 16 on 81,920
// triangles 129 -> 97 ms.  (Groups of 8 lanes on a 16-ary tree: 1.60 and 154 ms
// in 2D.)
//
// A search starts at the nodes of its point's grid cell (SceneView::grid) instead
// of the root: 2.9 instead of 6.1 node steps per query on 4,096 segments, 76 instead
// of 95 warp instructions.  The forward solve above 0.755 -> 0.706 ms, the 3D one
// (on the median-split order) 10.4 -> 8.9, the gradients 102.9 -> 100.8 and 60.8 ->
// 57.5.  The cell's boxes are taken in one of two ways (GATHER):
//   from the tree by their numbers, in a step of its own when the search begins:
//     16 bytes per cell, so most of what it reads is in L1; the walks do this;
//   from the cell's own block, as the first of the loop's node steps: 96 or 128
//     bytes per cell, mostly from L2, but hardly any code; the adjoint does, whose
//     loop is 40 KB of instructions and stalls on fetching them (gathering,
//     no_instruction stalls went from 1.1 to 2.8 cycles per issue).
// Each way in the other's place: the forward solves 0.773 and 9.2 ms, the gradients
// 103.4 and 63.0.  (Lower bounds per cell instead of boxes: 2D solve 0.93 ms, as
// leaves are visited that their boxes rule out.)
//
// What bounds it: instruction issue (about 70 % of the slots), at 14 of 32 lanes
// per instruction, since lanes wait at the other kind of step; L1 is 55-60 % busy.
template <int D>
struct Search {
    float tol;     // pruning tolerance of the query point (search_bound)
    float bound;   // nodes farther than this (squared) are pruned
    float stop;    // a primitive this near (squared) ends the search (negative: none does)
    float d2;      // best squared distance so far, and its position (-1: none)
    int pos;
    unsigned idx;  // the node to visit next: index within its depth
    int dep;       // its depth, or SEARCH_*
    int sp;        // stack entries
};
enum { SEARCH_DONE = -1, SEARCH_NEED = -2 };  // no node left; no search begun

// Pruning bound: a node farther than this (squared) holds no primitive whose
// computed squared distance is below `best`: at least (d (1 + 2^-18) + e)^2 with d =
// sqrt(best) and e = prune_tol.  A computed distance is that of a point of the
// primitive -- whichever: a needle triangle's is often not its closest -- up to 2^-24
// of itself and of the primitive's length (at most 0.06 e: 96 million random triangles
// as large as the scene, aspects 1 to 1e-7, points near to 30 lengths away), and a box's
// computed bound exceeds the true one by at most 2^-20 of itself.
//   2D: just that, tol = e.  (A slack of 2^-10 in the squared distance costs a third more
// leaves: arcs a thousandth farther than the nearest are many.)  3D: without the root,
// best (1 + 2^-12) + tol with tol = 4300 e^2 (2 d e <= t d^2 + e^2 / t).  (With 2^-10
// a query near a sphere's centre visits a large part of the sphere.)
// Clamped to the largest float: infinitely far boxes are never visited, even before a
// first candidate.
template <int D>
__device__ __forceinline__ float search_tol(float e) {
    return D == 2 ? e : 4300.0f * (e * e);
}
__device__ __forceinline__ float search_bound2(float d, float e) {
    const float r = fmaf(d, 1.0f + 0x1p-18f, e);
    return fminf((r * r) * (1.0f + 0x1p-22f), FLT_MAX);
}
template <int D>
__device__ __forceinline__ float search_bound(float best, float tol) {
    if constexpr (D == 2) return search_bound2(sqrtf(best), tol);
    return fminf(fmaf(best, 1.0f + 0x1p-12f, tol), FLT_MAX);
}

// Squared distance to an oriented box, a lower bound for its primitives.  With
// |u_k.(y - c)| <= e_k for every point y and axes whose matrix has norm below 1,
// the exact value is at most |q - y|^2; the float roundings of q - c and of the
// dot products (relative 2^-22 of |q - c|) are covered by the 1e-6 |y - c|
// margin in e_k for the |y - c| part and by search_bound for the rest.
__device__ __forceinline__ float obb_d2(float4 a, float e0, float e1, const float *q) {
    const float vx = q[0] - a.z, vy = q[1] - a.w;
    const float a0 = fmaxf(fabsf(dot2(a.x, a.y, vx, vy)) - e0, 0.0f);
    const float a1 = fmaxf(fabsf(dot2(-a.y, a.x, vx, vy)) - e1, 0.0f);
    return fmaf(a0, a0, a1 * a1);
}
// Third axis of a 3D box from the other two in units of 2^-15 (so itself in
// units of 2^-30), evaluated alike here and where the box is built.
__device__ __forceinline__ void obb_axis2(const float *a, const float *b, float *o) {
    o[0] = fmaf(a[1], b[2], -(a[2] * b[1]));
    o[1] = fmaf(a[2], b[0], -(a[0] * b[2]));
    o[2] = fmaf(a[0], b[1], -(a[1] * b[0]));
}
// The float q of a 16-bit q + 32768, from a word's lower or upper half: as the
// low bits of 2^23 + 32768 + q.
__device__ __forceinline__ float obb_axis_lo(unsigned w) {
    return __uint_as_float(__byte_perm(w, 0x4b000000u, 0x7610)) - 8421376.0f;
}
__device__ __forceinline__ float obb_axis_hi(unsigned w) {
    return __uint_as_float(__byte_perm(w, 0x4b000000u, 0x7632)) - 8421376.0f;
}
struct Obb3 {
    float c[3];
    unsigned w[5];
};
__device__ __forceinline__ Obb3 load_obb3(const float4 *p) {
    Obb3 o;
    float w[5];
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(o.c[0]), "=f"(o.c[1]), "=f"(o.c[2]), "=f"(w[0]), "=f"(w[1]), "=f"(w[2]), "=f"(w[3]), "=f"(w[4])
        : "l"(p));
#pragma unroll
    for (int k = 0; k < 5; ++k) o.w[k] = __float_as_uint(w[k]);
    return o;
}
__device__ __forceinline__ float obb_d2(const Obb3 &o, const float *q) {
    const float u0[3] = {obb_axis_lo(o.w[0]), obb_axis_hi(o.w[0]), obb_axis_lo(o.w[1])};
    const float u1[3] = {obb_axis_hi(o.w[1]), obb_axis_lo(o.w[2]), obb_axis_hi(o.w[2])};
    float u2[3];
    obb_axis2(u0, u1, u2);
    const float v[3] = {q[0] - o.c[0], q[1] - o.c[1], q[2] - o.c[2]};
    const float e0 = __uint_as_float(o.w[3] << 16), e1 = __uint_as_float(o.w[3] & 0xffff0000u);
    const float e2 = __uint_as_float(o.w[4]);
    const float a0 = fmaxf(fmaf(fabsf(dot3(u0[0], u0[1], u0[2], v[0], v[1], v[2])), 0x1p-15f, -e0), 0.0f);
    const float a1 = fmaxf(fmaf(fabsf(dot3(u1[0], u1[1], u1[2], v[0], v[1], v[2])), 0x1p-15f, -e1), 0.0f);
    const float a2 = fmaxf(fmaf(fabsf(dot3(u2[0], u2[1], u2[2], v[0], v[1], v[2])), 0x1p-30f, -e2), 0.0f);
    return fmaf(a0, a0, fmaf(a1, a1, a2 * a2));
}

// Cell of the entry grid that holds q.  The grid's place is read from memory: a
// view taken before vertices moved finds the current one.
template <int D>
__device__ __forceinline__ unsigned grid_cell(const SceneView &S, const float *q) {
    const float4 *head = reinterpret_cast<const float4 *>(S.grid_node) - 2;
    const float4 o = __ldg(head), inv = __ldg(head + 1);
    const float g = (float)(1 << S.grid_bits);
    const float x = (q[0] - o.x) * inv.x, y = (q[1] - o.y) * inv.y;
    bool in = x >= 0.0f && x < g && y >= 0.0f && y < g;
    unsigned cell = ((unsigned)y << S.grid_bits) + (unsigned)x;
    if (D == 3) {
        const float z = (q[2] - o.z) * inv.z;
        in = in && z >= 0.0f && z < g;
        cell += (unsigned)z << (2 * S.grid_bits);
    }
    return in ? cell : 1u << (D * S.grid_bits);
}

__device__ __forceinline__ unsigned grid_node(const SceneView &S, unsigned cell, unsigned c) {
    return __ldg(reinterpret_cast<const unsigned *>(S.grid_node + cell) + c);
}

// Next node from the stack: the last entry within the bound.  An entry is its
// node's squared distance, the low 6 bits replaced by its depth and its place
// among its siblings (rounded down, so pruning stays conservative); being on
// the stack of a depth-first descent, it is a sibling of the current path's
// node at that depth, which gives its index.  Depth 0 stands for the nodes of
// the query's grid cell.
constexpr unsigned ENTRY_LOW = 63u;
template <int D>
__device__ __forceinline__ void search_pop(Search<D> &s, const SceneView &S, const float *q, const unsigned *stack) {
    const unsigned b = __float_as_uint(s.bound) | ENTRY_LOW;
    for (;;) {
        if (s.sp == 0) {
            s.dep = SEARCH_DONE;
            return;
        }
        const unsigned e = stack[--s.sp * blockDim.x];
        if (e <= b) {
            const int dep = (int)((e >> 2) & 15u);
            if (dep == 0) {
                tree_place(grid_node(S, grid_cell<D>(S, q), e & 3u), s.dep, s.idx);
                return;
            }
            s.idx = ((s.idx >> (2 * (s.dep - dep))) & ~3u) | (e & 3u);
            s.dep = dep;
            return;
        }
    }
}

// Ascending.
__device__ __forceinline__ void sort4(unsigned *k) {
    auto order = [&](int i, int j) {
        const unsigned lo = min(k[i], k[j]), hi = max(k[i], k[j]);
        k[i] = lo;
        k[j] = hi;
    };
    order(0, 1);
    order(2, 3);
    order(0, 2);
    order(1, 3);
    order(1, 2);
}

// Squared distances to the four boxes of a node block.
template <int D>
__device__ __forceinline__ void block_distances(const float4 *b, const float *q, float *d) {
    if constexpr (D == 2) {
        const float4 e01 = __ldg(b + 4), e23 = __ldg(b + 5);
        d[0] = obb_d2(__ldg(b), e01.x, e01.y, q);
        d[1] = obb_d2(__ldg(b + 1), e01.z, e01.w, q);
        d[2] = obb_d2(__ldg(b + 2), e23.x, e23.y, q);
        d[3] = obb_d2(__ldg(b + 3), e23.z, e23.w, q);
    } else {
#pragma unroll
        for (int c = 0; c < 4; ++c) d[c] = obb_d2(load_obb3(b + 2 * c), q);
    }
}

// Visit an inner node, or at depth 0 (not after search_cell) the nodes of the
// query's grid cell: bound the four children, go to the nearest and leave the
// others within the bound on the stack, the farthest first.
template <int D, bool GATHER>
__device__ __forceinline__ void search_node(Search<D> &s, const SceneView &S, const float *q, unsigned *stack) {
    const bool top = !GATHER && s.dep == 0;
    float d[4];
    block_distances<D>((top ? S.grid : S.tree) + (size_t)tree_block(s.dep, s.idx) * Tree<D>::NODE_W, q, d);
    const unsigned low = top ? 0u : (unsigned)(s.dep + 1) << 2;
    unsigned k[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) k[c] = (__float_as_uint(d[c]) & ~ENTRY_LOW) | (low + c);
    sort4(k);
    const unsigned bound = __float_as_uint(s.bound) | ENTRY_LOW;
#pragma unroll
    for (int c = 3; c >= 1; --c)
        if (k[c] <= bound) stack[s.sp++ * blockDim.x] = k[c];
    if (k[0] > bound) {
        search_pop(s, S, q, stack);
    } else if (top) {
        tree_place(grid_node(S, s.idx, k[0] & 3u), s.dep, s.idx);
    } else {
        s.idx = 4u * s.idx + (k[0] & 3u);
        s.dep += 1;
    }
}

// Squared distance to the box of one node (tree_node).
template <int D>
__device__ __forceinline__ float node_distance(const SceneView &S, unsigned node, const float *q) {
    const float4 *b = S.tree + (size_t)(node >> 2) * Tree<D>::NODE_W;
    const int c = (int)(node & 3u);
    if constexpr (D == 2) {
        const float2 e = __ldg(reinterpret_cast<const float2 *>(b + 4) + c);
        return obb_d2(__ldg(b + c), e.x, e.y, q);
    } else {
        return obb_d2(load_obb3(b + 2 * c), q);
    }
}

// The first step of a search: the nodes of its grid cell, their boxes gathered
// from the tree.
template <int D>
__device__ __forceinline__ void search_cell(Search<D> &s, const SceneView &S, unsigned cell, const float *q,
                                            unsigned *stack) {
    const uint4 e = __ldg(S.grid_node + cell);
    const unsigned n[4] = {e.x, e.y, e.z, e.w};
    unsigned k[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const float d = node_distance<D>(S, n[c] == GRID_NONE ? 0u : n[c], q);
        k[c] = n[c] == GRID_NONE ? GRID_NONE : (__float_as_uint(d) & ~ENTRY_LOW) | c;
    }
    sort4(k);
    const unsigned bound = __float_as_uint(s.bound) | ENTRY_LOW;
#pragma unroll
    for (int c = 3; c >= 1; --c)
        if (k[c] <= bound) stack[s.sp++ * blockDim.x] = k[c];
    s.dep = SEARCH_DONE;
    if (k[0] <= bound) {
        const unsigned c = k[0] & 3u;
        tree_place(c == 0 ? n[0] : c == 1 ? n[1] : c == 2 ? n[2] : n[3], s.dep, s.idx);
    }
}

// Begin a search at q.  warm: a primitive whose distance bounds the nearest
// one's (that walk's previous nearest primitive), or -1; its own leaf lies
// within that bound, so it is found again if nothing is nearer.  ball_m > 0: the
// search is for a primitive blocking the ball of radius ball_m centred at q and
// may stop at any; primitives that do not block are of no interest.  GATHER: the
// cell's nodes are visited at once (search_cell), else by the first search_node.
template <int D, bool GATHER, class WK>
__device__ __forceinline__ void search_begin(Search<D> &s, const SceneView &S, const float *q, int warm,
                                             float ball_m, unsigned *stack, WK &wk) {
    const float e = prune_tol<D>(S, q);
    s.tol = search_tol<D>(e);
    s.stop = -1.0f;
    if (ball_m > 0.0f) {
        // a blocking primitive is nearer than m - 1e-5 (ball_blocks)
        s.bound = search_bound2(fmaxf(ball_m - 0.99e-5f, 0.0f) * (1.0f + 0x1p-20f), e);
        // blocking is monotone in the distance: if `stop` blocks, whatever is
        // nearer does
        const float t = ball_m - 1.1e-5f;
        if (t > 0.0f && ball_blocks(t * t, ball_m)) s.stop = t * t;
    } else {
        s.bound = warm >= 0 ? search_bound<D>(prim_d2<D>(S, warm, q), s.tol) : FLT_MAX;
    }
    s.d2 = INFINITY;
    s.pos = -1;
    s.idx = grid_cell<D>(S, q);
    s.sp = 0;
    // a point that is not finite has no primitive at a finite distance
    bool finite = true;
#pragma unroll
    for (int k = 0; k < D; ++k) finite = finite && fabsf(q[k]) <= FLT_MAX;
    s.dep = finite ? 0 : SEARCH_DONE;
    if (GATHER && finite) {
        wk.nb += 1;
        search_cell<D>(s, S, s.idx, q, stack);
    }
}

// Squared distances to the primitives of a leaf.
template <int D>
__device__ __forceinline__ void leaf_distances(const SceneView &S, unsigned leaf, const float *q, float *d2) {
    const float4 *b = S.prims + (size_t)leaf * Tree<D>::LEAF_W;
    if constexpr (D == 2) {
        const float4 inv = __ldg(b + 4);
        const float iv[4] = {inv.x, inv.y, inv.z, inv.w};
        float t;
#pragma unroll
        for (int c = 0; c < 4; ++c) d2[c] = seg_d2(__ldg(b + c), iv[c], q[0], q[1], t);
    } else {
#pragma unroll
        for (int c = 0; c < Tree<3>::LEAF; ++c)
            d2[c] = tri_d2_uniform(__ldg(b + 3 * c), __ldg(b + 3 * c + 1), __ldg(b + 3 * c + 2), q[0], q[1], q[2]);
    }
}

// Visit a leaf.  The search keeps the exact minimum of (d2, original index),
// as nearest_brute does: indices are looked up only where distances are equal.
template <int D>
__device__ __forceinline__ void search_leaf(Search<D> &s, const SceneView &S, const float *q, unsigned *stack) {
    constexpr int N = Tree<D>::LEAF;
    float d2[N];
    leaf_distances<D>(S, s.idx, q, d2);
    float m = d2[0];
#pragma unroll
    for (int c = 1; c < N; ++c) m = fminf(m, d2[c]);
    if (m <= s.d2 && m < INFINITY) {
        const int p0 = (int)s.idx * N;
        unsigned at = m == s.d2 ? 1u << N : 0u;  // who is at distance m: bit N the best so far
#pragma unroll
        for (int c = 0; c < N; ++c) at |= d2[c] == m ? 1u << c : 0u;
        int pos = p0 + __ffs(at) - 1;
        if ((at & (at - 1u)) != 0u) {
            // equal distances: the lowest original index
            int o = 0x7fffffff;
            for (; at != 0u; at &= at - 1u) {
                const int c = __ffs(at) - 1, p = c == N ? s.pos : p0 + c, op = __ldg(&S.torig[p]);
                if (op < o) {
                    o = op;
                    pos = p;
                }
            }
        }
        s.pos = pos;
        s.d2 = m;
        s.bound = fminf(s.bound, search_bound<D>(m, s.tol));
        if (m <= s.stop) s.sp = 0;
    }
    search_pop(s, S, q, stack);
}

// One step of the searches of a warp's lanes, unless at most `keep` of them still have a
// node to visit: then false.  S: the lane's scene.  Called by all 32 lanes.
template <int D, bool GATHER, class WK>
__device__ __forceinline__ bool search_step(Search<D> &s, const SceneView &S, const float *q, unsigned *stack,
                                            int keep, WK &wk) {
    const unsigned FULL = 0xffffffffu;
    const bool run = s.dep >= 0, leaf = run && s.dep == S.tree_depth;
    const int nr = __popc(__ballot_sync(FULL, run)), nl = __popc(__ballot_sync(FULL, leaf));
    if (nr <= keep) return false;
    if (2 * nl > nr) {
        if (leaf) {
            wk.np += 1;
            search_leaf<D>(s, S, q, stack);
        }
    } else if (run && !leaf) {
        wk.nb += 1;
        search_node<D, GATHER>(s, S, q, stack);
    }
    return true;
}

// Run the searches of a warp's lanes until at most `keep` of them still have a
// node to visit.  scenes[MULTI ? item : 0] is the lane's scene.
template <int D, bool GATHER, bool MULTI, class WK>
__device__ __forceinline__ void search_run(Search<D> &s, const SceneView *scenes, int item, const float *q,
                                           unsigned *stack, int keep, WK &wk) {
    const SceneView &S = scenes[MULTI ? item : 0];
    while (search_step<D, GATHER>(s, S, q, stack, keep, wk)) {
    }
}

// Finish the search of lane `owner` by all lanes that have no search of their own:
// each descends from a node of its own and they share the bound.  Per round, a lane
// with nothing left takes over the lowest -- so nearest to the root -- stack entry
// of the lane it is paired with, where that has one; the entry left behind is
// GRID_NONE, which a pop passes over.  A ball search ends for all when one has found a
// primitive at `stop` or nearer.  S: the owner's scene; called by all 32 lanes.
//
// What it is for: a query at about the same distance from much of a mesh visits
// thousands of nodes one after the other, long after its warp's others are done.
// 10,007 points on a mesh of 81,920 triangles, which it has just been moved to: 0.76
// -> 0.67 ms with the rebuild.
template <int D, bool GATHER, class WK>
__device__ __forceinline__ void search_share(Search<D> &s, const SceneView &S, const float *p, int owner,
                                             unsigned *stack, WK &wk) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const bool helps = lane == owner || s.dep < 0;
    float q[3] = {0.0f, 0.0f, 0.0f};
#pragma unroll
    for (int k = 0; k < D; ++k) q[k] = __shfl_sync(FULL, p[k], owner);
    Search<D> t;
    t.tol = __shfl_sync(FULL, s.tol, owner);
    t.bound = __shfl_sync(FULL, s.bound, owner);
    t.stop = __shfl_sync(FULL, s.stop, owner);
    t.d2 = lane == owner ? s.d2 : INFINITY;
    t.pos = lane == owner ? s.pos : -1;
    t.idx = lane == owner ? s.idx : 0u;
    t.dep = lane == owner ? s.dep : (int)SEARCH_DONE;
    t.sp = lane == owner ? s.sp : 0;
    int low = 0;  // entries given away
    for (int round = 0;; ++round) {
        const bool run = t.dep >= 0;
        if (!__any_sync(FULL, run)) break;
        // hand over
        int gd = -1;
        unsigned gi = 0u;
        if (low > t.sp) low = t.sp;
        if (run && low < t.sp) {
            const unsigned e = stack[low * blockDim.x];
            if (e <= (__float_as_uint(t.bound) | ENTRY_LOW)) {
                gd = (int)((e >> 2) & 15u);
                gi = ((t.idx >> (2 * (t.dep - gd))) & ~3u) | (e & 3u);
                if (gd == 0) tree_place(grid_node(S, grid_cell<D>(S, q), e & 3u), gd, gi);
            } else {
                ++low;
            }
        }
        const int other = 1 + (7 * round) % 31;
        const bool takes = helps && !run;
        const int d = __shfl_xor_sync(FULL, gd, other);
        const unsigned i = __shfl_xor_sync(FULL, gi, other);
        const bool taken = __shfl_xor_sync(FULL, (int)takes, other) != 0;
        if (takes && d >= 0) {
            t.dep = d;
            t.idx = i;
            t.sp = 0;
            low = 0;
        }
        if (gd >= 0 && taken) stack[low++ * blockDim.x] = GRID_NONE;
        // a step
        const bool on = t.dep >= 0, leaf = on && t.dep == S.tree_depth;
        const int nr = __popc(__ballot_sync(FULL, on)), nl = __popc(__ballot_sync(FULL, leaf));
        if (2 * nl > nr) {
            if (leaf) {
                wk.np += 1;
                search_leaf<D>(t, S, q, stack);
            }
        } else if (on && !leaf) {
            wk.nb += 1;
            search_node<D, GATHER>(t, S, q, stack);
        }
        t.bound = __uint_as_float(__reduce_min_sync(FULL, __float_as_uint(t.bound)));
        if (__any_sync(FULL, t.d2 <= t.stop)) break;
    }
    // the lowest original index at the least distance
    const unsigned best = __reduce_min_sync(FULL, __float_as_uint(t.d2));
    const bool at = t.pos >= 0 && __float_as_uint(t.d2) == best;
    const int o = at ? __ldg(&S.torig[t.pos]) : 0x7fffffff;
    const int least = __reduce_min_sync(FULL, o);
    const unsigned who = __ballot_sync(FULL, at && o == least);
    const int pos = __shfl_sync(FULL, t.pos, who != 0u ? __ffs(who) - 1 : 0);
    if (lane == owner) {
        s.d2 = __uint_as_float(best);
        s.pos = who != 0u ? pos : -1;
        s.dep = SEARCH_DONE;
        s.sp = 0;
    }
}

// search_run for a warp most of whose lanes may have nothing left to do (few): then, a
// few dozen steps on, the searches that are left, where they are more than `keep`, are
// shared.
//
// What it is for: an adjoint with fewer samples than lanes, and the end of any, lasts as
// long as its longest chain of searches, and balls that touch a mesh in much of it (the
// last bisection steps in a sphere) visit thousands of nodes each.  1,000 samples on a
// sphere of 81,920 triangles: 14.5 ms without sharing, 1.9 with it.  The lanes' limit and
// pace (8 and 1) hardly matter: 4 or 8 lanes, half or a quarter of the pace within 3 %; 2
// lanes take twice as long on a sphere with 30,000 samples, 16 lanes 10 % longer.
constexpr int FEW_LANES = 8, FEW_MORE = 1;
template <int D, bool GATHER, bool MULTI, class WK>
__device__ __forceinline__ void search_few(Search<D> &s, const SceneView *scenes, int item, const float *p,
                                           unsigned *stack, int keep, bool few, WK &wk) {
    const unsigned FULL = 0xffffffffu;
    // few: a lane more may be left every 32 / FEW_MORE steps
    const int more = few ? FEW_MORE : 0;
    for (int k = 32 * keep; search_step<D, GATHER>(s, scenes[MULTI ? item : 0], p, stack, k >> 5, wk); k += more) {
    }
    if (!few) return;
    unsigned left = __ballot_sync(FULL, s.dep >= 0);
    if (__popc(left) <= keep) return;
    for (; left != 0u; left &= left - 1u) {
        const int owner = __ffs(left) - 1;
        search_share<D, GATHER>(s, scenes[MULTI ? __shfl_sync(FULL, item, owner) : 0], p, owner, stack, wk);
    }
}

// The hit of a finished search: the original index of the nearest primitive
// (ball searches: of one that blocks, else -1).
template <int D>
__device__ __forceinline__ Hit search_hit(const Search<D> &s, const SceneView &S, float ball_m = -1.0f) {
    if (s.pos < 0 || (ball_m > 0.0f && !ball_blocks(s.d2, ball_m))) return Hit{-1, INFINITY};
    return Hit{__ldg(&S.torig[s.pos]), s.d2};
}

// ------------------------------------------------------------------ records
// Closest-point record at x for primitive prim (include/scene.cuh:180-223).
struct Rec {
    float p[3];
    float n[3];
    float t0, t1;  // 2D: (h, 0); 3D: (w_b, w_c)
    bool flip;     // the normal was negated to face the query point
};

// Per-walk boundary record stored by the forward pass for the adjoint:
// code = -1 (invalid walk) or prim | (flip << 30); t0, t1 as float bits.
struct WalkRec {
    int code;
    float t0, t1;
};
__host__ __device__ constexpr int walkrec_words(int D) { return D == 2 ? 2 : 4; }

template <int D>
__device__ __forceinline__ Rec closest_record(const SceneView &S, const float *x, int prim) {
    Rec r;
    if (D == 2) {
        const float4 s = __ldg(&S.seg[prim]);
        float h;
        seg_d2(s, __ldg(&S.seginv[prim]), x[0], x[1], h);
        const float pax = x[0] - s.x, pay = x[1] - s.y;
        r.p[0] = fmaf(s.z, h, s.x);
        r.p[1] = fmaf(s.w, h, s.y);
        float nx = s.w, ny = -s.z;
        const float len = sqrtf(dot2(nx, ny, nx, ny));
        nx = nx / len;
        ny = ny / len;
        r.flip = !(dot2(nx, ny, pax, pay) > 0.0f);
        if (r.flip) {
            nx = -nx;
            ny = -ny;
        }
        r.n[0] = nx;
        r.n[1] = ny;
        r.n[2] = 0.0f;
        r.p[2] = 0.0f;
        r.t0 = h;
        r.t1 = 0.0f;
    } else {
        const float4 t0 = __ldg(&S.tri[3 * prim]), t1 = __ldg(&S.tri[3 * prim + 1]), t2 = __ldg(&S.tri[3 * prim + 2]);
        float v, w, dx, dy, dz;
        tri_closest(t0, t1, t2, x[0], x[1], x[2], v, w, dx, dy, dz);
        r.p[0] = fmaf(t2.x, w, fmaf(t1.x, v, t0.x));
        r.p[1] = fmaf(t2.y, w, fmaf(t1.y, v, t0.y));
        r.p[2] = fmaf(t2.z, w, fmaf(t1.z, v, t0.z));
        float nx, ny, nz;
        cross3(t1.x, t1.y, t1.z, t2.x, t2.y, t2.z, nx, ny, nz);
        const float len = sqrtf(dot3(nx, ny, nz, nx, ny, nz));
        nx = nx / len;
        ny = ny / len;
        nz = nz / len;
        const float axx = x[0] - t0.x, axy = x[1] - t0.y, axz = x[2] - t0.z;
        r.flip = !(dot3(nx, ny, nz, axx, axy, axz) > 0.0f);
        const float sg = r.flip ? -1.0f : 1.0f;
        r.n[0] = sg * nx;
        r.n[1] = sg * ny;
        r.n[2] = sg * nz;
        r.t0 = v;
        r.t1 = w;
    }
    return r;
}

// The record of closest_record() rebuilt from (prim, t0, t1, flip): the same
// operations on the same inputs, so the same bits.
template <int D>
__device__ __forceinline__ Rec record_from(const SceneView &S, int prim, float t0, float t1, bool flip) {
    Rec r;
    r.flip = flip;
    r.t0 = t0;
    r.t1 = t1;
    if (D == 2) {
        const float4 s = __ldg(&S.seg[prim]);
        r.p[0] = fmaf(s.z, t0, s.x);
        r.p[1] = fmaf(s.w, t0, s.y);
        r.p[2] = 0.0f;
        float nx = s.w, ny = -s.z;
        const float len = sqrtf(dot2(nx, ny, nx, ny));
        nx = nx / len;
        ny = ny / len;
        r.n[0] = flip ? -nx : nx;
        r.n[1] = flip ? -ny : ny;
        r.n[2] = 0.0f;
    } else {
        const float4 a = __ldg(&S.tri[3 * prim]), b = __ldg(&S.tri[3 * prim + 1]), c = __ldg(&S.tri[3 * prim + 2]);
        r.p[0] = fmaf(c.x, t1, fmaf(b.x, t0, a.x));
        r.p[1] = fmaf(c.y, t1, fmaf(b.y, t0, a.y));
        r.p[2] = fmaf(c.z, t1, fmaf(b.z, t0, a.z));
        float nx, ny, nz;
        cross3(b.x, b.y, b.z, c.x, c.y, c.z, nx, ny, nz);
        const float len = sqrtf(dot3(nx, ny, nz, nx, ny, nz));
        const float sg = flip ? -1.0f : 1.0f;
        r.n[0] = sg * (nx / len);
        r.n[1] = sg * (ny / len);
        r.n[2] = sg * (nz / len);
    }
    return r;
}

// Signed distance and inside test (same composition as the oracle:
// include/scene.cuh:148-178 with wos/scene.py:325-339 and
// wos/scene3d.py:201-214).
template <int D>
__device__ __forceinline__ bool inside_test(const SceneView &S, const float *p, const Hit &hit, float *sd) {
    if (hit.prim < 0) {
        if (sd) *sd = INFINITY;
        return false;
    }
    const float d = sqrtf(hit.d2);
    if (D == 2) {
        const float4 s = __ldg(&S.seg[hit.prim]);
        float h;
        seg_d2(s, __ldg(&S.seginv[hit.prim]), p[0], p[1], h);
        const float pax = p[0] - s.x, pay = p[1] - s.y;
        const float vx = fmaf(-s.z, h, pax), vy = fmaf(-s.w, h, pay);
        const int ia = __ldg(&S.F[2 * hit.prim]), ib = __ldg(&S.F[2 * hit.prim + 1]);
        const float nax = __ldg(&S.N[2 * ia]), nay = __ldg(&S.N[2 * ia + 1]);
        const float nbx = __ldg(&S.N[2 * ib]), nby = __ldg(&S.N[2 * ib + 1]);
        const float nx = fmaf(nbx - nax, h, nax), ny = fmaf(nby - nay, h, nay);
        const float s2 = dot2(nx, ny, vx, vy);
        if (sd) *sd = s2 > 0.0f ? d : -d;
        return (s2 < 0.0f) && (hit.d2 > 0.0f);
    } else {
        const float4 t0 = __ldg(&S.tri[3 * hit.prim]), t1 = __ldg(&S.tri[3 * hit.prim + 1]),
                     t2 = __ldg(&S.tri[3 * hit.prim + 2]);
        float v, w, dx, dy, dz;
        tri_closest(t0, t1, t2, p[0], p[1], p[2], v, w, dx, dy, dz);
        float fx, fy, fz;
        cross3(t1.x, t1.y, t1.z, t2.x, t2.y, t2.z, fx, fy, fz);
        const float sf = dot3(fx, fy, fz, dx, dy, dz);
        const int ia = __ldg(&S.F[3 * hit.prim]), ib = __ldg(&S.F[3 * hit.prim + 1]),
                  ic = __ldg(&S.F[3 * hit.prim + 2]);
        const float w0 = (1.0f - v) - w;
        float nv[3];
#pragma unroll
        for (int k = 0; k < 3; ++k)
            nv[k] = fmaf(__ldg(&S.N[3 * ia + k]), w0, fmaf(__ldg(&S.N[3 * ib + k]), v, __ldg(&S.N[3 * ic + k]) * w));
        const float sv = dot3(nv[0], nv[1], nv[2], dx, dy, dz);
        if (sd) *sd = sf > 0.0f ? d : -d;
        return (hit.d2 > 0.0f) && (sv < 0.0f) && (sf <= 0.0f);
    }
}

// Dirichlet value (include/scene.cuh:251-264) and the vertex weights.
template <int D>
__device__ __forceinline__ float dirichlet(const SceneView &S, int prim, float t0, float t1, int *vid, float *wts) {
    if (D == 2) {
        const int ia = __ldg(&S.F[2 * prim]), ib = __ldg(&S.F[2 * prim + 1]);
        const float va = __ldg(&S.g[ia]), vb = __ldg(&S.g[ib]);
        if (vid) {
            vid[0] = ia;
            vid[1] = ib;
            wts[0] = 1.0f - t0;
            wts[1] = t0;
        }
        return fmaf(t0, vb - va, va);
    } else {
        const int ia = __ldg(&S.F[3 * prim]), ib = __ldg(&S.F[3 * prim + 1]), ic = __ldg(&S.F[3 * prim + 2]);
        const float va = __ldg(&S.g[ia]), vb = __ldg(&S.g[ib]), vc = __ldg(&S.g[ic]);
        const float w0 = (1.0f - t0) - t1;
        if (vid) {
            vid[0] = ia;
            vid[1] = ib;
            vid[2] = ic;
            wts[0] = w0;
            wts[1] = t0;
            wts[2] = t1;
        }
        return fmaf(va, w0, fmaf(vb, t0, vc * t1));
    }
}

// Source function and its parameter derivatives (include/scene.cuh:278-301).
__device__ __forceinline__ float source(const SceneView &S, float x, float y, float *df) {
    const float *q = S.src;
    if (S.src_type == 1) {
        const float tx = x - q[0], ty = y - q[1];
        const float sx2 = q[2] * q[2], sy2 = q[3] * q[3];
        const float dx = tx * tx / (2.0f * sx2);
        const float dy = ty * ty / (2.0f * sy2);
        const float E = wosm::exp_(-dx - dy);
        const float f = q[4] * E;
        if (df) {
            df[0] = f * (tx / sx2);
            df[1] = f * (ty / sy2);
            df[2] = f * (tx * tx / (sx2 * q[2]));
            df[3] = f * (ty * ty / (sy2 * q[3]));
            df[4] = E;
        }
        return f;
    }
    if (S.src_type == 2) {
        const float phi = fmaf(q[0], x, fmaf(q[1], y, q[2]));
        const float s = wosm::sin_(phi);
        if (df) {
            const float c = wosm::cos_(phi);
            df[0] = q[3] * c * x;
            df[1] = q[3] * c * y;
            df[2] = q[3] * c;
            df[3] = s;
            df[4] = 1.0f;
        }
        return fmaf(q[3], s, q[4]);
    }
    if (df) {
#pragma unroll
        for (int k = 0; k < 5; ++k) df[k] = 0.0f;
    }
    return 0.0f;
}

// Radius sample from the G CDF (include/wos.cuh:49-75).  The guide table
// (usually in shared memory) brackets the search; the bracket is checked and
// widened when it does not hold, so the result is always the first l with
// u < cdf[l], as a search over the whole table gives.
__device__ __forceinline__ float sample_G_radius(const float *cdf, int n, const unsigned short *guide, int ng,
                                                 float u, float R, float &pdf) {
    int k = (int)(u * (float)ng);
    k = min(max(k, 0), ng - 1);
    int l = guide[k], r = guide[k + 1];
    if (l > 0 && !(u >= __ldg(&cdf[l - 1]))) l = 0;
    if (!(u < __ldg(&cdf[r]))) r = n - 1;
    while (l < r) {
        const int mid = (l + r) >> 1;
        if (u < __ldg(&cdf[mid]))
            r = mid;
        else
            l = mid + 1;
    }
    const float pmf = l == 0 ? __ldg(&cdf[0]) : __ldg(&cdf[l]) - __ldg(&cdf[l - 1]);
    const float prev = l == 0 ? 0.0f : __ldg(&cdf[l - 1]);
    u = (u - prev) / pmf;
    pdf = pmf * (float)n / R;
    return R * ((float)l + u) / (float)n;
}

// Interior source term of one step (include/wos.cuh:115-139 with the
// importance-sampled branch of :121-130): returns the factor K with
// contrib += f(y) * K, and y.
__device__ __forceinline__ float source_step(const SceneView &S, const unsigned short *guide, bool use_IS, float px,
                                             float py, float d, uint32_t ra, uint32_t rb, float &yx, float &yy) {
    float dx, dy, pdf, weight;
    if (use_IS) {
        const float rad = sample_G_radius(S.cdf, S.n_cdf, guide, S.n_guide, wosm::u01(ra), d, pdf);
        float s, c;
        wosm::sincos_2pi(wosm::u01(rb), &s, &c);
        pdf = pdf / wosm::kTwoPi;
        dx = rad * c;
        dy = rad * s;
        weight = sqrtf(dot2(dx, dy, dx, dy));
    } else {
        float s, c;
        wosm::sincos_2pi(wosm::u01(ra), &s, &c);
        const float rr = sqrtf(wosm::u01(rb));
        dx = rr * c * d;
        dy = rr * s * d;
        pdf = 1.0f / (wosm::kPi * d * d);
        weight = 1.0f;
    }
    const float rn = sqrtf(dot2(dx, dy, dx, dy));
    const float G = wosm::log_(d / fmaxf(rn, 1e-4f)) * wosm::kInv2Pi;
    yx = px + dx;
    yy = py + dy;
    return pdf > 1e-5f ? G * weight / pdf : 0.0f;
}

}  // namespace wosd
