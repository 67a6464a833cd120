// Far fields by complex expansions over a binary tree of the sorted blobs.
//
// With Z = x + i z, the velocity of vortices Gamma_j at Z_j outside their cores
// is F(Z) = sum Gamma_j / (Z - Z_j), Re F = 2 pi w, Im F = 2 pi u.  The blobs of a
// simulation are sorted along a Hilbert curve and cut into leaves of kLeaf; a
// node of level l is 2^l consecutive leaves.  Each node keeps the moments
// a_k = sum Gamma_j ((Z_j - c) / s)^k, k < kTerms, about its box's centre c,
// scaled by a power of two s >= its radius R (no over- or underflow at any
// scale of the coordinates).  A target group (centre, radius R_t) takes a node
// by one moment-to-local translation when
//     R + R_t <= kTheta D   and the boxes are farther apart than the node's cores,
// D the distance of the centres, and otherwise looks at its two halves; a leaf
// that is still too near is summed pair by pair (Greengard & Rokhlin,
// J. Comput. Phys. 73 (1987) 325; the translations are theirs).  A group spread
// far wider than a node (the sparse fringe of a wake) takes it by the moments
// themselves, evaluated at every target, when each target on its own is far
// enough: without this a fringe leaf summed most of the wake pair by pair, and
// one such block held up the kernel (2^18 blobs: 2.4 ms, SMs busy 27 % of it).  All expansion
// arithmetic is FP64.  Truncation: a pair's term is off by at most
// kTheta^kTerms / (1 - kTheta) of |Gamma| / D, and in practice by two orders
// less (the bound has every blob on the rim of both circles).
//
// Target groups nest: a leaf, the node kFarStep levels above it, and so on (the
// leaf's chain).  A pair (group, node) that is too near is replaced by the
// node's halves when the node is the larger circle, else by the next narrower
// group with the same node; so wide groups meet wide nodes, their translations
// are shared (2^18 blobs of the wake: 203 per leaf without the chain, 67 with
// it), and a leaf adds up the local expansions of its chain.  The pairs follow
// from the geometry alone, so the kernels that walk for different purposes
// agree.
#pragma once
#include <cfloat>

#include "dvm_device.cuh"
#include "dvm_internal.h"

namespace dvmk {

constexpr double kTheta = 0.5;

// First node of level l in a simulation whose capacity holds C leaves, relative
// to its first node (room for (C >> l) + 1 nodes at every level).
__host__ __device__ __forceinline__ uint64_t node_level(uint32_t C, int l) {
    return 2ull * C - ((2ull * C) >> l) + (uint64_t)l;
}

__device__ __forceinline__ double exp2_int(int e) {  // 2^e, 0 below the normal range
    return e < -1022 ? 0.0 : __hiloint2double((1023 + min(e, 1023)) << 20, 0);
}

struct Cplx {
    double x, y;
};
__device__ __forceinline__ Cplx cmul(Cplx a, Cplx b) {
    return Cplx{fma(a.x, b.x, -(a.y * b.y)), fma(a.x, b.y, a.y * b.x)};
}
__device__ __forceinline__ Cplx cfma(Cplx a, Cplx b, Cplx c) {
    return Cplx{fma(a.x, b.x, fma(-a.y, b.y, c.x)), fma(a.x, b.y, fma(a.y, b.x, c.y))};
}
__device__ __forceinline__ Cplx cshfl(Cplx a, int src) {
    return Cplx{__shfl_sync(0xffffffffu, a.x, src), __shfl_sync(0xffffffffu, a.y, src)};
}

// q^n for n = 0 .. 31 (one per lane).
__device__ __forceinline__ Cplx cpow_lane(Cplx q, int n) {
    Cplx p{1.0, 0.0};
#pragma unroll
    for (int b = 0; b < 5; ++b) {
        const Cplx t = cmul(p, q);
        if ((n >> b) & 1) p = t;
        if (b < 4) q = Cplx{fma(q.x, q.x, -(q.y * q.y)), 2.0 * q.x * q.y};
    }
    return p;
}

// Block-wide exclusive prefix of count(k), k < n, into s_pre[0 .. n] (every
// thread must call it; ends with a barrier).
template <typename F>
__device__ __forceinline__ void list_prefix(unsigned* s_pre, int n, F count) {
    for (int k = threadIdx.x; k < n; k += blockDim.x) s_pre[k + 1] = count(k);
    __syncthreads();
    if (threadIdx.x < 32) {
        unsigned carry = 0;
        for (int b = 0; b < n; b += 32) {
            const int k = b + (int)threadIdx.x;
            unsigned v = k < n ? s_pre[k + 1] : 0u;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned t = __shfl_up_sync(0xffffffffu, v, o);
                if ((int)threadIdx.x >= o) v += t;
            }
            if (k < n) s_pre[k + 1] = v + carry;
            carry += __shfl_sync(0xffffffffu, v, 31);
        }
        if (threadIdx.x == 0) s_pre[0] = 0;
    }
    __syncthreads();
}

// A group of targets: centre, radius, half extents of its box, scale exponent.
struct TargetBox {
    double cx, cz, R, hx, hz;
    int e;
    int n;              // targets
    const double2* at;  // their positions (shared memory)
};
constexpr double kSpread = 3.0;  // a group this many times wider than a node may take its moments

// Squared gap between the boxes of a node and of a target group.
__device__ __forceinline__ double box_gap2(const TreeNode& m, const TargetBox& t) {
    const double gx = fmax(0.0, fabs(m.cx - t.cx) - (m.hx + t.hx));
    const double gz = fmax(0.0, fabs(m.cz - t.cz) - (m.hz + t.hz));
    return gx * gx + gz * gz;
}

constexpr int kFarStep = 2;       // tree levels between the groups of a chain
constexpr int kChainMax = 3;      // groups of a chain, the leaf first
constexpr uint32_t kChainMin = 256;  // leaves below which the leaf stands alone: its own
                                     // translations are few, and a pass over groups costs a launch

// Groups of a leaf's chain in a simulation of nleaves leaves.
__host__ __device__ __forceinline__ int chain_length(uint32_t nleaves) {
    return nleaves < kChainMin ? 1 : kChainMax;
}

__device__ __forceinline__ bool takes(const TargetBox& t, const TreeNode& m) {
    const double dx = m.cx - t.cx, dz = m.cz - t.cz, r = m.R + t.R;
    return r * r <= kTheta * kTheta * (dx * dx + dz * dz) &&
           box_gap2(m, t) > m.thr * 1.001 + 1e-30;
}

// Whether every target of a leaf can take the node's moments on its own (a
// target's distance to any of the node's blobs is at least half of d).
__device__ __forceinline__ bool takes_each(const TargetBox& t, const TreeNode& m) {
    double d2 = DBL_MAX;
    for (int q = 0; q < t.n; ++q) {
        const double2 p = t.at[q];
        const double ex = p.x - m.cx, ez = p.y - m.cz;
        d2 = fmin(d2, ex * ex + ez * ez);
    }
    return m.R * m.R <= kTheta * kTheta * d2 &&
           (1.0 - kTheta) * (1.0 - kTheta) * d2 > m.thr * 1.001 + 1e-30;
}

// Walks the tree for one target group with the block's kWalk threads and fills
// the block's lists: for FAR the nodes that this group translates, else the
// leaves to sum and the nodes to evaluate (chain[0] is then the leaf's own).
// chain[0 .. nchain): the group and the wider ones above it; a stack entry keeps
// the place in the chain that its node is to meet.  Every thread of
// the block must call step(); it returns false when the walk is over.  The
// lists' order depends on the tree and the chain only.  A step adds at most kWalk
// entries to each list.  The stack holds at most kWalk nodes left over per level
// (a step takes kWalk from the top and adds twice that one level down), and a
// walk starts at most 20 levels up (2^27 leaves under kWalk nodes).
constexpr int kWalk = 128;
constexpr int kListCap = 512;                // entries of a list before it is worked off
constexpr int kWalkStack = kWalk * 22;
struct TreeWalk {
    TargetBox chain[kChainMax];
    uint32_t stack[kWalkStack];
    uint8_t place[kWalkStack];
    uint32_t list[2][kListCap];  // FAR: [0] nodes to translate; else [0] leaves to sum, [1] nodes
                                 // to evaluate at every target (ids: level << 27 | index)
    unsigned cnt[3][kWalk / 32];
    int sp, n[2];
};

__device__ __forceinline__ TargetBox target_box(const TreeNode& m) {
    return TargetBox{m.cx, m.cz, m.R, m.hx, m.hz, m.e, 0, nullptr};
}

// Chain of node (level, idx); the targets' positions are needed for a leaf only.
__device__ __forceinline__ void walk_begin(TreeWalk& W, const TreeNode* __restrict__ nodes,
                                           uint32_t C, uint32_t nleaves, int level, uint32_t idx,
                                           int ntargets, const double2* at) {
    int l0 = 0;
    while (((nleaves + (1u << l0) - 1) >> l0) > (unsigned)kWalk) ++l0;
    const int top = (int)((nleaves + (1u << l0) - 1) >> l0);
    const int nchain = chain_length(nleaves) - level / kFarStep;
    for (int i = threadIdx.x; i < top; i += blockDim.x) {
        W.stack[i] = ((uint32_t)l0 << 27) | (uint32_t)i;
        W.place[i] = (uint8_t)(nchain - 1);
    }
    if ((int)threadIdx.x < nchain) {
        const int up = kFarStep * (int)threadIdx.x;
        TargetBox t = target_box(nodes[node_level(C, level + up) + (idx >> up)]);
        if (threadIdx.x == 0) {
            t.n = ntargets;
            t.at = at;
        }
        W.chain[threadIdx.x] = t;
    }
    if (threadIdx.x == 0) {
        W.sp = top;
        W.n[0] = W.n[1] = 0;
    }
    __syncthreads();
}

template <bool FAR>
__device__ __forceinline__ bool walk_step(TreeWalk& W, const TreeNode* __restrict__ nodes,
                                          uint32_t C, uint32_t nleaves) {
    const int sp = W.sp;
    if (sp == 0) return false;  // block-uniform
    const int take = min(kWalk, sp), base = sp - take;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    uint32_t id = 0;
    int kind = -1, c = 0;  // 0, 1: to that list; 2: split; -1: another group's
    if (tid < take) {
        id = W.stack[base + tid];
        c = W.place[base + tid];
        const int l = (int)(id >> 27);
        const uint32_t i = id & ((1u << 27) - 1);
        if (i < ((nleaves + (1u << l) - 1) >> l)) {
            const TreeNode m = nodes[node_level(C, l) + i];
            bool met = false;  // taken, or to be split
            while (c > 0 && !met) {
                const TargetBox& t = W.chain[c];
                if (takes(t, m)) {
                    met = true;
                } else if (l > 0 && m.R >= t.R) {
                    met = true;
                    kind = 2;
                } else {
                    --c;
                }
            }
            if (!met) {
                const TargetBox& t = W.chain[0];
                if (takes(t, m)) kind = FAR ? 0 : -1;
                else if (t.n == 0) kind = l > 0 && m.R >= t.R ? 2 : -1;  // a wide group
                else if (t.R > kSpread * m.R && takes_each(t, m)) kind = FAR ? -1 : 1;
                else kind = l > 0 ? 2 : (FAR ? -1 : 0);
            }
        }
    }
    unsigned ball[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        ball[k] = __ballot_sync(0xffffffffu, kind == k);
        if (lane == 0) W.cnt[k][wid] = __popc(ball[k]);
    }
    __syncthreads();
    if (kind >= 0) {
        const unsigned b = kind == 0 ? ball[0] : kind == 1 ? ball[1] : ball[2];
        int at = __popc(b & ((1u << lane) - 1u));
        for (int q = 0; q < wid; ++q) at += (int)W.cnt[kind][q];
        if (kind < 2) {
            W.list[kind][W.n[kind] + at] = id;
        } else {
            const uint32_t child = (((id >> 27) - 1) << 27) | ((id & ((1u << 27) - 1)) << 1);
            W.stack[base + 2 * at] = child;
            W.stack[base + 2 * at + 1] = child + 1;
            W.place[base + 2 * at] = W.place[base + 2 * at + 1] = (uint8_t)c;
        }
    }
    __syncthreads();
    if (tid < 3) {
        int n = 0;
        for (int q = 0; q < kWalk / 32; ++q) n += (int)W.cnt[tid][q];
        if (tid < 2) W.n[tid] += n;
        else W.sp = base + 2 * n;
    }
    __syncthreads();
    return true;
}

// Translation matrix C(l + k, k), exact in FP64: row k holds lanes l = 0 .. 31.
struct BinomialTable {
    double c[kTerms][32];
    constexpr BinomialTable() : c() {
        for (int l = 0; l < 32; ++l) c[0][l] = 1.0;
        for (int k = 1; k < kTerms; ++k) {
            c[k][0] = 1.0;
            for (int l = 1; l < 32; ++l) c[k][l] = c[k][l - 1] + c[k - 1][l];  // Pascal
        }
    }
};
static __device__ const BinomialTable g_binomial = BinomialTable();

__device__ __forceinline__ void binomial_row(double (&row)[kTerms], int l) {
#pragma unroll
    for (int k = 0; k < kTerms; ++k) row[k] = __ldg(&g_binomial.c[k][l]);
}

// Value of a node's moments at an offset (dx, dz) from its centre outside
// R / kTheta; A: the moments in shared memory.
__device__ __forceinline__ Cplx moment_value(const Cplx* __restrict__ A, double s, double dx,
                                             double dz) {
    const double r = 1.0 / fma(dx, dx, dz * dz);
    const Cplx q{s * (dx * r), -(s * (dz * r))};  // s / (Z - c)
    Cplx v = A[kTerms - 1];
#pragma unroll 4
    for (int k = kTerms - 2; k >= 0; --k) v = cfma(v, q, A[k]);
    return cmul(v, Cplx{dx * r, -(dz * r)});
}

// One moment-to-local translation by a warp: lane l adds node m's contribution
// to local coefficient l (scaled by 2^(e l) of the target group).  buf: the
// warp's kTerms entries of shared memory.
__device__ __forceinline__ void translate(const TreeNode& m, const double2* __restrict__ mom,
                                          const TargetBox& t, const double (&row)[kTerms],
                                          Cplx* __restrict__ buf, int lane, Cplx& b) {
    Cplx a{0.0, 0.0};
    if (lane < kTerms) {
        const double2 v = mom[lane];
        a = Cplx{v.x, v.y};
    }
    const double dx = t.cx - m.cx, dz = t.cz - m.cz;
    const int e = max(m.e, t.e);
    const double s = exp2_int(e);
    const double inv = s / fma(dx, dx, dz * dz);
    const Cplx q{dx * inv, -(dz * inv)};  // s / d
    const Cplx pw = cpow_lane(q, lane);
    const double fs = exp2_int((m.e - e) * lane);
    const Cplx c = cmul(a, pw);
    __syncwarp();  // the previous translation's reads of buf
    if (lane < kTerms) buf[lane] = Cplx{c.x * fs, c.y * fs};
    __syncwarp();
    Cplx s0{0.0, 0.0}, s1{0.0, 0.0};
#pragma unroll
    for (int k = 0; k < kTerms; k += 2) {
        const Cplx c0 = buf[k], c1 = buf[k + 1];
        s0.x = fma(row[k], c0.x, s0.x);
        s0.y = fma(row[k], c0.y, s0.y);
        s1.x = fma(row[k + 1], c1.x, s1.x);
        s1.y = fma(row[k + 1], c1.y, s1.y);
    }
    const double ft = exp2_int((t.e - e) * lane) * ((lane & 1) ? -1.0 : 1.0) / s;
    const Cplx f = cmul(pw, Cplx{q.x * ft, q.y * ft});
    b = cfma(Cplx{s0.x + s1.x, s0.y + s1.y}, f, b);
}

// Value of a local expansion at offset (dx, dz) from the group's centre.
__device__ __forceinline__ Cplx local_value(const Cplx* __restrict__ b, double dx, double dz,
                                            int e) {
    const double is = exp2_int(-e);
    const Cplx w{dx * is, dz * is};
    Cplx v = b[kTerms - 1];
#pragma unroll 4
    for (int k = kTerms - 2; k >= 0; --k) v = cfma(v, w, b[k]);
    return v;
}

}  // namespace dvmk
