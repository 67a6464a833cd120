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
//     R + R_t <= kTheta D   and the boxes are farther apart than the node's cores
//     (a node of panels: than their quadrature needs),
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

// Panel p as the FP32 sheet sums read it.
__device__ __forceinline__ PanelRec panel_record(const InstDesc& d, int p) {
    auto dup = [](double v) {
        const float f = (float)v;
        return f2pack(f, f);
    };
    const double ds = d.ds[p], g0 = d.gamma[p], g1 = d.gamma[p + 1 == d.np ? 0 : p + 1];
    PanelRec r;
    r.cs = make_ulonglong2(dup(d.cth[p]), dup(d.sth[p]));
    r.dd = make_ulonglong2(dup(ds), dup(1.0 / ds));
    r.cc = make_ulonglong2(dup(d.c2th[p]), dup(d.s2th[p]));
    r.gd = make_ulonglong2(dup(g0), dup(g1 - g0));
    r.xc = d.xc[p];
    r.zc = d.zc[p];
    r.ex = d.xc[p] + ds * d.cth[p];
    r.ez = d.zc[p] + ds * d.sth[p];
    return r;
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

__device__ __forceinline__ TargetBox target_box(const TreeNode& m) {
    return TargetBox{m.cx, m.cz, m.R, m.hx, m.hz, m.e, 0, nullptr};
}

// A warp's walk of the tree for one target group.  chain[0 .. nchain): the group
// and the wider ones above it; a stack entry keeps the place in the chain that
// its node is to meet.  step() takes up to 32 nodes from the stack, tells each
// lane what becomes of its node, and pushes the halves of those to be split.
// The order of the outcomes depends on the tree and the chain only.  The
// stack starts with at most kWalkTop nodes and holds at most 32 left over per
// level below (a step takes 32 from the top and adds twice that one level down;
// 20 levels: 2^26 leaves under kWalkTop nodes).
constexpr int kWalkTop = 128;
constexpr int kWalkStack = kWalkTop + 32 * 22;
enum WalkKind : int { kWalkNone = -1, kWalkFar = 0, kWalkNear = 1, kWalkMid = 2, kWalkSplit = 3 };
struct TreeWalk {
    TargetBox chain[kChainMax];
    uint32_t stack[kWalkStack];  // level << 27 | index
    uint8_t place[kWalkStack];
};

__host__ __device__ __forceinline__ uint32_t level_count(uint32_t nleaves, int l) {
    return (nleaves + (1u << l) - 1) >> l;
}

// Starts the walk of node (level, idx), a chain member; ntargets, at: a leaf's
// targets.  Returns the stack's height.
__device__ __forceinline__ int walk_begin(TreeWalk& W, const TreeNode* __restrict__ nodes,
                                          uint32_t C, uint32_t nleaves, int level, uint32_t idx,
                                          int ntargets, const double2* at, int lane) {
    int l0 = 0;
    while (level_count(nleaves, l0) > (uint32_t)kWalkTop) ++l0;
    const int top = (int)level_count(nleaves, l0);
    const int nchain = chain_length(nleaves) - level / kFarStep;
    __syncwarp();
    for (int i = lane; i < top; i += 32) {
        W.stack[i] = ((uint32_t)l0 << 27) | (uint32_t)i;
        W.place[i] = (uint8_t)(nchain - 1);
    }
    if (lane < nchain) {
        const int up = kFarStep * lane;
        TargetBox t = target_box(nodes[node_level(C, level + up) + (idx >> up)]);
        if (lane == 0) {
            t.n = ntargets;
            t.at = at;
        }
        W.chain[lane] = t;
    }
    __syncwarp();
    return top;
}

// Starts a walk for one group alone, given its box: the nodes first, first + step, ...
// of the lowest level with at most `most` nodes.
__device__ __forceinline__ int walk_begin(TreeWalk& W, uint32_t nleaves, const TargetBox& t,
                                          uint32_t most, uint32_t first, uint32_t step, int lane) {
    int l0 = 0;
    while (level_count(nleaves, l0) > most) ++l0;
    const uint32_t top = level_count(nleaves, l0);
    const uint32_t have = first < top ? (top - first + step - 1) / step : 0u;
    __syncwarp();
    for (uint32_t i = lane; i < have; i += 32) {
        W.stack[i] = ((uint32_t)l0 << 27) | (first + i * step);
        W.place[i] = 0;
    }
    if (lane == 0) W.chain[0] = t;
    __syncwarp();
    return (int)have;
}

// What the walk's own group (chain[0]) makes of the lane's node: translate (far),
// sum its pairs (near, a leaf), evaluate its moments at every target (mid); none:
// another group's, or no node.
__device__ __forceinline__ int walk_step(TreeWalk& W, const TreeNode* __restrict__ nodes,
                                         uint32_t C, uint32_t nleaves, int& sp, uint32_t& id,
                                         int lane) {
    const int take = min(32, sp), base = sp - take;
    int kind = kWalkNone, c = 0;
    id = 0;
    if (lane < take) {
        id = W.stack[base + lane];
        c = W.place[base + lane];
        const int l = (int)(id >> 27);
        const uint32_t i = id & ((1u << 27) - 1);
        if (i < level_count(nleaves, l)) {
            const TreeNode m = nodes[node_level(C, l) + i];
            bool met = false;  // taken by a wider group, or to be split
            while (c > 0 && !met) {
                const TargetBox& t = W.chain[c];
                if (takes(t, m)) {
                    met = true;
                } else if (l > 0 && m.R >= t.R) {
                    met = true;
                    kind = kWalkSplit;
                } else {
                    --c;
                }
            }
            if (!met) {
                const TargetBox& t = W.chain[0];
                if (takes(t, m)) kind = kWalkFar;
                else if (t.n == 0) kind = l > 0 && m.R >= t.R ? kWalkSplit : kWalkNone;  // a wide group
                else if (t.R > kSpread * m.R && takes_each(t, m)) kind = kWalkMid;
                else kind = l > 0 ? kWalkSplit : kWalkNear;
            }
        }
    }
    const unsigned split = __ballot_sync(0xffffffffu, kind == kWalkSplit);  // (all have read)
    if (kind == kWalkSplit) {
        const int at = base + 2 * __popc(split & ((1u << lane) - 1u));
        const uint32_t child = (((id >> 27) - 1) << 27) | ((id & ((1u << 27) - 1)) << 1);
        W.stack[at] = child;
        W.stack[at + 1] = child + 1;
        W.place[at] = W.place[at + 1] = (uint8_t)c;
    }
    sp = base + 2 * __popc(split);
    __syncwarp();
    return kind;
}

// The place of this lane's item among the warp's, and how many there are.
__device__ __forceinline__ int warp_place(bool mine, int lane, int& count) {
    const unsigned b = __ballot_sync(0xffffffffu, mine);
    count = __popc(b);
    return __popc(b & ((1u << lane) - 1u));
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

// Moment-to-local translations by a warp, kBatch nodes at a time.  Four lanes per
// node first write c_k = a_k (s_node / d)^k and f_l = (-s_group / d)^l / d to
// shared memory, a quarter of the powers each; then the constant translation matrix
// times the c of four nodes (real and imaginary parts: eight columns) goes to the
// FP64 matrix instruction, and a lane adds f_l times its share.  Every lane with
// a row of the matrix in registers, multiplying two nodes' c read from shared memory,
// was bound by those reads (82 % of the L1 pipe, FP64 34 %): k_far at 262 144 blobs 146
// us against 98, where latency bounds it (four warps per scheduler).  One buffer for c
// and f, for a fifth, spills: 125 us.
constexpr int kBatch = 8;
constexpr int kPowStride = kTerms + 1;  // 400-byte rows: the quarters' stores meet no bank twice
struct TransBuf {
    Cplx c[kBatch][kPowStride];
    Cplx f[kBatch][kPowStride];
};

// The lane's entries of the translation matrix, as m8n8k4 takes them: rows l = 8 i +
// lane / 4, columns k = 6 (lane % 4) + s (any order of the k will do, the same for c;
// this one reads c without bank conflicts).
struct Binomials {
    double a[kTerms / 8][kTerms / 4];
};
__device__ __forceinline__ Binomials binomials(int lane) {
    Binomials t;
#pragma unroll
    for (int i = 0; i < kTerms / 8; ++i)
#pragma unroll
        for (int s = 0; s < kTerms / 4; ++s)
            t.a[i][s] = __ldg(&g_binomial.c[(lane & 3) * (kTerms / 4) + s][8 * i + (lane >> 2)]);
    return t;
}

__device__ __forceinline__ void mma_f64(double (&d)[2], double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
        : "+d"(d[0]), "+d"(d[1])
        : "d"(a), "d"(b));
}

// A local expansion while it is summed: coefficient 8 i + lane / 4, the share of the
// nodes at places lane % 4 (mod 4) of their batches.
struct LocalSum {
    Cplx b[kTerms / 8];
};
// Lane l < kTerms: coefficient l.
__device__ __forceinline__ Cplx local_total(const LocalSum& t, int lane) {
    Cplx out{0.0, 0.0};
#pragma unroll
    for (int i = 0; i < kTerms / 8; ++i) {
        Cplx v = t.b[i];
#pragma unroll
        for (int o = 1; o <= 2; o <<= 1) {
            v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
            v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
        }
        const Cplx w = cshfl(v, (lane & 7) << 2);
        if ((lane >> 3) == i) out = w;
    }
    return out;
}

// Nodes list[0 .. cnt), cnt <= kBatch; N, mom: the simulation's.
__device__ __forceinline__ void translate(const TreeNode* __restrict__ N,
                                          const double2* __restrict__ mom, uint32_t C,
                                          const uint32_t* __restrict__ list, int cnt,
                                          const TargetBox& t, const Binomials& mat,
                                          TransBuf& buf, int lane, LocalSum& sum) {
    constexpr int Q = kTerms / 4;
    const int n = lane >> 2, part = lane & 3;
    __syncwarp();  // the previous batch's reads
    if (n < cnt) {
        const uint32_t id = list[n];
        const uint64_t at = node_level(C, (int)(id >> 27)) + (id & ((1u << 27) - 1));
        const double2* __restrict__ A = mom + at * kTerms + part * Q;
        double2 a[Q];
#pragma unroll
        for (int k = 0; k < Q; ++k) a[k] = A[k];
        const double dx = t.cx - N[at].cx, dz = t.cz - N[at].cz;
        const int en = N[at].e;
        const double inv = 1.0 / fma(dx, dx, dz * dz);
        const Cplx r{dx * inv, -(dz * inv)};  // 1 / d
        const double sn = exp2_int(en), st = -exp2_int(t.e);
        const Cplx qn{r.x * sn, r.y * sn}, qt{r.x * st, r.y * st};
        auto start = [&](Cplx q) {  // q^(part Q)
            static_assert(Q == 6, "powers of six");
            const Cplx q3 = cmul(cmul(q, q), q), q6 = cmul(q3, q3), q12 = cmul(q6, q6);
            Cplx p = (part & 1) ? q6 : Cplx{1.0, 0.0};
            const Cplx h = cmul(p, q12);
            if (part & 2) p = h;
            return p;
        };
        Cplx pn = start(qn), pt = cmul(start(qt), r);
#pragma unroll
        for (int k = 0; k < Q; ++k) {
            buf.c[n][part * Q + k] = cmul(Cplx{a[k].x, a[k].y}, pn);
            buf.f[n][part * Q + k] = pt;
            pn = cmul(pn, qn);
            pt = cmul(pt, qt);
        }
    } else if (n < ((cnt + 3) & ~3)) {
#pragma unroll
        for (int k = 0; k < Q; ++k) buf.c[n][part * Q + k] = buf.f[n][part * Q + k] = Cplx{0.0, 0.0};
    }
    __syncwarp();
#pragma unroll
    for (int j = 0; j < kBatch / 4; ++j) {
        if (4 * j >= cnt) break;
        const Cplx* c = &buf.c[4 * j + (lane >> 3)][part * Q];
        double d[kTerms / 8][2] = {};
#pragma unroll
        for (int s = 0; s < Q; ++s) {
            const double v = (lane & 4) ? c[s].y : c[s].x;
#pragma unroll
            for (int i = 0; i < kTerms / 8; ++i) mma_f64(d[i], mat.a[i][s], v);
        }
#pragma unroll
        for (int i = 0; i < kTerms / 8; ++i)
            sum.b[i] = cfma(Cplx{d[i][0], d[i][1]}, buf.f[4 * j + part][8 * i + n], sum.b[i]);
    }
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
