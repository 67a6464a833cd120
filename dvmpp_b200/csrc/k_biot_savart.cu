// Regularised 2-D Biot-Savart kernels (reference: src/VelocityKernel.cpp:30-109,
// src/VortexSheet.cpp:171-210).
//
// Pair kernel:  K(r2) = (1 - exp(-r2/sigma_j^2)) / r2   if r2 < 10 sigma_j^2
//                     = 1 / r2                          otherwise
//               u_i = -(1/2pi) sum_j K dz Gamma_j,  w_i = (1/2pi) sum_j K dx Gamma_j
//
// FP32 path (the throughput path): blobs of every listed simulation are sorted
// along a Hilbert curve, packed as FP64 (x, z) + FP32 (Gamma, 10 sigma^2,
// 1/sigma^2) and cut into leaves of 64 blobs.  A binary tree over the leaves
// carries FP64 expansions of the field outside the cores (dvm_tree.cuh).  k_far, a
// warp per group of targets, walks the tree, translates every node that is far
// enough into a local expansion about the group and lists the few leaves that
// remain; k_self_f32, a block per leaf of targets, sums those pair by pair in packed
// FP32x2 arithmetic, each with the core test only where a core can reach, and
// adds the local expansions.  Coordinates are FP32 offsets from the
// target leaf's first blob; sums are FP32 within a source leaf and FP64 across
// leaves, in an order that the simulation's own blobs fix: deterministic, and
// independent of the batch a simulation runs in and of the launch shape.
//
// FP64 path (the parity path): every pair with the reference's formula in FP64,
// over 256-blob tiles of the same sorted order.
#include <cfloat>
#include <mutex>
#include <string>

#include <cub/cub.cuh>

#include "dvm_device.cuh"
#include "dvm_internal.h"
#include "dvm_tree.cuh"

namespace dvmk {
namespace {

constexpr int kMaxList = kMaxBatch;  // simulations per batched launch

// Index along a Hilbert curve over 2^16 x 2^16 cells (the standard quadrant
// recursion: rotate and reflect the lower bits by the quadrant taken).  Runs of
// consecutive blobs are spatially connected, so the boxes of sort tiles and
// leaves stay compact where Morton order jumps.
__device__ __forceinline__ uint32_t curve_key(double x, double z, double x0, double z0,
                                              double inv) {
    double fx = (x - x0) * inv, fz = (z - z0) * inv;
    fx = fmin(fmax(fx, 0.0), 65535.0);
    fz = fmin(fmax(fz, 0.0), 65535.0);
    uint32_t a = (uint32_t)fx, b = (uint32_t)fz, key = 0;
#pragma unroll 4
    for (int k = 15; k >= 0; --k) {
        const uint32_t ra = (a >> k) & 1u, rb = (b >> k) & 1u;
        key = (key << 2) | ((3u * ra) ^ rb);
        if (!rb) {
            if (ra) {
                a = ~a;
                b = ~b;
            }
            const uint32_t t = a;
            a = b;
            b = t;
        }
    }
    return key == 0xFFFFFFFFu ? 0xFFFFFFFEu : key;
}

// Bounding box of n points as order-preserving bits: dom[0..3] = max of x, z,
// -x, -z over the finite points (0: none yet).
__device__ __forceinline__ unsigned long long ordered_bits(double v) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}
__device__ __forceinline__ double from_ordered_bits(unsigned long long o) {
    return __longlong_as_double((long long)((o >> 63) ? (o & 0x7FFFFFFFFFFFFFFFull) : ~o));
}
__global__ void __launch_bounds__(256) k_domain(const double* __restrict__ x,
                                                const double* __restrict__ z, uint32_t n,
                                                unsigned long long* __restrict__ dom) {
    double m[4] = {-DBL_MAX, -DBL_MAX, -DBL_MAX, -DBL_MAX};
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const double a = x[i], b = z[i];
        if (fabs(a) < 1e300 && fabs(b) < 1e300) {
            m[0] = fmax(m[0], a);
            m[1] = fmax(m[1], b);
            m[2] = fmax(m[2], -a);
            m[3] = fmax(m[3], -b);
        }
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        for (int o = 16; o > 0; o >>= 1) m[k] = fmax(m[k], __shfl_xor_sync(0xffffffffu, m[k], o));
        if ((threadIdx.x & 31) == 0 && m[k] > -DBL_MAX) atomicMax(&dom[k], ordered_bits(m[k]));
    }
}

// The lane with the r-th smallest value of a warp's.
__device__ __forceinline__ int ranked_lane(double v, int r, int lane) {
    int mine = 0;
#pragma unroll 4
    for (int k = 0; k < 32; ++k) {
        const double o = __shfl_sync(0xffffffffu, v, k);
        mine += o < v || (o == v && k < lane);
    }
    return __ffs(__ballot_sync(0xffffffffu, mine == r)) - 1;
}
// The sort domain of a simulation's descriptor from the largest x, z, -x and -z (-DBL_MAX:
// no finite point, and any domain will do), by a warp.  Of 32 blobs taken at equal
// distances in their order, s holds all but three around their median; where the box is
// far wider than that (64 s to a side), a few strays make it so, and it would put all others in a
// few cells: the domain is then 16 s to each side, and the strays share its edge cells (200 k blobs
// of a wake, one at 1e6: 18.9 ms by the box, 0.47 without that one).
__device__ __forceinline__ void set_domain_of(InstDesc* d, const double (&m)[4], const double* __restrict__ x,
                                              const double* __restrict__ z, uint32_t n, int lane) {
    if (m[0] == -DBL_MAX) return;
    double x0 = -m[2], z0 = -m[3], L = fmax(m[0] + m[2], m[1] + m[3]);
    const uint32_t i = (uint32_t)((uint64_t)lane * n / 32);
    // (a non-finite one counts as a stray)
    const double sx = isfinite(x[i]) ? x[i] : 1e300, sz = isfinite(z[i]) ? z[i] : 1e300;
    const double cx = __shfl_sync(0xffffffffu, sx, ranked_lane(sx, 16, lane));
    const double cz = __shfl_sync(0xffffffffu, sz, ranked_lane(sz, 16, lane));
    const double r = fmax(fabs(sx - cx), fabs(sz - cz));
    const double s = __shfl_sync(0xffffffffu, r, ranked_lane(r, 28, lane));
    if (n >= 64 && s > 0.0 && L > 128.0 * s) {
        x0 = cx - 16.0 * s;
        z0 = cz - 16.0 * s;
        L = 32.0 * s;
    }
    if (lane != 0) return;
    d->kx0 = x0;
    d->kz0 = z0;
    d->kinv = L > 0.0 ? 65535.0 / L : 1.0;
}
__global__ void k_set_domain(InstDesc* __restrict__ d, const unsigned long long* __restrict__ dom,
                             const double* __restrict__ x, const double* __restrict__ z, uint32_t n) {
    if (dom[0] == 0ull) return;
    const double m[4] = {from_ordered_bits(dom[0]), from_ordered_bits(dom[1]), from_ordered_bits(dom[2]),
                         from_ordered_bits(dom[3])};
    set_domain_of(d, m, x, z, n, (int)threadIdx.x);
}

// Both by one block, for a few blobs.
constexpr uint32_t kDomainOne = 8192;
__global__ void __launch_bounds__(1024) k_domain_one(const double* __restrict__ x, const double* __restrict__ z,
                                                     uint32_t n, InstDesc* __restrict__ d) {
    __shared__ double s_m[4][32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    double m[4] = {-DBL_MAX, -DBL_MAX, -DBL_MAX, -DBL_MAX};
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
        const double a = x[i], b = z[i];
        if (fabs(a) < 1e300 && fabs(b) < 1e300) {
            m[0] = fmax(m[0], a);
            m[1] = fmax(m[1], b);
            m[2] = fmax(m[2], -a);
            m[3] = fmax(m[3], -b);
        }
    }
    for (int pass = 0; pass < 2; ++pass) {  // within the warps, then over them
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            for (int o = 16; o > 0; o >>= 1) m[k] = fmax(m[k], __shfl_xor_sync(0xffffffffu, m[k], o));
            if (pass == 0 && lane == 0) s_m[k][wid] = m[k];
        }
        if (pass == 1) break;
        __syncthreads();
        if (wid != 0) return;
#pragma unroll
        for (int k = 0; k < 4; ++k) m[k] = s_m[k][lane];
    }
    set_domain_of(d, m, x, z, n, lane);
}

__device__ __forceinline__ int entry_of_slot(const ListEntry* list, int nlist, uint64_t g) {
    int lo = 0, hi = nlist - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (list[mid].coff <= g) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// Sort keys over the concatenated capacity space: (entry << 32 | curve index);
// unused slots sort to the end of their simulation's range.
__global__ void k_keys(const InstDesc* __restrict__ table, const InstState* __restrict__ st,
                       const ListEntry* __restrict__ list, int nlist, uint64_t total,
                       uint64_t* __restrict__ keys, uint32_t* __restrict__ vals) {
    for (uint64_t g = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; g < total;
         g += (uint64_t)gridDim.x * blockDim.x) {
        const int k = entry_of_slot(list, nlist, g);
        const ListEntry e = list[k];
        const uint32_t i = (uint32_t)(g - e.coff);
        const InstDesc& d = table[e.inst];
        uint32_t mk = 0xFFFFFFFFu;
        const InstState& S = st[e.inst];
        if (i < S.n) {
            double x0 = d.kx0, z0 = d.kz0, inv = d.kinv;
            if (S.level) {
                const double grow = 32768.0 / inv * (exp2_int(S.level) - 1.0);
                x0 -= grow;
                z0 -= grow;
                inv *= exp2_int(-S.level);
            }
            mk = curve_key(d.x[i], d.z[i], x0, z0, inv);
        }
        keys[g] = ((uint64_t)k << 32) | mk;
        vals[g] = i;
    }
}

// Gather (x, z, Gamma, sigma) into sorted order and record per-tile bounds (FP64
// path).
__global__ void __launch_bounds__(kBsST) k_pack(const InstDesc* __restrict__ table,
                                                const InstState* __restrict__ st,
                                                const ListEntry* __restrict__ list, int nlist,
                                                const uint32_t* __restrict__ perm,
                                                double4* __restrict__ packed,
                                                TileMeta* __restrict__ meta) {
    __shared__ unsigned s_pre[kMaxList + 1];
    __shared__ double s_red[5][kBsST / 32];
    list_prefix(s_pre, nlist, [&](int k) { return (st[list[k].inst].n + kBsST - 1) / kBsST; });
    const unsigned total = s_pre[nlist];
    for (unsigned item = blockIdx.x; item < total; item += gridDim.x) {
        const int k = locate(s_pre, nlist, item);
        const ListEntry e = list[k];
        const InstDesc& d = table[e.inst];
        const uint32_t n = st[e.inst].n;
        const uint32_t i = (item - s_pre[k]) * kBsST + threadIdx.x;
        double xmin = DBL_MAX, xmax = -DBL_MAX, zmin = DBL_MAX, zmax = -DBL_MAX, thr = 0.0;
        if (i < n) {
            const uint32_t p = perm[e.coff + i];
            const double4 v = make_double4(d.x[p], d.z[p], d.circ[p], d.sigma[p]);
            packed[e.coff + i] = v;
            xmin = xmax = v.x;
            zmin = zmax = v.y;
            thr = 10.0 * (v.w * v.w);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            xmin = fmin(xmin, __shfl_xor_sync(0xffffffffu, xmin, o));
            xmax = fmax(xmax, __shfl_xor_sync(0xffffffffu, xmax, o));
            zmin = fmin(zmin, __shfl_xor_sync(0xffffffffu, zmin, o));
            zmax = fmax(zmax, __shfl_xor_sync(0xffffffffu, zmax, o));
            thr = fmax(thr, __shfl_xor_sync(0xffffffffu, thr, o));
        }
        const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
        if (lane == 0) {
            s_red[0][wid] = xmin;
            s_red[1][wid] = xmax;
            s_red[2][wid] = zmin;
            s_red[3][wid] = zmax;
            s_red[4][wid] = thr;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            TileMeta m;
            m.xmin = s_red[0][0];
            m.xmax = s_red[1][0];
            m.zmin = s_red[2][0];
            m.zmax = s_red[3][0];
            m.thr = s_red[4][0];
            for (int q = 1; q < kBsST / 32; ++q) {
                m.xmin = fmin(m.xmin, s_red[0][q]);
                m.xmax = fmax(m.xmax, s_red[1][q]);
                m.zmin = fmin(m.zmin, s_red[2][q]);
                m.zmax = fmax(m.zmax, s_red[3][q]);
                m.thr = fmax(m.thr, s_red[4][q]);
            }
            m.pad0 = m.pad1 = m.pad2 = 0.0;
            meta[(e.coff + (uint64_t)(item - s_pre[k]) * kBsST) / kBsST] = m;
        }
        __syncthreads();
    }
}

// ---- far-field tree of the sorted blobs ----------------------------------------
// Sum over the warp of 8 complex values per lane: each step halves the values a
// lane holds and the lanes that share one, so 8 sums cost 9 complex shuffles
// instead of 40.  Returns value ((lane >> 2) & 7, bit-reversed as the exchanges
// take them) complete in every lane.
__device__ __forceinline__ Cplx warp_sum8(Cplx (&v)[8], int lane) {
    const unsigned all = 0xffffffffu;
#pragma unroll
    for (int h = 4, o = 16; h >= 1; h >>= 1, o >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int k = 0; k < h; ++k) {
            const Cplx give = up ? v[k] : v[k + h], keep = up ? v[k + h] : v[k];
            v[k].x = keep.x + __shfl_xor_sync(all, give.x, o);
            v[k].y = keep.y + __shfl_xor_sync(all, give.y, o);
        }
    }
#pragma unroll
    for (int o = 2; o >= 1; o >>= 1) {
        v[0].x += __shfl_xor_sync(all, v[0].x, o);
        v[0].y += __shfl_xor_sync(all, v[0].y, o);
    }
    return v[0];
}

__device__ __forceinline__ int scale_exp(double R) {  // 2^e > R, clamped
    return R > 0.0 ? max(-300, min(300, ilogb(R) + 1)) : -300;
}

// Gather the blobs in sorted order, and build the tree bottom up.  A block makes
// 16 consecutive leaves (box, radius, moments; one warp each at a time) and the
// four levels above them in shared memory, one warp per node (moment-to-moment
// translations as a convolution with the factorials divided out).  Of 16
// neighbouring blocks the one that finishes last goes on with their 16 top nodes
// in the same way, and so on up to the root; nobody waits.  A node is always
// made from its halves in index order, so the result does not depend on who
// finishes when.
//
// What bounds it is latency (a gather, then a chain of small FP64 steps), so the
// levels inside a block meet no memory fence: with one arrival counter per
// node and a fence at each the kernel took 284 us for 2^20 blobs, 93 for 250 k and
// 38 for 5003, against 174, 55 and 29 us this way (32 leaves and five levels per
// block: 143, 75 and 36).
constexpr int kFan = 16;  // nodes of the lowest level of a block's share
constexpr int kFanLevels = 4;
struct TreeShared {
    TreeNode node[2 * kFan - 1];
    Cplx mom[2 * kFan - 1][kTerms];  // level j of the share starts at 2 kFan - (2 kFan >> j)
};

// A leaf's node and moments from its (up to) two blobs per lane, as offsets from
// its centre.
__device__ __forceinline__ void leaf_moments(const double (&px)[2], const double (&pz)[2],
                                             const double (&g)[2], int e, Cplx* __restrict__ out,
                                             int lane) {
    const double is = exp2_int(-e);
    const Cplx q0{px[0] * is, pz[0] * is}, q1{px[1] * is, pz[1] * is};
    // (even and odd powers as chains of their own, stepping by q^2)
    const Cplx s0 = cmul(q0, q0), s1 = cmul(q1, q1);
    Cplx t0[2] = {Cplx{g[0], 0.0}, Cplx{g[0] * q0.x, g[0] * q0.y}};
    Cplx t1[2] = {Cplx{g[1], 0.0}, Cplx{g[1] * q1.x, g[1] * q1.y}};
    const int own = ((lane >> 4) & 1) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1);
#pragma unroll
    for (int c = 0; c < kTerms / 8; ++c) {
        Cplx v[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            v[q] = Cplx{t0[q & 1].x + t1[q & 1].x, t0[q & 1].y + t1[q & 1].y};
            t0[q & 1] = cmul(t0[q & 1], s0);
            t1[q & 1] = cmul(t1[q & 1], s1);
        }
        const Cplx sum = warp_sum8(v, lane);
        if ((lane & 3) == 0) out[c * 8 + own] = sum;
    }
}

// A node from its halves (b == a when there is one), by a warp; fact = lane!.
__device__ __forceinline__ void parent_node(const TreeNode& a, const TreeNode& b,
                                            const Cplx* __restrict__ ma,
                                            const Cplx* __restrict__ mb, bool two, double fact,
                                            double ifact, int lane, TreeNode& m, Cplx& acc) {
    const double bx0 = fmin(a.cx - a.hx, b.cx - b.hx), bx1 = fmax(a.cx + a.hx, b.cx + b.hx);
    const double bz0 = fmin(a.cz - a.hz, b.cz - b.hz), bz1 = fmax(a.cz + a.hz, b.cz + b.hz);
    m.cx = 0.5 * (bx0 + bx1);
    m.cz = 0.5 * (bz0 + bz1);
    m.hx = 0.5 * (bx1 - bx0);
    m.hz = 0.5 * (bz1 - bz0);
    m.thr = fmax(a.thr, b.thr);
    const double ra = a.R + sqrt((a.cx - m.cx) * (a.cx - m.cx) + (a.cz - m.cz) * (a.cz - m.cz));
    const double rb = b.R + sqrt((b.cx - m.cx) * (b.cx - m.cx) + (b.cz - m.cz) * (b.cz - m.cz));
    m.R = fmin(fmax(ra, rb), sqrt(m.hx * m.hx + m.hz * m.hz)) * (1.0 + 1e-12);
    m.e = scale_exp(m.R);
    m.pad = 0;
    m.pad2 = 0.0;
    const double is = exp2_int(-m.e);
    // both halves side by side: four independent chains of sums
    Cplx v[2], h[2], sum[4];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const TreeNode& ch = q ? b : a;
        v[q] = Cplx{0.0, 0.0};
        if (lane < kTerms && (q == 0 || two)) {
            const Cplx w = (q ? mb : ma)[lane];
            const double f = exp2_int((ch.e - m.e) * lane) * ifact;
            v[q] = Cplx{w.x * f, w.y * f};
        }
        h[q] = cpow_lane(Cplx{(ch.cx - m.cx) * is, (ch.cz - m.cz) * is}, lane);
        h[q].x *= ifact;
        h[q].y *= ifact;
        sum[2 * q] = sum[2 * q + 1] = Cplx{0.0, 0.0};
    }
#pragma unroll
    for (int j = 0; j < kTerms; ++j)
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const Cplx aj = cshfl(v[q], j), hj = cshfl(h[q], (lane - j) & 31);
            Cplx& t = sum[2 * q + (j & 1)];
            if (lane >= j) t = cfma(aj, hj, t);
        }
    acc.x = ((sum[0].x + sum[1].x) + (sum[2].x + sum[3].x)) * fact;
    acc.y = ((sum[0].y + sum[1].y) + (sum[2].y + sum[3].y)) * fact;
}

// Gauss points and weights of four-point quadrature on [0, 1].  Seen from a gap of
// 1, 2 or 3 of its lengths a panel is off by at most 6e-5, 6e-7 or 4e-8 of the sum of
// its absolute contributions, whatever its two end strengths (against 200 points),
// so the panels' nodes are taken from a gap of kPanelGap of their longest panel on (as
// TreeNode::thr) and their boxes and radii hold the panels' ends.  A leaf of 16 equal
// panels is farther away than that by its radius alone; one that a single panel
// dominates (a remainder of one or two, a contour with long straight panels) is not,
// and blobs near it were off by up to 2e-4 without the gap.
constexpr double kPanelGap = 3.0;
__device__ __constant__ const double kGaussT[kPanelPoints] = {
    0.06943184420297371, 0.33000947820757187, 0.66999052179242813, 0.93056815579702629};
__device__ __constant__ const double kGaussW[kPanelPoints] = {
    0.17392742256872693, 0.32607257743127307, 0.32607257743127307, 0.17392742256872693};

// PANELS: the same over the sheet's Gauss points (panel order; circulation -gamma ds
// dt each, which gives the sheet's velocity the blobs' convention), and the
// panels' records for the near sums.
constexpr int kTreeWarps = 8;
template <bool PANELS>
__global__ void __launch_bounds__(32 * kTreeWarps, 2)
    k_tree(const InstDesc* __restrict__ table, const InstState* __restrict__ st,
           const ListEntry* __restrict__ list, int nlist, const uint32_t* __restrict__ perm,
           double2* __restrict__ pxz, float4* __restrict__ pf, TreeNode* __restrict__ nodes,
           double2* __restrict__ mom, unsigned* __restrict__ arrived,
           PanelRec* __restrict__ pan) {
    __shared__ unsigned s_pre[kMaxList + 1];
    __shared__ TreeShared S;
    __shared__ unsigned s_last;
    list_prefix(s_pre, nlist, [&](int k) {
        const uint32_t n = PANELS ? (uint32_t)(kPanelPoints * table[list[k].inst].np)
                                  : st[list[k].inst].n;
        return (n + kLeaf * kFan - 1) / (kLeaf * kFan);
    });
    const unsigned total = s_pre[nlist], all = 0xffffffffu;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    double fact = 1.0;  // lane!
    for (int k = 2; k <= lane; ++k) fact *= (double)k;
    const double ifact = 1.0 / fact;
    for (unsigned item = blockIdx.x; item < total; item += gridDim.x) {
        const int k = locate(s_pre, nlist, item);
        const ListEntry e = list[k];
        const InstDesc& d = table[e.inst];
        const uint32_t n = PANELS ? (uint32_t)(kPanelPoints * d.np) : st[e.inst].n;
        const uint32_t C = PANELS ? panel_leaves(d.np) : e.cap / kLeaf;
        const uint32_t nl = (n + kLeaf - 1) / kLeaf;
        const uint64_t noff = PANELS ? e.pnoff : e.noff;
        TreeNode* __restrict__ N = nodes + noff;
        double2* __restrict__ A = mom + noff * kTerms;
        uint32_t g = item - s_pre[k];  // the block's share: nodes kFan g .. of its lowest level
        if (PANELS) {
            const uint32_t p = g * (kFan * kPanelLeaf) + threadIdx.x;
            static_assert(kFan * kPanelLeaf == 32 * kTreeWarps, "a record per thread");
            if (p < (uint32_t)d.np) pan[e.panoff + p] = panel_record(d, (int)p);
        }
        uint32_t next[2];  // the next leaf's blobs, ahead of its gather
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint32_t i = (g * kFan + wid) * kLeaf + h * 32 + lane;
            next[h] = !PANELS && i < n ? perm[e.coff + i] : 0u;
        }
        for (int w = wid; w < kFan && g * kFan + w < nl; w += kTreeWarps) {
            const uint32_t idx = g * kFan + w;
            const uint32_t here[2] = {next[0], next[1]};
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint32_t i = (idx + kTreeWarps) * kLeaf + h * 32 + lane;
                next[h] = !PANELS && i < n ? perm[e.coff + i] : 0u;
            }
            double px[2], pz[2], gc[2];
            double ex[2], ez[2];  // PANELS: what the box holds, for a panel's outer points its ends
            double x0 = DBL_MAX, x1 = -DBL_MAX, z0 = DBL_MAX, z1 = -DBL_MAX, thr = 0.0;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint32_t i = idx * kLeaf + h * 32 + lane;
                px[h] = pz[h] = gc[h] = ex[h] = ez[h] = 0.0;
                if (i < n) {
                    if (PANELS) {
                        const uint32_t p = i / kPanelPoints;
                        const double t = kGaussT[i % kPanelPoints], w = kGaussW[i % kPanelPoints];
                        const double dsp = d.ds[p], g0 = d.gamma[p];
                        const double g1 = d.gamma[p + 1 == (uint32_t)d.np ? 0 : p + 1];
                        px[h] = fma(dsp * t, d.cth[p], d.xc[p]);
                        pz[h] = fma(dsp * t, d.sth[p], d.zc[p]);
                        gc[h] = -(w * dsp) * fma(g1 - g0, t, g0);
                        const int q = i % kPanelPoints;
                        const double te = q == 0 ? 0.0 : q == kPanelPoints - 1 ? 1.0 : t;
                        ex[h] = fma(dsp * te, d.cth[p], d.xc[p]);
                        ez[h] = fma(dsp * te, d.sth[p], d.zc[p]);
                        thr = fmax(thr, (kPanelGap * dsp) * (kPanelGap * dsp));
                    } else {
                        const uint32_t p = here[h];
                        const double sg = d.sigma[p], s2 = sg * sg;
                        px[h] = d.x[p];
                        pz[h] = d.z[p];
                        gc[h] = d.circ[p];
                        pxz[e.coff + i] = make_double2(px[h], pz[h]);
                        pf[e.coff + i] =
                            make_float4((float)gc[h], (float)(10.0 * s2), (float)(1.0 / s2), 0.f);
                        thr = fmax(thr, 10.0 * s2);
                    }
                    const double bx = PANELS ? ex[h] : px[h], bz = PANELS ? ez[h] : pz[h];
                    x0 = fmin(x0, bx);
                    x1 = fmax(x1, bx);
                    z0 = fmin(z0, bz);
                    z1 = fmax(z1, bz);
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                x0 = fmin(x0, __shfl_xor_sync(all, x0, o));
                x1 = fmax(x1, __shfl_xor_sync(all, x1, o));
                z0 = fmin(z0, __shfl_xor_sync(all, z0, o));
                z1 = fmax(z1, __shfl_xor_sync(all, z1, o));
                thr = fmax(thr, __shfl_xor_sync(all, thr, o));
            }
            TreeNode m;
            m.cx = 0.5 * (x0 + x1);
            m.cz = 0.5 * (z0 + z1);
            m.hx = 0.5 * (x1 - x0);
            m.hz = 0.5 * (z1 - z0);
            m.thr = thr;
            double r2 = 0.0;
#pragma unroll
            for (int h = 0; h < 2; ++h)
                if (idx * kLeaf + h * 32 + lane < n) {
                    px[h] -= m.cx;
                    pz[h] -= m.cz;
                    const double bx = PANELS ? ex[h] - m.cx : px[h], bz = PANELS ? ez[h] - m.cz : pz[h];
                    r2 = fmax(r2, bx * bx + bz * bz);
                }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) r2 = fmax(r2, __shfl_xor_sync(all, r2, o));
            m.R = sqrt(r2) * (1.0 + 1e-12);
            m.e = scale_exp(m.R);
            m.pad = 0;
            m.pad2 = 0.0;
            leaf_moments(px, pz, gc, m.e, S.mom[w], lane);
            __syncwarp();
            if (lane < kTerms)
                A[(uint64_t)idx * kTerms + lane] = make_double2(S.mom[w][lane].x, S.mom[w][lane].y);
            if (lane == 0) S.node[w] = N[idx] = m;
        }
        __syncthreads();
        for (int base = 0;; base += kFanLevels) {  // level of the share's lowest nodes
            int l = base;
            for (int j = 1; j <= kFanLevels; ++j) {
                const uint32_t below = (nl + (1u << l) - 1) >> l;
                if (below <= 1u) break;  // the root is done
                ++l;
                const uint32_t here = (nl + (1u << l) - 1) >> l, first = g * (kFan >> j);
                const int at = 2 * kFan - (2 * kFan >> j), child = 2 * kFan - (2 * kFan >> (j - 1));
                for (int w = wid; w < (kFan >> j) && first + w < here; w += kTreeWarps) {
                    const bool two = 2 * (first + w) + 1 < below;
                    const int c0 = child + 2 * w, c1 = two ? c0 + 1 : c0;
                    TreeNode m;
                    Cplx a;
                    parent_node(S.node[c0], S.node[c1], S.mom[c0], S.mom[c1], two, fact, ifact,
                                lane, m, a);
                    const uint64_t to = node_level(C, l) + first + w;
                    if (lane < kTerms) {
                        S.mom[at + w][lane] = a;
                        A[to * kTerms + lane] = make_double2(a.x, a.y);
                    }
                    if (lane == 0) S.node[at + w] = N[to] = m;
                }
                __syncthreads();
            }
            const uint32_t tops = (nl + (1u << l) - 1) >> l;
            if (tops <= 1u) break;  // (then l is the root's level)
            // kFan neighbouring shares: the last to finish takes their top nodes
            __threadfence();
            __syncthreads();
            if (threadIdx.x == 0) {
                const uint32_t up = g / kFan, want = min((uint32_t)kFan, tops - up * kFan);
                s_last = atomicAdd(&arrived[noff + node_level(C, l + kFanLevels) + up], 1u) + 1 == want;
            }
            __syncthreads();
            if (!s_last) break;
            __threadfence();
            g /= kFan;
            // (__ldcg: written by other SMs during this launch)
            const uint32_t have = min((uint32_t)kFan, tops - g * kFan);
            const uint64_t from = node_level(C, l) + (uint64_t)g * kFan;
            for (uint32_t q = threadIdx.x; q < have * kTerms; q += blockDim.x) {
                const double2 v = __ldcg(&A[from * kTerms + q]);
                S.mom[q / kTerms][q % kTerms] = Cplx{v.x, v.y};
            }
            for (uint32_t q = threadIdx.x; q < have * (sizeof(TreeNode) / 16); q += blockDim.x)
                reinterpret_cast<double2*>(S.node)[q] =
                    __ldcg(reinterpret_cast<const double2*>(N + from) + q);
            __syncthreads();
        }
        __syncthreads();
    }
}

// FP64 path: sources per chunk (a multiple of 64) of n blobs cut into at most
// `chunks`, and how many chunks that makes.
__device__ __forceinline__ uint32_t chunk_size(uint32_t n, int chunks) {
    return max(64u, ((n + chunks - 1) / chunks + 63) / 64 * 64);
}
__device__ __forceinline__ uint32_t chunk_count(uint32_t n, int chunks) {
    const uint32_t cs = chunk_size(n, chunks);
    return (n + cs - 1) / cs;
}

// ---- FP32 pair loops --------------------------------------------------------
// A warp sums one staged source leaf at the 64 targets of a leaf, two targets
// per lane.  Two SOURCES share a packed FP32x2 instruction: their values come
// out of shared memory as register pairs (no duplicating moves), the targets'
// are duplicated once per item.
constexpr int kNearThreads = 640;  // per SM at full occupancy (96 registers)
constexpr double kStray = 64.0;
constexpr int kNearSlots = 8;   // partial sums of an item: list entries q, q + 8, ...

__device__ __forceinline__ void split_hi_lo(double v, float& hi, float& lo) {
    hi = (float)v;
    lo = (float)(v - (double)hi);
}

struct StagedLeaf {
    float4 pos[kLeaf / 2];   // (x a, x b, z a, z b) of sources 2i, 2i + 1 (offsets)
    float2 gam[kLeaf / 2];   // Gamma of both
    float2 thr[kLeaf / 2];   // 10 sigma^2 of both
    float2 rs[kLeaf / 2];    // 1 / sigma^2 of both
    float4 low[kLeaf / 2];   // WIDE: what pos leaves of the offsets, same order
};

// Core kernel (1 - exp(-r2/sigma^2)) / r2 in FP32, written as rs phi(t) with
// t = r2 rs, rs = 1/sigma^2 and phi(t) = (1 - e^-t) / t.  For t < 1/2 phi is
// a degree-5 polynomial, minimax in relative error on [0, 1/2] (Lawson's
// algorithm, csrc/fit_polys.py: 6.1e-8 relative in FP32 Horner form, the
// degree-8 Taylor series it replaced gave 6.5e-8 with three more FMAs per
// half).  Its constant term 1 = phi(0) gives the r -> 0 limit 1/sigma^2: the
// self pair then contributes exactly zero, as the reference's i != j skip
// gives, and distinct blobs closer than FP32 resolves stay finite, as the
// FP64 reference is.  For t >= 1/2 it is (1 - e) / r2 with e = 2^(-t log2 e)
// from one MUFU ex2; 1 - e >= 0.39 there, so the ex2 error stays below 4e-7
// relative.  Two pairs at once, packed.
__device__ __forceinline__ uint64_t core_kernel2(uint64_t r2, uint64_t rs, uint64_t rcp_r2) {
    auto dup = [](float v) { return f2pack(v, v); };
    const uint64_t t = f2mul(r2, rs);
    uint64_t p = dup(-1.121634850e-03f);
    p = f2fma(p, t, dup(8.187386207e-03f));
    p = f2fma(p, t, dup(-4.162909091e-02f));
    p = f2fma(p, t, dup(1.666622460e-01f));
    p = f2fma(p, t, dup(-4.999998212e-01f));
    p = f2fma(p, t, dup(1.0f));
    const uint64_t m = f2mul(t, dup(-1.44269504088896341f));
    const uint64_t e = f2pack(ex2_approx(f2lo(m)), ex2_approx(f2hi(m)));
    const uint64_t in = f2mul(rs, p), out = f2mul(f2sub(dup(1.0f), e), rcp_r2);
    return f2pack(f2lo(t) < 0.5f ? f2lo(in) : f2lo(out), f2hi(t) < 0.5f ? f2hi(in) : f2hi(out));
}

// The same core kernel through expm1f (about 1 ulp): the blob-on-collocation
// right-hand side keeps it, since that sum is a small residual of nearly
// cancelling terms.  Below FLT_MIN the r -> 0 limit 1/sigma^2 is used.
__device__ __forceinline__ float core_kernel_expm1(float r2, float rs, float rcp_r2) {
    const float e = expm1f(-r2 * rs);
    return r2 > 1e-30f ? -e * rcp_r2 : rs;
}

// The staged leaf against the lane's two targets.  MODE 0: no core reaches (the
// 1/r^2 branch without a test); 1: the reference's exact test per pair; 2: the
// same for the targets' own leaf, where a pair at r2 == 0 adds nothing -- the
// reference's i != j skip for the self pair whatever the core size (sigma = 0
// would otherwise give 1/0 times dz = 0).  A pair outside the core gets the
// same bits in every mode; the core kernel runs for both halves, branch-free,
// whenever any lane of the warp has a pair inside a core, and a select keeps it
// only for those pairs, so a pair's value does not depend on its neighbours.
// Accumulates -u and w, even and odd sources apart.
//
// WIDE: for a target leaf much wider than the source leaf, or than its
// neighbours (blobs of two distant clusters, a sparse fringe; against every source leaf
// when a stray makes it kStray times wider than a neighbour).  Offsets from
// its first blob would carry the rounding of its extent into close pairs, so
// they are kept in two FP32 parts, hi + low: dx = (t_hi - s_hi) + (t_low -
// s_low), exact before its last rounding for close pairs.
template <int MODE, bool WIDE>
__device__ __forceinline__ void leaf_sum(const StagedLeaf& __restrict__ src,
                                         const uint64_t (&tx2)[2], const uint64_t (&tz2)[2],
                                         const uint64_t (&lx2)[2], const uint64_t (&lz2)[2],
                                         uint64_t (&nu2)[2], uint64_t (&w2)[2]) {
#pragma unroll 4
    for (int i = 0; i < kLeaf / 2; ++i) {
        const float4 P = src.pos[i];
        const float2 G = src.gam[i];
        const uint64_t sx = f2pack(P.x, P.y), sz = f2pack(P.z, P.w), sg = f2pack(G.x, G.y);
        const float4 L = WIDE ? src.low[i] : make_float4(0.f, 0.f, 0.f, 0.f);
        float2 T = make_float2(0.f, 0.f), S = make_float2(0.f, 0.f);
        if (MODE) {
            T = src.thr[i];
            S = src.rs[i];
        }
#pragma unroll
        for (int t = 0; t < 2; ++t) {
            uint64_t dx = f2sub(tx2[t], sx);
            uint64_t dz = f2sub(tz2[t], sz);
            if (WIDE) {
                dx = f2add(dx, f2sub(lx2[t], f2pack(L.x, L.y)));
                dz = f2add(dz, f2sub(lz2[t], f2pack(L.z, L.w)));
            }
            const uint64_t r2 = f2fma(dx, dx, f2mul(dz, dz));
            const float ra = f2lo(r2), rb = f2hi(r2);
            // one MUFU reciprocal per pair (padded sources: rcp of ~2e36, Gamma 0)
            float ka = rcp_approx(ra), kb = rcp_approx(rb);
            if (MODE) {
                const bool ca = ra < T.x, cb = rb < T.y;
                if (__any_sync(0xffffffffu, ca || cb)) {
                    const uint64_t q = core_kernel2(r2, f2pack(S.x, S.y), f2pack(ka, kb));
                    ka = ca ? f2lo(q) : ka;
                    kb = cb ? f2hi(q) : kb;
                }
                if (MODE == 2) {
                    ka = ra > 0.0f ? ka : 0.0f;
                    kb = rb > 0.0f ? kb : 0.0f;
                }
            }
            const uint64_t g = f2mul(f2pack(ka, kb), sg);
            nu2[t] = f2fma(g, dz, nu2[t]);
            w2[t] = f2fma(g, dx, w2[t]);
        }
    }
}

// The same from the FP64 positions, for a leaf whose sum came out non-finite: two blobs of
// different leaves that lie closer than their FP32 offsets resolve give r2 == 0 there, and
// with a core size below that 1/0 times 0 (a blob's own leaf skips such pairs, above).  Pairs
// whose squared distance is below FP32's range and that no core covers add nothing; what
// is non-finite by its inputs stays so.  (The test, one for a lane's two targets: 0.5 % of a
// call of 2^20 blobs; one per target and component 1.1 %.)
__device__ __forceinline__ void leaf_sum_close(const double2* __restrict__ X, const float4* __restrict__ F,
                                               uint32_t j0, uint32_t j1, double2 p, double& nu, double& w) {
#pragma unroll 1
    for (uint32_t j = j0; j < j1; ++j) {
        const float4 f = F[j];
        const float dx = (float)(p.x - X[j].x), dz = (float)(p.y - X[j].y);
        const float r2 = fmaf(dx, dx, dz * dz);
        float k = r2 >= FLT_MIN ? rcp_approx(r2) : 0.0f;
        if (r2 < f.y && r2 > 0.0f) k = core_kernel_expm1(r2, f.z, k);
        const double g = (double)k * f.x;
        nu += g * dz;
        w += g * dx;
    }
}

// Local expansions of every target group of every listed simulation, one warp per
// group (the wide groups first, they have the most to translate).  A leaf's walk
// also meets the leaves to be summed pair by pair and the nodes to be evaluated
// at every target; it leaves them to k_self_f32 in the leaf's row of `near`:
// leaves from the front, nodes from the back.  A row that is too short (cores
// that reach over hundreds of leaves) has kNearOver as its count, and k_self_f32
// walks again.
constexpr int kFarWarps = 4;
constexpr int kFarBlocks = 4;  // blocks per SM (the translation matrix: 36 registers)
constexpr int kFarList = 64;   // at least kBatch + 32
struct FarShared {
    TreeWalk walk;
    TransBuf buf;
    double2 at[kLeaf];
    uint32_t far[kFarList];
};

__device__ __forceinline__ uint32_t groups_at(uint32_t nl, int c) {  // groups of chain place c
    return c < chain_length(nl) ? level_count(nl, kFarStep * c) : 0u;
}

__global__ void __launch_bounds__(32 * kFarWarps, kFarBlocks)
    k_far(const InstState* __restrict__ st, const ListEntry* __restrict__ list, int nlist,
          const double2* __restrict__ pxz, const TreeNode* __restrict__ nodes,
          const double2* __restrict__ mom, double2* __restrict__ loc, NearRow* __restrict__ near,
          unsigned* __restrict__ work) {
    __shared__ unsigned s_pre[kMaxList + 1];
    extern __shared__ __align__(16) unsigned char s_far[];  // FarShared per warp
    list_prefix(s_pre, nlist, [&](int k) {
        const uint32_t nl = (st[list[k].inst].n + kLeaf - 1) / kLeaf;
        uint32_t g = 0;
        for (int c = 0; c < kChainMax; ++c) g += groups_at(nl, c);
        return g;
    });
    const unsigned total = s_pre[nlist];
    const int lane = threadIdx.x & 31;
    FarShared& S = reinterpret_cast<FarShared*>(s_far)[threadIdx.x >> 5];
    const Binomials mat = binomials(lane);
    for (;;) {
        unsigned item = 0;
        if (lane == 0) item = atomicAdd(work, 1u);
        item = __shfl_sync(0xffffffffu, item, 0);
        if (item >= total) break;
        const int k = locate(s_pre, nlist, item);
        const ListEntry e = list[k];
        const uint32_t n = st[e.inst].n, C = e.cap / kLeaf;
        const uint32_t nl = (n + kLeaf - 1) / kLeaf;
        const TreeNode* __restrict__ N = nodes + e.noff;
        const double2* __restrict__ A = mom + e.noff * kTerms;
        uint32_t idx = item - s_pre[k];
        int c = chain_length(nl) - 1;
        while (idx >= groups_at(nl, c)) idx -= groups_at(nl, c--);
        const int level = kFarStep * c;
        const uint32_t t0 = idx * kLeaf;  // (a leaf's)
        NearRow* row_out = c == 0 ? near + e.coff / kLeaf + idx : nullptr;
        if (c == 0)
            for (int q = lane; q < kLeaf; q += 32) S.at[q] = pxz[e.coff + min(t0 + q, n - 1)];
        int sp = walk_begin(S.walk, N, C, nl, level, idx, c == 0 ? (int)min((uint32_t)kLeaf, n - t0) : 0,
                            S.at, lane);
        const TargetBox tb = S.walk.chain[0];
        LocalSum sum{};
        int nfar = 0, nnear = 0, nmid = 0;
        while (sp > 0) {
            uint32_t id;
            const int kind = walk_step(S.walk, N, C, nl, sp, id, lane);
            int cnt;
            int at = warp_place(kind == kWalkFar, lane, cnt);
            if (kind == kWalkFar) S.far[nfar + at] = id;
            nfar += cnt;
            if (row_out) {
                at = warp_place(kind == kWalkNear, lane, cnt);
                if (kind == kWalkNear && nnear + at < kNearRow) row_out->id[nnear + at] = id;
                nnear += cnt;
                at = warp_place(kind == kWalkMid, lane, cnt);
                if (kind == kWalkMid && nmid + at < kNearRow) row_out->id[kNearRow - 1 - (nmid + at)] = id;
                nmid += cnt;
            }
            __syncwarp();
            while (nfar >= kBatch || (sp == 0 && nfar > 0)) {  // from the list's end
                const int m = min(kBatch, nfar);
                nfar -= m;
                translate(N, A, C, S.far + nfar, m, tb, mat, S.buf, lane, sum);
            }
        }
        const Cplx b = local_total(sum, lane);
        if (lane < kTerms)
            loc[(e.noff + node_level(C, level) + idx) * kTerms + lane] = make_double2(b.x, b.y);
        if (row_out && lane == 0) {
            const bool fits = nnear + nmid <= kNearRow;
            row_out->nnear = fits ? (uint32_t)nnear : kNearOver;
            row_out->nmid = (uint32_t)nmid;
        }
    }
}

// Near pairs, and the sum of everything: one block per leaf of 64 targets, taken
// from a counter.  The list's entries go to kNearSlots partial sums by their place
// in it (a warp serves several slots in turn), which are added in slot order.
// The local expansions of the leaf's chain are evaluated at the targets at the
// end.
//
// Measured (B200, wake of 2^20 blobs, sigma 0.0169): the whole velocity call
// 1.87 ms, of which this kernel 1.18, k_far 0.36 and k_tree 0.17, against
// 215 ms for all pairs in mutual FP32x2 tiles at 80 % of the FP32 peak.  Relative
// L2 error against FP64 1.3e-7 (all pairs: 5.7e-7 to 7.6e-7) at 2^18.  At 2^18
// the MUFU pipe is 60 % and the FMA pipe 53 % busy, issue 57 %: latency bounds
// it (6 blocks per SM at 80 registers were no faster at 2^20 and slower below).
//
// WARPS does not change a result; few leaves take eight, so that a leaf's chain of
// near sums is half as long (k_far and this kernel, 5003 blobs: 78 -> 60 us; 20 k:
// 118 -> 86).
template <int WARPS>
struct NearShared {
    StagedLeaf src[WARPS];
    Cplx buf[WARPS][kTerms];
    double2 at[kLeaf];
    double2 sum[kNearSlots][kLeaf];
    uint32_t near[kNearRow], mid[kNearRow];
    TreeWalk walk;  // for rows that overflowed
    int count[2], more;
};

template <int WARPS>
__global__ void __launch_bounds__(32 * WARPS, kNearThreads / (32 * WARPS))
    k_self_f32(const InstDesc* __restrict__ table, const InstState* __restrict__ st,
               const ListEntry* __restrict__ list, int nlist, const double2* __restrict__ pxz,
               const float4* __restrict__ pf, const uint32_t* __restrict__ perm,
               const TreeNode* __restrict__ nodes, const double2* __restrict__ mom,
               const double2* __restrict__ loc, const NearRow* __restrict__ near,
               double* __restrict__ dry_u, double* __restrict__ dry_w,
               unsigned* __restrict__ work) {
    __shared__ unsigned s_pre[kMaxList + 1];
    __shared__ NearShared<WARPS> S;
    __shared__ unsigned s_item;
    list_prefix(s_pre, nlist, [&](int k) { return (st[list[k].inst].n + kLeaf - 1) / kLeaf; });
    const unsigned total = s_pre[nlist];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    for (;;) {
        __syncthreads();
        if (tid == 0) s_item = atomicAdd(work, 1u);
        __syncthreads();
        const unsigned item = s_item;
        if (item >= total) break;
        const int k = locate(s_pre, nlist, item);
        const ListEntry e = list[k];
        const uint32_t n = st[e.inst].n, C = e.cap / kLeaf;
        const uint32_t nl = (n + kLeaf - 1) / kLeaf, leaf = item - s_pre[k];
        const TreeNode* __restrict__ N = nodes + e.noff;
        const double2* __restrict__ X = pxz + e.coff;
        const float4* __restrict__ F = pf + e.coff;
        const uint32_t t0 = leaf * kLeaf;
        const int nchain = chain_length(nl), nt = (int)min((uint32_t)kLeaf, n - t0);
        const NearRow& R = near[e.coff / kLeaf + leaf];
        const bool over = R.nnear == kNearOver;
        const double2 o = X[t0];  // FP32 offsets from the leaf's first blob
        uint64_t tx2[2], tz2[2];
#pragma unroll
        for (int t = 0; t < 2; ++t) {
            const uint32_t i = t0 + t * 32 + lane;
            float x = 0.0f, z = 0.0f;  // padding targets sit on the origin
            if (i < n) {
                const double2 p = X[i];
                x = (float)(p.x - o.x);
                z = (float)(p.y - o.y);
            }
            tx2[t] = f2pack(x, x);
            tz2[t] = f2pack(z, z);
        }
        if (tid < kLeaf) S.at[tid] = X[min(t0 + tid, n - 1)];
        for (int q = tid; q < kNearSlots * kLeaf; q += 32 * WARPS)
            S.sum[q / kLeaf][q % kLeaf] = make_double2(0.0, 0.0);
        TargetBox tb = target_box(N[leaf]);
        const double nr = fmin(leaf > 0 ? N[leaf - 1].R : DBL_MAX,
                               leaf + 1 < nl ? N[leaf + 1].R : DBL_MAX);
        if (tb.R > kStray * nr) tb.R = DBL_MAX;  // (only `wide` below reads it)
        int sp = 0;
        if (over) {
            __syncthreads();  // S.at is complete
            if (wid == 0) sp = walk_begin(S.walk, N, C, nl, 0, leaf, nt, S.at, lane);
        } else {
            const uint32_t a = R.nnear, m = R.nmid;
            for (uint32_t q = tid; q < a; q += 32 * WARPS) S.near[q] = R.id[q];
            for (uint32_t q = tid; q < m; q += 32 * WARPS) S.mid[q] = R.id[kNearRow - 1 - q];
            if (tid == 0) {
                S.count[0] = (int)a;
                S.count[1] = (int)m;
                S.more = 0;
            }
        }
        for (;;) {
            if (over && wid == 0) {  // the next part of the walk
                int a = 0, m = 0;
                while (sp > 0 && max(a, m) + 32 <= kNearRow) {
                    uint32_t id;
                    const int kind = walk_step(S.walk, N, C, nl, sp, id, lane);
                    int cnt;
                    int at = warp_place(kind == kWalkNear, lane, cnt);
                    if (kind == kWalkNear) S.near[a + at] = id;
                    a += cnt;
                    at = warp_place(kind == kWalkMid, lane, cnt);
                    if (kind == kWalkMid) S.mid[m + at] = id;
                    m += cnt;
                }
                if (lane == 0) {
                    S.count[0] = a;
                    S.count[1] = m;
                    S.more = sp > 0;
                }
            }
            __syncthreads();
            const int nnear = S.count[0], nmid = S.count[1];
            for (int slot = wid; slot < kNearSlots && slot < max(nnear, nmid); slot += WARPS) {
                double su[2] = {0.0, 0.0}, sw[2] = {0.0, 0.0};
                for (int q = slot; q < nmid; q += kNearSlots) {
                    const uint32_t id = S.mid[q];
                    const uint64_t at = node_level(C, (int)(id >> 27)) + (id & ((1u << 27) - 1));
                    const TreeNode& m = N[at];
                    __syncwarp();
                    if (lane < kTerms) {
                        const double2 v = mom[(e.noff + at) * kTerms + lane];
                        S.buf[wid][lane] = Cplx{v.x, v.y};
                    }
                    __syncwarp();
#pragma unroll
                    for (int t = 0; t < 2; ++t) {
                        const double2 p = S.at[t * 32 + lane];
                        const Cplx f = moment_value(S.buf[wid], exp2_int(m.e), p.x - m.cx, p.y - m.cz);
                        su[t] -= f.y;
                        sw[t] += f.x;
                    }
                }
                for (int q = slot; q < nnear; q += kNearSlots) {
                    const uint32_t sl = S.near[q], j0 = sl * kLeaf;
                    const TreeNode& sm = N[sl];
                    const bool wide = tb.R > kSpread * (sl == leaf ? nr : sm.R);
                    const bool far = box_gap2(sm, tb) > sm.thr * 1.001 + 1e-30;
                    float4 P = make_float4(1e18f, 1e18f, 1e18f, 1e18f);  // padding: far away
                    float4 L = make_float4(0.f, 0.f, 0.f, 0.f);
                    float2 G = make_float2(0.f, 0.f), T = make_float2(-1.f, -1.f), V = G;
                    const uint32_t ja = j0 + 2 * lane, jb = ja + 1;
                    if (ja < n) {
                        const double2 p = X[ja];
                        const float4 f = F[ja];
                        split_hi_lo(p.x - o.x, P.x, L.x);
                        split_hi_lo(p.y - o.y, P.z, L.z);
                        G.x = f.x;
                        T.x = f.y;
                        V.x = f.z;
                    }
                    if (jb < n) {
                        const double2 p = X[jb];
                        const float4 f = F[jb];
                        split_hi_lo(p.x - o.x, P.y, L.y);
                        split_hi_lo(p.y - o.y, P.w, L.w);
                        G.y = f.x;
                        T.y = f.y;
                        V.y = f.z;
                    }
                    StagedLeaf& w = S.src[wid];
                    __syncwarp();
                    w.pos[lane] = P;
                    w.gam[lane] = G;
                    w.thr[lane] = T;
                    w.rs[lane] = V;
                    if (wide) w.low[lane] = L;
                    __syncwarp();
                    uint64_t nu2[2] = {0ull, 0ull}, w2[2] = {0ull, 0ull};
                    if (wide) {
                        uint64_t lx2[2], lz2[2];
#pragma unroll
                        for (int t = 0; t < 2; ++t) {
                            const double2 p = S.at[t * 32 + lane];
                            float h, lo;
                            split_hi_lo(p.x - o.x, h, lo);
                            lx2[t] = f2pack(lo, lo);
                            split_hi_lo(p.y - o.y, h, lo);
                            lz2[t] = f2pack(lo, lo);
                        }
                        if (sl != leaf) leaf_sum<1, true>(w, tx2, tz2, lx2, lz2, nu2, w2);
                        else leaf_sum<2, true>(w, tx2, tz2, lx2, lz2, nu2, w2);
                    } else if (far) {
                        leaf_sum<0, false>(w, tx2, tz2, tx2, tz2, nu2, w2);
                    } else if (sl != leaf) {
                        leaf_sum<1, false>(w, tx2, tz2, tx2, tz2, nu2, w2);
                    } else {
                        leaf_sum<2, false>(w, tx2, tz2, tx2, tz2, nu2, w2);
                    }
                    float fu[2], fw[2], bad = 0.0f;  // (NaN where a sum is not finite)
#pragma unroll
                    for (int t = 0; t < 2; ++t) {
                        fu[t] = f2lo(nu2[t]) + f2hi(nu2[t]);
                        fw[t] = f2lo(w2[t]) + f2hi(w2[t]);
                        bad = fmaf(fu[t], 0.0f, fmaf(fw[t], 0.0f, bad));
                    }
                    if (bad == 0.0f) {
#pragma unroll
                        for (int t = 0; t < 2; ++t) {
                            su[t] += (double)fu[t];
                            sw[t] += (double)fw[t];
                        }
                    } else {
                        leaf_sum_close(X, F, j0, min(n, j0 + kLeaf), S.at[lane], su[0], sw[0]);
                        leaf_sum_close(X, F, j0, min(n, j0 + kLeaf), S.at[32 + lane], su[1], sw[1]);
                    }
                }
#pragma unroll
                for (int t = 0; t < 2; ++t) {  // only this warp touches the slot
                    double2& v = S.sum[slot][t * 32 + lane];
                    v.x += su[t];
                    v.y += sw[t];
                }
            }
            const int more = S.more;
            __syncthreads();
            if (!more) break;
        }
        for (int q = tid; q < nchain * kTerms; q += 32 * WARPS) {
            const int c = q / kTerms, up = kFarStep * c;
            const double2 v = loc[(e.noff + node_level(C, up) + (leaf >> up)) * kTerms + q % kTerms];
            S.buf[c][q % kTerms] = Cplx{v.x, v.y};
        }
        __syncthreads();
        if (tid < nt) {
            const double2 p = S.at[tid];
            double nu = 0.0, w = 0.0;
            for (int c = 0; c < nchain; ++c) {
                const TreeNode& t = N[node_level(C, kFarStep * c) + (leaf >> (kFarStep * c))];
                const Cplx f = local_value(S.buf[c], p.x - t.cx, p.y - t.cz, t.e);
                nu -= f.y;
                w += f.x;
            }
            for (int q = 0; q < kNearSlots; ++q) {
                nu += S.sum[q][tid].x;
                w += S.sum[q][tid].y;
            }
            const double u = -nu * kRpi2;
            w *= kRpi2;
            const uint32_t i = t0 + tid;
            if (dry_u) {  // timing runs leave the simulations alone
                dry_u[e.coff + i] = u;
                dry_w[e.coff + i] = w;
            } else {
                const InstDesc& d = table[e.inst];
                const uint32_t g = perm[e.coff + i];
                d.u[g] = u;
                d.w[g] = w;
            }
        }
    }
}
static_assert(kChainMax <= 4, "a chain's expansions fit the warps' buffers");

// ---- FP64 pairs ---------------------------------------------------------------
// 1 / v in FP64: the hardware's approximation (about 20 bits) and two steps of
// Newton's iteration y += y (1 - v y), each error the square of the one before;
// the last step's rounding is all that is left (within one ulp; an IEEE
// reciprocal takes three times the instructions).  For v in [1e-290, 1e290].
__device__ __forceinline__ double rcp_newton(double v) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(v));
    y = fma(y, fma(-v, y, 1.0), y);
    return fma(y, fma(-v, y, 1.0), y);
}

// K(r2) of src/VelocityKernel.cpp:51-57 with rs = 1 / sigma^2, thr = 10 sigma^2; a division
// where the iteration has no range (zero, infinite, NaN or near the ends of the
// exponents: below 5.6e-309 a reciprocal overflows and would make NaN of a core's 0).
// Called, not inlined: with it in line, or a test of the common path's result, a probe of
// 3001 points and 60 k blobs takes 430 us instead of 400 (an IEEE reciprocal in line 418),
// velocities of 40 k blobs 1515 instead of 1481 (1511).
__device__ __noinline__ double kernel_f64_any(double r2, double thr, double rs) {
    return ddiv(r2 < thr ? dsub(1.0, exp(dmul(-r2, rs))) : 1.0, r2);
}
__device__ __forceinline__ double kernel_f64(double r2, double thr, double rs) {
    const unsigned h = (unsigned)__double2hiint(r2);
    if (h - 0x03d00000u >= 0x78000000u) return kernel_f64_any(r2, thr, rs);
    const double y = rcp_newton(r2);
    return r2 < thr ? dmul(dsub(1.0, exp(dmul(-r2, rs))), y) : y;
}

// Every pair, over the 256-blob tiles of the sorted order; each pair is the
// reference's formula (src/VelocityKernel.cpp:44-60) in FP64.  A source stage
// whose tile box is beyond 10 sigma^2 of the target tile's box holds no core pair
// and no self pair, and runs the 1/r^2 branch without the per-pair test.
//
// The FP64 pipe bounds it (64 lanes per clock and SM): 12 operations per far
// pair, where an IEEE reciprocal and unfused products took 27; 72 % busy at 40 k.  A work item is one
// tile of targets (two per thread) against one source chunk; chunks are as
// short as leaves a single simulation about five rounds of blocks
// (nbody_chunks).  Measured (whole call): 40 k blobs 2.55 -> 1.52 ms, 262 k 75 -> 51,
// 5003 blobs 0.64 -> 0.16 (before: items of 1024 targets, at least 256 sources).
constexpr int kF64Threads = 128;
constexpr int kF64Ctas = 6;
__global__ void __launch_bounds__(kF64Threads, kF64Ctas)
    k_self_f64(const InstState* __restrict__ st, const ListEntry* __restrict__ list, int nlist,
               const double4* __restrict__ packed, const TileMeta* __restrict__ meta,
               double2* __restrict__ part, unsigned* __restrict__ work) {
    static_assert(2 * kF64Threads == kBsST, "a work item's targets are one sort tile");
    __shared__ unsigned s_pre[kMaxList + 1];
    __shared__ double4 s_src[kBsST];  // x, z, circ, threshold
    __shared__ double s_rs[kBsST];
    __shared__ unsigned s_item;
    list_prefix(s_pre, nlist, [&](int k) {
        const uint32_t n = st[list[k].inst].n;
        return (n + kBsST - 1) / kBsST * chunk_count(n, list[k].chunks);
    });
    const unsigned total = s_pre[nlist];
    const int tid = threadIdx.x;
    for (;;) {
        if (tid == 0) s_item = atomicAdd(work, 1u);
        __syncthreads();
        const unsigned item = s_item;
        __syncthreads();
        if (item >= total) break;
        const int k = locate(s_pre, nlist, item);
        const ListEntry e = list[k];
        const uint32_t n = st[e.inst].n;
        const unsigned local = item - s_pre[k], chunks = chunk_count(n, e.chunks);
        const uint32_t tile = local / chunks, c = local % chunks;
        const uint32_t cs = chunk_size(n, e.chunks);
        const uint32_t j0 = c * cs, j1 = min(n, j0 + cs);
        const double4* __restrict__ P = packed + e.coff;
        const TileMeta tm = meta[(e.coff + (uint64_t)tile * kBsST) / kBsST];
        const uint32_t tb = tile * kBsST + tid;
        double tx[2], tz[2], uu[2], ww[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const uint32_t t = tb + r * kF64Threads;
            const double4 p = t < n ? P[t] : make_double4(0, 0, 0, 1);
            tx[r] = p.x;
            tz[r] = p.y;
            uu[r] = ww[r] = 0.0;
        }
        for (uint32_t s0 = j0; s0 < j1;) {
            const int cnt = (int)min((uint32_t)kBsST - s0 % kBsST, j1 - s0);  // within one tile
            const TileMeta& m = meta[(e.coff + s0) / kBsST];
            const double gx = fmax(0.0, fmax(m.xmin - tm.xmax, tm.xmin - m.xmax));
            const double gz = fmax(0.0, fmax(m.zmin - tm.zmax, tm.zmin - m.zmax));
            const double ex = fmax(m.xmax, tm.xmax) - fmin(m.xmin, tm.xmin);
            const double ez = fmax(m.zmax, tm.zmax) - fmin(m.zmin, tm.zmin);
            // (the last: every r^2 of the stage is in rcp_newton's range)
            const bool far = gx * gx + gz * gz > m.thr * 1.001 + 1e-30 && ex * ex + ez * ez < 1e290;
            __syncthreads();
            for (int q = tid; q < cnt; q += kF64Threads) {
                const double4 p = P[s0 + q];
                const double s2 = dmul(p.w, p.w);
                s_src[q] = make_double4(p.x, p.y, p.z, dmul(10.0, s2));
                if (!far) s_rs[q] = ddiv(1.0, s2);
            }
            __syncthreads();
            if (far) {
#pragma unroll 4
                for (int jj = 0; jj < cnt; ++jj) {
                    const double4 sj = s_src[jj];
#pragma unroll
                    for (int r = 0; r < 2; ++r) {
                        const double dx = dsub(tx[r], sj.x), dz = dsub(tz[r], sj.y);
                        const double g = dmul(rcp_newton(fma(dx, dx, dmul(dz, dz))), sj.z);
                        uu[r] = fma(-g, dz, uu[r]);
                        ww[r] = fma(g, dx, ww[r]);
                    }
                }
            } else {
                for (int jj = 0; jj < cnt; ++jj) {
                    const double4 sj = s_src[jj];
#pragma unroll
                    for (int r = 0; r < 2; ++r) {
                        if (tb + r * kF64Threads == s0 + jj) continue;  // i != j (src/VelocityKernel.cpp:43)
                        const double dx = dsub(tx[r], sj.x), dz = dsub(tz[r], sj.y);
                        const double K = kernel_f64(fma(dx, dx, dmul(dz, dz)), sj.w, s_rs[jj]);
                        const double g = dmul(K, sj.z);
                        uu[r] = fma(-g, dz, uu[r]);
                        ww[r] = fma(g, dx, ww[r]);
                    }
                }
            }
            s0 += cnt;
        }
        double2* __restrict__ out = part + e.poff + (uint64_t)c * e.cap;
#pragma unroll
        for (int r = 0; r < 2; ++r)
            if (tb + r * kF64Threads < n) out[tb + r * kF64Threads] = make_double2(uu[r], ww[r]);
    }
}

// FP64 path, per blob: the chunk partials in chunk order, scaled by 1/(2 pi),
// scattered to blob order.
__global__ void k_self_combine(const InstDesc* __restrict__ table,
                               const InstState* __restrict__ st,
                               const ListEntry* __restrict__ list, int nlist,
                               const uint32_t* __restrict__ perm,
                               const double2* __restrict__ part) {
    __shared__ unsigned s_pre[kMaxList + 1];
    list_prefix(s_pre, nlist,
                [&](int k) { return (st[list[k].inst].n + blockDim.x - 1) / blockDim.x; });
    const unsigned total = s_pre[nlist];
    for (unsigned item = blockIdx.x; item < total; item += gridDim.x) {
        const int k = locate(s_pre, nlist, item);
        const ListEntry e = list[k];
        const uint32_t n = st[e.inst].n;
        const uint32_t t = (item - s_pre[k]) * blockDim.x + threadIdx.x;
        if (t >= n) continue;
        double su = 0.0, sw = 0.0;
        const uint32_t chunks = chunk_count(n, e.chunks);
#pragma unroll 4
        for (uint32_t c = 0; c < chunks; ++c) {
            const double2 v = part[e.poff + (uint64_t)c * e.cap + t];
            su += v.x;
            sw += v.y;
        }
        const InstDesc& d = table[e.inst];
        const uint32_t p = perm[e.coff + t];
        d.u[p] = su * kRpi2;
        d.w[p] = sw * kRpi2;
    }
}

// ---- arbitrary targets --------------------------------------------------------
// One item = (job, a tile of 256 targets, a chunk of `chunk` sources: at_chunk(...)
// for at-target calls, rhs_chunk_for(...) for a simulation's right-hand side).
struct AtJob {
    const double* tx;
    const double* tz;
    uint32_t nt;
    int skip_close;  // 1: pairs with r2 <= 1e-15 skipped (computeInducedAt)
    const double* sx;
    const double* sz;
    const double* sc;
    const double* ss;
    const uint32_t* pns;  // source count on the device, or null -> ns
    uint32_t ns;
    int npad;             // partial row length
    uint32_t chunk;       // sources per work item (64, 128 or a multiple of 256)
    double2* part;        // [chunk][npad]
    double* circ_part;    // [chunk], or null
};

// Kahan sum of packed pairs with the compensation kept negated (e = -c):
// y = x + e, t = s + y, e = y - (t - s), s = t -- each half the scalar
// algorithm; x = a b enters through one fused multiply-add.
__device__ __forceinline__ void kahan2_fma(uint64_t& s, uint64_t& e, uint64_t a, uint64_t b) {
    const uint64_t y = f2fma(a, b, e);
    const uint64_t t = f2add(s, y);
    e = f2sub(y, f2sub(t, s));
    s = t;
}

// Velocity at targets from a chunk of J.chunk sources per work item, 256
// targets per item, one per thread.
//
// FP32 jobs pack two SOURCES per FP32x2 instruction, so no lane idles however few
// targets a job has.  Offsets are formed without per-pair conversions: every
// position is taken relative to the tile's origin (its first finite target) in FP64
// and split into an FP32 pair, hi of 16 bits and lo = the remainder (40 bits
// together); dx = (t_hi - s_hi) + (t_lo - s_lo), where the first difference is exact
// unless one position is 2^8 times farther out than the other, so dx is rounded
// once (hi of 24 bits rounds it twice: error against 64 bits 4 % up, this 7 % down
// against FP64 differences rounded once).  40 bits are not enough for a pair much
// closer than its distance from the origin: below kSplitClose of that distance (where
// the split's own error is 3e-8 at most) dx and dz come from the FP64 positions.
// Targets need not lie together, so a tile may span everything; without this
// offsets of 1e-4 were off by 3e-7 to 1.8e-5 at 10 to 1000 from the origin.
// Each pair keeps its compensated update (the right-hand side is the small residual
// normal velocity, so its rounding must stay relative to the few large near-blob
// terms, not compound): one Kahan sum per half, the halves added at the end.  The
// core kernel runs for both halves when any lane of the warp has a pair inside a
// core.  Sources are staged as packed pairs (two 16-byte loads bring positions, two
// more the circulations and core constants).  Where close pairs are skipped, a pair
// with not r2 > 1e-15 (NaN included) adds nothing.
constexpr double kSplitClose = 1.0 / 8192.0;
__device__ __forceinline__ void split_16(double v, float& hi, float& lo) {
    const float f = (float)v;
    if (!(fabsf(f) <= FLT_MAX)) {  // infinite or NaN: all of it
        hi = f;
        lo = 0.0f;
        return;
    }
    hi = __int_as_float((__float_as_int(f) + 0x80) & ~0xFF);
    lo = (float)(v - (double)hi);
}
// Squared distance below which a target's pairs need FP64 offsets; dx, dz: from the
// origin.  A source's, twice over, is above that of any target it is so close to, so
// the larger of it and 10 sigma^2 settles for most pairs with one comparison that
// neither matters (comparisons of their own: 4 % of the call).
__device__ __forceinline__ float split_close2(double dx, double dz) {
    return (float)(fma(dx, dx, dz * dz) * (kSplitClose * kSplitClose));
}
__device__ __forceinline__ float look_closer2(double dx, double dz, float thr) {
    return fmaxf(thr, 2.0f * split_close2(dx, dz));
}
// The pair loops' r2 of one source (hi, lo: its entries of AtStage, z two further on),
// bit for bit.
__device__ __forceinline__ float split_dist2(float txh, float txl, float tzh, float tzl, const float* hi,
                                             const float* lo) {
    const float dx = __fadd_rn(__fsub_rn(txh, hi[0]), __fsub_rn(txl, lo[0]));
    const float dz = __fadd_rn(__fsub_rn(tzh, hi[2]), __fsub_rn(tzl, lo[2]));
    return __fmaf_rn(dx, dx, __fmul_rn(dz, dz));
}
// One pair from its FP64 offsets, added to half h of the packed sums; the caller's own
// term for it is zero.
__device__ __forceinline__ void close_pair(double ddx, double ddz, float rs, float thr, float circ, int h,
                                           bool skip, uint64_t& snu, uint64_t& enu, uint64_t& sw,
                                           uint64_t& ew) {
    const float dx = (float)ddx, dz = (float)ddz, r2 = fmaf(dx, dx, dz * dz);
    if (skip && !(r2 > 1e-15f)) return;
    float k = rcp_approx(r2);
    if (r2 < thr) k = core_kernel_expm1(r2, rs, k);
    const float g = k * circ;
    const uint64_t G = h ? f2pack(0.0f, g) : f2pack(g, 0.0f);
    kahan2_fma(snu, enu, G, f2pack(dz, dz));
    kahan2_fma(sw, ew, G, f2pack(dx, dx));
}
struct AtStage {
    float4 pos_hi[128];  // (x_hi a, x_hi b, z_hi a, z_hi b) of sources 2i, 2i+1
    float4 pos_lo[128];  // (x_lo a, x_lo b, z_lo a, z_lo b)
    float4 cst[128];     // (circ a, circ b, squared distance a, b below which to look closer)
    float4 core[128];    // (1/sigma^2 a, 1/sigma^2 b, 10 sigma^2 a, 10 sigma^2 b)
};

// (FP32: three blocks fit an SM by themselves, but told so the compiler's loop is 4 %
// faster: 256 targets against 2^20 sources 288 us, 300.  FP64: four, at 64 registers; at 68
// a probe of 3001 points and 60 k blobs took 478 us instead of 416, before kernel_f64_any)
template <bool F32>
__global__ void __launch_bounds__(256, F32 ? 3 : 4) k_at(const AtJob* __restrict__ jobs, int njobs) {
    __shared__ unsigned s_pre[kMaxList + 1];
    // FP64: x, z, circ, 10 sigma^2 and 1 / sigma^2; FP32: packed pairs
    __shared__ union Stage {
        struct {
            double4 src[256];
            double rs[256];
        } d;
        AtStage f;
        __device__ Stage() {}
    } S;
    __shared__ double s_red[8];
    list_prefix(s_pre, njobs, [&](int k) {
        const uint32_t ns = jobs[k].pns ? *jobs[k].pns : jobs[k].ns;
        return ((jobs[k].nt + 255) / 256) * ((ns + jobs[k].chunk - 1) / jobs[k].chunk);
    });
    const unsigned total = s_pre[njobs];
    for (unsigned item = blockIdx.x; item < total; item += gridDim.x) {
        const int k = locate(s_pre, njobs, item);
        const AtJob J = jobs[k];
        const bool skip = J.skip_close != 0;
        const uint32_t ns = J.pns ? *J.pns : J.ns;
        const uint32_t nchunk = (ns + J.chunk - 1) / J.chunk;
        const unsigned local = item - s_pre[k];
        const uint32_t ttile = local / nchunk, c = local % nchunk;
        const uint32_t t = ttile * 256 + threadIdx.x;
        const double tx = t < J.nt ? J.tx[t] : 0.0, tz = t < J.nt ? J.tz[t] : 0.0;
        uint32_t o = ttile * 256;  // the tile's origin (block-uniform)
        if (F32)
            while (o + 1 < min(J.nt, ttile * 256 + 256) && !(isfinite(J.tx[o]) && isfinite(J.tz[o]))) ++o;
        const double ox = J.tx[o], oz = J.tz[o];
        float txh, txl, tzh, tzl;
        split_16(tx - ox, txh, txl);
        split_16(tz - oz, tzh, tzl);
        const uint64_t TXH = f2pack(txh, txh), TXL = f2pack(txl, txl);
        const uint64_t TZH = f2pack(tzh, tzh), TZL = f2pack(tzl, tzl);
        const float close2 = split_close2(tx - ox, tz - oz);
        const uint32_t j0 = c * J.chunk, j1 = min(ns, j0 + J.chunk);
        double uu = 0.0, ww = 0.0, csum = 0.0;
        const uint64_t zero2 = f2pack(0.0f, 0.0f);
        uint64_t snu = zero2, enu = zero2, sw = zero2, ew = zero2;  // -u and w, packed Kahan
        for (uint32_t s0 = j0; s0 < j1; s0 += 256) {
            __syncthreads();
            const uint32_t j = s0 + threadIdx.x;
            if (F32) {
                // slot (pair i = tid / 2, half h = tid % 2); a slot past the
                // chunk holds a far, circulation-free source (it adds 0)
                float xh = 1.0e18f, xl = 0.f, zh = 0.f, zl = 0.f, cf = 0.f, thr = 0.f, rsf = 0.f, look = 0.f;
                if (j < j1) {
                    const double sg = J.ss[j];
                    const double s2 = dmul(sg, sg);
                    split_16(J.sx[j] - ox, xh, xl);
                    split_16(J.sz[j] - oz, zh, zl);
                    cf = (float)J.sc[j];
                    thr = (float)dmul(10.0, s2);
                    rsf = (float)ddiv(1.0, s2);
                    look = look_closer2(J.sx[j] - ox, J.sz[j] - oz, thr);
                    if (ttile == 0) csum += J.sc[j];
                }
                const int i = threadIdx.x >> 1, h = threadIdx.x & 1;
                float* ph = reinterpret_cast<float*>(&S.f.pos_hi[i]);
                float* pl = reinterpret_cast<float*>(&S.f.pos_lo[i]);
                float* pc = reinterpret_cast<float*>(&S.f.cst[i]);
                float* pr = reinterpret_cast<float*>(&S.f.core[i]);
                ph[h] = xh;
                ph[2 + h] = zh;
                pl[h] = xl;
                pl[2 + h] = zl;
                pc[h] = cf;
                pc[2 + h] = look;
                pr[h] = rsf;
                pr[2 + h] = thr;
            } else if (j < j1) {
                const double sg = J.ss[j];
                const double s2 = dmul(sg, sg);
                S.d.src[threadIdx.x] = make_double4(J.sx[j], J.sz[j], J.sc[j], dmul(10.0, s2));
                S.d.rs[threadIdx.x] = ddiv(1.0, s2);
                if (ttile == 0) csum += J.sc[j];
            }
            __syncthreads();
            const int cnt = (int)min(256u, j1 - s0);
            if (F32) {
                int first = 256, last = -1;  // of the pairs with a source that is too close
#pragma unroll 4
                for (int i = 0; i < (cnt + 1) / 2; ++i) {
                    const float4 H = S.f.pos_hi[i], L = S.f.pos_lo[i], Cs = S.f.cst[i];
                    uint64_t DX = f2add(f2sub(TXH, f2pack(H.x, H.y)), f2sub(TXL, f2pack(L.x, L.y)));
                    uint64_t DZ = f2add(f2sub(TZH, f2pack(H.z, H.w)), f2sub(TZL, f2pack(L.z, L.w)));
                    const uint64_t R2 = f2fma(DX, DX, f2mul(DZ, DZ));
                    const float ra = f2lo(R2), rb = f2hi(R2);
                    float ka = rcp_approx(ra), kb = rcp_approx(rb);
                    if (__any_sync(0xffffffffu, ra < Cs.z || rb < Cs.w)) {
                        const float4 R = S.f.core[i];
                        const bool ca = ra < R.z, cb = rb < R.w;
                        const float qa = core_kernel_expm1(ra, R.x, ka);
                        const float qb = core_kernel_expm1(rb, R.y, kb);
                        ka = ca ? qa : ka;
                        kb = cb ? qb : kb;
                        if (fminf(ra, rb) < close2) {  // left to the loop below
                            ka = ra < close2 ? 0.0f : ka;
                            kb = rb < close2 ? 0.0f : kb;
                            first = min(first, i);
                            last = i;
                        }
                    }
                    if (skip) {  // computeInducedAt (src/VelocityKernel.cpp:89)
                        const bool oa = ra > 1e-15f, ob = rb > 1e-15f;
                        ka = oa ? ka : 0.f;
                        kb = ob ? kb : 0.f;
                        DX = f2pack(oa ? f2lo(DX) : 0.f, ob ? f2hi(DX) : 0.f);
                        DZ = f2pack(oa ? f2lo(DZ) : 0.f, ob ? f2hi(DZ) : 0.f);
                    }
                    const uint64_t G = f2mul(f2pack(ka, kb), f2pack(Cs.x, Cs.y));
                    kahan2_fma(snu, enu, G, DZ);
                    kahan2_fma(sw, ew, G, DX);
                }
#pragma unroll 1
                for (int h = 2 * first; h < min(2 * last + 2, cnt); ++h) {
                    const float* hi = reinterpret_cast<const float*>(&S.f.pos_hi[h >> 1]) + (h & 1);
                    const float* lo = reinterpret_cast<const float*>(&S.f.pos_lo[h >> 1]) + (h & 1);
                    const float* co = reinterpret_cast<const float*>(&S.f.core[h >> 1]) + (h & 1);
                    if (split_dist2(txh, txl, tzh, tzl, hi, lo) < close2)
                        close_pair(tx - J.sx[s0 + h], tz - J.sz[s0 + h], co[0], co[2],
                                   reinterpret_cast<const float*>(&S.f.cst[h >> 1])[h & 1], h & 1, skip, snu,
                                   enu, sw, ew);
                }
            } else {
                for (int jj = 0; jj < cnt; ++jj) {
                    const double4 sj = S.d.src[jj];
                    const double dx = dsub(tx, sj.x), dz = dsub(tz, sj.y);
                    const double r2 = fma(dx, dx, dmul(dz, dz));
                    if (skip && !(r2 > 1e-15)) continue;
                    const double g = dmul(kernel_f64(r2, sj.w, S.d.rs[jj]), sj.z);
                    uu = fma(-g, dz, uu);
                    ww = fma(g, dx, ww);
                }
            }
        }
        if (F32) {
            uu = -(((double)f2lo(snu) + (double)f2lo(enu)) + ((double)f2hi(snu) + (double)f2hi(enu)));
            ww = ((double)f2lo(sw) + (double)f2lo(ew)) + ((double)f2hi(sw) + (double)f2hi(ew));
        }
        if (t < J.nt) J.part[(uint64_t)c * J.npad + t] = make_double2(uu, ww);
        if (ttile == 0 && J.circ_part) {
            for (int o = 16; o > 0; o >>= 1) csum += __shfl_xor_sync(0xffffffffu, csum, o);
            if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = csum;
            __syncthreads();
            if (threadIdx.x == 0) {
                double a = 0.0;
                for (int q = 0; q < 8; ++q) a += s_red[q];
                J.circ_part[c] = a;
            }
        }
    }
}

// Sums a job's chunk partials: a block finishes 32 targets, warp w adding chunks
// w, w + W, ... for its lane's target and the W warp sums added in warp order.
__global__ void __launch_bounds__(1024) k_at_combine(const AtJob* __restrict__ jobs,
                                                     double* __restrict__ u,
                                                     double* __restrict__ w) {
    __shared__ double2 s_sum[32][32];
    const AtJob J = jobs[0];
    const uint32_t ns = J.pns ? *J.pns : J.ns;
    const uint32_t nchunk = (ns + J.chunk - 1) / J.chunk;
    const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5, warps = blockDim.x >> 5;
    for (uint32_t t0 = blockIdx.x * 32; t0 < J.nt; t0 += gridDim.x * 32) {
        const uint32_t t = t0 + lane;
        double su = 0.0, sw = 0.0;
        if (t < J.nt) {
#pragma unroll 4
            for (uint32_t c = wid; c < nchunk; c += warps) {
                const double2 v = J.part[(uint64_t)c * J.npad + t];
                su += v.x;
                sw += v.y;
            }
        }
        s_sum[wid][lane] = make_double2(su, sw);
        __syncthreads();
        if (wid == 0 && t < J.nt) {
            for (uint32_t q = 1; q < warps; ++q) {
                su += s_sum[q][lane].x;
                sw += s_sum[q][lane].y;
            }
            u[t] = su * kRpi2;
            w[t] = sw * kRpi2;
        }
        __syncthreads();
    }
}

// b_i = (Ux + u_i) enx_i + (Uz + w_i) enz_i, b_np = -sum(circ)
// (src/VortexSheet.cpp:206-210).  Block (x, k) finishes targets 32x .. 32x+31
// of simulation k: warp w sums chunks w, w + 8, ... for its lane's target and
// the eight warp sums are added in warp order; block x = 0 also sums the
// Kelvin row's circulation partials (thread t takes chunks t, t + 256, ...,
// then a fixed shuffle tree and the warp sums in order).  The order depends
// only on the simulation's chunk count, never on the batch.
__global__ void __launch_bounds__(256) k_rhs_combine(const InstDesc* __restrict__ table,
                                                     InstState* __restrict__ st,
                                                     const ListEntry* __restrict__ list,
                                                     const AtJob* __restrict__ jobs) {
    __shared__ double s_u[8][32], s_w[8][32], s_c[8];
    const int k = blockIdx.y;
    const ListEntry e = list[k];
    const InstDesc& d = table[e.inst];
    const AtJob J = jobs[k];
    const uint32_t ns = st[e.inst].n;
    const uint32_t nchunk = (ns + J.chunk - 1) / J.chunk;
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int i = blockIdx.x * 32 + lane;
    const bool targets = (int)(blockIdx.x * 32) < d.np;  // block-uniform
    if (targets) {
        double su = 0.0, sw = 0.0;
        if (i < d.np)
            for (uint32_t c = wid; c < nchunk; c += 8) {
                const double2 v = J.part[(uint64_t)c * J.npad + i];
                su += v.x;
                sw += v.y;
            }
        s_u[wid][lane] = su;
        s_w[wid][lane] = sw;
    }
    __syncthreads();
    if (targets && threadIdx.x < 32 && i < d.np) {
        double su = 0.0, sw = 0.0;
        for (int q = 0; q < 8; ++q) {
            su += s_u[q][lane];
            sw += s_w[q][lane];
        }
        const double ui = dmul(su, kRpi2), wi = dmul(sw, kRpi2);
        d.b[i] = dadd(dmul(dadd(d.ux, ui), d.enx[i]), dmul(dadd(d.uz, wi), d.enz[i]));
    }
    if (blockIdx.x == 0) {  // block-uniform
        double tc = 0.0;
        for (uint32_t c = threadIdx.x; c < nchunk; c += 256) tc += J.circ_part[c];
        for (int o = 16; o > 0; o >>= 1) tc += __shfl_xor_sync(0xffffffffu, tc, o);
        if (lane == 0) s_c[wid] = tc;
        __syncthreads();
        if (threadIdx.x == 0) {
            double a = 0.0;
            for (int q = 0; q < 8; ++q) a += s_c[q];
            d.b[d.np] = -a;
            st[e.inst].totalcirc = a;
        }
    }
}

// The same right-hand side for FP32 simulations, over the tree of the blobs: one
// block per group of 32 collocation points, lane t of every warp at point t (of
// eight points for bodies of up to 128 panels, whose few blocks would otherwise each
// see half of the near leaves: lane t at point t % 8, with every fourth pair of
// sources).
// The tree's top nodes are dealt out to the warps, and each walks its own: far
// nodes are translated, near leaves summed pair by pair as in k_at (offsets in
// two parts, one compensated sum per half), their sums added in FP64; the
// warps' results are added in order.  The circulations' sum is the root's first
// moment.  Depends only on the simulation, never on the batch.
//
// Near leaves go to a queue that all warps share out, or the warps with the
// nearest top nodes would work alone.  Measured (B200, 2^17 blobs, RHS of a step):
// 64, 128, 512, 1024 panels 29, 23, 27, 25 us; without the queue and with 32 points
// per block throughout 142, 109, -, 39; all pairs 72, 70, 87, 129.
constexpr int kRhsWarps = 8;
constexpr int kRhsGroup = 32;
constexpr int kRhsNear = 128;  // near leaves a warp leaves to all; more it sums at once
__host__ __device__ __forceinline__ int rhs_group(int np) { return np <= 128 ? 8 : kRhsGroup; }
struct RhsWarp {
    TreeWalk walk;
    TransBuf buf;
    uint32_t far[kFarList], near[kRhsNear];
    float4 pos_hi[kLeaf / 2], pos_lo[kLeaf / 2];  // (x a, x b, z a, z b) of sources 2i, 2i + 1
    float4 cst[kLeaf / 2], core[kLeaf / 2];       // (as AtStage's)
    double2 sum[kRhsGroup];
};
struct RhsShared {
    RhsWarp w[kRhsWarps];
    double2 at[kRhsGroup];
    int nnear[kRhsWarps];
};
__global__ void __launch_bounds__(32 * kRhsWarps, 2)
    k_rhs_tree(const InstDesc* __restrict__ table, InstState* __restrict__ st,
               const ListEntry* __restrict__ list, const double2* __restrict__ pxz,
               const float4* __restrict__ pf, const TreeNode* __restrict__ nodes,
               const double2* __restrict__ mom) {
    extern __shared__ __align__(16) unsigned char s_raw[];
    RhsShared& S = *reinterpret_cast<RhsShared*>(s_raw);
    const ListEntry e = list[blockIdx.y];
    const InstDesc& d = table[e.inst];
    const int group = rhs_group(d.np), i0 = (int)blockIdx.x * group;
    if (i0 >= d.np) return;  // block-uniform
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const unsigned all = 0xffffffffu;
    RhsWarp& W = S.w[wid];
    const uint32_t n = st[e.inst].n, C = e.cap / kLeaf, nl = (n + kLeaf - 1) / kLeaf;
    const TreeNode* __restrict__ N = nodes + e.noff;
    const double2* __restrict__ A = mom + e.noff * kTerms;
    const double2* __restrict__ X = pxz + e.coff;
    const float4* __restrict__ F = pf + e.coff;
    const int i = min(i0 + (lane & (group - 1)), d.np - 1);
    const double tx = d.xc[i], tz = d.zc[i];
    if (wid == 0) S.at[lane] = make_double2(tx, tz);
    double x0 = tx, x1 = tx, z0 = tz, z1 = tz;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        x0 = fmin(x0, __shfl_xor_sync(all, x0, o));
        x1 = fmax(x1, __shfl_xor_sync(all, x1, o));
        z0 = fmin(z0, __shfl_xor_sync(all, z0, o));
        z1 = fmax(z1, __shfl_xor_sync(all, z1, o));
    }
    TargetBox tb;
    tb.cx = 0.5 * (x0 + x1);
    tb.cz = 0.5 * (z0 + z1);
    tb.hx = 0.5 * (x1 - x0);
    tb.hz = 0.5 * (z1 - z0);
    tb.R = sqrt(tb.hx * tb.hx + tb.hz * tb.hz) * (1.0 + 1e-12);
    tb.e = scale_exp(tb.R);
    tb.n = kRhsGroup;
    tb.at = S.at;
    const double ox = __shfl_sync(all, tx, 0), oz = __shfl_sync(all, tz, 0);  // the group's origin
    float txh, txl, tzh, tzl;
    split_16(tx - ox, txh, txl);
    split_16(tz - oz, tzh, tzl);
    const uint64_t TXH = f2pack(txh, txh), TXL = f2pack(txl, txl);
    const uint64_t TZH = f2pack(tzh, tzh), TZL = f2pack(tzl, tzl);
    const float close2 = split_close2(tx - ox, tz - oz);
    __syncthreads();
    const Binomials mat = binomials(lane);
    LocalSum sum{};              // this warp's share
    double nu = 0.0, sw = 0.0;   // -u and w at the lane's point, near and mid
    auto near_leaf = [&](uint32_t leaf) {  // sums a leaf's pairs with the 32 points
        const uint32_t j0 = leaf * kLeaf;
        // (padding: far away, no circulation)
        float xh[2] = {1e18f, 1e18f}, xl[2] = {0.f, 0.f}, zh[2] = {0.f, 0.f}, zl[2] = {0.f, 0.f};
        float g[2] = {0.f, 0.f}, thr[2] = {0.f, 0.f}, rs[2] = {0.f, 0.f}, look[2] = {0.f, 0.f};
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint32_t j = j0 + 2 * lane + h;
            if (j < n) {
                const double2 p = X[j];
                const float4 f = F[j];
                split_16(p.x - ox, xh[h], xl[h]);
                split_16(p.y - oz, zh[h], zl[h]);
                g[h] = f.x;
                thr[h] = f.y;
                rs[h] = f.z;
                look[h] = look_closer2(p.x - ox, p.y - oz, f.y);
            }
        }
        __syncwarp();
        W.pos_hi[lane] = make_float4(xh[0], xh[1], zh[0], zh[1]);
        W.pos_lo[lane] = make_float4(xl[0], xl[1], zl[0], zl[1]);
        W.cst[lane] = make_float4(g[0], g[1], look[0], look[1]);
        W.core[lane] = make_float4(rs[0], rs[1], thr[0], thr[1]);
        __syncwarp();
        const uint64_t zero2 = f2pack(0.0f, 0.0f);
        uint64_t snu = zero2, enu = zero2, s2 = zero2, e2 = zero2;
        int first = kLeaf, last = -1;  // (as in k_at)
#pragma unroll 4
        for (int q = lane / group; q < kLeaf / 2; q += kRhsGroup / group) {
            const float4 H = W.pos_hi[q], L = W.pos_lo[q], Cs = W.cst[q];
            const uint64_t DX = f2add(f2sub(TXH, f2pack(H.x, H.y)), f2sub(TXL, f2pack(L.x, L.y)));
            const uint64_t DZ = f2add(f2sub(TZH, f2pack(H.z, H.w)), f2sub(TZL, f2pack(L.z, L.w)));
            const uint64_t R2 = f2fma(DX, DX, f2mul(DZ, DZ));
            const float ra = f2lo(R2), rb = f2hi(R2);
            float ka = rcp_approx(ra), kb = rcp_approx(rb);
            if (__any_sync(all, ra < Cs.z || rb < Cs.w)) {
                const float4 R = W.core[q];
                const bool ca = ra < R.z, cb = rb < R.w;
                const float qa = core_kernel_expm1(ra, R.x, ka);
                const float qb = core_kernel_expm1(rb, R.y, kb);
                ka = ca ? qa : ka;
                kb = cb ? qb : kb;
                if (fminf(ra, rb) < close2) {  // left to the loop below
                    ka = ra < close2 ? 0.0f : ka;
                    kb = rb < close2 ? 0.0f : kb;
                    first = min(first, q);
                    last = q;
                }
            }
            const uint64_t G = f2mul(f2pack(ka, kb), f2pack(Cs.x, Cs.y));
            kahan2_fma(snu, enu, G, DZ);
            kahan2_fma(s2, e2, G, DX);
        }
#pragma unroll 1
        for (int q = first; q <= last; q += kRhsGroup / group)
            for (int h = 0; h < 2; ++h) {
                const uint32_t j = j0 + 2 * q + h;
                const float* hi = reinterpret_cast<const float*>(&W.pos_hi[q]) + h;
                const float* lo = reinterpret_cast<const float*>(&W.pos_lo[q]) + h;
                const float* co = reinterpret_cast<const float*>(&W.core[q]) + h;
                if (j < n && split_dist2(txh, txl, tzh, tzl, hi, lo) < close2)
                    close_pair(tx - X[j].x, tz - X[j].y, co[0], co[2],
                               reinterpret_cast<const float*>(&W.cst[q])[h], h, false, snu, enu, s2, e2);
            }
        nu += ((double)f2lo(snu) + (double)f2lo(enu)) + ((double)f2hi(snu) + (double)f2hi(enu));
        sw += ((double)f2lo(s2) + (double)f2lo(e2)) + ((double)f2hi(s2) + (double)f2hi(e2));
    };
    int sp = nl ? walk_begin(W.walk, nl, tb, kWalkTop, (uint32_t)wid, kRhsWarps, lane) : 0;
    int nfar = 0, nnear = 0;
    while (sp > 0) {
        uint32_t id;
        const int kind = walk_step(W.walk, N, C, nl, sp, id, lane);
        int cnt;
        const int at = warp_place(kind == kWalkFar, lane, cnt);
        if (kind == kWalkFar) W.far[nfar + at] = id;
        nfar += cnt;
        __syncwarp();
        while (nfar >= kBatch || (sp == 0 && nfar > 0)) {
            const int m = min(kBatch, nfar);
            nfar -= m;
            translate(N, A, C, W.far + nfar, m, tb, mat, W.buf, lane, sum);
        }
        for (unsigned todo = __ballot_sync(all, kind == kWalkMid); todo; todo &= todo - 1) {
            const uint32_t q = __shfl_sync(all, id, __ffs(todo) - 1);
            const uint64_t at = node_level(C, (int)(q >> 27)) + (q & ((1u << 27) - 1));
            __syncwarp();
            if (lane < kTerms) W.buf.c[0][lane] = Cplx{A[at * kTerms + lane].x, A[at * kTerms + lane].y};
            __syncwarp();
            const Cplx f = moment_value(W.buf.c[0], exp2_int(N[at].e), tx - N[at].cx, tz - N[at].cz);
            if (lane < group) {
                nu -= f.y;
                sw += f.x;
            }
        }
        int cnear;
        const int place = warp_place(kind == kWalkNear, lane, cnear);
        const bool kept = kind == kWalkNear && nnear + place < kRhsNear;
        if (kept) W.near[nnear + place] = id;
        for (unsigned todo = __ballot_sync(all, kind == kWalkNear && !kept); todo; todo &= todo - 1)
            near_leaf(__shfl_sync(all, id, __ffs(todo) - 1));  // (no room)
        nnear = min(nnear + cnear, kRhsNear);
    }
    if (lane == 0) S.nnear[wid] = nnear;
    __syncthreads();
    for (int q = 0, at = 0; q < kRhsWarps; at += S.nnear[q++])  // every warp's, dealt out by place
        for (int k = (wid - at) & (kRhsWarps - 1); k < S.nnear[q]; k += kRhsWarps)
            near_leaf(S.w[q].near[k]);
    __syncwarp();
    W.sum[lane] = make_double2(nu, sw);
    Cplx b = local_total(sum, lane);
    if (lane < kTerms) W.buf.c[0][lane] = b;
    __syncthreads();
    if (wid != 0) return;
    if (lane < kTerms) {
        for (int q = 1; q < kRhsWarps; ++q) {
            b.x += S.w[q].buf.c[0][lane].x;
            b.y += S.w[q].buf.c[0][lane].y;
        }
        W.buf.c[0][lane] = b;
    }
    __syncwarp();
    const Cplx f = local_value(W.buf.c[0], tx - tb.cx, tz - tb.cz, tb.e);
    for (int q = 1; q < kRhsWarps; ++q) {
        nu += S.w[q].sum[lane].x;
        sw += S.w[q].sum[lane].y;
    }
    for (int o = group; o < 32; o <<= 1) {  // a point's lanes
        nu += __shfl_xor_sync(all, nu, o);
        sw += __shfl_xor_sync(all, sw, o);
    }
    nu -= f.y;
    sw += f.x;
    if (lane < group && i0 + lane < d.np) {
        const double ui = dmul(-nu, kRpi2), wi = dmul(sw, kRpi2);
        d.b[i] = dadd(dmul(dadd(d.ux, ui), d.enx[i]), dmul(dadd(d.uz, wi), d.enz[i]));
    }
    if (i0 == 0 && lane == 0) {
        int l = 0;
        while (level_count(nl, l) > 1u) ++l;
        const double a = nl ? A[node_level(C, l) * kTerms].x : 0.0;
        d.b[d.np] = -a;
        st[e.inst].totalcirc = a;
    }
}

__global__ void k_build_rhs_jobs(const InstDesc* __restrict__ table, InstState* __restrict__ st,
                                 const ListEntry* __restrict__ list, int nlist,
                                 double2* rhs_part, double* circ_part, AtJob* jobs) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nlist) return;
    const ListEntry e = list[k];
    const InstDesc& d = table[e.inst];
    AtJob J;
    J.tx = d.xc;
    J.tz = d.zc;
    J.nt = (uint32_t)d.np;
    J.skip_close = 0;  // solvevortexsheet has no close-pair skip (src/VortexSheet.cpp:186-203)
    J.sx = d.x;
    J.sz = d.z;
    J.sc = d.circ;
    J.ss = d.sigma;
    J.pns = &st[e.inst].n;
    J.ns = 0;
    J.npad = e.npad;
    J.chunk = e.rhs_chunk;
    J.part = rhs_part + e.roff;
    J.circ_part = circ_part + e.cofs;
    jobs[k] = J;
}

}  // namespace

void set_domain(InstDesc* d, const double* x, const double* z, uint32_t n, const Workspace& ws,
                int sms, cudaStream_t s) {
    if (n <= kDomainOne) {
        k_domain_one<<<1, 1024, 0, s>>>(x, z, n, d);
        return;
    }
    unsigned long long* dom = reinterpret_cast<unsigned long long*>(ws.work + 32);
    cudaMemsetAsync(dom, 0, 4 * sizeof(*dom), s);
    k_domain<<<std::min<uint32_t>((n + 1023) / 1024, sms * 4), 256, 0, s>>>(x, z, n, dom);
    k_set_domain<<<1, 32, 0, s>>>(d, dom, x, z, n);
}

size_t cub_sort_bytes(uint64_t total) {
    size_t bytes = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, bytes, (const uint64_t*)nullptr, (uint64_t*)nullptr,
                                    (const uint32_t*)nullptr, (uint32_t*)nullptr, (int64_t)total,
                                    0, 48);
    return bytes;
}

void biot_savart_prepare(const InstDesc* table, InstState* st, const ListEntry* list, int nlist,
                         int precision, const Workspace& ws, int sms, cudaStream_t s) {
    {  // both precisions evaluate over sorted tiles
        const int g = (int)std::min<uint64_t>((ws.total_cap + 255) / 256, (uint64_t)sms * 16);
        k_keys<<<g, 256, 0, s>>>(table, st, list, nlist, ws.total_cap, ws.keys_in, ws.vals_in);
        size_t bytes = ws.cub_bytes;
        cub::DeviceRadixSort::SortPairs(ws.cub_tmp, bytes, ws.keys_in, ws.keys_out, ws.vals_in,
                                        ws.perm, (int64_t)ws.total_cap, 0, ws.key_bits, s);
    }
    if (precision == kF32) {
        cudaMemsetAsync(ws.arrived, 0, sizeof(unsigned) * (2 * ws.total_cap / kLeaf + (uint64_t)kNodeSlack * nlist), s);
        k_tree<false><<<sms * 2, 32 * kTreeWarps, 0, s>>>(
            table, st, list, nlist, ws.perm, reinterpret_cast<double2*>(ws.packed),
            reinterpret_cast<float4*>(ws.packed + ws.packed_cap / 2), ws.nodes, ws.mom, ws.arrived,
            nullptr);
    } else {
        k_pack<<<sms * 8, kBsST, 0, s>>>(table, st, list, nlist, ws.perm, ws.packed, ws.meta);
    }
}

void biot_savart_compute(const InstDesc* table, InstState* st, const ListEntry* list, int nlist,
                         int precision, const Workspace& ws, int sms, cudaStream_t s,
                         const PairConfig& cfg, bool dry) {
    if (precision == kF32) {
        const double2* pxz = reinterpret_cast<const double2*>(ws.packed);
        cudaMemsetAsync(ws.work, 0, 2 * sizeof(unsigned), s);
        constexpr size_t far_smem = sizeof(FarShared) * kFarWarps;
        cudaFuncSetAttribute(k_far, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)far_smem);
        k_far<<<sms * kFarBlocks, 32 * kFarWarps, far_smem, s>>>(st, list, nlist, pxz, ws.nodes,
                                                                 ws.mom, ws.loc, ws.near,
                                                                 ws.work + 1);
        auto near = [&](auto kernel, int warps) {
            // cfg.ctas = 1 .. 4 quarters of full occupancy
            const int full = sms * (kNearThreads / (32 * warps));
            const int g = std::max(1, full * std::max(1, std::min(cfg.ctas, 4)) / 4);
            kernel<<<g, 32 * warps, 0, s>>>(
                table, st, list, nlist, pxz,
                reinterpret_cast<const float4*>(ws.packed + ws.packed_cap / 2), ws.perm, ws.nodes,
                ws.mom, ws.loc, ws.near, dry ? reinterpret_cast<double*>(ws.keys_in) : nullptr,
                dry ? reinterpret_cast<double*>(ws.keys_out) : nullptr, ws.work);
        };
        if (ws.total_cap / kLeaf <= (uint64_t)sms * 4) near(k_self_f32<8>, 8);
        else near(k_self_f32<4>, 4);
    } else {
        cudaMemsetAsync(ws.work, 0, sizeof(unsigned), s);
        k_self_f64<<<sms * kF64Ctas, kF64Threads, 0, s>>>(st, list, nlist, ws.packed, ws.meta,
                                                             ws.part, ws.work);
    }
}

void biot_savart_finish(const InstDesc* table, InstState* st, const ListEntry* list, int nlist,
                        int precision, const Workspace& ws, int sms, cudaStream_t s) {
    if (precision == kF32) return;  // the pair kernel writes the blobs' velocities itself
    k_self_combine<<<sms * 8, 256, 0, s>>>(table, st, list, nlist, ws.perm, ws.part);
}

void biot_savart_self(const InstDesc* table, InstState* st, const ListEntry* list, int nlist,
                      int precision, const Workspace& ws, int sms, cudaStream_t s,
                      const PairConfig& cfg) {
    biot_savart_prepare(table, st, list, nlist, precision, ws, sms, s);
    biot_savart_compute(table, st, list, nlist, precision, ws, sms, s, cfg);
    biot_savart_finish(table, st, list, nlist, precision, ws, sms, s);
}

void sheet_rhs(const InstDesc* table, InstState* st, const ListEntry* list, int nlist,
               int max_np, int precision, const Workspace& ws, int sms, cudaStream_t s, bool pairs) {
    if (precision == kF32 && !pairs) {
        cudaFuncSetAttribute(k_rhs_tree, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sizeof(RhsShared));
        // (a list's smaller bodies may have up to 16 groups of eight points)
        k_rhs_tree<<<dim3(std::max((max_np + kRhsGroup - 1) / kRhsGroup,
                                   std::min((max_np + 7) / 8, 16)), nlist), 32 * kRhsWarps,
                     sizeof(RhsShared), s>>>(
            table, st, list, reinterpret_cast<const double2*>(ws.packed),
            reinterpret_cast<const float4*>(ws.packed + ws.packed_cap / 2), ws.nodes, ws.mom);
        return;
    }
    static_assert(sizeof(AtJob) <= 256, "job record size");
    AtJob* jobs = reinterpret_cast<AtJob*>(ws.jobs);
    k_build_rhs_jobs<<<(nlist + 127) / 128, 128, 0, s>>>(table, st, list, nlist, ws.rhs_part,
                                                         ws.circ_part, jobs);
    if (precision == kF32) k_at<true><<<sms * 4, 256, 0, s>>>(jobs, nlist);
    else k_at<false><<<sms * 4, 256, 0, s>>>(jobs, nlist);
    k_rhs_combine<<<dim3((max_np + 31) / 32, nlist), 256, 0, s>>>(table, st, list, jobs);
}

// Sources per work item of an at-target call: a multiple of 256, at most kAtChunk,
// that leaves about 1184 items, two to three rounds of the resident blocks (256
// targets against 2^20 sources: 256 items of 4096 left half of the blocks idle, the
// call 685 us; 303 now; chunks in multiples of 64, 348).
static uint32_t at_chunk(uint64_t ns, uint64_t nt) {
    const uint64_t want = (ns * ((nt + 255) / 256) + 1183) / 1184;
    return (uint32_t)std::max<uint64_t>(256, std::min<uint64_t>(kAtChunk, (want + 255) / 256 * 256));
}

// Warps per block of k_at_combine: about four chunks each.
static unsigned combine_threads(uint64_t nchunk) {
    unsigned w = 1;
    while (w < 32 && 4ull * w < nchunk) w *= 2;
    return 32 * w;
}

void panel_tree(const InstDesc* table, const InstState* st, const ListEntry* list, int nlist,
                int max_np, const Workspace& ws, int sms, cudaStream_t s) {
    const int shares = ((int)panel_leaves(max_np) + kFan - 1) / kFan;
    cudaMemsetAsync(ws.parrived, 0, sizeof(unsigned) * ws.pnodes_used, s);
    k_tree<true><<<std::min(sms * 2, nlist * shares), 32 * kTreeWarps, 0, s>>>(
        table, st, list, nlist, nullptr, nullptr, nullptr, ws.pnodes, ws.pmom,
        ws.parrived, ws.pan);
}

size_t direct_at_part_elems(uint32_t ns, uint32_t nt) {
    const size_t chunk = at_chunk(ns, nt);
    const size_t nchunk = (ns + chunk - 1) / chunk;
    const size_t npad = (nt + 255) / 256 * 256;
    return std::max<size_t>(1, nchunk) * std::max<size_t>(npad, 256) + 64;
}

namespace {
__global__ void k_write_job(AtJob* dst, AtJob job) { *dst = job; }
}  // namespace

static void launch_at(const AtJob* job, const AtJob& J, int precision, double* u, double* w, int sms,
                      cudaStream_t s) {
    if (precision == kF32) k_at<true><<<sms * 4, 256, 0, s>>>(job, 1);
    else k_at<false><<<sms * 4, 256, 0, s>>>(job, 1);
    const unsigned blocks = (unsigned)std::min<uint64_t>(((uint64_t)J.nt + 31) / 32, (uint64_t)sms * 16);
    k_at_combine<<<std::max(1u, blocks), combine_threads((J.ns + J.chunk - 1) / J.chunk), 0, s>>>(
        job, u, w);
}

void direct_at_raw(const double* x, const double* z, const double* circ, const double* sigma,
                   uint32_t ns, const double* tx, const double* tz, uint32_t nt, double* u,
                   double* w, int precision, int skip_close, double2* part, int sms,
                   cudaStream_t s) {
    // The job record sits in the last 64 entries of the partials buffer.
    const size_t elems = direct_at_part_elems(ns, nt);
    AtJob* job = reinterpret_cast<AtJob*>(part + elems - 64);
    AtJob J;
    J.tx = tx;
    J.tz = tz;
    J.nt = nt;
    J.skip_close = skip_close;
    J.sx = x;
    J.sz = z;
    J.sc = circ;
    J.ss = sigma;
    J.pns = nullptr;
    J.ns = ns;
    J.npad = (int)std::max<size_t>((nt + 255) / 256 * 256, 256);
    J.chunk = at_chunk(ns, nt);
    J.part = part;
    J.circ_part = nullptr;
    if (ns > 0) {
        k_write_job<<<1, 1, 0, s>>>(job, J);
        launch_at(job, J, precision, u, w, sms, s);
    } else {
        cudaMemsetAsync(u, 0, sizeof(double) * nt, s);
        cudaMemsetAsync(w, 0, sizeof(double) * nt, s);
    }
}

// ---- at-target velocity with fixed, library-owned scratch -------------------
// For callers that must not allocate device memory (see
// dvm_biot_savart_at_noalloc in include/dvm_cuda.h).  The chunk partials of
// k_at live in this file-scope array instead of a caller- or context-owned
// buffer; every GPU that loads the library holds it until the process exits.
namespace {

constexpr size_t kNoAllocElems = 262144;  // double2 entries: 4 MiB per device
constexpr size_t kNoAllocJobElems = 64;   // tail entries that hold the job record
static __device__ __align__(256) double2 g_noalloc_scratch[kNoAllocElems];

}  // namespace

}  // namespace dvmk

extern "C" int dvm_biot_savart_at_noalloc(const double* x, const double* z, const double* circ,
                                          const double* sigma, uint64_t ns, const double* tx,
                                          const double* tz, uint64_t nt, double* u, double* w,
                                          int precision, int skip_close, void* stream) {
    using namespace dvmk;
    if (nt && (!tx || !tz || !u || !w)) return report_error(1, "null target or output array");
    if (ns && (!x || !z || !circ || !sigma)) return report_error(1, "null source array");
    if (precision != kF64 && precision != kF32) return report_error(1, "bad precision");
    if (nt == 0) return 0;
    const size_t nchunk = (ns + kAtChunk - 1) / kAtChunk;
    const size_t npad = std::max<size_t>((nt + 255) / 256 * 256, 256);
    if (ns > 0xF0000000ull || nt > 0xF0000000ull ||
        nchunk * npad > kNoAllocElems - kNoAllocJobElems) {
        return report_error(
            1, "dvm_biot_savart_at_noalloc: ceil(ns/4096) * ceil(nt/256) * 256 must not exceed "
               "262080 (fixed 4 MiB scratch); use dvm_biot_savart_at_device for larger sizes");
    }
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0)
        return report_error(3, "dvm_biot_savart_at_noalloc: no current CUDA device");
    // The array's device address, looked up with the device current on every
    // call (host code cannot use the symbol itself).  Not cached: a device
    // reset reloads the library's device code, and the array may then move.
    // The first call on a device also loads that code, which is why it should
    // come before any stream capture.
    void* scratch_p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&scratch_p, g_noalloc_scratch);
    if (e != cudaSuccess)
        return report_error(3, (std::string("cudaGetSymbolAddress: ") + cudaGetErrorString(e)).c_str());
    int sms = 0;
    e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess)
        return report_error(3, (std::string("cudaDeviceGetAttribute: ") + cudaGetErrorString(e)).c_str());
    double2* const scratch = static_cast<double2*>(scratch_p);
    if (ns == 0) {  // no sources: zero velocity, as the reference's empty loop gives
        if (cudaMemsetAsync(u, 0, sizeof(double) * nt, s) != cudaSuccess ||
            cudaMemsetAsync(w, 0, sizeof(double) * nt, s) != cudaSuccess)
            return report_error(3, "cudaMemsetAsync failed");
        return 0;
    }
    AtJob J;
    J.tx = tx;
    J.tz = tz;
    J.nt = (uint32_t)nt;
    J.skip_close = skip_close ? 1 : 0;
    J.sx = x;
    J.sz = z;
    J.sc = circ;
    J.ss = sigma;
    J.pns = nullptr;
    J.ns = (uint32_t)ns;
    J.npad = (int)npad;
    // (kAtChunk fits, by the check above; shorter chunks as far as the scratch holds them)
    const uint64_t most = (kNoAllocElems - kNoAllocJobElems) / npad;
    J.chunk = std::max<uint32_t>(at_chunk(ns, nt),
                                 (uint32_t)std::min<uint64_t>(kAtChunk, ((ns + most - 1) / most + 255) / 256 * 256));
    J.part = scratch;  // every entry read by k_at_combine is written by k_at first
    J.circ_part = nullptr;
    AtJob* job = reinterpret_cast<AtJob*>(scratch + (kNoAllocElems - kNoAllocJobElems));
    k_write_job<<<1, 1, 0, s>>>(job, J);
    launch_at(job, J, precision, u, w, sms, s);
    e = cudaGetLastError();
    if (e != cudaSuccess)
        return report_error(3, (std::string("dvm_biot_savart_at_noalloc launch: ") +
                                cudaGetErrorString(e)).c_str());
    return 0;
}
